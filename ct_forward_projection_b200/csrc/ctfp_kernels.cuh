// ctfp_kernels.cuh — kernel parameter blocks and launcher declarations.
#pragma once

#include "ctfp_device.cuh"

namespace ctfp {

// One problem as the march kernels see it.
struct MarchParams {
    GeomParams g;
    const float* vol[kMaxM];          // material densities [nz][ny][nx]
    cudaTextureObject_t tex[kMaxM];   // same volumes as 3D textures (TEXTURE mode)
    cudaTextureObject_t ltex[kMaxM];  // same volumes as layered 2D textures (SAMPLER_LAYERED)
    cudaTextureObject_t xtex[kMaxM];  // SAMPLER_AXIS: layered along x (layer x, texel (y, z))
    cudaTextureObject_t ytex[kMaxM];  // SAMPLER_AXIS: layered along y (layer y, texel (x, z))
    const float* cvol;                // SAMPLER_AXIS, four materials: the column copy instead (ctfp_column.cuh)
    float* L;                         // [P][V][U][M] path integrals (out, may be null)
    const float* Lin;                 // [P][V][U][M] path integrals (in, epilogue/adjoint)
    float* I;                         // [P][V][U] (may be null)
    float* IAbs;                      // [P][V][U] (may be null)
    const float* W;                   // energy weights I0Val*S*G*D of every pixel (pixel_weights)
    const float* mu;                  // [E][M] attenuation per density, 1/mm per g/cm^3
    const float* gI;                  // [P][V][U] dLoss/dI (adjoint)
    const float* gIAbs;               // [P][V][U] dLoss/dIAbsorb (adjoint, may be null)
    float* gvol[kMaxM];               // gradient volumes (adjoint)
    float* gcol;                      // gradient accumulators of every material (adjoint, ctfp_column.cuh)
    int sets;                         // sets of them, set_floats apart: as many parts of the views as
    int set_columns;                  // set_columns (a power of two) goes into, times columns taking turns (accum_sets)
    size_t set_floats;
    int E;
    int view0;                        // first view of this launch
    int n_views;                      // views in this launch
    int views_per_cta;                // views each CTA marches for its pixel tile
    int out_view0;                    // view stored at index 0 of I, IAbs, L, Lin, gI, gIAbs (0: full arrays)
    const uint8_t* occ;               // empty-space skipping: brick occupancy (null: march every sample)
    int occ_x, occ_y;                 // bricks along x, y (see launch_occupancy)
    unsigned* status;                 // plan-owned word; kCtfpStatusWaitTimeout is or-ed in when a bounded wait ran out
    int wait_limit;                   // polls of a TMA completion before a CTA gives up on staging
};

// Bits of the plan's device status word (ctfp_plan_check_status; the same
// values as CTFP_STATUS_* in ctfp.h).  WaitTimeout: a CTA gave up waiting for
// a TMA load and read the volume instead (outputs correct).  ExitWaitTimeout:
// the CTA's bounded wait at exit for that load ran out as well, so the copy may
// have landed in shared memory another CTA owned (outputs not trusted).
constexpr unsigned kCtfpStatusWaitTimeout = 1u;
constexpr unsigned kCtfpStatusExitWaitTimeout = 2u;

// Bricks of kOccShift^2 voxels per axis for empty-space skipping.  Brick
// (bx, by, bz) is marked when any material has a non-zero voxel in
// [8b - 1, 8b + 7] on every axis: exactly the voxels a footprint with base
// corner ix in [8b - 1, 8b + 6] (brick of ix + 1) can read.
constexpr int kOccShift = 3;
inline int occ_dim(int n) { return ((n + 1) >> kOccShift) + 1; }

struct LaunchShape {
    int tile_u = 16, tile_v = 8, views_per_cta = 2;
    int min_ctas = 4;  // register cap of the forward march: 65536 / (256 * min_ctas) per thread
};

// Launchers; all return cudaGetLastError() of the launch.  sampler selects
// SAMPLER_GLOBAL or SAMPLER_LAYERED for the software interp modes.
cudaError_t launch_forward(const MarchParams& prm, int M, int interp, int sampler, bool do_spectral,
                           const LaunchShape& ls, cudaStream_t st);
cudaError_t launch_spectral_from_L(const MarchParams& prm, int M, cudaStream_t st);
// Whether this forward shares rays among lanes (axis_split), in its own launch shape.
bool forward_splits(const MarchParams& prm, int M, int interp, int sampler);
// Floats of one set of the adjoint's accumulators (accum_width).
size_t accum_floats(int nx, int ny, int nz, int M);
int accum_set_count(const GeomParams& g, int n_views, int M);  // accum_sets, any number of sets
void set_accum_sets(MarchParams& prm, int M, int most);        // prm.sets and prm.set_columns for prm.n_views, at most so many
bool accum_fits(int nx, int ny, int nz);  // false: launch_backward adds into prm.gvol (prm.gcol null)
// Adjoint scatter into the accumulators prm.gcol (zeroed by the caller),
// followed by launch_fold into prm.gvol.
cudaError_t launch_backward(const MarchParams& prm, int M, int interp, bool from_gL, const LaunchShape& ls,
                            cudaStream_t st);
cudaError_t launch_fold(const MarchParams& prm, int M, cudaStream_t st);
cudaError_t launch_weights(const float* spectrum, const float* grid, int grid_layout, const float* det,
                           float I0Val, int E, int U, int V, float* W, float* I0, cudaStream_t st);
cudaError_t launch_finalize(int64_t n_pix, int64_t n_views, const float* I, const float* IAbs, const float* I0,
                            uint32_t* Ipoly, uint32_t* IAbsPoly, float* proj, cudaStream_t st);
cudaError_t launch_sample_points(const float* vol, cudaTextureObject_t tex, int nx, int ny, int nz, int interp,
                                 const float* pts, int64_t n, float* out, cudaStream_t st);
cudaError_t launch_count_support(const GeomParams& g, unsigned long long* out, cudaStream_t st);
// Focal-spot re-alignment of compact line-integral images [n_views][V][U][M]
// of views view0.. (interp selects exact or texture-unit bilinear weights).
cudaError_t launch_shift_views(const float* in, float* out, const GeomParams& g, int M, int interp, int view0,
                               int n_views, cudaStream_t st);
// SAMPLER_AXIS: whether M materials use the column copy, its floats, and its
// interior from the volumes (the border stays as allocated: zero).
bool axis_uses_columns(int M);
size_t column_floats(int nx, int ny, int nz);
cudaError_t launch_column_fill(const float* const* vol, int nx, int ny, int nz, float* cvol, cudaStream_t st);
// Otherwise: writes each volume [nz][ny][nx] into its x-layered copy (surface
// xs: texture layer x + 1, texel (y, z)) and its y-layered copy (ys: texture
// layer y + 1, texel (x, z)).
struct AxisCopies {
    const float* vol[kMaxM];
    cudaSurfaceObject_t xs[kMaxM], ys[kMaxM];
};
cudaError_t launch_axis_fill(const AxisCopies& copies, int M, int nx, int ny, int nz, cudaStream_t st);
// The axis march's texture quad-gathers over every view of a problem, with the
// launch shape's tile and lane layout: out[0] += quads, out[1] += samples.
cudaError_t launch_axis_gather_count(const GeomParams& g, int interp, const LaunchShape& ls, unsigned long long* out,
                                     cudaStream_t st);
// Zeros the pad layers (0 and the last) of both copies; once per array.
cudaError_t launch_axis_zero_pads(int nx, int ny, int nz, cudaSurfaceObject_t xs, cudaSurfaceObject_t ys,
                                  cudaStream_t st);
// Fills occ [occ_dim(nz)][occ_dim(ny)][occ_dim(nx)] from the M volumes
// (vol: host array of M device pointers; occ is zeroed first).
cudaError_t launch_occupancy(const float* const* vol, int M, int nx, int ny, int nz, uint8_t* occ, cudaStream_t st);

}  // namespace ctfp
