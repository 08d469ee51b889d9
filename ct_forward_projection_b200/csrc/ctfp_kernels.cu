// ctfp_kernels.cu — the march kernels (K1 ray march fused with the K2
// spectral epilogue), the adjoint scatter, and small helper kernels.
//
// K1+K2 replaces, for every (view, pixel) ray, the reference's
//   transformKernel (CBCTPolyProjGPU.cu:1902-1924)  K*U*V samples to HBM per view
//   forward*Kernel  (CBCTPolyProjGPU.cu:1980-2169)  per-ray sum + Beer-Lambert per energy
//   host energy loop (CBCTPolyForwardProjGrid.cpp:159-177, CBCTForwardProj.cpp:65-76)
// with one pass: samples stay in registers, each material is marched once for
// all energies (sum_m mu[e][m] * L_m equals the reference's per-energy
// mu_E-volume integral because trilinear interpolation is linear in the voxel
// values), and the energy sum runs on the device in compensated FP32.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "ctfp_axis.cuh"
#include "ctfp_column.cuh"
#include "ctfp_kernels.cuh"

namespace ctfp {

namespace {

struct VolPtrs {
    const float* p[kMaxM];
};

template <int M, int SAMPLER>
__device__ __forceinline__ void load_corners(const MarchParams& prm, const Corner& c, float (*v)[8])
{
    if (SAMPLER == SAMPLER_LAYERED || SAMPLER == SAMPLER_LAYERED_SKIP) load8_layered<M>(prm.ltex, prm.g.nz, c, v);
    else load8_global<M>(prm.vol, prm.g.nx, prm.g.ny, prm.g.nz, c, v);
}

// Whether the footprint with base corner c can read a non-zero voxel (brick
// occupancy); bases outside [-1, n - 1] read only the border.
__device__ __forceinline__ bool footprint_occupied(const MarchParams& prm, const Corner& c)
{
    const unsigned x = (unsigned)(c.ix + 1), y = (unsigned)(c.iy + 1), z = (unsigned)(c.iz + 1);
    if (x > (unsigned)prm.g.nx || y > (unsigned)prm.g.ny || z > (unsigned)prm.g.nz) return false;
    const size_t b = ((size_t)(z >> kOccShift) * prm.occ_y + (y >> kOccShift)) * prm.occ_x + (x >> kOccShift);
    return __ldg(prm.occ + b) != 0;
}

// One sample of a software-interpolated march: fetch the footprint,
// interpolate, accumulate.  With empty-space skipping, a footprint inside an
// all-zero brick contributes exactly zero and is not fetched.
template <int M, int MODE, int SAMPLER>
__device__ __forceinline__ void sample_acc(const MarchParams& prm, const Corner& c, float* acc, float* cmp)
{
    if (SAMPLER == SAMPLER_LAYERED_SKIP && !footprint_occupied(prm, c)) return;
    float v[M][8];
    load_corners<M, SAMPLER>(prm, c, v);
#pragma unroll
    for (int m = 0; m < M; m++) kahan_add(acc[m], cmp[m], interp8<MODE>(c, v[m]));
}

// L_m for one ray, compensated FP32 sum times dx.  TRILINEAR samples at FP64
// coordinates; the compat samplers at the reference's FP32 coordinates.
template <int M, int MODE, int SAMPLER>
__device__ __forceinline__ void march_ray(const MarchParams& prm, int p, int v, int u, float* L)
{
    const RaySeg s = ray_segment(prm.g, p, v, u);
    float acc[M], cmp[M];
#pragma unroll
    for (int m = 0; m < M; m++) { acc[m] = 0.f; cmp[m] = 0.f; }
    if (MODE == INTERP_TRILINEAR) {
#pragma unroll 2
        for (int i = s.i0; i < s.i1; i++) {
            const double t = (double)i;
            sample_acc<M, MODE, SAMPLER>(
                prm, corner_of<INTERP_TRILINEAR>(fma(t, s.bx, s.ax), fma(t, s.by, s.ay), fma(t, s.bz, s.az)), acc, cmp);
        }
    } else if (MODE == INTERP_TEXTURE) {
        // the reference's own fetch: tex3D on a border/linear texture
        const RayRef32 r = ray_ref32(prm.g, p, v, u);
#pragma unroll 2
        for (int i = s.i0; i < s.i1; i++) {
            const float3 x = ref32_coords<false>(prm.g, r, i);
            // with empty-space skipping: the unit's own footprint (base texel
            // of its fixed-point coordinate) in an all-zero brick filters to 0
            if (SAMPLER == SAMPLER_LAYERED_SKIP && !footprint_occupied(prm, corner_tex(x))) continue;
#pragma unroll
            for (int m = 0; m < M; m++) kahan_add(acc[m], cmp[m], tex3D<float>(prm.tex[m], x.x, x.y, x.z));
        }
    } else {
        const RayRef32 r = ray_ref32(prm.g, p, v, u);
#pragma unroll 2
        for (int i = s.i0; i < s.i1; i++) sample_acc<M, MODE, SAMPLER>(prm, corner_tex(ref32_coords(prm.g, r, i)), acc, cmp);
    }
#pragma unroll
    for (int m = 0; m < M; m++) L[m] = prm.g.dx * (acc[m] - cmp[m]);
}

__device__ __forceinline__ void load_mu(float* s_mu, const float* mu, int E, int M)
{
    stage_mu(s_mu, mu, E, M, threadIdx.y * blockDim.x + threadIdx.x, blockDim.x * blockDim.y);
    __syncthreads();
}

template <int M>
__device__ __forceinline__ void store_L(float* L, int64_t ray, const float* l)
{
    float* q = L + ray * M;
    if (M == 4) {
        *reinterpret_cast<float4*>(q) = make_float4(l[0], l[1], l[2], l[3]);
    } else if (M == 2) {
        *reinterpret_cast<float2*>(q) = make_float2(l[0], l[1]);
    } else {
#pragma unroll
        for (int m = 0; m < M; m++) q[m] = l[m];
    }
}

template <int M>
__device__ __forceinline__ void load_L(const float* L, int64_t ray, float* l)
{
    const float* q = L + ray * M;
    if (M == 4) {
        const float4 a = *reinterpret_cast<const float4*>(q);
        l[0] = a.x; l[1] = a.y; l[2] = a.z; l[3] = a.w;
    } else if (M == 2) {
        const float2 a = *reinterpret_cast<const float2*>(q);
        l[0] = a.x; l[1] = a.y;
    } else {
#pragma unroll
        for (int m = 0; m < M; m++) l[m] = q[m];
    }
}

// K1+K2. Grid: x = pixel tiles along u, y = along v, z = view groups.
template <int M, int MODE, int SAMPLER, bool SPECTRAL, int MINB>
__global__ void __launch_bounds__(256, MINB) k_forward(const MarchParams prm)
{
    extern __shared__ __align__(16) float s_mu[];
    if (SPECTRAL) load_mu(s_mu, prm.mu, prm.E, M);
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y * blockDim.y + threadIdx.y;
    if (u >= prm.g.U || v >= prm.g.V) return;
    const int64_t npix = (int64_t)prm.g.U * prm.g.V;
    const int64_t pix = (int64_t)v * prm.g.U + u;
    const int pend = prm.view0 + prm.n_views;
    for (int k = 0; k < prm.views_per_cta; k++) {
        const int p = prm.view0 + blockIdx.z * prm.views_per_cta + k;
        if (p >= pend) break;
        float L[M];
        march_ray<M, MODE, SAMPLER>(prm, p, v, u, L);
        const int64_t ray = (int64_t)(p - prm.out_view0) * npix + pix;
        if (prm.L) store_L<M>(prm.L, ray, L);
        if (SPECTRAL) {
            float I, A;
            spectral<M>(s_mu, prm.E, pixel_weights(prm.W, prm.g.U, prm.E, u, v), L, I, A);
            if (prm.I) prm.I[ray] = I;
            if (prm.IAbs) prm.IAbs[ray] = A;
        }
    }
}

// K1+K2 with the axis sampler.  One-dimensional CTAs of tile_u * tile_v
// threads (tile_v a multiple of 4) cover a tile_u x tile_v pixel tile: lane
// quads run down 4 detector rows of one column, so a warp covers 8 columns x
// 4 rows.  Grid: x = pixel tiles along u, y = along v, z = view groups.
template <int M, int MODE, bool SKIP, bool SPECTRAL, int MINB>
__global__ void __launch_bounds__(256, MINB) k_forward_axis(const MarchParams prm, int tile_u, int warp_rows)
{
    extern __shared__ __align__(16) float s_mu[];
    if (SPECTRAL) load_mu(s_mu, prm.mu, prm.E, M);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int tile_v = (int)blockDim.x / tile_u;
    // a warp covers wcols columns x warp_rows rows, lane quads down 4 rows
    const int wcols = 32 / warp_rows, warps_u = tile_u / wcols;
    const int col = (lane >> 2) % wcols, row = 4 * ((lane >> 2) / wcols) + (lane & 3);
    const int u = blockIdx.x * tile_u + (w % warps_u) * wcols + col;
    const int v = blockIdx.y * tile_v + (w / warps_u) * warp_rows + row;
    if (u >= prm.g.U || v >= prm.g.V) return;
    const int64_t npix = (int64_t)prm.g.U * prm.g.V;
    const int64_t pix = (int64_t)v * prm.g.U + u;
    const int pend = prm.view0 + prm.n_views;
    for (int k = 0; k < prm.views_per_cta; k++) {
        const int p = prm.view0 + blockIdx.z * prm.views_per_cta + k;
        if (p >= pend) break;
        float L[M];
        const OccView ov{prm.occ, prm.occ_x, prm.occ_y, prm.g.nx, prm.g.ny, prm.g.nz, kOccShift};
        march_axis<M, MODE, SKIP>(prm.g, prm.xtex, prm.ytex, prm.cvol, ov, p, v, u, L);
        const int64_t ray = (int64_t)(p - prm.out_view0) * npix + pix;
        if (prm.L) store_L<M>(prm.L, ray, L);
        if (SPECTRAL) {
            float I, A;
            spectral<M>(s_mu, prm.E, pixel_weights(prm.W, prm.g.U, prm.E, u, v), L, I, A);
            if (prm.I) prm.I[ray] = I;
            if (prm.IAbs) prm.IAbs[ray] = A;
        }
    }
}

// K1+K2 with the axis sampler for a plan of few rays (axis_split), where a
// thread per ray leaves most of the chip idle and the time is one ray's chain
// of gathers: 1 << shift lanes share a ray, each marching an equal run of its
// samples and taking a fourth of the energies.  A warp covers 32 >> shift rays,
// rows of a column (lane quads down 4 rows, as k_forward_axis) or, where the
// detector has fewer rows, that many rows of several columns; a CTA 4 warps.
// The energies' partial sums are spectral()'s four accumulators, combined in
// its order, so I and IAbs equal its values for the same L.
template <int M, int MODE, bool SKIP, bool SPECTRAL>
__global__ void __launch_bounds__(128, uses_columns(M) ? 6 : 8) k_forward_axis_split(const MarchParams prm, int shift, int rows)
{
    extern __shared__ __align__(16) float s_mu[];
    if (SPECTRAL) load_mu(s_mu, prm.mu, prm.E, M);
    const int lane = threadIdx.x & 31, rays = 32 >> shift, part = lane / rays, ray_at = lane % rays, cols = rays / rows;
    const int u = (blockIdx.x * 4 + (threadIdx.x >> 5)) * cols + ray_at / rows, v = blockIdx.y * rows + ray_at % rows;
    const int p = prm.view0 + blockIdx.z;
    const bool on = u < prm.g.U && v < prm.g.V;
    const int64_t npix = (int64_t)prm.g.U * prm.g.V;
    const int64_t pix = (int64_t)v * prm.g.U + u;
    const int64_t ray = (int64_t)(p - prm.out_view0) * npix + pix;
    float L[M], cmp[M];  // the sum's Kahan pair, then L
#pragma unroll
    for (int m = 0; m < M; m++) L[m] = cmp[m] = 0.f;
    if (on) {
        const OccView ov{prm.occ, prm.occ_x, prm.occ_y, prm.g.nx, prm.g.ny, prm.g.nz, kOccShift};
        march_axis_sums<M, MODE, SKIP>(prm.g, prm.xtex, prm.ytex, prm.cvol, ov, p, v, u, L, cmp, part, 1 << shift);
    }
    for (int d = rays; d < 32; d <<= 1)
#pragma unroll
        for (int m = 0; m < M; m++)
            kahan_join(L[m], cmp[m], __shfl_xor_sync(0xffffffffu, L[m], d), __shfl_xor_sync(0xffffffffu, cmp[m], d));
#pragma unroll
    for (int m = 0; m < M; m++) L[m] = prm.g.dx * (L[m] - cmp[m]);
    if (on && part == 0 && prm.L) store_L<M>(prm.L, ray, L);
    if (SPECTRAL) {
        // accumulators of this lane: two of the four (2 lanes per ray) or one
        const int first = shift == 1 ? 2 * part : part, own = shift == 1 ? 2 : 1;
        float sI = 0.f, sA = 0.f;
        if (on && first < 4) {
            const PixelWeights W = pixel_weights(prm.W, prm.g.U, prm.E, u, v);
            const int full = prm.E >> 2, Ep = energy_groups(prm.E) * 4;
            for (int a = 0; a < own; a++) {
                float tI = 0.f, tA = 0.f;
                const auto term = [&](int e, const float* at) {
                    float att = 0.f, ex, om;
#pragma unroll
                    for (int m = 0; m < M; m++) att = fmaf(s_mu[m * Ep + e], L[m], att);
                    const float w = __ldg(at);
                    transmit(att, ex, om);
                    tI = fmaf(w, ex, tI);
                    tA = fmaf(w, om, tA);
                };
#pragma unroll 4
                for (int g = 0; g < full; g++) term(4 * g + first + a, (const float*)(W.full + g * 32) + first + a);
                if (first + a == 0)
                    for (int e = 4 * full; e < prm.E; e++) term(e, W.rest + e * 32);
                sI += tI;
                sA += tA;
            }
        }
        for (int d = rays; d < 4 * rays / own; d <<= 1) {
            sI += __shfl_xor_sync(0xffffffffu, sI, d);
            sA += __shfl_xor_sync(0xffffffffu, sA, d);
        }
        if (on && part == 0) {
            if (prm.I) prm.I[ray] = sI;
            if (prm.IAbs) prm.IAbs[ray] = sA;
        }
    }
}

// Texture quad-gathers of the axis march (count_ray_axis) over every view,
// with k_forward_axis's CTA tile and lane layout; out[0] += quads, out[1] +=
// samples.  Grid: x = pixel tiles along u, y = along v, z = views.
template <int MODE>
__global__ void __launch_bounds__(256) k_axis_gather_count(const GeomParams g, int tile_u, int warp_rows,
                                                           unsigned long long* out)
{
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int tile_v = (int)blockDim.x / tile_u;
    const int wcols = 32 / warp_rows, warps_u = tile_u / wcols;
    const int col = (lane >> 2) % wcols, row = 4 * ((lane >> 2) / wcols) + (lane & 3);
    const int u = blockIdx.x * tile_u + (w % warps_u) * wcols + col;
    const int v = blockIdx.y * tile_v + (w / warps_u) * warp_rows + row;
    const bool valid = u < g.U && v < g.V;
    const unsigned warp_mask = __ballot_sync(0xffffffffu, valid);
    if (!valid) return;
    const int p = blockIdx.z;
    unsigned long long r[2];
    if (axis_is_x(g, p)) count_ray_axis<MODE, 0>(g, p, v, u, warp_mask, r);
    else count_ray_axis<MODE, 1>(g, p, v, u, warp_mask, r);
    if (lane == __ffs(warp_mask) - 1) {
        atomicAdd(out, r[0]);
        atomicAdd(out + 1, r[1]);
    }
}

// The x- and y-layered copies of one volume, through a 32 x 32 (x, y) tile
// of one z slice in shared memory so that both copies are written along their
// texel rows; voxel layer l is texture layer l + 1 (layer 0 and the last
// layer are zeros, k_axis_zero_layers).  Block (32, 8); grid (ceil(nx / 32),
// ceil(ny / 32), nz * materials): one launch for all of them (two launches of
// 5 us were a third of the smallest forward).
__global__ void __launch_bounds__(256) k_axis_fill(const AxisCopies c, int nx, int ny, int nz)
{
    __shared__ float t[32][33];
    const int m = blockIdx.z / nz, z = blockIdx.z - m * nz;
    const float* __restrict__ vol = c.vol[m];
    const cudaSurfaceObject_t xs = c.xs[m], ys = c.ys[m];
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
    const int tx = threadIdx.x;
    for (int ty = threadIdx.y; ty < 32; ty += 8) {
        const int x = x0 + tx, y = y0 + ty;
        t[ty][tx] = (x < nx && y < ny) ? __ldg(vol + ((size_t)z * ny + y) * nx + x) : 0.f;
    }
    __syncthreads();
    for (int ty = threadIdx.y; ty < 32; ty += 8) {
        {
            const int x = x0 + tx, y = y0 + ty;  // y-layered: layer y, texel (x, z)
            if (x < nx && y < ny) surf2DLayeredwrite(t[ty][tx], ys, x * (int)sizeof(float), z, y + 1);
        }
        {
            const int y = y0 + tx, x = x0 + ty;  // x-layered: layer x, texel (y, z)
            if (x < nx && y < ny) surf2DLayeredwrite(t[tx][ty], xs, y * (int)sizeof(float), z, x + 1);
        }
    }
}

// The column copy's interior: for one y, a 32 x 32 (x, z) tile of the four
// materials through shared memory, read along x and written along z as 16-byte
// elements.  Block (32, 8); one block per tile, column_tile.
__global__ void __launch_bounds__(256) k_column_fill(const VolPtrs vol, int nx, int ny, int nz, float* __restrict__ cvol)
{
    __shared__ float t[4][32][33];
    int x0, y, z0;
    column_tile(blockIdx.x, nx, nz, x0, y, z0);
    const int tx = threadIdx.x;
    for (int k = threadIdx.y; k < 32; k += 8) {
        const int x = x0 + tx, z = z0 + k;
        if (x < nx && z < nz) {
#pragma unroll
            for (int m = 0; m < 4; m++) t[m][k][tx] = __ldg(vol.p[m] + ((size_t)z * ny + y) * nx + x);
        }
    }
    __syncthreads();
    const ColumnDims cd = column_dims(nx, ny, nz);
    for (int k = threadIdx.y; k < 32; k += 8) {
        const int x = x0 + k, z = z0 + tx;
        if (x < nx && z < nz)
            ((float4*)cvol)[(size_t)x * cd.sx + (size_t)y * cd.sy + (size_t)z + cd.origin] =
                make_float4(t[0][tx][k], t[1][tx][k], t[2][tx][k], t[3][tx][k]);
    }
}

// Zeros texture layer `layer` (width x height texels) of a layered surface.
__global__ void k_axis_zero_layer(cudaSurfaceObject_t sf, int width, int height, int layer)
{
    const int n = width * height;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        surf2DLayeredwrite(0.0f, sf, (k % width) * (int)sizeof(float), k / width, layer);
}

// K2 on stored line integrals.  Bound by memory for few energies (8 + 4 M bytes
// a ray) and by the epilogue's issue for many.  A thread takes a pixel and walks
// views, so that no ray costs a division; a warp is 32 pixels of a row (whole
// sectors of W, and L, I and IAbs in one piece).  512 x 256 pixels, 90 views, 1
// material, 1 / 61 energies: 54 / 539 us; 1000 x 1, 360 views, 61 energies: 23 us
// (walking W's blocks of 4 x 8 pixels, a division per ray: 95 / 539 and 140 us).
// 6 CTAs (40 registers): 2 materials, 1 energy 73 -> 56 us against 58 registers.
// A detector has fewer than 2^32 pixels.  Grid: x = pixels, y = views.
template <int M>
__global__ void __launch_bounds__(256, 6) k_spectral_from_L(const MarchParams prm)
{
    extern __shared__ __align__(16) float s_mu[];
    load_mu(s_mu, prm.mu, prm.E, M);
    const unsigned U = (unsigned)prm.g.U, npix = U * (unsigned)prm.g.V;
    const int64_t pix = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (pix >= npix) return;
    const unsigned v = (unsigned)pix / U, u = (unsigned)pix - v * U;
    const PixelWeights W = pixel_weights(prm.W, prm.g.U, prm.E, (int)u, (int)v);
    for (int p = blockIdx.y; p < prm.g.P; p += gridDim.y) {
        const int64_t ray = (int64_t)p * npix + pix;
        float L[M];
        load_L<M>(prm.Lin, ray, L);
        float I, A;
        spectral<M>(s_mu, prm.E, W, L, I, A);
        if (prm.I) prm.I[ray] = I;
        if (prm.IAbs) prm.IAbs[ray] = A;
    }
}

// Adjoint: spectral-weight recompute from the checkpoint, then the matched
// ray march scattering the transposed trilinear weights with vector
// reductions.  FROM_GL: the input is dLoss/dL directly (transpose of the line
// integrals).
//
// Grid: x = pixel tiles along u, y = the view groups of one part of the views,
// z = pixel tiles along v of every part, so that the CTAs resident at any time
// cover one band of detector rows for many views.  The rays of a row band cross a thin z-slab of the volume (the cone
// angle is small), so the accumulator cells they reduce into stay in L2; with
// views outermost every view would sweep the whole accumulator through DRAM.
// Register cap for 4 CTAs of 256 threads (64 registers): more warps hide the
// reductions' latency.
// KIND: kEach, kMerge (merge_faces) or kDirect: no accumulators (prm.gcol null),
// the gradients take the sums.
enum { kEach, kMerge, kDirect };
template <int M, int MODE, bool FROM_GL, int KIND>
__global__ void __launch_bounds__(256, 4)
    k_backward(const MarchParams prm, int tile_u, int warp_rows, int tiles_v, int group0, bool parts_in_y)
{
    extern __shared__ __align__(16) float s_mu[];
    if (!FROM_GL) load_mu(s_mu, prm.mu, prm.E, M);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int tile_v = (int)blockDim.x / tile_u;
    const int wcols = 32 / warp_rows, warps_u = tile_u / wcols;
    const int u = blockIdx.x * tile_u + (w % warps_u) * wcols + lane / warp_rows;
    // the parts of the views: z, or interleaved in y (parts_in_y)
    const int parts = prm.sets / prm.set_columns;
    const int part = parts_in_y ? blockIdx.y % parts : blockIdx.z / tiles_v;
    const int group = group0 + (int)(parts_in_y ? blockIdx.y / parts : blockIdx.y), band = parts_in_y ? blockIdx.z : blockIdx.z % tiles_v;
    const int v = band * tile_v + (w / warps_u) * warp_rows + lane % warp_rows;
    const bool ray_on = u < prm.g.U && v < prm.g.V;
    const int64_t npix = (int64_t)prm.g.U * prm.g.V;
    const int64_t pix = (int64_t)v * prm.g.U + u;
    // the part's views, each part's as many as another's or one more
    const int first = prm.view0 + (int)((int64_t)prm.n_views * part / parts);
    const int pend = prm.view0 + (int)((int64_t)prm.n_views * (part + 1) / parts);
    const int set = part * prm.set_columns + (u & (prm.set_columns - 1));
    for (int k = 0; k < prm.views_per_cta; k++) {
        const int p = first + group * prm.views_per_cta + k;
        if (p >= pend) break;
        const int64_t ray = (int64_t)(p - prm.out_view0) * npix + pix;
        float g[M];
        bool any = false;
#pragma unroll
        for (int m = 0; m < M; m++) g[m] = 0.f;
        if (ray_on) {
            if (FROM_GL) {
                load_L<M>(prm.Lin, ray, g);
#pragma unroll
                for (int m = 0; m < M; m++) g[m] *= prm.g.dx;
            } else {
                float L[M], S[M];
                load_L<M>(prm.Lin, ray, L);
#pragma unroll
                for (int m = 0; m < M; m++) S[m] = 0.f;
                // the spectral weights as the forward formed them (transmit, the
                // same order), so S matches the fused kernels' exactly
                const int Ep = energy_groups(prm.E) * 4;
                for_energies<M>(s_mu, prm.E, pixel_weights(prm.W, prm.g.U, prm.E, u, v), L,
                                [&](int, int e, float att, float wt) {
                                    float ex, om;
                                    transmit(att, ex, om);
                                    const float Ie = wt * ex;
#pragma unroll
                                    for (int m = 0; m < M; m++) S[m] = fmaf(s_mu[m * Ep + e], Ie, S[m]);
                                });
                const float gd = ((prm.gIAbs ? prm.gIAbs[ray] : 0.f) - (prm.gI ? prm.gI[ray] : 0.f)) * prm.g.dx;
#pragma unroll
                for (int m = 0; m < M; m++) g[m] = gd * S[m];
            }
#pragma unroll
            for (int m = 0; m < M; m++) any |= (g[m] != 0.f);
        }
        // the transposed weights of the forward's sampler (for the texture
        // modes, the texture unit's, at the reference's FP32 coordinates)
        constexpr int SM = MODE == INTERP_TRILINEAR ? INTERP_TRILINEAR : INTERP_TEXEMU;
        if (KIND == kDirect) scatter_direct<M, SM>(prm.g, prm.gvol, any, p, v, u, g);
        else scatter_columns<M, SM, KIND == kMerge>(prm.g, prm.gcol + (size_t)set * prm.set_floats, any, p, v, u, g);
    }
}

// Adds the accumulators into the gradient volumes (fold_tile).  Block (32, 8);
// one block per tile, column_tile.
template <int M>
__global__ void __launch_bounds__(256) k_fold(const MarchParams prm)
{
    __shared__ float t[M][32][33];
    int x0, y, z0;
    column_tile(blockIdx.x, prm.g.nx, prm.g.nz, x0, y, z0);
    fold_tile<M>(prm.gcol, prm.sets, prm.set_floats, prm.gvol, prm.g.nx, prm.g.ny, prm.g.nz, x0, y, z0, t);
}

// W[e][k] = ((I0Val * S_e) * G_e) * D_e in the reference's multiplication order
// (CBCTPolyProjGPU.cu:1994), laid out as pixel_weights reads it; I0[k] = the sum over e
// (CBCTPolyForwardProjGrid.cpp:330-339).
__global__ void k_weights(const float* __restrict__ S, const float* __restrict__ G, int grid_layout,
                          const float* __restrict__ D, float I0Val, int E, int U, int V, float* W, float* I0)
{
    const int64_t npix = (int64_t)U * V;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < npix; k += (int64_t)gridDim.x * blockDim.x) {
        const int u = (int)(k % U), v = (int)(k / U);
        // the spectral epilogue's summation order (energy e into accumulator
        // e mod 4, E rounded down to a multiple of 4 first, the rest into
        // accumulator 0, combined pairwise), so that a ray with no attenuation
        // gives exactly I0
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        const auto Wp = pixel_weights_at<float4>(W, U, E, u, v);
        const auto weight = [&](int e) {
            float w = I0Val * S[e];
            if (grid_layout == 1) w = w * G[(int64_t)e * U + u];
            if (grid_layout == 2) w = w * G[(int64_t)e * npix + k];
            if (D) w = w * D[(int64_t)e * npix + k];
            return w;
        };
        const int full = E >> 2;
        for (int g = 0; g < full; g++) {
            float w[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                w[j] = weight(4 * g + j);
                s[j] += w[j];
            }
            Wp.full[g * 32] = make_float4(w[0], w[1], w[2], w[3]);
        }
        for (int e = 4 * full; e < E; e++) {
            const float w = weight(e);
            s[0] += w;
            Wp.rest[e * 32] = w;
        }
        I0[k] = (s[0] + s[1]) + (s[2] + s[3]);
    }
}

// Ipoly = (uint32)floorf(I); proj = logf(I0 / Ipoly) (CBCTForwardProj.cpp:79-90, 376-387).
__global__ void k_finalize(int64_t n_pix, int64_t n, const float* __restrict__ I, const float* __restrict__ IAbs,
                           const float* __restrict__ I0, uint32_t* Ipoly, uint32_t* IAbsPoly, float* proj)
{
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        if (I) {
            const uint32_t ip = (uint32_t)floorf(I[k]);
            if (Ipoly) Ipoly[k] = ip;
            if (proj && I0) proj[k] = logf(I0[k % n_pix] / (float)ip);
        }
        if (IAbs && IAbsPoly) IAbsPoly[k] = (uint32_t)floorf(IAbs[k]);
    }
}

__global__ void k_sample_points(const float* vol, cudaTextureObject_t tex, int nx, int ny, int nz, int interp,
                                const float* pts, int64_t n, float* out)
{
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const double cx = pts[3 * k], cy = pts[3 * k + 1], cz = pts[3 * k + 2];
        float val;
        if (interp == INTERP_TEXTURE) {
            val = tex3D<float>(tex, (float)(cx + 0.5), (float)(cy + 0.5), (float)(cz + 0.5));
        } else {
            const float* vp[1] = {vol};
            if (interp == INTERP_TEXEMU)
                gather_interp<1, INTERP_TEXEMU>(vp, nx, ny, nz, corner_of<INTERP_TEXEMU>(cx, cy, cz), &val);
            else
                gather_interp<1, INTERP_TRILINEAR>(vp, nx, ny, nz, corner_of<INTERP_TRILINEAR>(cx, cy, cz), &val);
        }
        out[k] = val;
    }
}

// Exact count of samples whose trilinear footprint touches the volume.
__global__ void k_count_support(const GeomParams g, unsigned long long* out)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y * blockDim.y + threadIdx.y;
    unsigned long long n = 0;
    if (u < g.U && v < g.V) {
        for (int p = blockIdx.z; p < g.P; p += gridDim.z) {
            const RaySeg s = ray_segment(g, p, v, u);
            for (int i = s.i0; i < s.i1; i++) {
                const double t = (double)i;
                const double cx = fma(t, s.bx, s.ax), cy = fma(t, s.by, s.ay), cz = fma(t, s.bz, s.az);
                n += (cx > -1.0 && cy > -1.0 && cz > -1.0 && cx < (double)g.nx && cy < (double)g.ny &&
                      cz < (double)g.nz);
            }
        }
    }
    // warp reduce then one atomic per warp
    for (int o = 16; o > 0; o >>= 1) n += __shfl_down_sync(0xffffffffu, n, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, n);
}

// ---------------------------------------------------------------------------
// Brick sampler: the CTA stages, for every segment of kBS consecutive samples,
// the box of voxels its ray bundle crosses in shared memory, and each sample
// reads its 8 corners from there (LDS) instead of through the texture unit.
// Rays of one CTA step through the same sample indices, so at any index their
// samples lie on a small patch: kBU x kBV rays about one voxel apart, swept
// kBS/2 voxels along the rays per segment.  The box origin and fit are
// computed per segment from the rays' first and last footprints (FP64
// coordinates are affine in the sample index, so their floors are monotone;
// the FP32 compat coordinates get a one-voxel margin).  A segment whose box
// does not fit, and any sample outside the box, reads the caller's volume
// instead, so the result never depends on the fit.
constexpr int kBU = 8, kBV = 16;             // rays per CTA: u x v
constexpr int kBX = 16, kBY = 16, kBZ = 20;  // box, voxels
constexpr int kBXp = 17;                     // row pitch (floats)
constexpr int kBZp = 296;                    // slice pitch: 17 * 16 + 24 = 8 (mod 32 banks)
constexpr int kBS = 16;                      // samples per segment
constexpr int kBoxFloats = kBZp * kBZ;       // one material's box

template <int MODE>
__device__ __forceinline__ Corner corner_at(const MarchParams& prm, const RaySeg& s, const RayRef32& r, int i)
{
    if (MODE == INTERP_TRILINEAR) {
        const double t = (double)i;
        return corner_of<INTERP_TRILINEAR>(fma(t, s.bx, s.ax), fma(t, s.by, s.ay), fma(t, s.bz, s.az));
    }
    return corner_tex(ref32_coords(prm.g, r, i));
}

template <int M, int MODE, bool SPECTRAL, int MINB>
__global__ void __launch_bounds__(kBU * kBV, MINB) k_forward_brick(const MarchParams prm)
{
    extern __shared__ __align__(16) float smem[];
    float* s_box = smem;                   // [M][kBZ][kBY][kBXp] (slices kBZp apart)
    float* s_mu = smem + M * kBoxFloats;   // [E][M]
    __shared__ int s_red[8];
    if (SPECTRAL) load_mu(s_mu, prm.mu, prm.E, M);
    const int tid = threadIdx.y * kBU + threadIdx.x;
    const int u = blockIdx.x * kBU + threadIdx.x;
    const int v = blockIdx.y * kBV + threadIdx.y;
    const bool live = u < prm.g.U && v < prm.g.V;
    const int64_t npix = (int64_t)prm.g.U * prm.g.V;
    const int64_t pix = (int64_t)v * prm.g.U + u;
    const int pend = prm.view0 + prm.n_views;
    constexpr int margin = MODE == INTERP_TRILINEAR ? 0 : 1;
    for (int k = 0; k < prm.views_per_cta; k++) {
        const int p = prm.view0 + blockIdx.z * prm.views_per_cta + k;
        if (p >= pend) break;
        RaySeg s;
        s.i0 = s.i1 = 0;
        if (live) s = ray_segment(prm.g, p, v, u);
        RayRef32 r;
        if (MODE != INTERP_TRILINEAR && live) r = ray_ref32(prm.g, p, v, u);
        if (tid == 0) {
            s_red[0] = INT_MAX;
            s_red[1] = INT_MIN;
        }
        __syncthreads();
        if (s.i1 > s.i0) {
            atomicMin(&s_red[0], s.i0);
            atomicMax(&s_red[1], s.i1);
        }
        __syncthreads();
        const int I0 = s_red[0], I1 = s_red[1];
        __syncthreads();
        float acc[M], cmp[M];
#pragma unroll
        for (int m = 0; m < M; m++) { acc[m] = 0.f; cmp[m] = 0.f; }
        for (int seg = I0; seg < I1; seg += kBS) {
            const int a0 = max(seg, s.i0), a1 = min(min(seg + kBS, I1), s.i1);
            if (tid == 0) {
                s_red[0] = s_red[1] = s_red[2] = INT_MAX;
                s_red[3] = s_red[4] = s_red[5] = INT_MIN;
            }
            __syncthreads();
            if (a0 < a1) {
                const Corner c0 = corner_at<MODE>(prm, s, r, a0), c1 = corner_at<MODE>(prm, s, r, a1 - 1);
                atomicMin(&s_red[0], min(c0.ix, c1.ix) - margin);
                atomicMin(&s_red[1], min(c0.iy, c1.iy) - margin);
                atomicMin(&s_red[2], min(c0.iz, c1.iz) - margin);
                atomicMax(&s_red[3], max(c0.ix, c1.ix) + margin);
                atomicMax(&s_red[4], max(c0.iy, c1.iy) + margin);
                atomicMax(&s_red[5], max(c0.iz, c1.iz) + margin);
            }
            __syncthreads();
            const int ox = s_red[0], oy = s_red[1], oz = s_red[2];
            const bool fits = s_red[3] >= ox && s_red[3] + 1 - ox < kBX && s_red[4] + 1 - oy < kBY &&
                              s_red[5] + 1 - oz < kBZ;
            if (fits) {
                // stage the box; voxels outside the volume read as 0 (border)
                const int nx = prm.g.nx, ny = prm.g.ny, nz = prm.g.nz;
                for (int idx = tid; idx < kBX * kBY * kBZ; idx += kBU * kBV) {
                    const int x = idx % kBX, y = (idx / kBX) % kBY, z = idx / (kBX * kBY);
                    const int gx = ox + x, gy = oy + y, gz = oz + z;
                    const bool in = (unsigned)gx < (unsigned)nx && (unsigned)gy < (unsigned)ny &&
                                    (unsigned)gz < (unsigned)nz;
                    const int64_t off = ((int64_t)gz * ny + gy) * nx + gx;
                    const int so = z * kBZp + y * kBXp + x;
#pragma unroll
                    for (int m = 0; m < M; m++) s_box[m * kBoxFloats + so] = in ? __ldg(prm.vol[m] + off) : 0.f;
                }
            }
            __syncthreads();
            for (int i = a0; i < a1; i++) {
                const Corner c = corner_at<MODE>(prm, s, r, i);
                const int bx = c.ix - ox, by = c.iy - oy, bz = c.iz - oz;
                float cv[M][8];
                if (fits && (unsigned)bx < (unsigned)(kBX - 1) && (unsigned)by < (unsigned)(kBY - 1) &&
                    (unsigned)bz < (unsigned)(kBZ - 1)) {
                    const int b = bz * kBZp + by * kBXp + bx;
#pragma unroll
                    for (int m = 0; m < M; m++) {
                        const float* q = s_box + m * kBoxFloats + b;
                        cv[m][0] = q[0]; cv[m][1] = q[1]; cv[m][2] = q[kBXp]; cv[m][3] = q[kBXp + 1];
                        cv[m][4] = q[kBZp]; cv[m][5] = q[kBZp + 1]; cv[m][6] = q[kBZp + kBXp];
                        cv[m][7] = q[kBZp + kBXp + 1];
                    }
                } else {
                    load8_global<M>(prm.vol, prm.g.nx, prm.g.ny, prm.g.nz, c, cv);
                }
#pragma unroll
                for (int m = 0; m < M; m++) kahan_add(acc[m], cmp[m], interp8<MODE>(c, cv[m]));
            }
            __syncthreads();
        }
        if (!live) continue;
        float L[M];
#pragma unroll
        for (int m = 0; m < M; m++) L[m] = prm.g.dx * (acc[m] - cmp[m]);
        const int64_t ray = (int64_t)(p - prm.out_view0) * npix + pix;
        if (prm.L) store_L<M>(prm.L, ray, L);
        if (SPECTRAL) {
            float I, A;
            spectral<M>(s_mu, prm.E, pixel_weights(prm.W, prm.g.U, prm.E, u, v), L, I, A);
            if (prm.I) prm.I[ray] = I;
            if (prm.IAbs) prm.IAbs[ray] = A;
        }
    }
}

// ---------------------------------------------------------------------------
// Brick sampler with TMA staging: the same boxes, the same fit rule and the
// same reads as k_forward_brick, but each box is one tensor load per material
// (cp.async.bulk.tensor.3d, issued by one thread, completion counted on an
// mbarrier) instead of 128 threads' scalar loads.  The box's x origin is
// rounded down to a multiple of 4 voxels, because a tiled tensor load must
// start on a 16-byte boundary in x, so kTX = 16 + 3 + 1 columns are staged;
// y and z start at the box origin, and voxels outside the volume (negative or
// past the end) arrive as zeros, the texture border.  The dense box layout is
// the one TMA writes: rows of kTX floats, slices of kTX * kBY floats.
//
// Every wait is bounded: thread 0 issues, all threads poll the mbarrier at
// most prm.wait_limit times; when any gives up, the CTA reads that segment and
// all later ones from the volume (same results), ors kCtfpStatusWaitTimeout
// into the plan's status word, and before exiting waits, again bounded, for
// the load still in flight so that it cannot land in shared memory the CTA no
// longer owns; when that exit wait runs out as well, it ors
// kCtfpStatusExitWaitTimeout, an error (outputs not trusted).
constexpr int kTX = 20;
constexpr int kTRow = kTX, kTSlice = kTX * kBY;
constexpr int kTBoxFloats = kTSlice * kBZ;  // 6400 floats = 25600 bytes, a multiple of 128
constexpr int kExitPolls = 1 << 22;

struct BrickMaps {
    CUtensorMap tm[kMaxM];
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded poll of one mbarrier phase; true when it completed.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, int limit)
{
    for (int k = 0; k < limit; k++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

__device__ __forceinline__ void tma_load_box(float* dst, const CUtensorMap* tm, int x, int y, int z, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar))
        : "memory");
}

template <int M, int MODE, bool SPECTRAL, int MINB>
__global__ void __launch_bounds__(kBU * kBV, MINB)
    k_forward_brick_tma(const MarchParams prm, const __grid_constant__ BrickMaps maps)
{
    extern __shared__ unsigned char smem_raw[];
    float* s_box = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    float* s_mu = s_box + M * kTBoxFloats;  // [E][M]
    __shared__ int s_red[8];
    __shared__ __align__(8) uint64_t s_bar;
    const int tid = threadIdx.y * kBU + threadIdx.x;
    if (tid == 0) mbar_init(&s_bar, 1);
    if (SPECTRAL) load_mu(s_mu, prm.mu, prm.E, M);
    __syncthreads();
    uint32_t phase = 0;
    bool staging = true;   // CTA-uniform: false once a wait ran out
    bool in_flight = false;  // CTA-uniform: a load whose completion was not seen
    const int u = blockIdx.x * kBU + threadIdx.x;
    const int v = blockIdx.y * kBV + threadIdx.y;
    const bool live = u < prm.g.U && v < prm.g.V;
    const int64_t npix = (int64_t)prm.g.U * prm.g.V;
    const int64_t pix = (int64_t)v * prm.g.U + u;
    const int pend = prm.view0 + prm.n_views;
    constexpr int margin = MODE == INTERP_TRILINEAR ? 0 : 1;
    for (int k = 0; k < prm.views_per_cta; k++) {
        const int p = prm.view0 + blockIdx.z * prm.views_per_cta + k;
        if (p >= pend) break;
        RaySeg s;
        s.i0 = s.i1 = 0;
        if (live) s = ray_segment(prm.g, p, v, u);
        RayRef32 r;
        if (MODE != INTERP_TRILINEAR && live) r = ray_ref32(prm.g, p, v, u);
        if (tid == 0) {
            s_red[0] = INT_MAX;
            s_red[1] = INT_MIN;
        }
        __syncthreads();
        if (s.i1 > s.i0) {
            atomicMin(&s_red[0], s.i0);
            atomicMax(&s_red[1], s.i1);
        }
        __syncthreads();
        const int I0 = s_red[0], I1 = s_red[1];
        __syncthreads();
        float acc[M], cmp[M];
#pragma unroll
        for (int m = 0; m < M; m++) { acc[m] = 0.f; cmp[m] = 0.f; }
        for (int seg = I0; seg < I1; seg += kBS) {
            const int a0 = max(seg, s.i0), a1 = min(min(seg + kBS, I1), s.i1);
            if (tid == 0) {
                s_red[0] = s_red[1] = s_red[2] = INT_MAX;
                s_red[3] = s_red[4] = s_red[5] = INT_MIN;
            }
            __syncthreads();
            if (a0 < a1) {
                const Corner c0 = corner_at<MODE>(prm, s, r, a0), c1 = corner_at<MODE>(prm, s, r, a1 - 1);
                atomicMin(&s_red[0], min(c0.ix, c1.ix) - margin);
                atomicMin(&s_red[1], min(c0.iy, c1.iy) - margin);
                atomicMin(&s_red[2], min(c0.iz, c1.iz) - margin);
                atomicMax(&s_red[3], max(c0.ix, c1.ix) + margin);
                atomicMax(&s_red[4], max(c0.iy, c1.iy) + margin);
                atomicMax(&s_red[5], max(c0.iz, c1.iz) + margin);
            }
            __syncthreads();
            const int ox = s_red[0], oy = s_red[1], oz = s_red[2];
            bool fits = staging && s_red[3] >= ox && s_red[3] + 1 - ox < kBX && s_red[4] + 1 - oy < kBY &&
                        s_red[5] + 1 - oz < kBZ;
            const int ox4 = ox & ~3;  // floor to a multiple of 4: the load starts on a 16-byte boundary
            if (fits) {
                if (tid == 0) {
                    mbar_expect_tx(&s_bar, (uint32_t)(M * kTBoxFloats * sizeof(float)));
#pragma unroll
                    for (int m = 0; m < M; m++) tma_load_box(s_box + m * kTBoxFloats, &maps.tm[m], ox4, oy, oz, &s_bar);
                }
                const bool done = mbar_wait_bounded(&s_bar, phase, prm.wait_limit);
                if (__syncthreads_and(done)) {
                    phase ^= 1u;
                } else {
                    // give up staging in this CTA; the load may still land
                    staging = false;
                    in_flight = true;
                    fits = false;
                    if (tid == 0 && prm.status) atomicOr(prm.status, kCtfpStatusWaitTimeout);
                }
            }
            const int dxa = ox - ox4;
            for (int i = a0; i < a1; i++) {
                const Corner c = corner_at<MODE>(prm, s, r, i);
                const int bx = c.ix - ox, by = c.iy - oy, bz = c.iz - oz;
                float cv[M][8];
                if (fits && (unsigned)bx < (unsigned)(kBX - 1) && (unsigned)by < (unsigned)(kBY - 1) &&
                    (unsigned)bz < (unsigned)(kBZ - 1)) {
                    const int b = bz * kTSlice + by * kTRow + bx + dxa;
#pragma unroll
                    for (int m = 0; m < M; m++) {
                        const float* q = s_box + m * kTBoxFloats + b;
                        cv[m][0] = q[0]; cv[m][1] = q[1]; cv[m][2] = q[kTRow]; cv[m][3] = q[kTRow + 1];
                        cv[m][4] = q[kTSlice]; cv[m][5] = q[kTSlice + 1]; cv[m][6] = q[kTSlice + kTRow];
                        cv[m][7] = q[kTSlice + kTRow + 1];
                    }
                } else {
                    load8_global<M>(prm.vol, prm.g.nx, prm.g.ny, prm.g.nz, c, cv);
                }
#pragma unroll
                for (int m = 0; m < M; m++) kahan_add(acc[m], cmp[m], interp8<MODE>(c, cv[m]));
            }
            __syncthreads();  // the box is read; the next segment may overwrite it
        }
        if (!live) continue;
        float L[M];
#pragma unroll
        for (int m = 0; m < M; m++) L[m] = prm.g.dx * (acc[m] - cmp[m]);
        const int64_t ray = (int64_t)(p - prm.out_view0) * npix + pix;
        if (prm.L) store_L<M>(prm.L, ray, L);
        if (SPECTRAL) {
            float I, A;
            spectral<M>(s_mu, prm.E, pixel_weights(prm.W, prm.g.U, prm.E, u, v), L, I, A);
            if (prm.I) prm.I[ray] = I;
            if (prm.IAbs) prm.IAbs[ray] = A;
        }
    }
    // a load given up on may still be writing the box: wait for it (bounded)
    // before the CTA's shared memory is released; if that wait runs out too,
    // the copy may land in shared memory another CTA then owns, which the
    // plan's status word reports as an error (kCtfpStatusExitWaitTimeout)
    if (in_flight) {
        const bool landed = mbar_wait_bounded(&s_bar, phase, kExitPolls);
        if (!landed && tid == 0 && prm.status) atomicOr(prm.status, kCtfpStatusExitWaitTimeout);
    }
}

// The dynamic shared-memory opt-in is per device and per kernel; plans on
// other threads may get here at the same time (setting it twice is harmless).
template <typename K>
cudaError_t opt_in_smem(K kernel, std::atomic<unsigned long long>& done)
{
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && (done.load() >> dev & 1ull)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e == cudaSuccess && dev < 64) done.fetch_or(1ull << dev);
    return e;
}

template <int M, int MODE, bool SPEC>
cudaError_t brick_launch(const MarchParams& prm, const BrickMaps* maps, dim3 grid, size_t smem_loads, size_t smem_tma,
                         cudaStream_t st)
{
    static std::atomic<unsigned long long> set_loads{0}, set_tma{0};
    if (maps) {
        const cudaError_t e = opt_in_smem(k_forward_brick_tma<M, MODE, SPEC, 4>, set_tma);
        if (e != cudaSuccess) return e;
        k_forward_brick_tma<M, MODE, SPEC, 4><<<grid, dim3(kBU, kBV), smem_tma, st>>>(prm, *maps);
    } else {
        const cudaError_t e = opt_in_smem(k_forward_brick<M, MODE, SPEC, 4>, set_loads);
        if (e != cudaSuccess) return e;
        k_forward_brick<M, MODE, SPEC, 4><<<grid, dim3(kBU, kBV), smem_loads, st>>>(prm);
    }
    return cudaGetLastError();
}

template <int M>
cudaError_t brick_dispatch(const MarchParams& prm, int interp, bool spec, const BrickMaps* maps, dim3 grid,
                           size_t smem_loads, size_t smem_tma, cudaStream_t st)
{
    if (interp == INTERP_TRILINEAR)
        return spec ? brick_launch<M, INTERP_TRILINEAR, true>(prm, maps, grid, smem_loads, smem_tma, st)
                    : brick_launch<M, INTERP_TRILINEAR, false>(prm, maps, grid, smem_loads, smem_tma, st);
    if (interp == INTERP_TEXEMU)
        return spec ? brick_launch<M, INTERP_TEXEMU, true>(prm, maps, grid, smem_loads, smem_tma, st)
                    : brick_launch<M, INTERP_TEXEMU, false>(prm, maps, grid, smem_loads, smem_tma, st);
    return cudaErrorInvalidValue;
}

// cuTensorMapEncodeTiled from the driver, looked up once through the runtime
// (no link-time dependency on libcuda).
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled()
{
    static std::once_flag once;
    static EncodeTiledFn fn = nullptr;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(f);
    });
    return fn;
}

// Tensor maps of the M volumes for the TMA-staged boxes, when the volumes
// allow them: rows of a multiple of 16 bytes (pNumX % 4 == 0) and every base
// address on a 16-byte boundary.  False: stage with plain loads.
bool brick_maps(const MarchParams& prm, int M, BrickMaps& bm)
{
    const char* mode = std::getenv("CTFP_BRICK_STAGING");
    if (mode && std::strcmp(mode, "loads") == 0) return false;
    const EncodeTiledFn fn = encode_tiled();
    if (!fn) return false;
    const int nx = prm.g.nx, ny = prm.g.ny, nz = prm.g.nz;
    if (nx % 4 != 0) return false;
    std::memset(&bm, 0, sizeof(bm));
    for (int m = 0; m < M; m++) {
        if (reinterpret_cast<uintptr_t>(prm.vol[m]) % 16 != 0) return false;
        const cuuint64_t dims[3] = {(cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz};
        const cuuint64_t strides[2] = {(cuuint64_t)nx * sizeof(float), (cuuint64_t)nx * ny * sizeof(float)};
        const cuuint32_t box[3] = {(cuuint32_t)kTX, (cuuint32_t)kBY, (cuuint32_t)kBZ};
        const cuuint32_t estride[3] = {1, 1, 1};
        if (fn(&bm.tm[m], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(prm.vol[m]), dims, strides, box,
               estride, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    return true;
}

template <int M, int MODE, int SAMPLER, int MINB>
cudaError_t fwd_launch(const MarchParams& prm, bool spec, dim3 grid, dim3 block, size_t smem, cudaStream_t st)
{
    if (spec) k_forward<M, MODE, SAMPLER, true, MINB><<<grid, block, smem, st>>>(prm);
    else k_forward<M, MODE, SAMPLER, false, MINB><<<grid, block, 0, st>>>(prm);
    return cudaGetLastError();
}

template <int M, int MODE, int SAMPLER>
cudaError_t fwd_dispatch_spec(const MarchParams& prm, bool spec, int minb, dim3 grid, dim3 block, size_t smem,
                              cudaStream_t st)
{
    switch (minb) {
        case 3: return fwd_launch<M, MODE, SAMPLER, 3>(prm, spec, grid, block, smem, st);
        case 4:
        case 5: return fwd_launch<M, MODE, SAMPLER, 4>(prm, spec, grid, block, smem, st);
        default: return fwd_launch<M, MODE, SAMPLER, 2>(prm, spec, grid, block, smem, st);
    }
}

template <int M>
cudaError_t fwd_dispatch_mode(const MarchParams& prm, int interp, int sampler, bool spec, int minb, dim3 grid,
                              dim3 block, size_t smem, cudaStream_t st)
{
    const bool lay = sampler == SAMPLER_LAYERED;
    switch (interp) {
        case INTERP_TRILINEAR:
            if (lay && prm.occ)
                return fwd_dispatch_spec<M, INTERP_TRILINEAR, SAMPLER_LAYERED_SKIP>(prm, spec, minb, grid, block, smem, st);
            return lay ? fwd_dispatch_spec<M, INTERP_TRILINEAR, SAMPLER_LAYERED>(prm, spec, minb, grid, block, smem, st)
                       : fwd_dispatch_spec<M, INTERP_TRILINEAR, SAMPLER_GLOBAL>(prm, spec, minb, grid, block, smem, st);
        case INTERP_TEXEMU:
            if (lay && prm.occ)
                return fwd_dispatch_spec<M, INTERP_TEXEMU, SAMPLER_LAYERED_SKIP>(prm, spec, minb, grid, block, smem, st);
            return lay ? fwd_dispatch_spec<M, INTERP_TEXEMU, SAMPLER_LAYERED>(prm, spec, minb, grid, block, smem, st)
                       : fwd_dispatch_spec<M, INTERP_TEXEMU, SAMPLER_GLOBAL>(prm, spec, minb, grid, block, smem, st);
        case INTERP_TEXTURE:
            if (prm.occ)
                return fwd_dispatch_spec<M, INTERP_TEXTURE, SAMPLER_LAYERED_SKIP>(prm, spec, minb, grid, block, smem, st);
            return fwd_dispatch_spec<M, INTERP_TEXTURE, SAMPLER_GLOBAL>(prm, spec, minb, grid, block, smem, st);
    }
    return cudaErrorInvalidValue;
}

// Rows of the detector a warp of the axis kernel covers (32 / rows columns):
// 8 rows x 4 columns measured 1-2 % faster than 4 x 8 and 16 x 2 on
// poly_grid_256 (53.6 against 54.1 and 54.5 ms).
constexpr int kAxisWarpRows = 8;

template <int M, int MODE, bool SKIP, int MINB>
cudaError_t axis_launch(const MarchParams& prm, bool spec, int tile_u, dim3 grid, dim3 block, size_t smem,
                        cudaStream_t st)
{
    int wr = kAxisWarpRows;
    const int tile_v = (int)block.x / tile_u;
    if (tile_u % (32 / wr) != 0 || tile_v % wr != 0) wr = 4;
    if (spec) k_forward_axis<M, MODE, SKIP, true, MINB><<<grid, block, smem, st>>>(prm, tile_u, wr);
    else k_forward_axis<M, MODE, SKIP, false, MINB><<<grid, block, 0, st>>>(prm, tile_u, wr);
    return cudaGetLastError();
}

template <int M, int MODE, bool SKIP>
cudaError_t axis_dispatch_minb(const MarchParams& prm, bool spec, int minb, int tile_u, dim3 grid, dim3 block,
                               size_t smem, cudaStream_t st)
{
    switch (minb) {
        case 3: return axis_launch<M, MODE, SKIP, 3>(prm, spec, tile_u, grid, block, smem, st);
        case 4: return axis_launch<M, MODE, SKIP, 4>(prm, spec, tile_u, grid, block, smem, st);
        case 5: return axis_launch<M, MODE, SKIP, 5>(prm, spec, tile_u, grid, block, smem, st);
        default: return axis_launch<M, MODE, SKIP, 2>(prm, spec, tile_u, grid, block, smem, st);
    }
}

template <int M>
cudaError_t axis_dispatch(const MarchParams& prm, int interp, bool spec, int minb, int tile_u, dim3 grid,
                          dim3 block, size_t smem, cudaStream_t st)
{
    const bool skip = prm.occ != nullptr;
    if (interp == INTERP_TRILINEAR)
        return skip ? axis_dispatch_minb<M, INTERP_TRILINEAR, true>(prm, spec, minb, tile_u, grid, block, smem, st)
                    : axis_dispatch_minb<M, INTERP_TRILINEAR, false>(prm, spec, minb, tile_u, grid, block, smem, st);
    if (interp == INTERP_TEXEMU)
        return skip ? axis_dispatch_minb<M, INTERP_TEXEMU, true>(prm, spec, minb, tile_u, grid, block, smem, st)
                    : axis_dispatch_minb<M, INTERP_TEXEMU, false>(prm, spec, minb, tile_u, grid, block, smem, st);
    return cudaErrorInvalidValue;
}

// Whether the scatter of three or four materials hands sums over between rows
// (flush_voxels): the shuffles pay while neighbouring rows mostly flush
// neighbouring voxels (spacing), there are neighbours in a warp (rows), and the
// L2's reductions bind rather than a ray's own chain: from a full chip of rays
// on, and for the texture emulation, whose samples cost more instructions, where
// the accumulators are large or the rays dense.  Measured, adjoint + fold, each
// lane on its own / merged, ms -- trilinear, 3 materials: 64^3, row spacing 1.3
// voxels 0.392 / 0.346, 176^3, 1.0 5.69 / 4.37, 128^3, 2.0 1.00 / 1.08; 96 x 96 x
// 16, 180 views of 1 / 2 / 3 / 5 / 8 / 13 rows 0.19 / 0.29, 0.20 / 0.30, 0.28 / 0.35,
// 0.36 / 0.43, 0.55 / 0.46, 0.67 / 0.53; 32^3, 46 k rays 0.085 / 0.103; texture emulation: 96^3, 1.0
// 1.03 / 1.06, 0.8 (180 views) 4.63 / 3.77, 128^3, 0.5 3.76 / 3.22, 256^3, 1.3 9.47 /
// 8.66, 128^3, 2.0 1.03 / 1.13, 96 x 96 x 16, 8 rows 0.8 0.59 / 0.51.
bool merge_faces(const MarchParams& prm, int interp)
{
    const GeomParams& g = prm.g;
    const float rows = g.dSize * g.sod / (g.sdd * g.pSizeZ);
    if (rows >= 1.8f || g.V < 8 || (int64_t)prm.n_views * g.U * g.V < 150000) return false;
    return interp == INTERP_TRILINEAR || rows < 0.9f || (int64_t)g.nx * g.ny * g.nz > 2000000;
}

struct BwdGrid {
    int tile_u, rows, tiles_v, group0;
    bool parts_in_y;
    dim3 grid, block;
    size_t smem;
};

template <int M, int MODE, bool FROM_GL>
cudaError_t bwd_launch(const MarchParams& prm, const BwdGrid& b, cudaStream_t st)
{
    const size_t smem = FROM_GL ? 0 : b.smem;
    auto k = k_backward<M, MODE, FROM_GL, kEach>;
    if (!prm.gcol) k = k_backward<M, MODE, FROM_GL, kDirect>;
    else if (M > 2 && merge_faces(prm, MODE)) k = k_backward<M, MODE, FROM_GL, (M > 2 ? kMerge : kEach)>;
    k<<<b.grid, b.block, smem, st>>>(prm, b.tile_u, b.rows, b.tiles_v, b.group0, b.parts_in_y);
    return cudaGetLastError();
}

// log2 of the lanes per ray of a plan's march: 0 is k_forward_axis, one thread
// per ray.  It depends on the plan alone, so that every call of it (a range of its
// views, any launch shape) sums a ray the same way.  The chip holds 148 x 1024
// threads of the march at a time (148 x 768 of four materials'): while the rays
// leave it part empty, the time is one ray's chain of gathers, and as many lanes
// share a ray as fit.  Past that 2 lanes still pay, by a shorter last wave, the
// longer the rays are: up to some 5500 rays for each voxel of nx + ny (2 samples a
// voxel; where empty space is skipped, half of them).  Measured, us a forward with 1
// / 2 / 4 / 8 lanes per ray, 2 materials -- 18 k rays of 32^3 50 / 29 / 28 / 28, 64^3 89 /
// 46 / 31 / 31, 128^3 204 / 90 / 67 / 56 (4 materials 183 / 68 / 49 / 63), 256^3 769 / 352 /
// 269 / 233; 55 k of 32^3 48 / 31 / 35 / 44, 128^3 199 / 91 / 99 / 99; 197 k of 32^3 77 / 72 /
// 85 / 117, 128^3 272 / 219 / 220 / 249; 390 k of 32^3 124 / 126 / 152 / 218, 64^3 220 / 202 /
// 228 / 295, 256^3 1303 / 1039 / 1098 / 1221; 688 k of 32^3 197 / 210 / 258 / 376, 64^3 349 /
// 340 / 389 / 510 (half of it empty and skipped 356 / 379), 128^3 691 / 631 / 659 / 771;
// 897 k of 64^3 440 / 434, 128^3 849 / 804, 256^3 2189 / 2135, 3 and 4 materials 3789 / 3940, 3272 / 3656.
int axis_split(const GeomParams& g, int M, bool skip)
{
    const int64_t rays = (int64_t)g.U * g.V * g.P, chip = 148 * (uses_columns(M) ? 768 : 1024);
    const int64_t voxels = (int64_t)(g.nx + g.ny) >> (skip ? 1 : 0);
    if (rays > std::max<int64_t>(chip, std::min<int64_t>(700000, 5500 * voxels))) return 0;
    return 8 * rays <= chip ? 3 : 4 * rays <= chip ? 2 : 1;
}

template <int M, int MODE, bool SKIP>
cudaError_t split_launch(const MarchParams& prm, bool spec, int shift, cudaStream_t st)
{
    const size_t smem = spec ? sizeof(float) * (size_t)energy_groups(prm.E) * 4 * M : 0;
    // no more rows than the detector has (one row of 400 pixels, 360 views of 128^2,
    // 4 lanes a ray, 8 rows / 1: 830 / 168 us)
    int rows = 32 >> shift;
    while (rows > 1 && rows / 2 >= prm.g.V) rows /= 2;
    const int cols = 4 * (32 >> shift) / rows;  // of a CTA
    const dim3 grid((prm.g.U + cols - 1) / cols, (prm.g.V + rows - 1) / rows, prm.n_views);
    if (grid.x == 0 || grid.y == 0 || grid.z == 0) return cudaSuccess;
    if (spec) k_forward_axis_split<M, MODE, SKIP, true><<<grid, 128, smem, st>>>(prm, shift, rows);
    else k_forward_axis_split<M, MODE, SKIP, false><<<grid, 128, smem, st>>>(prm, shift, rows);
    return cudaGetLastError();
}

template <int M>
cudaError_t split_dispatch(const MarchParams& prm, int interp, bool spec, int shift, cudaStream_t st)
{
    const bool skip = prm.occ != nullptr;
    if (interp == INTERP_TRILINEAR)
        return skip ? split_launch<M, INTERP_TRILINEAR, true>(prm, spec, shift, st)
                    : split_launch<M, INTERP_TRILINEAR, false>(prm, spec, shift, st);
    return skip ? split_launch<M, INTERP_TEXEMU, true>(prm, spec, shift, st)
                : split_launch<M, INTERP_TEXEMU, false>(prm, spec, shift, st);
}

template <int M>
cudaError_t bwd_dispatch(const MarchParams& prm, int interp, bool from_gL, const BwdGrid& b, cudaStream_t st)
{
    const bool tri = interp == INTERP_TRILINEAR;
    if (from_gL)
        return tri ? bwd_launch<M, INTERP_TRILINEAR, true>(prm, b, st) : bwd_launch<M, INTERP_TEXEMU, true>(prm, b, st);
    return tri ? bwd_launch<M, INTERP_TRILINEAR, false>(prm, b, st) : bwd_launch<M, INTERP_TEXEMU, false>(prm, b, st);
}

dim3 march_grid(const MarchParams& prm, const LaunchShape& ls)
{
    return dim3((prm.g.U + ls.tile_u - 1) / ls.tile_u, (prm.g.V + ls.tile_v - 1) / ls.tile_v,
                (prm.n_views + ls.views_per_cta - 1) / ls.views_per_cta);
}

}  // namespace

namespace {

// One launch over prm.n_views views (at most 65535 view groups: grid.z).
cudaError_t launch_forward_once(const MarchParams& prm, int M, int interp, int sampler, bool do_spectral,
                                const LaunchShape& ls, cudaStream_t st)
{
    if (sampler == SAMPLER_BRICK && interp != INTERP_TEXTURE) {
        const dim3 grid((prm.g.U + kBU - 1) / kBU, (prm.g.V + kBV - 1) / kBV,
                        (prm.n_views + ls.views_per_cta - 1) / ls.views_per_cta);
        if (grid.z == 0) return cudaSuccess;
        const size_t mu_floats = do_spectral ? (size_t)energy_groups(prm.E) * 4 * M : 0;
        const size_t smem = sizeof(float) * ((size_t)M * kBoxFloats + mu_floats);
        const size_t smem_tma = 128 + sizeof(float) * ((size_t)M * kTBoxFloats + mu_floats);  // + alignment slack
        BrickMaps bm;
        const BrickMaps* maps = brick_maps(prm, M, bm) ? &bm : nullptr;
        switch (M) {
            case 1: return brick_dispatch<1>(prm, interp, do_spectral, maps, grid, smem, smem_tma, st);
            case 2: return brick_dispatch<2>(prm, interp, do_spectral, maps, grid, smem, smem_tma, st);
            case 3: return brick_dispatch<3>(prm, interp, do_spectral, maps, grid, smem, smem_tma, st);
            case 4: return brick_dispatch<4>(prm, interp, do_spectral, maps, grid, smem, smem_tma, st);
        }
        return cudaErrorInvalidValue;
    }
    if (forward_splits(prm, M, interp, sampler)) {
        const int shift = axis_split(prm.g, M, prm.occ);
        switch (M) {
            case 1: return split_dispatch<1>(prm, interp, do_spectral, shift, st);
            case 2: return split_dispatch<2>(prm, interp, do_spectral, shift, st);
            case 3: return split_dispatch<3>(prm, interp, do_spectral, shift, st);
            case 4: return split_dispatch<4>(prm, interp, do_spectral, shift, st);
        }
        return cudaErrorInvalidValue;
    }
    if (sampler == SAMPLER_AXIS && interp != INTERP_TEXTURE) {
        // lane quads run down 4 detector rows and a warp covers 8 columns:
        // tiles whose height is not a multiple of 4, or whose width is not a
        // multiple of 8, use 16 x 16
        LaunchShape as = ls;
        if (as.tile_v % 4 != 0 || as.tile_u % 8 != 0 || as.tile_u * as.tile_v > 256 ||
            (as.tile_u * as.tile_v) % 32 != 0) {
            as.tile_u = 16;
            as.tile_v = 16;
        }
        const dim3 block(as.tile_u * as.tile_v), grid = march_grid(prm, as);
        const size_t smem = do_spectral ? sizeof(float) * (size_t)energy_groups(prm.E) * 4 * M : 0;
        if (grid.x == 0 || grid.y == 0 || grid.z == 0) return cudaSuccess;
        switch (M) {
            case 1: return axis_dispatch<1>(prm, interp, do_spectral, as.min_ctas, as.tile_u, grid, block, smem, st);
            case 2: return axis_dispatch<2>(prm, interp, do_spectral, as.min_ctas, as.tile_u, grid, block, smem, st);
            case 3: return axis_dispatch<3>(prm, interp, do_spectral, as.min_ctas, as.tile_u, grid, block, smem, st);
            case 4: return axis_dispatch<4>(prm, interp, do_spectral, as.min_ctas, as.tile_u, grid, block, smem, st);
        }
        return cudaErrorInvalidValue;
    }
    const dim3 block(ls.tile_u, ls.tile_v), grid = march_grid(prm, ls);
    const size_t smem = do_spectral ? sizeof(float) * (size_t)energy_groups(prm.E) * 4 * M : 0;
    if (grid.x == 0 || grid.y == 0 || grid.z == 0) return cudaSuccess;
    switch (M) {
        case 1: return fwd_dispatch_mode<1>(prm, interp, sampler, do_spectral, ls.min_ctas, grid, block, smem, st);
        case 2: return fwd_dispatch_mode<2>(prm, interp, sampler, do_spectral, ls.min_ctas, grid, block, smem, st);
        case 3: return fwd_dispatch_mode<3>(prm, interp, sampler, do_spectral, ls.min_ctas, grid, block, smem, st);
        case 4: return fwd_dispatch_mode<4>(prm, interp, sampler, do_spectral, ls.min_ctas, grid, block, smem, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

bool forward_splits(const MarchParams& prm, int M, int interp, int sampler)
{
    return sampler == SAMPLER_AXIS && interp != INTERP_TEXTURE && axis_split(prm.g, M, prm.occ) > 0;
}

cudaError_t launch_forward(const MarchParams& prm_in, int M, int interp, int sampler, bool do_spectral,
                           const LaunchShape& ls, cudaStream_t st)
{
    // view groups run along grid.z, at most 65535 per launch
    const int vpc = forward_splits(prm_in, M, interp, sampler) ? 1 : ls.views_per_cta;
    const int max_views = 65535 * vpc;
    for (int v0 = 0; v0 < prm_in.n_views; v0 += max_views) {
        MarchParams prm = prm_in;
        prm.views_per_cta = vpc;
        prm.view0 = prm_in.view0 + v0;
        prm.n_views = std::min(max_views, prm_in.n_views - v0);
        const cudaError_t e = launch_forward_once(prm, M, interp, sampler, do_spectral, ls, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_axis_gather_count(const GeomParams& g, int interp, const LaunchShape& ls, unsigned long long* out,
                                     cudaStream_t st)
{
    LaunchShape as = ls;
    if (as.tile_v % 4 != 0 || as.tile_u % 8 != 0 || as.tile_u * as.tile_v > 256 || (as.tile_u * as.tile_v) % 32 != 0) {
        as.tile_u = 16;
        as.tile_v = 16;
    }
    int wr = kAxisWarpRows;
    if (as.tile_u % (32 / wr) != 0 || as.tile_v % wr != 0) wr = 4;
    for (int p0 = 0; p0 < g.P; p0 += 65535) {
        GeomParams gv = g;
        const int n = std::min(65535, g.P - p0);
        gv.trig = g.trig + p0;  // views p0 .. p0 + n - 1 as views 0 .. n - 1
        gv.trigf = g.trigf + p0;
        if (g.fspot) gv.fspot = g.fspot + p0;
        gv.P = n;
        const dim3 grid((g.U + as.tile_u - 1) / as.tile_u, (g.V + as.tile_v - 1) / as.tile_v, n);
        if (interp == INTERP_TRILINEAR) k_axis_gather_count<INTERP_TRILINEAR><<<grid, as.tile_u * as.tile_v, 0, st>>>(gv, as.tile_u, wr, out);
        else k_axis_gather_count<INTERP_TEXEMU><<<grid, as.tile_u * as.tile_v, 0, st>>>(gv, as.tile_u, wr, out);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_axis_zero_pads(int nx, int ny, int nz, cudaSurfaceObject_t xs, cudaSurfaceObject_t ys,
                                  cudaStream_t st)
{
    // x-layered: texels (y, z), layers 0 and nx + 1; y-layered: texels (x, z), layers 0 and ny + 1
    k_axis_zero_layer<<<64, 256, 0, st>>>(xs, ny, nz, 0);
    k_axis_zero_layer<<<64, 256, 0, st>>>(xs, ny, nz, nx + 1);
    k_axis_zero_layer<<<64, 256, 0, st>>>(ys, nx, nz, 0);
    k_axis_zero_layer<<<64, 256, 0, st>>>(ys, nx, nz, ny + 1);
    return cudaGetLastError();
}

cudaError_t launch_axis_fill(const AxisCopies& copies, int M, int nx, int ny, int nz, cudaStream_t st)
{
    // grid.z holds at most 65535 slices
    const int per = std::max(1, std::min(M, 65535 / nz));
    for (int m = 0; m < M; m += per) {
        const int n = std::min(per, M - m);
        AxisCopies c = copies;
        for (int k = 0; k < n; k++) {
            c.vol[k] = copies.vol[m + k];
            c.xs[k] = copies.xs[m + k];
            c.ys[k] = copies.ys[m + k];
        }
        k_axis_fill<<<dim3((nx + 31) / 32, (ny + 31) / 32, nz * n), dim3(32, 8), 0, st>>>(c, nx, ny, nz);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

bool axis_uses_columns(int M) { return uses_columns(M); }

size_t column_floats(int nx, int ny, int nz) { return column_dims(nx, ny, nz).elems * 4; }

cudaError_t launch_column_fill(const float* const* vol, int nx, int ny, int nz, float* cvol, cudaStream_t st)
{
    VolPtrs vp = {};
    for (int m = 0; m < kMaxM; m++) vp.p[m] = vol[m];
    k_column_fill<<<(unsigned)column_tiles(nx, ny, nz), dim3(32, 8), 0, st>>>(vp, nx, ny, nz, cvol);
    return cudaGetLastError();
}

cudaError_t launch_spectral_from_L(const MarchParams& prm, int M, cudaStream_t st)
{
    const dim3 block(256, 1);
    const int64_t npix = (int64_t)prm.g.U * prm.g.V;
    if (npix == 0 || prm.g.P == 0) return cudaSuccess;
    // some blocks per SM, each over several views: a block's start is paid for by
    // them, and with few energies by more of them (32 / 64 blocks per SM, 512 x 256
    // pixels, 90 views: 1 energy 54 / 56 us, 61 energies 552 / 539)
    const int64_t gx = (npix + 255) / 256, blocks = 148 * (prm.E < 16 ? 32 : 64);
    const dim3 nb((unsigned)gx, (unsigned)std::max<int64_t>(1, std::min<int64_t>(prm.g.P, blocks / gx)));
    const size_t smem = sizeof(float) * (size_t)energy_groups(prm.E) * 4 * M;
    switch (M) {
        case 1: k_spectral_from_L<1><<<nb, block, smem, st>>>(prm); break;
        case 2: k_spectral_from_L<2><<<nb, block, smem, st>>>(prm); break;
        case 3: k_spectral_from_L<3><<<nb, block, smem, st>>>(prm); break;
        case 4: k_spectral_from_L<4><<<nb, block, smem, st>>>(prm); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

bool accum_fits(int nx, int ny, int nz) { return column_fits(nx, ny, nz); }

int accum_set_count(const GeomParams& g, int n_views, int M) { return accum_sets(g, n_views, M, kMostSets).total(); }

void set_accum_sets(MarchParams& prm, int M, int most)
{
    const AccumSets s = accum_sets(prm.g, prm.n_views, M, most);
    prm.sets = s.total();
    prm.set_columns = s.columns;
}

size_t accum_floats(int nx, int ny, int nz, int M) { return column_dims(nx, ny, nz).elems * accum_width(M); }

cudaError_t launch_backward(const MarchParams& prm_in, int M, int interp, bool from_gL, const LaunchShape& ls,
                            cudaStream_t st)
{
    // Rows of the detector a warp covers (32 / rows columns).  Its lanes' z
    // neighbours share sectors, so taller is better until the rows stop
    // crossing layers together: 16 rows, and 32 where the rows lie close
    // together and several lanes flush the same cell.  Measured, adjoint +
    // fold of 24 views of 128^3, row spacing in voxels: 8 / 16 / 32 rows, ms --
    // 1 material 0.25: 4.72 / 3.78 / 3.75, 0.6: 1.05 / 1.02 / 1.09, 1.05: 0.46 /
    // 0.47 / 0.49; 3 materials 0.25: 11.96 / 10.07 / 9.17, 1.05: 0.86 / 0.84 / 0.88.
    // A detector of fewer rows: no more than hold them all (one row, 96 x 96 x 16, 180
    // views, 4 rows / 1, 1 material 0.167 / 0.131, 3 materials 0.345 / 0.192).
    const GeomParams& g = prm_in.g;
    int rows = g.dSize * g.sod < 0.35f * g.sdd * g.pSizeZ ? 32 : 16;
    while (rows > 1 && rows / 2 >= g.V) rows /= 2;
    const int threads = ls.tile_u * ls.tile_v;
    LaunchShape bs = ls;
    if (bs.tile_v % rows != 0 || bs.tile_u % (32 / rows) != 0) {
        bs.tile_v = rows;
        bs.tile_u = threads / rows;  // a multiple of 32 / rows: whole warps
    }
    BwdGrid b;
    b.tile_u = bs.tile_u;
    b.rows = rows;
    b.tiles_v = (prm_in.g.V + bs.tile_v - 1) / bs.tile_v;
    b.block = dim3(threads);
    b.smem = sizeof(float) * (size_t)energy_groups(prm_in.E) * 4 * M;
    const unsigned tiles_u = (unsigned)((prm_in.g.U + bs.tile_u - 1) / bs.tile_u);
    // a part's view groups run along grid.y, at most 65535 per launch
    MarchParams prm = prm_in;
    if (!prm.gcol) prm.sets = prm.set_columns = 1;
    const int parts = prm.sets / prm.set_columns, views = (prm.n_views + parts - 1) / parts;  // of the largest part
    prm.views_per_cta = std::max(1, std::min(ls.views_per_cta, views));
    const int groups = (views + prm.views_per_cta - 1) / prm.views_per_cta;
    // One band of rows and elements of 16 bytes: the parts at the same time, since the
    // CTAs of neighbouring views reduce into the same few voxels (8 rows, 3 materials
    // 0.457 -> 0.424 ms, 5 rows 0.357 -> 0.334; pair cells lose, 1 material, 2 rows 0.125 -> 0.135).
    b.parts_in_y = M > 2 && b.tiles_v == 1;
    const int most = b.parts_in_y ? 65535 / parts : 65535;
    for (b.group0 = 0; b.group0 < groups; b.group0 += most) {
        const int n = std::min(most, groups - b.group0);
        b.grid = b.parts_in_y ? dim3(tiles_u, n * parts, 1) : dim3(tiles_u, n, b.tiles_v * parts);
        if (b.grid.x == 0 || b.grid.y == 0 || b.grid.z == 0) return cudaSuccess;
        cudaError_t e = cudaErrorInvalidValue;
        switch (M) {
            case 1: e = bwd_dispatch<1>(prm, interp, from_gL, b, st); break;
            case 2: e = bwd_dispatch<2>(prm, interp, from_gL, b, st); break;
            case 3: e = bwd_dispatch<3>(prm, interp, from_gL, b, st); break;
            case 4: e = bwd_dispatch<4>(prm, interp, from_gL, b, st); break;
        }
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_fold(const MarchParams& prm, int M, cudaStream_t st)
{
    if (!prm.gcol) return cudaSuccess;
    const dim3 grid((unsigned)column_tiles(prm.g.nx, prm.g.ny, prm.g.nz)), block(32, 8);
    switch (M) {
        case 1: k_fold<1><<<grid, block, 0, st>>>(prm); break;
        case 2: k_fold<2><<<grid, block, 0, st>>>(prm); break;
        case 3: k_fold<3><<<grid, block, 0, st>>>(prm); break;
        case 4: k_fold<4><<<grid, block, 0, st>>>(prm); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_weights(const float* spectrum, const float* grid, int grid_layout, const float* det, float I0Val,
                           int E, int U, int V, float* W, float* I0, cudaStream_t st)
{
    const int64_t npix = (int64_t)U * V;
    int64_t nb = (npix + 255) / 256;
    if (nb > 148 * 32) nb = 148 * 32;
    if (nb == 0) return cudaSuccess;
    k_weights<<<(unsigned)nb, 256, 0, st>>>(spectrum, grid, grid_layout, det, I0Val, E, U, V, W, I0);
    return cudaGetLastError();
}

cudaError_t launch_finalize(int64_t n_pix, int64_t n_views, const float* I, const float* IAbs, const float* I0,
                            uint32_t* Ipoly, uint32_t* IAbsPoly, float* proj, cudaStream_t st)
{
    const int64_t n = n_pix * n_views;
    int64_t nb = (n + 255) / 256;
    if (nb > 148 * 32) nb = 148 * 32;
    if (nb == 0) return cudaSuccess;
    k_finalize<<<(unsigned)nb, 256, 0, st>>>(n_pix, n, I, IAbs, I0, Ipoly, IAbsPoly, proj);
    return cudaGetLastError();
}

cudaError_t launch_sample_points(const float* vol, cudaTextureObject_t tex, int nx, int ny, int nz, int interp,
                                 const float* pts, int64_t n, float* out, cudaStream_t st)
{
    int64_t nb = (n + 255) / 256;
    if (nb > 148 * 32) nb = 148 * 32;
    if (nb == 0) return cudaSuccess;
    k_sample_points<<<(unsigned)nb, 256, 0, st>>>(vol, tex, nx, ny, nz, interp, pts, n, out);
    return cudaGetLastError();
}

namespace {

// One thread per voxel: a non-zero voxel marks every brick whose dilated
// range [8b - 1, 8b + 7] holds it (b = (x + 1) >> 3, and b - 1 when x + 1 is a
// multiple of 8), per axis.  Concurrent stores all write 1.
__global__ void k_occupancy(const VolPtrs vol, int M, int nx, int ny, int nz, int ox, int oy, uint8_t* occ)
{
    const int64_t n = (int64_t)nx * ny * nz;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        bool any = false;
        for (int m = 0; m < M; m++) any |= __ldg(vol.p[m] + k) != 0.f;
        if (!any) continue;
        const int x = (int)(k % nx), y = (int)((k / nx) % ny), z = (int)(k / ((int64_t)nx * ny));
        const int bx = (x + 1) >> kOccShift, by = (y + 1) >> kOccShift, bz = (z + 1) >> kOccShift;
        const int lx = ((x + 1) & ((1 << kOccShift) - 1)) == 0 && bx > 0;
        const int ly = ((y + 1) & ((1 << kOccShift) - 1)) == 0 && by > 0;
        const int lz = ((z + 1) & ((1 << kOccShift) - 1)) == 0 && bz > 0;
        for (int dz = 0; dz <= lz; dz++)
            for (int dy = 0; dy <= ly; dy++)
                for (int dx = 0; dx <= lx; dx++)
                    occ[((size_t)(bz - dz) * oy + (by - dy)) * ox + (bx - dx)] = 1;
    }
}

}  // namespace

namespace {

// Focal-spot re-alignment of the line-integral images (projOffsetMatchKernel,
// CBCTPolyProjGPU.cu:1956-1978): out[p][v][u][m] = in[p] sampled at
// (u + offU[p] / dSize, v + offV[p] / dSize), bilinear, 0 outside the image.
// The compat modes reproduce the texture unit (8-bit weights at the FP32
// coordinate u + offU/dSize + 0.5 it receives); TRILINEAR interpolates
// exactly at the FP64 position.
template <int M, int MODE>
__global__ void k_shift_views(const float* __restrict__ in, float* __restrict__ out, const float2* __restrict__ fspot,
                              int U, int V, float dSize, int view0, int n_views)
{
    const int64_t npix = (int64_t)U * V;
    const int64_t n = npix * n_views;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = t / npix, pix = t % npix;
        const int u = (int)(pix % U), v = (int)(pix / U);
        const float2 f = fspot[view0 + k];
        int ix, iy;
        float w[4];  // (ix, iy), (ix + 1, iy), (ix, iy + 1), (ix + 1, iy + 1)
        if (MODE == INTERP_TRILINEAR) {
            const double cx = (double)u + (double)f.x / (double)dSize, cy = (double)v + (double)f.y / (double)dSize;
            const double fx = floor(cx), fy = floor(cy);
            ix = (int)fx;
            iy = (int)fy;
            float wx, ux, wy, uy;
            frac_pair(cx - fx, wx, ux);
            frac_pair(cy - fy, wy, uy);
            w[0] = ux * uy; w[1] = wx * uy; w[2] = ux * wy; w[3] = wx * wy;
        } else {
            const float x = __fadd_rn(__fadd_rn((float)u, __fdiv_rn(f.x, dSize)), 0.5f);
            const float y = __fadd_rn(__fadd_rn((float)v, __fdiv_rn(f.y, dSize)), 0.5f);
            const int X = tex_fixed(x), Y = tex_fixed(y);
            ix = X >> 8;
            iy = Y >> 8;
            float w8[8];
            texunit_weights(X & 255, Y & 255, 0, w8);  // the view coordinate p + 0.5 has fraction 0
            w[0] = w8[0]; w[1] = w8[1]; w[2] = w8[2]; w[3] = w8[3];
        }
        const float* src = in + k * npix * M;
        float acc[M];
#pragma unroll
        for (int m = 0; m < M; m++) acc[m] = 0.f;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int x = ix + (c & 1), y = iy + (c >> 1);
            if ((unsigned)x >= (unsigned)U || (unsigned)y >= (unsigned)V) continue;
            const float* q = src + ((int64_t)y * U + x) * M;
#pragma unroll
            for (int m = 0; m < M; m++) acc[m] = fmaf(w[c], __ldg(q + m), acc[m]);
        }
        float* d = out + t * M;
#pragma unroll
        for (int m = 0; m < M; m++) d[m] = acc[m];
    }
}

template <int MODE>
cudaError_t shift_dispatch(int M, const float* in, float* out, const float2* fspot, int U, int V, float dSize,
                           int view0, int n_views, unsigned nb, cudaStream_t st)
{
    switch (M) {
        case 1: k_shift_views<1, MODE><<<nb, 256, 0, st>>>(in, out, fspot, U, V, dSize, view0, n_views); break;
        case 2: k_shift_views<2, MODE><<<nb, 256, 0, st>>>(in, out, fspot, U, V, dSize, view0, n_views); break;
        case 3: k_shift_views<3, MODE><<<nb, 256, 0, st>>>(in, out, fspot, U, V, dSize, view0, n_views); break;
        case 4: k_shift_views<4, MODE><<<nb, 256, 0, st>>>(in, out, fspot, U, V, dSize, view0, n_views); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_shift_views(const float* in, float* out, const GeomParams& g, int M, int interp, int view0,
                               int n_views, cudaStream_t st)
{
    if (!g.fspot) return cudaErrorInvalidValue;
    const int64_t n = (int64_t)g.U * g.V * n_views;
    if (n == 0) return cudaSuccess;
    int64_t nb = (n + 255) / 256;
    if (nb > 148 * 32) nb = 148 * 32;
    if (interp == INTERP_TRILINEAR)
        return shift_dispatch<INTERP_TRILINEAR>(M, in, out, g.fspot, g.U, g.V, g.dSize, view0, n_views, (unsigned)nb, st);
    return shift_dispatch<INTERP_TEXEMU>(M, in, out, g.fspot, g.U, g.V, g.dSize, view0, n_views, (unsigned)nb, st);
}

cudaError_t launch_occupancy(const float* const* vol, int M, int nx, int ny, int nz, uint8_t* occ, cudaStream_t st)
{
    const int ox = occ_dim(nx), oy = occ_dim(ny), oz = occ_dim(nz);
    cudaError_t e = cudaMemsetAsync(occ, 0, (size_t)ox * oy * oz, st);
    if (e != cudaSuccess) return e;
    VolPtrs vp = {};
    for (int m = 0; m < M && m < kMaxM; m++) vp.p[m] = vol[m];
    const int64_t n = (int64_t)nx * ny * nz;
    int64_t nb = (n + 255) / 256;
    if (nb > 148 * 32) nb = 148 * 32;
    k_occupancy<<<(unsigned)nb, 256, 0, st>>>(vp, M, nx, ny, nz, ox, oy, occ);
    return cudaGetLastError();
}

cudaError_t launch_count_support(const GeomParams& g, unsigned long long* out, cudaStream_t st)
{
    const dim3 block(32, 8);
    int gz = g.P < 64 ? g.P : 64;
    const dim3 grid((g.U + 31) / 32, (g.V + 7) / 8, gz > 0 ? gz : 1);
    if (g.P == 0 || g.U == 0 || g.V == 0) return cudaSuccess;
    k_count_support<<<grid, block, 0, st>>>(g, out);
    return cudaGetLastError();
}

}  // namespace ctfp
