// ctfp_column.cuh — the z-fastest layout of the volumes' voxels: the four-material
// march of the axis sampler, and the adjoint's scatter (that sampler's march
// transposed) into accumulators; shared by the plan kernels and the batched
// persistent kernels.
#pragma once

#include <algorithm>
#include <cmath>

#include "ctfp_axis.cuh"
#include "ctfp_device.cuh"

namespace ctfp {

// The layout: voxel (x, y, z) is element ((x + 2) * ny' + (y + 2)) * nz' +
// (z + 2), ny' = ny + 4, nz' = nz + 4.  Two border voxels surround the volume on
// every side, so a footprint with its base in [-2, n] on each axis lies in
// bounds with no test: the march reads the border as zeros, what the adjoint
// adds there is never read.  One array serves the views marched along x and
// those marched along y, and with lanes down the detector's rows (z) a warp's
// loads and reductions are runs of memory.
constexpr int kColPad = 2;
struct ColumnDims {
    unsigned sx, sy, origin;  // element strides of x and y; element of voxel (0, 0, 0)
    size_t elems;
};
__host__ __device__ __forceinline__ ColumnDims column_dims(int nx, int ny, int nz)
{
    ColumnDims d;
    d.sy = (unsigned)(nz + 2 * kColPad);
    d.sx = d.sy * (unsigned)(ny + 2 * kColPad);
    d.origin = kColPad * (d.sx + d.sy + 1u);
    d.elems = (size_t)d.sx * (size_t)(nx + 2 * kColPad);
    return d;
}
// Whether 32-bit elements reach the whole set.  Every volume of the axis sampler
// fits; others of under 2^31 voxels may not where two extents are small (1 x 1 x
// 172 000 000, 5 x 5 x 53 100 000) or one is and the others are long (32768 x 26240 x 1).
__host__ __device__ __forceinline__ bool column_fits(int nx, int ny, int nz)
{
    return (double)(nx + 2 * kColPad) * (ny + 2 * kColPad) * (nz + 2 * kColPad) < 4294967040.0;
}
// 32 x 32 (x, z) tiles of every y: how the copy is filled and the gradients folded; block k's tile.
__host__ __device__ __forceinline__ long long column_tiles(int nx, int ny, int nz)
{
    return (long long)((nx + 31) / 32) * ((nz + 31) / 32) * ny;
}
__device__ __forceinline__ void column_tile(unsigned k, int nx, int nz, int& x0, int& y, int& z0)
{
    const unsigned bx = (unsigned)(nx + 31) / 32, bz = (unsigned)(nz + 31) / 32;
    x0 = (int)(k % bx) * 32;
    z0 = (int)((k / bx) % bz) * 32;
    y = (int)(k / (bx * bz));
}
// Clip of one axis to lo < a + b i < hi in samples, r = 1 / b: the first and
// last sample are exact up to 1e-6 of a sample (outwards), so a footprint at
// either end overhangs the volume by its border only.
__device__ __forceinline__ void clip_tight(double a, double b, double lo, double hi, int& i0, int& i1)
{
    if (fabs(b) < 1e-12) {
        if (!(a > lo && a < hi)) i1 = i0;
        return;
    }
    const double r = 1.0 / b;
    const double t0 = (lo - a) * r, t1 = (hi - a) * r;
    const double f0 = ceil(fmin(t0, t1) - 1e-6), f1 = floor(fmax(t0, t1) + 1e-6) + 1.0;
    if (f0 > (double)i0) i0 = (f0 > 2e9) ? 2000000000 : (int)f0;
    if (f1 < (double)i1) i1 = (f1 < -2e9) ? -2000000000 : (int)f1;
}

// ray_segment's coordinates with one reciprocal of R and the plan's
// reciprocals of the voxel sizes (each within 2^-52 relative of the quotient:
// 1e-13 voxel), clipped by clip_tight.  For the exact coordinates only: the
// texture emulation's FP32 ones may lie voxels away from these, so there
// ray_segment's samples count, as in every other sampler, and each footprint
// is moved to the border where it lies beyond it.
__device__ __forceinline__ RaySeg column_segment(const GeomParams& g, int p, int v, int u)
{
    const double dsz = g.dSize, sdd = g.sdd, sod = g.sod;
    const double detU = (double)g.dHalfLU - dsz / 2 - (double)u * dsz;
    const double detV = (double)g.dHalfLV - dsz / 2 - (double)v * dsz;
    const double s2 = sdd * sdd, u2 = detU * detU, v2 = detV * detV;
    const double rR = 1.0 / sqrt(s2 + u2 + v2);
    const double cosG = sqrt(s2 + u2) * rR;
    const double A = cosG * (sqrt(s2 + v2) * rR), B = cosG * (detU * rR), C = detV * rR;
    const double t0 = sod - (double)g.FOVR + (double)g.dx / 2, dt = g.dx;
    const double2 cs = g.trig[p];
    const double cth = cs.x, sth = cs.y;
    double fu = 0.0, fv = 0.0;
    if (g.fspot) {
        const float2 f = g.fspot[p];
        fu = f.x;
        fv = f.y;
    }
    const double ku = A * cth - B * sth, cu = -sod * cth + (double)g.pHalfX;
    const double kv = -(A * sth + B * cth), cv = sod * sth + (double)g.pHalfY + fu;
    const double kw = -C, cw = (double)g.pHalfZ + fv;
    RaySeg s;
    s.ax = (ku * t0 + cu) * g.qx; s.bx = ku * dt * g.qx;
    s.ay = (kv * t0 + cv) * g.qy; s.by = kv * dt * g.qy;
    s.az = (kw * t0 + cw) * g.qz; s.bz = kw * dt * g.qz;
    s.i0 = 0;
    s.i1 = g.K;
    clip_tight(s.ax, s.bx, -1.0, (double)g.nx, s.i0, s.i1);
    clip_tight(s.ay, s.by, -1.0, (double)g.ny, s.i0, s.i1);
    clip_tight(s.az, s.bz, -1.0, (double)g.nz, s.i0, s.i1);
    // The coordinates are linear in i, so the first and the last sample within
    // the border mean that all are.  Where 1e-6 of a sample is no longer a
    // fraction of a voxel (voxels a millionth of the step flat), or a coordinate
    // is no number, the clip alone does not place them there.
    const auto inside = [&](int i) {
        const double t = (double)i;
        const double x = fma(t, s.bx, s.ax), y = fma(t, s.by, s.ay), z = fma(t, s.bz, s.az);
        return x > -1.75 && y > -1.75 && z > -1.75 && x < (double)g.nx + 0.75 && y < (double)g.ny + 0.75 &&
               z < (double)g.nz + 0.75;
    };
    while (s.i0 < s.i1 && !inside(s.i0)) s.i0++;
    while (s.i0 < s.i1 && !inside(s.i1 - 1)) s.i1--;
    if (s.i1 < s.i0) s.i1 = s.i0;
    return s;
}

// Whether the axis sampler marches M materials over the column copy: 16-byte
// elements of the four materials side by side, instead of two layered texture
// copies of each.  A footprint's voxel is then one load for all materials,
// where the gathers cost the texture unit their time once per material: 48
// views of 512^3, 219 -> 151 ms (texture returns 90 % busy before).  For fewer
// materials the loads' lines cost the L1 as much as the gathers: 256^3, 90
// views, 2 materials 11.9 against 12.1 ms, 3 materials 14.1 against 12.1.
__host__ __device__ constexpr bool uses_columns(int M) { return M == 4; }

// The sums of one ray over the column copy (or of its part-th of parts equal runs
// of samples): march_ray_axis with each slot's four corners held for all
// materials, loaded when the slot's layer or in-layer base changes.
template <int M, int MODE, bool SKIP>
__device__ __forceinline__ void march_ray_columns(const GeomParams& g, const float* __restrict__ cvol, const OccView& occ,
                                                  int p, int v, int u, float* acc, float* cmp, int part, int parts)
{
    static_assert(M == 4, "elements of four floats");
    constexpr bool tri = MODE == INTERP_TRILINEAR;
    RaySeg s = tri ? column_segment(g, p, v, u) : ray_segment(g, p, v, u);
    if (parts > 1) {
        const int len = (s.i1 - s.i0 + parts - 1) / parts;
        s.i0 += part * len;
        s.i1 = min(s.i1, s.i0 + len);
    }
    RayRef32 r;
    if (!tri) r = ray_ref32(g, p, v, u);
    const ColumnDims cd = column_dims(g.nx, g.ny, g.nz);
    const bool xl = axis_is_x(g, p);
    const double bl = xl ? s.bx : s.by, ba = xl ? s.by : s.bx, bz = s.bz, i0 = (double)s.i0;
    double cl = fma(i0, bl, xl ? s.ax : s.ay), ca = fma(i0, ba, xl ? s.ay : s.ax), cz = fma(i0, bz, s.az);
    const unsigned sL = xl ? cd.sx : cd.sy, sA = xl ? cd.sy : cd.sx;
    const float4* const vol = (const float4*)cvol;
    float4 q0[4], q1[4];  // slots of the even and the odd layer: (a, b), (a + 1, b), (a, b + 1), (a + 1, b + 1)
#pragma unroll
    for (int j = 0; j < 4; j++) q0[j] = q1[j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int m = 0; m < M; m++) acc[m] = cmp[m] = 0.f;
    unsigned h0 = 0xffffffffu, h1 = 0xffffffffu;
    const auto fetch = [&](unsigned at, float4* q) {
        const float4 *c0 = vol + at, *c1 = vol + (at + sA);
        q[0] = __ldg(c0);
        q[2] = __ldg(c0 + 1);
        q[1] = __ldg(c1);
        q[3] = __ldg(c1 + 1);
    };
    constexpr int kBlock = 16;
    for (int ib = s.i0; ib < s.i1; ib += kBlock) {
        const int ie = min(ib + kBlock, s.i1);
        float blk[M] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
        for (int i = ib; i < ie; i++) {
            unsigned lo;
            bool odd;
            // tri: the in-layer weights and the layers' own; else the corners'
            // weights of the lower and the upper layer
            float w[4], wl, ul, g0[4], g1[4];
            if (tri) {
                float wa, ua, wz, uz;
                const int il = axis_weights(cl, wl, ul), ia = axis_weights(ca, wa, ua), iz = axis_weights(cz, wz, uz);
                cl += bl;
                ca += ba;
                cz += bz;
                if (SKIP) {
                    Corner c = {};
                    c.ix = xl ? il : ia;
                    c.iy = xl ? ia : il;
                    c.iz = iz;
                    if (!occ.occupied(c)) continue;
                }
                lo = (unsigned)il * sL + ((unsigned)ia * sA + (unsigned)(iz + (int)cd.origin));
                odd = il & 1;
                w[0] = ua * uz;
                w[1] = wa * uz;
                w[2] = ua * wz;
                w[3] = wa * wz;
            } else {
                const Corner c = corner_tex(ref32_coords(g, r, i));
                if (SKIP && !occ.occupied(c)) continue;
                // an FP32 coordinate may lie outside the border
                const int x = __vimin_s32_relu(c.ix + kColPad, g.nx + kColPad);
                const int y = __vimin_s32_relu(c.iy + kColPad, g.ny + kColPad);
                const int z = __vimin_s32_relu(c.iz + kColPad, g.nz + kColPad);
                lo = (unsigned)x * cd.sx + (unsigned)y * cd.sy + (unsigned)z;
                odd = (xl ? x : y) & 1;
                float t[8];
                texunit_weights(c.qx, c.qy, c.qz, t);
                g0[0] = t[0]; g0[2] = t[4]; g1[1] = t[3]; g1[3] = t[7];
                g0[1] = xl ? t[2] : t[1]; g0[3] = xl ? t[6] : t[5];
                g1[0] = xl ? t[1] : t[2]; g1[2] = xl ? t[5] : t[6];
            }
            const unsigned hi = lo + sL, f0 = odd ? hi : lo, f1 = odd ? lo : hi;
            if (f0 != h0) fetch(f0, q0);
            if (f1 != h1) fetch(f1, q1);
            h0 = f0;
            h1 = f1;
            // A sample is summed before it meets the block's sum, as in
            // march_ray_axis: products added to the block's sum one by one are
            // rounded at its size (RMS error of L 1.5 times that).
            const auto dot = [](const float* a, float x0, float x1, float x2, float x3) {
                return fmaf(x3, a[3], fmaf(x2, a[2], fmaf(x1, a[1], x0 * a[0])));
            };
            if (tri) {
                const float a = odd ? wl : ul, b = odd ? ul : wl;
                blk[0] = fmaf(dot(w, q1[0].x, q1[1].x, q1[2].x, q1[3].x), b, fmaf(dot(w, q0[0].x, q0[1].x, q0[2].x, q0[3].x), a, blk[0]));
                blk[1] = fmaf(dot(w, q1[0].y, q1[1].y, q1[2].y, q1[3].y), b, fmaf(dot(w, q0[0].y, q0[1].y, q0[2].y, q0[3].y), a, blk[1]));
                blk[2] = fmaf(dot(w, q1[0].z, q1[1].z, q1[2].z, q1[3].z), b, fmaf(dot(w, q0[0].z, q0[1].z, q0[2].z, q0[3].z), a, blk[2]));
                blk[3] = fmaf(dot(w, q1[0].w, q1[1].w, q1[2].w, q1[3].w), b, fmaf(dot(w, q0[0].w, q0[1].w, q0[2].w, q0[3].w), a, blk[3]));
            } else {
                float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float a = odd ? g1[j] : g0[j], b = odd ? g0[j] : g1[j];
                    v[0] = fmaf(q1[j].x, b, fmaf(q0[j].x, a, v[0]));
                    v[1] = fmaf(q1[j].y, b, fmaf(q0[j].y, a, v[1]));
                    v[2] = fmaf(q1[j].z, b, fmaf(q0[j].z, a, v[2]));
                    v[3] = fmaf(q1[j].w, b, fmaf(q0[j].w, a, v[3]));
                }
#pragma unroll
                for (int m = 0; m < M; m++) blk[m] += v[m];
            }
        }
#pragma unroll
        for (int m = 0; m < M; m++) kahan_add(acc[m], cmp[m], blk[m]);
    }
}

// The sums of one ray of the axis sampler, or of one part of it, over whichever
// copies M materials use.
template <int M, int MODE, bool SKIP>
__device__ __forceinline__ void march_axis_sums(const GeomParams& g, const cudaTextureObject_t* xtex,
                                                const cudaTextureObject_t* ytex, const float* cvol,
                                                const OccView& occ, int p, int v, int u, float* acc, float* cmp,
                                                int part = 0, int parts = 1)
{
    if constexpr (uses_columns(M)) march_ray_columns<M, MODE, SKIP>(g, cvol, occ, p, v, u, acc, cmp, part, parts);
    else if (axis_is_x(g, p)) march_ray_axis<M, MODE, 0, SKIP>(g, xtex, ytex, occ, p, v, u, acc, cmp, part, parts);
    else march_ray_axis<M, MODE, 1, SKIP>(g, xtex, ytex, occ, p, v, u, acc, cmp, part, parts);
}

// L_m of one ray.
template <int M, int MODE, bool SKIP>
__device__ __forceinline__ void march_axis(const GeomParams& g, const cudaTextureObject_t* xtex,
                                           const cudaTextureObject_t* ytex, const float* cvol, const OccView& occ, int p,
                                           int v, int u, float* L)
{
    float acc[M], cmp[M];
    march_axis_sums<M, MODE, SKIP>(g, xtex, ytex, cvol, occ, p, v, u, acc, cmp);
#pragma unroll
    for (int m = 0; m < M; m++) L[m] = g.dx * (acc[m] - cmp[m]);
}

// ---------------------------------------------------------------------------
// Adjoint: the transposed weights of one ray's samples into the accumulators.
// For one and two materials an element is a pair cell, the sums of voxels z and
// z + 1 of its column (2 M floats); for three and four it is voxel z (4 floats).
// Either way a face of 2 x 2 voxels is two columns, and a column one reduction
// of at most 16 bytes (pair cells) or two.
//
// What binds the scatter is the L2's rate of reduced sectors (a probe: 1.9e11
// scattered reductions of 4 to 16 bytes a second, 3.5e11 of 16 bytes in runs of
// 8 lanes or more, 1.4e12 floats a second at most) and, once the accumulators
// outgrow the L2, DRAM.  Hence z-fastest elements with lanes down the rows
// (runs), no copy of a voxel per face corner or march axis (2 or 1.3 floats per
// voxel and material instead of 8), pair cells where an element would be less
// than half a sector, and for 16-byte elements the hand-over in flush_voxels.
// Against the face-expanded layout this replaced (adjoint + fold): 256^3, 90
// views, 2 materials 18.4 -> 14.0 ms; 3 materials 34.3 -> 17.0 ms; 128^3, 60
// views, 1 material 3.2 -> 2.4 ms; 512^3, 48 views, 4 materials 558 -> 260 ms.
__host__ __device__ constexpr int accum_width(int M) { return M <= 2 ? 2 * M : 4; }

// Sets of accumulators an adjoint over n views sums into, folded together in
// FP64: views equal parts of the views, by columns of the detector within each.
// An FP32 sum of many small terms loses about sqrt(terms) ulp of itself, and K
// sets of a K-th of the terms lose a K-th (positive terms) to a sqrt(K)-th
// (signed ones) of that.  As many as leave the gradients' error against FP64 no
// larger than that of 8 separate accumulators per voxel, one per face corner and
// march axis, which took each a share of every view's rays: the more, the more
// rays of one view meet a voxel's face, the fewer, the fewer views there are; and
// where a view's rays alone outnumber what the views can be split into, its
// columns take turns.  2-norm relative error of 4 / 5 / 6 / 7 / 8 sets of single voxels
// against those 8: 256^3, 0.6 rays a face, 90 views 11.4 10.6 10.2 10.0 9.8 /
// 10.4e-8; 128^3, 4.1, 53 views 15.9 14.3 13.3 12.5 12.1 / 12.5e-8; 66^3, 19, 182
// views 56 45 38 33 29.9 / 28.8e-8; 65^3, 74, 7 views 27 24 22 17.7 - / 15.7e-8.
// Pair cells hold two sums a voxel: 48^3, 8.2 rays, 60 views, 4 / 5 / 6 sets 36 32
// 29 / 32e-8, 1 ray, 13.9 12.8 11.9 / 13.4e-8; 20 views 9.4 8.8 8.4 / 9.6e-8, 7 views 3
// sets 7.9 / 8.1e-8.
struct AccumSets {
    int views, columns;
    int total() const { return views * columns; }
};
inline AccumSets accum_sets(const GeomParams& g, int n, int M, int most)
{
    const float pitch = g.dSize * g.sod / g.sdd, across = fminf(g.pSizeX, g.pSizeY);
    const float face = g.pSizeZ * across / (pitch * pitch), rays = fminf((float)n * face, 1e6f);
    const int full = M <= 2 ? (face > 8.f ? 6 : 5) : (face > 8.f ? 10 : face > 1.7f ? 8 : 6);
    int k = full;
    if (face <= 1.7f) {
        int lg = 1;  // 1 + floor(log2 n)
        for (int j = n; j > 1; j >>= 1) lg++;
        if (face < 0.3f && lg > 3) lg--;
        k = std::max(std::min(k, lg), std::min((int)ceilf(rays / 6.f), M <= 2 ? 4 : 6));
    }
    AccumSets s;
    s.views = std::max(1, std::min(std::min(k, (int)ceilf(rays) + 1), std::min(n, most)));
    s.columns = 1;
    const int want = M <= 2 ? 2 : full;
    if (face > 1.7f && pitch < 0.75f * across)
        while (s.columns < 4 && 6 * s.total() < 5 * want && 2 * s.total() <= most) s.columns *= 2;
    return s;
}
constexpr int kMostSets = 18;  // more than any plan's

__device__ __forceinline__ void red_v2(float* q, float a, float b)
{
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(q), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void red_v4(float* q, float a, float b, float c, float d)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(q), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void red_v4_if(bool on, float* q, float a, float b, float c, float d)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t"
                 "@p red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n\t}" ::"l"(q), "f"(a), "f"(b), "f"(c), "f"(d),
                 "r"((unsigned)on)
                 : "memory");
}

// One ray's face sums on their way into memory: slot 0 the even layer, slot 1
// the odd one of its current pair, each the summed weights of (a, b),
// (a + 1, b), (a, b + 1), (a + 1, b + 1); a slot is flushed when its layer or
// the in-layer base changes.  MERGE: the whole warp calls move() and finish()
// together.
template <int M, bool MERGE>
struct ColumnScatter {
    static constexpr bool warp_wide = MERGE;
    float* acc;
    const float* g;  // dLoss/dL_m times dx
    unsigned sA;
    unsigned h0, h1;  // element of the slot's face, kNone before the first sample
    float s0[4], s1[4];
    static constexpr unsigned kNone = 0xffffffffu;

    __device__ __forceinline__ void begin(float* a, const float* gg, unsigned sa)
    {
        acc = a;
        g = gg;
        sA = sa;
        h0 = h1 = kNone;
#pragma unroll
        for (int j = 0; j < 4; j++) s0[j] = s1[j] = 0.f;
    }

    // One lane on its own.
    __device__ __forceinline__ void flush_cells(unsigned at, const float* s) const
    {
        constexpr int W = accum_width(M);
#pragma unroll
        for (int c = 0; c < 2; c++) {
            float* q = acc + (size_t)(at + (c ? sA : 0u)) * W;
            if (M == 1) {
                red_v2(q, s[c] * g[0], s[c + 2] * g[0]);
            } else if (M == 2) {
                red_v4(q, s[c] * g[0], s[c] * g[M - 1], s[c + 2] * g[0], s[c + 2] * g[M - 1]);
            } else {
                red_v4(q, s[c] * g[0], s[c] * g[1 % M], s[c] * g[2 % M], M == 4 ? s[c] * g[M - 1] : 0.f);
                red_v4(q + W, s[c + 2] * g[0], s[c + 2] * g[1 % M], s[c + 2] * g[2 % M], M == 4 ? s[c + 2] * g[M - 1] : 0.f);
            }
        }
    }

    // Single voxels, the lanes with need set.  Lanes run down the detector's
    // rows, about one voxel apart in z, so a lane's upper voxel is mostly the
    // next lane's lower one: where both flush the same column together, the
    // lane hands its upper sums over and one reduction covers both.
    __device__ __forceinline__ void flush_voxels(bool need, unsigned at, const float* s) const
    {
        constexpr unsigned full = 0xffffffffu;
        const unsigned key = need ? at : kNone;
        const unsigned below = __shfl_up_sync(full, key, 1);
        const bool take = need && below + 1u == key;
        const unsigned takers = __ballot_sync(full, take);  // (every lane: not in a short-circuited operand)
        const bool alone = need && !(takers >> 1 >> (threadIdx.x & 31u) & 1u);
#pragma unroll
        for (int c = 0; c < 2; c++) {
            float* q = acc + (size_t)((need ? at : 0u) + (c ? sA : 0u)) * 4;
            float lo[4], hi[4];
#pragma unroll
            for (int m = 0; m < 4; m++) {
                lo[m] = hi[m] = 0.f;
                if (m < M) {
                    hi[m] = s[c + 2] * g[m < M ? m : 0];
                    const float r = __shfl_up_sync(full, hi[m], 1);
                    lo[m] = fmaf(s[c], g[m < M ? m : 0], take ? r : 0.f);
                }
            }
            red_v4_if(need, q, lo[0], lo[1], lo[2], lo[3]);
            red_v4_if(alone, q + 4, hi[0], hi[1], hi[2], hi[3]);
        }
    }

    __device__ __forceinline__ void flush(bool need, unsigned at, const float* s) const
    {
        if (MERGE) flush_voxels(need, at, s);
        else if (need) flush_cells(at, s);
    }

    __device__ __forceinline__ void slot(bool live, unsigned f, unsigned& h, float* s)
    {
        const bool change = live && f != h;
        if (warp_wide ? __any_sync(0xffffffffu, change) : change) {
            flush(change && h != kNone, h, s);
#pragma unroll
            for (int j = 0; j < 4; j++) s[j] = change ? 0.f : s[j];
            if (change) h = f;
        }
    }
    __device__ __forceinline__ void move(bool live, unsigned f0, unsigned f1)
    {
        slot(live, f0, h0, s0);
        slot(live, f1, h1, s1);
    }
    __device__ __forceinline__ void finish() const
    {
        flush(h0 != kNone, h0, s0);
        flush(h1 != kNone, h1, s1);
    }
    // The samples a ray of n steps through: those of the warp's longest ray
    // when the warp flushes together.
    static __device__ __forceinline__ int steps(int n)
    {
        return warp_wide ? __reduce_max_sync(0xffffffffu, n) : n;
    }
};

template <int M, bool MERGE>
__device__ __forceinline__ void scatter_trilinear(const GeomParams& gp, float* acc, bool on, int p, int v, int u,
                                                  const float* g)
{
    RaySeg s = column_segment(gp, p, v, u);
    const ColumnDims cd = column_dims(gp.nx, gp.ny, gp.nz);
    const bool xl = axis_is_x(gp, p);
    const double bl = xl ? s.bx : s.by, ba = xl ? s.by : s.bx, bz = s.bz;
    const double i0 = (double)s.i0;
    double cl = fma(i0, bl, xl ? s.ax : s.ay), ca = fma(i0, ba, xl ? s.ay : s.ax), cz = fma(i0, bz, s.az);
    const unsigned sL = xl ? cd.sx : cd.sy, sA = xl ? cd.sy : cd.sx;
    using Scatter = ColumnScatter<M, MERGE>;
    const int n = on ? s.i1 - s.i0 : 0, steps = Scatter::steps(n);
    Scatter k;
    k.begin(acc, g, sA);
#pragma unroll(Scatter::warp_wide ? 1 : 2)
    for (int i = 0; i < steps; i++) {
        float wl, ul, wa, ua, wz, uz;
        const int il = axis_weights(cl, wl, ul), ia = axis_weights(ca, wa, ua), iz = axis_weights(cz, wz, uz);
        cl += bl;
        ca += ba;
        cz += bz;
        const unsigned lo = (unsigned)il * sL + ((unsigned)ia * sA + (unsigned)(iz + (int)cd.origin)), hi = lo + sL;
        const bool par = il & 1, live = !Scatter::warp_wide || i < n;
        k.move(live, par ? hi : lo, par ? lo : hi);
        if (!live) continue;
        const float w0 = par ? wl : ul, w1 = par ? ul : wl;
        const float w[4] = {ua * uz, wa * uz, ua * wz, wa * wz};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            k.s0[j] = fmaf(w[j], w0, k.s0[j]);
            k.s1[j] = fmaf(w[j], w1, k.s1[j]);
        }
    }
    k.finish();
}

template <int M, bool MERGE, bool XL>
__device__ __forceinline__ void scatter_texemu(const GeomParams& gp, float* acc, bool on, int p, int v, int u,
                                               const float* g)
{
    const RaySeg s = ray_segment(gp, p, v, u);
    const RayRef32 r = ray_ref32(gp, p, v, u);
    const ColumnDims cd = column_dims(gp.nx, gp.ny, gp.nz);
    const unsigned sL = XL ? cd.sx : cd.sy, sA = XL ? cd.sy : cd.sx;
    using Scatter = ColumnScatter<M, MERGE>;
    const int n = on ? s.i1 - s.i0 : 0, steps = Scatter::steps(n);
    Scatter k;
    k.begin(acc, g, sA);
    for (int i = 0; i < steps; i++) {
        const Corner c = corner_tex(ref32_coords(gp, r, s.i0 + i));
        const int x = __vimin_s32_relu(c.ix + kColPad, gp.nx + kColPad);
        const int y = __vimin_s32_relu(c.iy + kColPad, gp.ny + kColPad);
        const int z = __vimin_s32_relu(c.iz + kColPad, gp.nz + kColPad);
        const unsigned lo = (unsigned)x * cd.sx + (unsigned)y * cd.sy + (unsigned)z, hi = lo + sL;
        const bool par = (XL ? x : y) & 1, live = !Scatter::warp_wide || i < n;
        k.move(live, par ? hi : lo, par ? lo : hi);
        if (!live) continue;
        float w[8];
        texunit_weights(c.qx, c.qy, c.qz, w);
        constexpr int lb = XL ? 1 : 2, ab = XL ? 2 : 1;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int q = (j & 2 ? 4 : 0) + (j & 1 ? ab : 0);
            k.s0[j] += par ? w[q + lb] : w[q];
            k.s1[j] += par ? w[q] : w[q + lb];
        }
    }
    k.finish();
}

// The adjoint of one ray's march, scaled by g[m] = dLoss/dL_m times dx, for
// the lanes with on set; every lane of the warp calls it, for the same view.
template <int M, int MODE, bool MERGE>
__device__ __forceinline__ void scatter_columns(const GeomParams& gp, float* acc, bool on, int p, int v, int u,
                                                const float* g)
{
    if (!MERGE && !on) return;
    if (MODE == INTERP_TRILINEAR) scatter_trilinear<M, MERGE>(gp, acc, on, p, v, u, g);
    else if (axis_is_x(gp, p)) scatter_texemu<M, MERGE, true>(gp, acc, on, p, v, u, g);
    else scatter_texemu<M, MERGE, false>(gp, acc, on, p, v, u, g);
}

// The same for a volume that column_fits refuses: every voxel of every sample
// by an atomic addition into the gradients.  A batch's tuning runs have none.
template <int M, int MODE>
__device__ __noinline__ void scatter_direct(const GeomParams& gp, float* const* gvol, bool on, int p, int v, int u,
                                            const float* g)
{
    if (!on || !gvol[0]) return;
    const RaySeg s = ray_segment(gp, p, v, u);
    const RayRef32 r = ray_ref32(gp, p, v, u);
    for (int i = s.i0; i < s.i1; i++) {
        const double t = (double)i;
        const Corner c = MODE == INTERP_TRILINEAR
                             ? corner_of<INTERP_TRILINEAR>(fma(t, s.bx, s.ax), fma(t, s.by, s.ay), fma(t, s.bz, s.az))
                             : corner_tex(ref32_coords(gp, r, i));
        float w[8];
        corner_weights<MODE>(c, w);
        for (int k = 0; k < 8; k++) {
            const int x = c.ix + (k & 1), y = c.iy + (k >> 1 & 1), z = c.iz + (k >> 2);
            if ((unsigned)x >= (unsigned)gp.nx || (unsigned)y >= (unsigned)gp.ny || (unsigned)z >= (unsigned)gp.nz) continue;
            const size_t at = ((size_t)z * gp.ny + y) * gp.nx + x;
            for (int m = 0; m < M; m++) atomicAdd(gvol[m] + at, w[k] * g[m]);
        }
    }
}

// Adds `sets` sets of accumulators, stride floats apart, of a 32 x 32 (x, z)
// tile of one y into the gradients: read along z, turned in shared memory
// t[M][32][33], written along x.  The block is 32 x 8 threads.
template <int M>
__device__ __forceinline__ void fold_tile(const float* __restrict__ acc, int sets, size_t stride, float* const* g, int nx,
                                          int ny, int nz, int x0, int y, int z0, float (*t)[32][33])
{
    const ColumnDims cd = column_dims(nx, ny, nz);
    const int tx = threadIdx.x;
    for (int k = threadIdx.y; k < 32; k += 8) {
        const int x = x0 + k, z = z0 + tx;
        if (x < nx && z < nz) {
            const float* q =
                acc + ((size_t)x * cd.sx + (size_t)y * cd.sy + (size_t)z + cd.origin) * accum_width(M);
            // pair cells: voxel z is the first half of cell z and the second of cell z - 1;
            // in FP64, so that only the sums themselves have been rounded
            double v[4] = {0.0, 0.0, 0.0, 0.0};
            for (int j = 0; j < sets; j++, q += stride) {
                if (M == 1) {
                    v[0] += (double)q[0] + (double)q[-1];
                } else if (M == 2) {
                    const float2 e = *(const float2*)q, f = *(const float2*)(q - 2);
                    v[0] += (double)e.x + (double)f.x;
                    v[1] += (double)e.y + (double)f.y;
                } else {
                    const float4 e = *(const float4*)q;
                    v[0] += (double)e.x;
                    v[1] += (double)e.y;
                    v[2] += (double)e.z;
                    v[3] += (double)e.w;
                }
            }
#pragma unroll
            for (int m = 0; m < M; m++) t[m][tx][k] = (float)v[m];
        }
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += 8) {
        const int x = x0 + tx, z = z0 + k;
        if (x < nx && z < nz) {
#pragma unroll
            for (int m = 0; m < M; m++) g[m][((size_t)z * ny + y) * nx + x] += t[m][k][tx];
        }
    }
}

}  // namespace ctfp
