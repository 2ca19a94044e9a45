// Cone-beam Siddon kernels (forward and transpose) and their launch
// dispatch, shared by cb_forward.cu and cb_backward.cu, which instantiate
// them (one direction per translation unit), and siddon.cu (host side).
//
// Two walks, chosen per direction by NEFCT_TUNE_CB_WALK:
//  * thread per ray (cb_forward_kernel / cb_backward_kernel): 32 adjacent
//    detector columns x blockDim.y rows per CTA, each warp 32 neighbouring
//    columns of one row; volume x-fastest plus a y-fastest copy for x-driven
//    rays;
//  * column warps (colwarp_forward / colwarp_backward, FP32): each warp 32 R
//    rows of one column, R per lane, blockDim.y columns per CTA, over a
//    z-fastest copy of the volume (colwarp.cuh).
// The grid runs (column tile, view, row band) with the row band slowest, or
// (column tile, row band, view).  Per-view cos/sin/z-offset ride in the
// kernel parameters.
#pragma once

#include <math.h>
#include <algorithm>
#include <type_traits>

#include "colwarp.cuh"

namespace nefct {

template <typename T> struct CBParams {
    GridDev<T> g;
    int na, nb, nvc, v0, nv_total;
    RayGeom<T> rg;
    int band_major;
    int row0;                            // column warps: first detector row of the launch
    uint32_t flags;
    const T *vol;        // x-fastest volume (forward source)
    const T *volT;       // y-fastest copy for x-driven rays (thread walk) or z-fastest copy (column warps)
    const T *sino;       // backward source, full sinogram
    T *out;              // forward: full sinogram; backward: x-fastest volume
    T *outT;             // backward: y-fastest or z-fastest accumulator, or nullptr
    unsigned long long *fix, *fixT;   // deterministic backward: integer accumulators
    const float *fix_scale;           // deterministic backward: power-of-two scale (device)
    unsigned long long *count;
    ViewTable<T> tab;
};

template <typename T>
__device__ __forceinline__ void cb_ray(const CBParams<T> &p, int ia, int ib, int iv, T *r)
{
    cb_ray(p.rg, p.tab.cs[iv], p.tab.sn[iv], p.tab.off[iv], ia, ib, r);
}

// Detector cell of this thread (thread walk): 32 columns x blockDim.y rows
// per CTA; grid (column tile, view, row band) when band_major, else (column
// tile, row band, view).
template <typename T>
__device__ __forceinline__ void cb_cell(const CBParams<T> &p, int &ia, int &ib, int &iv)
{
    ia = blockIdx.x * 32 + threadIdx.x;
    if (p.band_major) { iv = blockIdx.y; ib = blockIdx.z * blockDim.y + threadIdx.y; }
    else { ib = blockIdx.y * blockDim.y + threadIdx.y; iv = blockIdx.z; }
}

// Sinogram value of a ray for the transpose; Q8: the reference's cylindrical
// backprojection reads ia + iv*na + ib*na*nb (reads past the end count as 0).
template <typename T> __device__ __forceinline__ T cb_sino_value(const CBParams<T> &p, int ia, int ib, int iv)
{
    const size_t total = (size_t)p.na * p.nb * p.nv_total;
    const size_t vg = (size_t)(p.v0 + iv);
    const size_t id = (p.flags & NEFCT_Q8_INDEX) ? (size_t)ia + vg * p.na + (size_t)ib * p.na * p.nb
                                                 : vg * p.na * p.nb + (size_t)ib * p.na + ia;
    return id < total ? p.sino[id] : (T)0;
}

// Whether a call's z splits follow the reference's rounding (colwarp.cuh, REF).
__host__ __device__ __forceinline__ bool ref_rounding(uint32_t flags) { return (flags & NEFCT_TIE_GT) != 0; }

// Sum of the volume along one ray again, without reading the voxels whose
// share is exactly 0 (in the grid, next to a voxel the ray passes): taken when
// a fast sum is not finite, so that an infinity or a NaN of a voxel the ray
// does not pass cannot enter it.
__device__ __noinline__ static float ray_resum(const GridDev<float> &g, float x1, float y1, float z1, float x2,
                                               float y2, float z2, uint32_t flags, const float *vol, unsigned su,
                                               unsigned sv, unsigned sw)
{
    const float r[6] = {x1, y1, z1, x2, y2, z2};
    Walk<float> w;
    if (!setup_walk(g, r, flags, w)) return 0.f;
    GatherSink f(vol);
    const ColWalk c = col_walk_of(g, w, su, sv);
    const ZGrid zg = z_grid(g);
    if (ref_rounding(flags))
        ray_slabs<true, true, false, -1, true, false>(c, z_ray<true>(w, zg, z_source<true>(w, zg), true), zg, w.k0, w.k1, sw, f);
    else
        ray_slabs<false, true, false, -1, true, false>(c, z_ray<false>(w, zg, z_source<false>(w, zg), true), zg, w.k0, w.k1, sw, f);
    f.close();
    return f.whole * w.W;
}

// Strides of the thread walk along (u, v): x-driven rays use the y-fastest
// copy when there is one.
__device__ __forceinline__ void thread_strides(int nx, int ny, bool xdrive, bool copy, unsigned &su, unsigned &sv)
{
    su = !xdrive ? (unsigned)nx : copy ? (unsigned)ny : 1u;
    sv = !xdrive || copy ? 1u : (unsigned)nx;
}

// Forward value of one ray: gathers x-driven rays from the y-fastest copy
// volT when there is one (COPY: there is), everything else from the x-fastest
// volume.  VAR: float: the reference's rounding; double: the voxels are not cubic.
template <typename T, bool VAR, bool EXACT = false, bool COPY = true>
__device__ __forceinline__ T ray_forward(const GridDev<T> &g, const T *r, uint32_t flags, const T *vol, const T *volT)
{
    if (EXACT) return exact_forward(g, r, flags, vol, volT);
    Walk<T> w;
    if (!setup_walk(g, r, flags, w)) return (T)0;
    const int sw = g.nx * g.ny;
    if constexpr (std::is_same<T, float>::value) {
        const float *const v = COPY && w.xdrive ? volT : vol;
        unsigned su, sv;
        thread_strides(g.nx, g.ny, w.xdrive, COPY, su, sv);
        GatherSink f(v);
        ray_walk<VAR, COPY>(g, w, su, sv, (unsigned)sw, f);
        const float sum = f.whole;
        if (!isfinite(sum)) return ray_resum(g, r[0], r[1], r[2], r[3], r[4], r[5], flags, v, su, sv, (unsigned)sw);
        return sum * w.W;
    } else {
        if (!w.xdrive) return gather_walk<T, VAR, true>(w, g, vol, g.nx, 1, sw);
        if (volT) return gather_walk<T, VAR, true>(w, g, volT, g.ny, 1, sw);
        return gather_walk<T, VAR, false>(w, g, vol, 1, g.nx, sw);
    }
}

// Transpose contribution of one ray with value y: x-driven rays reduce into
// the y-fastest accumulator outT when there is one.
template <typename T, bool VAR, bool EXACT = false>
__device__ __forceinline__ void ray_backward(const GridDev<T> &g, const T *r, uint32_t flags, T y, T *out, T *outT)
{
    if (EXACT) {
        exact_backward(g, r, flags, y, out, outT);
        return;
    }
    Walk<T> w;
    if (!setup_walk(g, r, flags, w)) return;
    const int sw = g.nx * g.ny;
    if constexpr (std::is_same<T, float>::value) {
        unsigned su, sv;
        thread_strides(g.nx, g.ny, w.xdrive, outT != nullptr, su, sv);
        ScatterSink f{w.xdrive && outT ? outT : out, y * w.W};
        ray_walk<VAR, true>(g, w, su, sv, (unsigned)sw, f);
    } else {
        if (!w.xdrive) scatter_walk<T, VAR, true>(w, g, out, g.nx, 1, sw, y);
        else if (outT) scatter_walk<T, VAR, true>(w, g, outT, g.ny, 1, sw, y);
        else scatter_walk<T, VAR, false>(w, g, out, 1, g.nx, sw, y);
    }
}

template <typename T, bool VAR, bool EXACT = false, bool COPY = true>
__global__ void __launch_bounds__(256, sizeof(T) == 4 && !EXACT ? 4 : 1) cb_forward_kernel(const __grid_constant__ CBParams<T> p)
{
    int ia, ib, iv;
    cb_cell(p, ia, ib, iv);
    if (ia >= p.na || ib >= p.nb) return;
    T r[6];
    cb_ray(p, ia, ib, iv, r);
    const T acc = ray_forward<T, VAR, EXACT, COPY>(p.g, r, p.flags, p.vol, p.volT);
    p.out[(size_t)(p.v0 + iv) * p.na * p.nb + (size_t)ib * p.na + ia] = acc;
}

template <typename T, bool VAR, bool EXACT = false>
__global__ void __launch_bounds__(256) cb_backward_kernel(const __grid_constant__ CBParams<T> p)
{
    int ia, ib, iv;
    cb_cell(p, ia, ib, iv);
    if (ia >= p.na || ib >= p.nb) return;
    const T y = cb_sino_value(p, ia, ib, iv);
    if (y == (T)0) return;
    T r[6];
    cb_ray(p, ia, ib, iv, r);
    ray_backward<T, VAR, EXACT>(p.g, r, p.flags, y, p.out, p.outT);
}

// What a kernel does with steep rays: there are none (cb_may_be_steep); they are
// walked in line; by a call.
enum Steep { kNoSteep, kSteepInline, kSteepCall };

// Forward of one row per lane (the whole warp calls it) of a warp with steep
// rays, not inlined: for the batch kernel, whose walk it would cost registers
// (64^3 to 384^3 problems: 7.68 against 9.47 ms; the single-problem kernels are
// the faster with it inlined: 256^3, 48 views, 1.55 against 1.61 ms, steep rays
// 0.221 against 0.240).
template <bool REF>
__device__ __noinline__ static float colwarp_gather_steep(const GridDev<float> &g, float x1, float y1, float z1, float x2,
                                                          float y2, float z2, bool has, uint32_t flags,
                                                          const float *__restrict__ volZ)
{
    const float r[1][6] = {{x1, y1, z1, x2, y2, z2}};
    const bool h[1] = {has};
    ColRays<1> q;
    if (!col_rays<1, REF, true>(g, r, h, flags, q)) return 0.f;
    GatherSink f[1] = {GatherSink(volZ)};
    col_gather<1, REF, true, true>(q, volZ, f);
    if (!q.z[0].live) return 0.f;
    if (isfinite(f[0].whole)) return f[0].whole * q.W[0];
    return ray_resum(g, x1, y1, z1, x2, y2, z2, flags, volZ, q.c.su, q.c.sv, 1u);
}

// Forward of R rows per lane of one detector column (the whole warp calls
// it) over the z-fastest copy volZ.  row(i, r): the lane's i-th ray (false: it
// has none); store(i, v): takes its value.
template <int R, bool REF, Steep STEEP, class Row, class Store>
__device__ __forceinline__ void colwarp_forward(const GridDev<float> &g, uint32_t flags, const float *__restrict__ volZ,
                                                Row row, Store store)
{
    ColRays<R> q;
    unsigned has = 0;
    {
        float r[R][6];
        bool h[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            h[i] = row(i, r[i]);
            has |= (unsigned)h[i] << i;
        }
        if (!col_rays<R, REF, true>(g, r, h, flags, q)) {
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (h[i]) store(i, 0.f);
            return;
        }
    }
    if (STEEP == kSteepCall && q.steep) {
#pragma unroll 1
        for (int i = 0; i < R; ++i) {
            float r[6];
            const bool h = row(i, r);
            const float v = colwarp_gather_steep<REF>(g, r[0], r[1], r[2], r[3], r[4], r[5], h, flags, volZ);
            if (h) store(i, v);
        }
        return;
    }
    GatherSink f[R];
#pragma unroll
    for (int i = 0; i < R; ++i) f[i] = GatherSink(volZ);
    if (STEEP == kSteepInline && q.steep) col_gather<R, REF, true, true>(q, volZ, f);
    else if (q.rising && q.falling) col_gather<R, REF, true, false>(q, volZ, f);
    else col_gather<R, REF, false, false>(q, volZ, f);
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (!(has >> i & 1u)) continue;
        float v = f[i].whole;
        if (!q.z[i].live) v = 0.f;
        else if (isfinite(v)) v *= q.W[i];
        else {
            float r[6];
            row(i, r);
            v = ray_resum(g, r[0], r[1], r[2], r[3], r[4], r[5], flags, volZ, q.c.su, q.c.sv, 1u);
        }
        store(i, v);
    }
}

__device__ __forceinline__ ScatterSink ray_sink(const FloatAcc &a, float yw) { return ScatterSink{a.vol, yw}; }
__device__ __forceinline__ FixedSink ray_sink(const FixedAcc &a, float yw) { return FixedSink{a.vol, yw, a.scale}; }

// Transpose of one row per lane (the whole warp calls it) of the warps that the
// walk below does not take: with steep rays, or with a value that is not finite
// (then every slab range checked and no voxel without a share touched).  Not
// inlined, and only in the kernels for scans that may have steep rays: the call
// costs the walk below 1 to 2 %, in line it would cost 1 % more.
template <bool REF, class Acc>
__device__ __noinline__ static void colwarp_scatter_rare(const GridDev<float> &g, float x1, float y1, float z1, float x2,
                                                         float y2, float z2, bool has, uint32_t flags, float y,
                                                         const Acc acc)
{
    const float r[1][6] = {{x1, y1, z1, x2, y2, z2}};
    const bool h[1] = {has};
    ColRays<1> q;
    if (!col_rays<1, REF, false>(g, r, h, flags, q)) return;
    const float yw[1] = {q.z[0].live ? y * q.W[0] : 0.f};
    if (__all_sync(0xffffffffu, isfinite(yw[0]))) {
        col_scatter<1, REF, true, true, kSingle>(q, acc, yw);
    } else if (q.z[0].live) {
        auto f = ray_sink(acc, yw[0]);
        ray_slabs<REF, true, false, -1, true, false>(q.c, q.z[0], q.zg, q.K0, q.K1, 1u, f);
    }
}

// Transpose of R rows per lane of one detector column: y[i] times the ray's
// weights into the z-fastest accumulator acc.  NEXT: the rows are neighbours
// in z order and merge their reductions.  STEEP: there may be steep rays.
template <int R, bool REF, bool NEXT, bool STEEP, class Acc>
__device__ __forceinline__ void colwarp_backward(const GridDev<float> &g, const float (&r)[R][6], bool (&has)[R],
                                                 uint32_t flags, const float (&y)[R], const Acc &acc)
{
    ColRays<R> q;
#pragma unroll
    for (int i = 0; i < R; ++i) has[i] = has[i] && y[i] != 0.f;
    if (!col_rays<R, REF, false>(g, r, has, flags, q)) return;
    float yw[R];
    bool finite = true;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        yw[i] = q.z[i].live ? y[i] * q.W[i] : 0.f;
        finite = finite && isfinite(yw[i]);
    }
    const bool plain = __all_sync(0xffffffffu, finite);
    if constexpr (STEEP) {
        if (q.steep || !plain) {
#pragma unroll
            for (int i = 0; i < R; ++i)
                colwarp_scatter_rare<REF>(g, r[i][0], r[i][1], r[i][2], r[i][3], r[i][4], r[i][5], has[i], flags, y[i],
                                          acc);
            return;
        }
    } else if (!plain) {
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (q.z[i].live) {
                auto f = ray_sink(acc, yw[i]);
                ray_slabs<REF, true, false, -1, true, false>(q.c, q.z[i], q.zg, q.K0, q.K1, 1u, f);
            }
        return;
    }
    const bool mixed = q.rising && q.falling;
    if constexpr (NEXT) {
        // a row that takes no part walks along with a neighbour, with value 0
        bool copy[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            copy[i] = !q.z[i].live;
            if (i > 0 && copy[i]) {
                q.z[i] = q.z[i - 1];
                q.z[i].live = false;
            }
        }
#pragma unroll
        for (int i = R - 2; i >= 0; --i)
            if (copy[i] && (i == 0 || copy[i - 1])) {
                q.z[i] = q.z[i + 1];
                q.z[i].live = false;
            }
        // the gap between two rays is linear along the walk: in order, and
        // within a voxel of the first ray, at both ends, by more than the
        // positions' rounding, it is so in every slab
        const float d0 = col_plane(q.c, q.K0), d1 = col_plane(q.c, q.K1 + 1);
        float size = fabsf(q.z[0].z0) + fabsf(q.z[0].kz) * (fabsf(q.c.pu) + fabsf(q.c.nu2));
        if (REF) size += fabsf(q.z[0].pw) * q.zg.rdz + q.zg.nz2;
        const float m = 1e-3f + 1e-6f * size;
        bool near = true;
#pragma unroll
        for (int i = 1; i < R; ++i) {
            const float a = fmaf(q.z[i].kz - q.z[i - 1].kz, d0, q.z[i].z0 - q.z[i - 1].z0);
            const float b = fmaf(q.z[i].kz - q.z[i - 1].kz, d1, q.z[i].z0 - q.z[i - 1].z0);
            near = near && (copy[i] || copy[i - 1] ? fminf(a, b) >= 0.f : fminf(a, b) > m);
        }
        const float a = fmaf(q.z[R - 1].kz - q.z[0].kz, d0, q.z[R - 1].z0 - q.z[0].z0);
        const float b = fmaf(q.z[R - 1].kz - q.z[0].kz, d1, q.z[R - 1].z0 - q.z[0].z0);
        near = near && fmaxf(a, b) < 1.f - m;
        if (!__all_sync(0xffffffffu, near)) col_scatter<R, REF, true, false, R == 2 ? kAny : kSingle>(q, acc, yw);
        else if (mixed) col_scatter<R, REF, true, false, kNear>(q, acc, yw);
        else col_scatter<R, REF, false, false, kNear>(q, acc, yw);
    } else {
        if (mixed) col_scatter<R, REF, true, false, kSingle>(q, acc, yw);
        else col_scatter<R, REF, false, false, kSingle>(q, acc, yw);
    }
}

// Row i of lane `lane` of a column warp whose rows start at `first`, with R
// rows per lane: rows 32 apart, or (NEXT) neighbours, in z order (rows fall in
// z when the row pitch is negative).
template <int R, bool NEXT> __device__ __forceinline__ int col_row(int first, int lane, int i, bool falling)
{
    return NEXT ? first + lane * R + (falling ? R - 1 - i : i) : first + i * 32 + lane;
}

// Launch shape of the thread walk for nvc views (see cb_cell).
template <typename T>
static inline void cb_shape(CBParams<T> &p, int na, int nb, int nvc, dim3 &grid, dim3 &block)
{
    const int rows = tune_get(NEFCT_TUNE_CB_ROWS);
    p.band_major = tune_get(NEFCT_TUNE_CB_ORDER) == 0;
    block = dim3(32, rows);
    const unsigned bands = (unsigned)((nb + rows - 1) / rows);
    grid = p.band_major ? dim3((na + 31) / 32, nvc, bands) : dim3((na + 31) / 32, bands, nvc);
}

// Launch shape of the column warps: NEFCT_TUNE_CB_ROWS columns (warps) per
// CTA, 32 rays_per_lane rows per warp.
template <typename T>
static inline void cb_colwarp_shape(CBParams<T> &p, int na, int nb, int nvc, dim3 &grid, dim3 &block,
                                    int rays_per_lane = 1)
{
    const int cols = tune_get(NEFCT_TUNE_CB_ROWS);
    p.band_major = tune_get(NEFCT_TUNE_CB_ORDER) == 0;
    block = dim3(32, cols);
    const unsigned tiles = (unsigned)((nb + 32 * rays_per_lane - 1) / (32 * rays_per_lane));
    grid = p.band_major ? dim3((na + cols - 1) / cols, nvc, tiles) : dim3((na + cols - 1) / cols, tiles, nvc);
}

// The walk skips its divisions when both transverse pitches equal the x pitch.
template <typename T> static inline bool cubic(const GridDev<T> &g) { return g.dy == (T)1 && g.dz == (T)1; }

// The rows per lane (least .. most) whose warps cover nb rows with the fewest
// slab steps: cost[R] for every full warp of 32 R rows, and for the last rows a
// warp with the fewest rows per lane that hold them (cb_row_launches).
static inline int cb_rows_per_lane(int nb, int least, int most, const int *cost)
{
    auto steps = [&](int r) {
        const int full = nb / (32 * r), few = (nb % (32 * r) + 31) / 32;
        // (a second launch ends with nearly empty waves of its own: 6 %)
        return ((long long)full * cost[r] + cost[few]) * (full > 0 && few > 0 && few < r ? 106 : 100);
    };
    int best = least;
    for (int r = least + 1; r <= most; ++r)
        if (steps(r) <= steps(best)) best = r;
    return best;
}

// Launches a column's rows with R rows per lane, and what is left of them with
// as few as hold it: launch(rows, rows per lane) takes rows from p.row0 on.
// 96^3, 120 views of 160 x 130 (130 rows as 96 + 34 instead of five 32-row warps
// in the forward, two 64-row warps and one of 32 instead of three 64-row warps in
// the transpose): forward 0.293 -> 0.275 ms, transpose 0.365 -> 0.329 ms.
template <class Launch>
static inline cudaError_t cb_row_launches(CBParams<float> &p, int nb, int R, Launch launch)
{
    const int left = nb % (32 * R), few = (left + 31) / 32;
    const int rows = few == R ? nb : nb - left;            // with R rows per lane
    p.row0 = 0;
    cudaError_t e = rows > 0 ? launch(rows, R) : cudaSuccess;
    if (e != cudaSuccess || rows == nb) return e;
    p.row0 = rows;
    e = launch(left, few);
    p.row0 = 0;
    return e;
}

// Neighbouring rows per lane that share the transpose's reductions.
//  * 1 while the row pitch at the rotation axis is 0.9 voxel or more: rows that
//    far apart rarely meet in a voxel, and 32 consecutive rows per warp then
//    touch fewer sectors than 32 pairs (256^3, 24 views, pitch 0.7 / 0.85 /
//    0.95 / 1.1 voxels: pairs 0.95 / 0.84 / 0.71 / 0.74 ms, single rows 1.27 /
//    0.91 / 0.67 / 0.55 ms);
//  * else two, or up to four if so many stay within a voxel at the far side of
//    the grid (thick slices), whichever covers the nb rows with the fewest slab
//    steps: a warp of 32 R rows takes about 1 / 1.45 / 1.85 times as long with R
//    = 2 / 3 / 4 (200 x 200 x 44 voxels of 2.5 mm, 60 views: 77 rows 0.50 / 0.38
//    / - ms, 120 rows 0.50 / 0.65 / 0.46 ms).
static inline int col_rows_next(const GridDev<float> &g, const RayGeom<float> &rg, int nb)
{
    if (!(rg.src_iso > 0.f && rg.src_det > 0.f)) return 1;
    const double rad = 0.5 * sqrt((double)g.nx * g.nx + (double)g.ny * g.dy * g.ny * g.dy) * g.dx_;
    const double pitch = fabs((double)rg.db) / rg.src_det / ((double)g.dz * g.dx_);       // voxels per unit distance
    if (pitch * rg.src_iso >= 0.9) return 1;
    const int most = std::min(4.0, 1.0 + 0.98 / (pitch * (rg.src_iso + rad)));
    static constexpr int cost[5] = {0, 67, 100, 145, 185};
    return cb_rows_per_lane(nb, 2, most, cost);
}

// Whether a scan may have steep rays (kSteep): |kz| <= sqrt(2) max |b| / src_det
// in units of the z and x pitch, since a ray runs at least src_det in x and y, of
// it 1 / sqrt(2) along its driving axis.  The transposes and the batch kernels
// without them are about 1 % faster (256^3, 48 views, transpose 2.008 against 2.031
// ms; 7 problems of 16^3 to 64^3, 84.9 + 94.8 against 86.1 + 95.5 us).
static inline bool cb_may_be_steep(const GridDev<float> &g, const RayGeom<float> &rg, int nb)
{
    if (!(rg.src_det > 0.f)) return true;
    const double b0 = (double)rg.bi * rg.db - rg.half_b, b1 = (nb - 1 + (double)rg.bi) * rg.db - rg.half_b;
    return !(sqrt(2.0) * std::max(fabs(b0), fabs(b1)) / rg.src_det / g.dz < 0.98);
}

// Column warps apply to FP32 slab walks with a workspace; the z-fastest
// copy's transposes launch ny planes (grid z: at most 65535); grids as wide keep
// the thread walk too, the only one run at that width.  Up to 8 detector rows
// leave most lanes of a column warp idle: the thread walk takes them (512^2 x 1 to
// 64, 120 views of 800 columns: 1 row 1.5 -> 0.26 ms forward and 1.7 -> 0.22
// transpose, 8 rows 1.6 -> 0.7 and 1.9 -> 0.7 to 0.8, 16 rows 1.6 / 1.3 and 1.9 /
// 1.5; 128^2: 75 -> 48 and 85 -> 46 us, 75 -> 58 and 92 -> 63, 78 / 82 and 93 / 98).
// (NEFCT_DETERMINISTIC changes nothing for the forward; its transpose has
// kernels of its own.)  nb: detector rows, where that counts.
template <typename T>
static inline bool cb_use_colwarp(const nefct_grid &g, uint32_t flags, bool forward, int nb = 65535)
{
    return sizeof(T) == sizeof(float) && (tune_get(NEFCT_TUNE_CB_WALK) & (forward ? 1 : 2)) != 0 &&
           !(flags & (NEFCT_EXACT | NEFCT_NO_TRANSPOSE)) && (forward || !(flags & NEFCT_DETERMINISTIC)) &&
           g.nx < 65533 && g.ny < 65533 && nb > 8;
}

// Launches the thread-walk forward (FWD) or transpose kernel for the views
// set in p.
template <typename T, bool FWD>
static inline cudaError_t cb_launch(CBParams<T> &p, int na, int nb, int nvc, uint32_t flags, cudaStream_t s)
{
    dim3 grid, block;
    cb_shape(p, na, nb, nvc, grid, block);
    const bool exact = (flags & NEFCT_EXACT) != 0;
    const bool var = sizeof(T) == 4 ? ref_rounding(flags) : !cubic(p.g);
    if constexpr (FWD) {
        if (exact) cb_forward_kernel<T, false, true><<<grid, block, 0, s>>>(p);
        else if (p.volT == nullptr && sizeof(T) == 4) {
            if (var) cb_forward_kernel<T, true, false, sizeof(T) != 4><<<grid, block, 0, s>>>(p);
            else cb_forward_kernel<T, false, false, sizeof(T) != 4><<<grid, block, 0, s>>>(p);
        } else if (var) cb_forward_kernel<T, true><<<grid, block, 0, s>>>(p);
        else cb_forward_kernel<T, false><<<grid, block, 0, s>>>(p);
    } else {
        if (exact) cb_backward_kernel<T, false, true><<<grid, block, 0, s>>>(p);
        else if (var) cb_backward_kernel<T, true><<<grid, block, 0, s>>>(p);
        else cb_backward_kernel<T, false><<<grid, block, 0, s>>>(p);
    }
    return cudaGetLastError();
}

// Launches the forward / transpose kernels for the views set in p: the
// thread walk, or the column warps when colwarp (p.volT / p.outT then hold
// the z-fastest copy / accumulator).  Defined in cb_forward.cu /
// cb_backward.cu for float and double.
template <typename T>
cudaError_t cb_launch_forward(CBParams<T> &p, int na, int nb, int nvc, uint32_t flags, cudaStream_t s,
                              bool colwarp = false);
template <typename T>
cudaError_t cb_launch_backward(CBParams<T> &p, int na, int nb, int nvc, uint32_t flags, cudaStream_t s,
                               bool colwarp = false);

// The deterministic transpose's column warps (p.fix: z-fastest accumulator).
cudaError_t cb_launch_backward_fixed(CBParams<float> &p, int na, int nb, int nvc, uint32_t flags, cudaStream_t s);

}  // namespace nefct
