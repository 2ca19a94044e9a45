// Distance-driven FDK backprojection on sm_100a (the detector-driven
// back_project_fdk_kernel of nefct/cc/distance_3d/dist_3d_back_fdk.cu.cc:17-255)
// and its C-ABI entry points (declared in include/nefct_b200.h).
//
// Semantics, per detector bin (ia, ib, iv), in the reference's order of
// operations (explicit round-to-nearest, no contraction):
//  * the bin centre ((i + 0.5) * d + offset - n * d / 2, evaluated in double
//    and rounded, :45-60) and the source give x21, y21, z21; the driving axis
//    is x when |x21| > |y21| (:66);
//  * for every slab of the driving axis the transverse footprint is the span
//    of the four rays through the bin's left/right edges with their x and y
//    components paired both ways (:72-123, :173-223), the z footprint the
//    span of the bin's lower/upper z edges (:125-139);
//  * every voxel inside both footprints gets value * (overlap fraction in v)
//    * (overlap fraction in z) / |u21| * |p2 - p1| * SAD^2 / (SAD + x cos +
//    y sin)^2 (:141-154).  The transverse footprint is evaluated with the
//    reference's operations (in double the z footprint too); the weights divide
//    by multiplying with approximate reciprocals and group the per-column
//    factors (a few ulp per weight).
//
// GPU structure (not the reference's), float: one warp walks the rows of one
// detector column at one view, several per lane, over a z-fastest volume copy
// (forward) or accumulator (backward), as the column warps of colwarp.cuh do.
//  * The x and y parts of those rays are identical (the bin's x and y do not
//    depend on the row), so each slab's transverse footprint, overlap
//    fractions and FDK weights are evaluated once per warp: lane j fills the
//    table entry of slab kc + j of a 32-slab chunk.
//  * A bin's z footprint has the same width 2 h in every row of the column (h =
//    |db / 2 / u21 * u|): its lower edge is affine along the walk and the share
//    of the lowest voxel is sat((floor(z) + 1 - z) / 2h), the rest falls on the
//    voxel above while 2h < 1 (wider footprints loop over their voxels).
//  * The backward sums the shares of two neighbouring rows in registers before
//    it reduces them.
// The double build (checks) evaluates every footprint per row, two rows per lane,
// over the x-fastest volume.  Per-view cos/sin/offset ride in the kernel parameters.
#include <math.h>
#include <algorithm>

#include "colwarp.cuh"

namespace nefct {

nefct_status zfold(const float *acc, float *vol, const nefct_grid &g, cudaStream_t s);
nefct_status zmajor_copy(const float *in, float *out, const nefct_grid &g, cudaStream_t s);

template <typename T> struct DDParams {
    int nx, ny, nz, na, nb, nvc, v0, cyl, fdk;
    T sid, sad;                   // source-detector, source-axis (the reference's SID, SAD)
    T da, ai, db, bi;
    const T *src;                 // backward: bins [nv][nb][na] (full); forward: the volume
    T *dst;                       // backward: accumulator; forward: bins [nv][nb][na] (full)
    unsigned long long sx, sy, sz;  // volume strides of (ix, iy, iz): z-fastest copy (float) or x-fastest (double)
    ViewTable<T> tab;
};

// (i + 0.5) * d + o - n * d / 2 with the reference's promotions: the first
// part in double, n * d / 2 in float (:45-60); all double in the FP64 build
__device__ __forceinline__ float dd_center(int i, float d, float o, int n)
{
    const float half = __fdiv_rn(__fmul_rn((float)n, d), 2.f);
    return (float)__dsub_rn(__dadd_rn(__dmul_rn((double)i + 0.5, (double)d), (double)o), (double)half);
}
__device__ __forceinline__ double dd_center(int i, double d, double o, int n)
{
    return __dsub_rn(__dadd_rn(__dmul_rn((double)i + 0.5, d), o), __dmul_rn((double)n, d) * 0.5);
}

// i * d + o - n * d / 2 (:78-80)
template <typename T> __device__ __forceinline__ T dd_edge(int i, T d, T o, int n)
{
    return FP<T>::sub(FP<T>::add(FP<T>::mul((T)i, d), o), FP<T>::div(FP<T>::mul((T)n, d), (T)2));
}

// cos/sin of a detector angle: the double-precision functions (rounded for float)
template <typename T> __device__ __forceinline__ void dd_trig(T a, T &c, T &s)
{
    double sd, cd;
    sincos((double)a, &sd, &cd);
    c = (T)cd;
    s = (T)sd;
}

// detector point (x20, y20) of lateral coordinate a (flat: a is the offset
// along the detector; cylindrical: the angle)
template <typename T> __device__ __forceinline__ void dd_det(const DDParams<T> &p, T a, T &x20, T &y20)
{
    if (p.cyl) {
        T c, s;
        dd_trig(a, c, s);
        x20 = FP<T>::sub(FP<T>::mul(p.sid, c), p.sad);
        y20 = FP<T>::mul(p.sid, s);
    } else {
        x20 = FP<T>::sub(p.sid, p.sad);
        y20 = a;
    }
}

template <typename T> __device__ __forceinline__ T dd_min(T a, T b) { return a < b ? a : b; }
template <typename T> __device__ __forceinline__ T dd_max(T a, T b) { return a > b ? a : b; }
template <typename T> __device__ __forceinline__ T dd_abs(T a) { return a > (T)0 ? a : -a; }
// reciprocal for the weight divisions: approximate in float (<= 1 ulp), exact in double
__device__ __forceinline__ float dd_rcp(float x) { return rcp_approx(x); }
__device__ __forceinline__ double dd_rcp(double x) { return __drcp_rn(x); }
__device__ __forceinline__ int dd_floor(float x) { return (int)floorf(x); }
__device__ __forceinline__ int dd_floor(double x) { return (int)floor(x); }

// The double build: one warp walks 32 R rows (bins) of one detector column at
// one view, R per lane (rows l, l + 32, ...), over the slabs of the column's
// driving axis; a slab's transverse part is evaluated once for the R rows
// (128^3, 24 views of 256 x 192, R = 1 / 2 / 4: forward 1.73 / 1.23 / 1.32 ms,
// backward 1.54 / 1.44 / 1.48).
// FWD false: each lane reduces value * weight into the voxels of its bins'
// footprints (the reference's kernel); FWD true: each lane sums voxel * weight
// over the same voxels with the same weights (the exact transpose) into its
// bins.  With p.fdk false the weight lacks the FDK factor SAD^2 / (SAD + x cos +
// y sin)^2.
static constexpr int kDDRows = 2;

template <bool FWD>
__global__ void __launch_bounds__(128) dd_kernel(const __grid_constant__ DDParams<double> p)
{
    using T = double;
    using F = FP<T>;
    constexpr int R = kDDRows;
    const int ia = blockIdx.x * blockDim.y + threadIdx.y;
    const int row = blockIdx.y * 32 * R + threadIdx.x;
    const int iv = blockIdx.z;
    if (ia >= p.na) return;
    const size_t bin = ((size_t)(p.v0 + iv) * p.nb + row) * p.na + ia, next = (size_t)32 * p.na;
    T value[R];
    bool live[R], any = false;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        live[i] = row + 32 * i < p.nb;
        value[i] = FWD || !live[i] ? (T)0 : p.src[bin + i * next];
        live[i] = live[i] && (FWD || value[i] != (T)0);
        any = any || live[i];
    }
    if (!any) return;

    const T cphi = p.tab.cs[iv], sphi = p.tab.sn[iv], off = p.tab.off[iv];
    const T x1 = F::mul(-p.sad, cphi), y1 = F::mul(-p.sad, sphi), z1 = off;
    T x20, y20;
    dd_det(p, dd_center(ia, p.da, p.ai, p.na), x20, y20);
    const T x2 = F::sub(F::mul(x20, cphi), F::mul(y20, sphi));
    const T y2 = F::add(F::mul(x20, sphi), F::mul(y20, cphi));
    const T x21 = F::sub(x2, x1), y21 = F::sub(y2, y1);
    T e[2][2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        T ex, ey;
        dd_det(p, dd_edge(ia + s, p.da, p.ai, p.na), ex, ey);
        e[s][0] = F::sub(F::sub(F::mul(ex, cphi), F::mul(ey, sphi)), x1);
        e[s][1] = F::sub(F::add(F::mul(ex, sphi), F::mul(ey, cphi)), y1);
    }
    const bool xdrive = dd_abs(x21) > dd_abs(y21);
    const int nu = xdrive ? p.nx : p.ny, nvt = xdrive ? p.ny : p.nx;
    const T u1 = xdrive ? x1 : y1, v1 = xdrive ? y1 : x1, u21 = xdrive ? x21 : y21;
    const T ul = xdrive ? e[0][0] : e[0][1], vl = xdrive ? e[0][1] : e[0][0];
    const T ur = xdrive ? e[1][0] : e[1][1], vr = xdrive ? e[1][1] : e[1][0];
    // the reference divides inside the slab loop; the quotients do not depend on the slab
    const T r0 = F::div(vl, ul), r1 = F::div(vl, ur), r2 = F::div(vr, ul), r3 = F::div(vr, ur);
    const T hdb = F::div(p.db, (T)2);
    T rzl[R], rzr[R], len_au[R], acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const T z2 = F::add(dd_center(row + 32 * i, p.db, p.bi, p.nb), off), z21 = F::sub(z2, z1);
        const T len = F::sqrt(F::add(F::add(F::mul(x21, x21), F::mul(y21, y21)), F::mul(z21, z21)));
        rzl[i] = F::div(F::sub(z21, hdb), u21);
        rzr[i] = F::div(F::add(z21, hdb), u21);
        len_au[i] = F::div(len, dd_abs(u21));
        acc[i] = (T)0;
    }
    const T vhalf = (T)(nvt / 2), zhalf = (T)(p.nz / 2), uhalf = F::div((T)nu, (T)2);
    const T sad2 = F::mul(p.sad, p.sad);
    const T xhalf = (T)(p.nx / 2), yhalf = (T)(p.ny / 2);
    for (int iu = 0; iu < nu; ++iu) {
        const T uc = F::sub(F::sub(F::add((T)iu, (T)0.5), uhalf), u1);
        const T c0 = F::add(F::add(F::mul(r0, uc), v1), vhalf);
        const T c1 = F::add(F::add(F::mul(r1, uc), v1), vhalf);
        const T c2 = F::add(F::add(F::mul(r2, uc), v1), vhalf);
        const T c3 = F::add(F::add(F::mul(r3, uc), v1), vhalf);
        const T vi1 = dd_min(dd_min(c0, c1), dd_min(c2, c3));
        const T vi2 = dd_max(dd_max(c0, c1), dd_max(c2, c3));
        const int va = max(0, dd_floor(vi1)), vb = min(nvt - 1, dd_floor(vi2));
        if (va > vb) continue;                      // footprint outside the grid
        const T ivspan = dd_rcp(F::sub(vi2, vi1));
        T zi1[R], zi2[R], izspan[R];
        int za[R], zb[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const T czl = F::add(F::add(F::mul(rzl[i], uc), z1), zhalf);
            const T czr = F::add(F::add(F::mul(rzr[i], uc), z1), zhalf);
            zi1[i] = dd_min(czl, czr);
            zi2[i] = dd_max(czl, czr);
            za[i] = max(0, dd_floor(zi1[i]));
            zb[i] = live[i] ? min(p.nz - 1, dd_floor(zi2[i])) : -1;
            izspan[i] = dd_rcp(F::sub(zi2[i], zi1[i]));
        }
        for (int iv2 = va; iv2 <= vb; ++iv2) {
            const T wv = F::mul(F::sub(dd_min((T)iv2 + (T)1, vi2), dd_max((T)iv2, vi1)), ivspan);
            const int ix = xdrive ? iu : iv2, iy = xdrive ? iv2 : iu;
            T fw = (T)1;
            if (p.fdk) {
                // (ix + 0.5 - nx / 2): exact
                const T xc = F::sub(F::add((T)ix, (T)0.5), xhalf);
                const T yc = F::sub(F::add((T)iy, (T)0.5), yhalf);
                const T iden = dd_rcp(F::add(F::add(p.sad, F::mul(xc, cphi)), F::mul(yc, sphi)));
                fw = F::mul(F::mul(sad2, iden), iden);
            }
            const size_t col = (size_t)iy * p.sy + (size_t)ix * p.sx;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                // (value *) wv * (len / |u21|) * fw per voxel of the column, times wz
                const T cw = F::mul(F::mul(FWD ? wv : F::mul(value[i], wv), len_au[i]), fw);
                for (int iz = za[i]; iz <= zb[i]; ++iz) {
                    const T wz = F::mul(F::sub(dd_min((T)iz + (T)1, zi2[i]), dd_max((T)iz, zi1[i])), izspan[i]);
                    if (FWD) acc[i] = F::add(acc[i], F::mul(__ldg(p.src + col + (size_t)iz * p.sz), F::mul(cw, wz)));
                    else atomicAdd(p.dst + col + (size_t)iz * p.sz, F::mul(cw, wz));
                }
            }
        }
    }
    if (FWD) {
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (live[i]) p.dst[bin + i * next] = acc[i];
    }
}

// ---- float: column warps ----

// Table of one chunk's slabs, for two of their voxel columns at most: a =
// (address of the first column less one element per floor bias, plane offset
// u, position of a footprint's lower edge less rz u), b = (weight of the first
// column, 1 / width, width, weight of the second), c = address of the second.
struct DDTable {
    uint4 a[32];
    float4 b[32];
    uint2 c[32];
};

// How a chunk's z footprints are walked: over two voxels (narrower than one
// voxel), inside the grid; the same with range checks; the same for rows that
// do not merge their reductions; over three voxels (narrower than two),
// checked; over any number.  Wider footprints do not merge either.
enum DDMode { kInner, kChecked, kApart, kThree, kWide };

// Lowest voxel (biased floor m) of the footprint whose lower edge is at rz * u
// + c, and t = (its lower plane) - (that edge), in (-1, 0].
template <bool CHECK> __device__ __forceinline__ void dd_low(float rz, float u, float c, float &m, float &t)
{
    float z = __fmaf_rn(rz, u, c);
    if (CHECK) z = fminf(fmaxf(z, -kFloorClamp), kFloorClamp);
    m = __fadd_rd(z, kFloorMagic);
    t = __fadd_rn(__fadd_rn(m, -kFloorMagic), -z);
}

// Walks table rows [0, single) with one voxel column and [single, n) with two,
// of the lane's two rows: FWD sums voxel * weight into acc, else reduces
// y * weight into the columns.
template <bool FWD, DDMode MODE>
__device__ __forceinline__ void dd_rows(const DDTable &tab, int single, int n, int nz, const float (&rz)[2],
                                        const float (&y)[2], float (&acc)[2])
{
    const Inside in(nz);
    if constexpr (MODE == kWide) {
#pragma unroll 1
        for (int j = 0; j < n; ++j) {
            const uint4 te = tab.a[j];
            const float4 tb = tab.b[j];
            const uint2 tc = tab.c[j];
            const int voxels = (int)fminf(tb.z, 4e6f) + 2;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float m, t;
                dd_low<true>(rz[i], __uint_as_float(te.z), __uint_as_float(te.w), m, t);
                const int f = __float_as_int(m) - kFloorMagicBits;
                const int k0 = max(0, -f), k1 = min(voxels, nz - f);         // voxels f + k in the grid
                float below = __saturatef(__fmul_rn(t + (float)k0, tb.y));
#pragma unroll 1
                for (int k = k0; k < k1; ++k) {
                    const float upto = __saturatef(__fmul_rn(t + (float)(k + 1), tb.y)), wz = upto - below;
                    below = upto;
                    if (wz == 0.f) continue;
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        if (c && j < single) continue;
                        float *const p = (c ? col_voxel(tc.x, tc.y, m) : col_voxel(te.x, te.y, m)) + k;
                        const float wv = c ? tb.w : tb.x;
                        if (FWD) acc[i] = __fmaf_rn(__ldg(p), wz * wv, acc[i]);
                        else FloatAcc::red(p, y[i] * wv * wz);
                    }
                }
            }
        }
    } else {
        constexpr int NV = MODE == kThree ? 3 : 2;
        constexpr bool CHECK = MODE != kInner;
        // the two rows' shares of the voxels m, m + 1(, m + 2) in one column at (lo, hi)
        auto column = [&](unsigned lo, unsigned hi, const float (&m)[2], const float (&w)[2][NV], float wv) {
            if constexpr (FWD) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float *const p = col_voxel(lo, hi, m[i]);
                    float sum = 0.f;
#pragma unroll
                    for (int k = 0; k < NV; ++k) {
                        const bool read = !CHECK || (w[i][k] != 0.f && in.low(m[i] + (float)k));
                        sum = __fmaf_rn(read ? __ldg(p + k) : 0.f, w[i][k], sum);
                    }
                    acc[i] = __fmaf_rn(sum, wv, acc[i]);
                }
            } else {
                float v[2][NV];
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int k = 0; k < NV; ++k) {
                        v[i][k] = (y[i] * wv) * w[i][k];
                        if (CHECK && (w[i][k] == 0.f || !in.low(m[i] + (float)k))) v[i][k] = 0.f;
                    }
                float *const p = col_voxel(lo, hi, m[0]);
                if constexpr (MODE == kInner || MODE == kChecked) {
                    // row 1's lowest voxel is row 0's or the one above
                    const bool same = m[0] == m[1];
                    v[0][0] += same ? v[1][0] : 0.f;
                    v[0][1] += same ? v[1][1] : v[1][0];
                    FloatAcc::red(p + 2, same ? 0.f : v[1][1]);
                } else {
                    float *const q = col_voxel(lo, hi, m[1]);
#pragma unroll
                    for (int k = 0; k < NV; ++k) FloatAcc::red(q + k, v[1][k]);
                }
#pragma unroll
                for (int k = 0; k < NV; ++k) FloatAcc::red(p + k, v[0][k]);
            }
        };
        auto shares = [&](const uint4 &te, float ispan, float (&m)[2], float (&w)[2][NV]) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float t;
                dd_low<CHECK>(rz[i], __uint_as_float(te.z), __uint_as_float(te.w), m[i], t);
                const float s1 = __saturatef(__fmaf_rn(t, ispan, ispan));
                w[i][0] = s1;
                if constexpr (NV == 2) {
                    w[i][1] = __fsub_rn(1.f, s1);
                } else {
                    const float s2 = __saturatef(__fmul_rn(t + 2.f, ispan));
                    w[i][1] = __fsub_rn(s2, s1);
                    w[i][2] = __fsub_rn(1.f, s2);
                }
            }
        };
#pragma unroll 2
        for (int j = 0; j < single; ++j) {
            const uint4 te = tab.a[j];
            const float2 tb = *reinterpret_cast<const float2 *>(&tab.b[j]);
            float m[2], w[2][NV];
            shares(te, tb.y, m, w);
            column(te.x, te.y, m, w, tb.x);
        }
#pragma unroll 2
        for (int j = single; j < n; ++j) {
            const uint4 te = tab.a[j];
            const float4 tb = tab.b[j];
            const uint2 tc = tab.c[j];
            float m[2], w[2][NV];
            shares(te, tb.y, m, w);
            column(te.x, te.y, m, w, tb.x);
            column(tc.x, tc.y, m, w, tb.w);
        }
    }
}

// One warp per 64 rows, two per lane, of detector column ia at view iv: rows l
// and l + 32, or (backward, while every footprint of the column is narrower
// than a voxel) neighbours, whose reductions merge.  256^3, 48 views of 512 x 384:
// forward 1.83 ms, bound by the gathers' L1 path (69 %) and latency, backward
// 2.87 ms, by the reductions' request path (88 %); with every footprint
// evaluated per ray (four edges, floors and overlaps per bin and slab, ~105
// instructions) 9.55 and 8.32 ms, bound by issue.  FWD false: value * weight into the z-fastest accumulator p.dst;
// FWD true: the sum of voxel * weight over the z-fastest copy p.src, the exact
// transpose.  With p.fdk false the weight lacks the FDK factor SAD^2 / (SAD + x
// cos + y sin)^2.
template <bool FWD>
__global__ void __launch_bounds__(128) dd_colwarp_kernel(const __grid_constant__ DDParams<float> p)
{
    using F = FP<float>;
    __shared__ DDTable tables[4];
    DDTable &tab = tables[threadIdx.y];
    const int lane = threadIdx.x;
    const int ia = blockIdx.x * blockDim.y + threadIdx.y;
    const int iv = blockIdx.z;
    if (ia >= p.na) return;                       // uniform across the warp
    const float cphi = p.tab.cs[iv], sphi = p.tab.sn[iv], off = p.tab.off[iv];
    const float x1 = F::mul(-p.sad, cphi), y1 = F::mul(-p.sad, sphi), z1 = off;
    // lane 0, 1: the bin's edges; the others: its centre (the reference
    // recomputes them in every slab)
    float ex, ey;
    dd_det(p, lane < 2 ? dd_edge(ia + lane, p.da, p.ai, p.na) : dd_center(ia, p.da, p.ai, p.na), ex, ey);
    const float px = F::sub(F::sub(F::mul(ex, cphi), F::mul(ey, sphi)), x1);
    const float py = F::sub(F::add(F::mul(ex, sphi), F::mul(ey, cphi)), y1);
    const float x21 = __shfl_sync(0xffffffffu, px, 2), y21 = __shfl_sync(0xffffffffu, py, 2);
    const bool xdrive = dd_abs(x21) > dd_abs(y21);
    const float pu = xdrive ? px : py, pv = xdrive ? py : px;
    const float ul = __shfl_sync(0xffffffffu, pu, 0), vl = __shfl_sync(0xffffffffu, pv, 0);
    const float ur = __shfl_sync(0xffffffffu, pu, 1), vr = __shfl_sync(0xffffffffu, pv, 1);
    const int nu = xdrive ? p.nx : p.ny, nvt = xdrive ? p.ny : p.nx;
    const float u1 = xdrive ? x1 : y1, v1 = xdrive ? y1 : x1, u21 = xdrive ? x21 : y21;
    const float r0 = F::div(vl, ul), r1 = F::div(vl, ur), r2 = F::div(vr, ul), r3 = F::div(vr, ur);
    const float hz = F::div(F::mul(p.db, 0.5f), u21);
    const float vhalf = (float)(nvt / 2), uhalf = F::mul((float)nu, 0.5f), zc = F::add(z1, (float)(p.nz / 2));
    const float sad2 = F::mul(p.sad, p.sad), xhalf = (float)(p.nx / 2), yhalf = (float)(p.ny / 2);
    // the widest footprint of the column, and whether all of it is in front of
    // the source
    const float uA = F::sub(F::sub(0.5f, uhalf), u1), uB = F::sub(F::sub((float)nu - 0.5f, uhalf), u1);
    const bool ahead = uA * u21 > 0.f && uB * u21 > 0.f;
    // (neighbouring footprints start that far apart, to the rounding of their
    // positions, which grows with the grid: less than a voxel, or the rows do not merge)
    const float apart = 1.f - (1e-3f + 1e-6f * ((float)p.nz + 2.f * dd_abs(z1)));
    const bool pairs = !FWD && ahead && 2.f * dd_abs(hz) * fmaxf(dd_abs(uA), dd_abs(uB)) < apart;
    // the rows: their z slope, length and value
    float rz[2], y[2], len[2], acc[2] = {0.f, 0.f};
    bool has[2], any = false, finite = true;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int row = blockIdx.y * 64 + (pairs ? lane * 2 + (p.db < 0.f ? 1 - i : i) : i * 32 + lane);
        has[i] = row < p.nb;
        const int ib = min(row, p.nb - 1);        // a row past the detector walks along with the last one
        const float z21 = F::sub(F::add(dd_center(ib, p.db, p.bi, p.nb), off), z1);
        rz[i] = F::div(z21, u21);
        len[i] = F::div(F::sqrt(F::add(F::add(F::mul(x21, x21), F::mul(y21, y21)), F::mul(z21, z21))), dd_abs(u21));
        y[i] = !FWD && has[i] ? p.src[((size_t)(p.v0 + iv) * p.nb + ib) * p.na + ia] : 0.f;
        any = any || y[i] != 0.f;
        y[i] *= len[i];
        finite = finite && isfinite(y[i]);
    }
    if (!FWD && !__any_sync(0xffffffffu, any)) return;
    bool checked = !FWD && !__all_sync(0xffffffffu, finite);
    const float *const vol = FWD ? p.src : p.dst;
    const char *const base = reinterpret_cast<const char *>(vol) - sizeof(float) * (size_t)(unsigned)kFloorMagicBits;
    // (forward: a sum that is not finite is walked again, range checked, which
    // reads no voxel of share 0)
    for (int pass = 0; pass < 2; ++pass) {
        for (int kc = 0; kc < nu; kc += 32) {
            const int iu = kc + lane;
            const float uc = F::sub(F::sub(F::add((float)min(iu, nu - 1), 0.5f), uhalf), u1);
            const float c0 = F::add(F::add(F::mul(r0, uc), v1), vhalf), c1 = F::add(F::add(F::mul(r1, uc), v1), vhalf);
            const float c2 = F::add(F::add(F::mul(r2, uc), v1), vhalf), c3 = F::add(F::add(F::mul(r3, uc), v1), vhalf);
            const float vi1 = fminf(fminf(c0, c1), fminf(c2, c3)), vi2 = fmaxf(fmaxf(c0, c1), fmaxf(c2, c3));
            const int va = max(0, dd_floor(vi1)), vb = min(nvt - 1, dd_floor(vi2));
            const int cols = iu < nu ? max(0, vb - va + 1) : 0;
            const int most = __reduce_max_sync(0xffffffffu, cols);
            if (most == 0) continue;
            const float h = dd_abs(F::mul(hz, uc)), zlow = F::sub(zc, h), span = 2.f * h, ispan = dd_rcp(span);
            const float ivspan = dd_rcp(F::sub(vi2, vi1));
            // the footprints' lower edges are linear over the chunk unless it
            // passes the source
            const float ua = __shfl_sync(0xffffffffu, uc, 0), ub = __shfl_sync(0xffffffffu, uc, 31);
            const float za = __shfl_sync(0xffffffffu, zlow, 0), zb = __shfl_sync(0xffffffffu, zlow, 31);
            const float wide = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(span)));
            const bool front = ua * u21 > 0.f && ub * u21 > 0.f;
            bool inner = true, out = true;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float a = __fmaf_rn(rz[i], ua, za), b = __fmaf_rn(rz[i], ub, zb);
                const float lo = fminf(a, b), hi = fmaxf(a, b) + wide, mg = 0.01f + 1e-5f * (dd_abs(lo) + dd_abs(hi));
                inner = inner && lo >= mg && hi <= (float)(p.nz - 1) - mg;
                out = out && (hi < -mg || lo > (float)p.nz + mg);
            }
            if (front && __all_sync(0xffffffffu, out)) continue;
            const bool safe = !checked && front && __all_sync(0xffffffffu, inner) && (FWD || pairs);
            const DDMode mode = !(wide < 1.999f && wide > 0.f) || !front ? kWide
                                : wide >= 0.999f ? kThree : safe ? kInner : FWD || pairs ? kChecked : kApart;
            // two voxel columns of every slab at a time
            for (int t = 0; t < most; t += 2) {
                const int rem = cols - t;
                const unsigned one = __ballot_sync(0xffffffffu, rem == 1), two = __ballot_sync(0xffffffffu, rem >= 2);
                const unsigned below = (1u << lane) - 1u;
                const int single = __popc(one), n = single + __popc(two);
                __syncwarp();
                if (rem >= 1) {
                    const int row = rem == 1 ? __popc(one & below) : single + __popc(two & below);
                    unsigned long long adr[2];
                    float wt[2];
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int iw = min(va + t + c, vb), ix = xdrive ? iu : iw, iy = xdrive ? iw : iu;
                        wt[c] = F::mul(F::sub(fminf((float)iw + 1.f, vi2), fmaxf((float)iw, vi1)), ivspan);
                        if (p.fdk) {
                            // (ix + 0.5 - nx / 2): exact
                            const float xc = F::sub(F::add((float)ix, 0.5f), xhalf), yc = F::sub(F::add((float)iy, 0.5f), yhalf);
                            const float iden = dd_rcp(F::add(F::add(p.sad, F::mul(xc, cphi)), F::mul(yc, sphi)));
                            wt[c] = F::mul(wt[c], F::mul(F::mul(sad2, iden), iden));
                        }
                        adr[c] = (unsigned long long)(base + sizeof(float) * ((size_t)iy * p.sy + (size_t)ix * p.sx));
                    }
                    tab.a[row] = make_uint4((unsigned)adr[0], (unsigned)(adr[0] >> 32), __float_as_uint(uc),
                                            __float_as_uint(zlow));
                    tab.b[row] = make_float4(wt[0], ispan, span, wt[1]);
                    tab.c[row] = make_uint2((unsigned)adr[1], (unsigned)(adr[1] >> 32));
                }
                __syncwarp();
                if (mode == kInner) dd_rows<FWD, kInner>(tab, single, n, p.nz, rz, y, acc);
                else if (mode == kChecked) dd_rows<FWD, kChecked>(tab, single, n, p.nz, rz, y, acc);
                else if (!FWD && mode == kApart) dd_rows<FWD, kApart>(tab, single, n, p.nz, rz, y, acc);
                else if (mode == kThree) dd_rows<FWD, kThree>(tab, single, n, p.nz, rz, y, acc);
                else dd_rows<FWD, kWide>(tab, single, n, p.nz, rz, y, acc);
            }
        }
        if (!FWD || checked || !__any_sync(0xffffffffu, !isfinite(acc[0]) || !isfinite(acc[1]))) break;
        checked = true;
        acc[0] = acc[1] = 0.f;
    }
    if (FWD) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int ib = blockIdx.y * 64 + i * 32 + lane;
            if (has[i]) p.dst[((size_t)(p.v0 + iv) * p.nb + ib) * p.na + ia] = acc[i] * len[i];
        }
    }
}

static nefct_status check_dd(const nefct_dd_geom *g)
{
    if (!g) return fail(NEFCT_ERR_INVALID, "geometry is NULL");
    if (g->nx < 1 || g->ny < 1 || g->nz < 1) return fail(NEFCT_ERR_INVALID, "grid must be >= 1 voxel per axis");
    if (g->nx > (1 << 20) || g->ny > 65535 || g->nz > (1 << 20) || (long long)g->nx * g->ny * g->nz >= (1ll << 31))
        return fail(NEFCT_ERR_INVALID, "grid too large (%d x %d x %d)", g->nx, g->ny, g->nz);
    if (g->nv < 1 || !g->angles) return fail(NEFCT_ERR_INVALID, "need nv >= 1 view angles");
    if (g->na < 1 || g->nb < 1 || g->nb > 65535 * 32)
        return fail(NEFCT_ERR_INVALID, "detector must be >= 1 x 1 (got %d x %d)", g->na, g->nb);
    if (g->det_kind != NEFCT_DET_FLAT && g->det_kind != NEFCT_DET_CYL)
        return fail(NEFCT_ERR_INVALID, "det_kind must be NEFCT_DET_FLAT or NEFCT_DET_CYL");
    const float v[7] = {g->src_iso, g->src_det, g->da, g->a_offset, g->db, g->b_offset, 0.f};
    for (int i = 0; i < 6; ++i)
        if (!std::isfinite(v[i])) return fail(NEFCT_ERR_INVALID, "geometry must be finite");
    for (int i = 0; i < g->nv; ++i)
        if (!std::isfinite(g->angles[i]) || (g->z_offsets && !std::isfinite(g->z_offsets[i])))
            return fail(NEFCT_ERR_INVALID, "view %d: angle / offset not finite", i);
    return NEFCT_OK;
}

template <typename T>
static nefct_status dd_impl(const nefct_dd_geom *g, const T *src, T *dst, uint32_t flags, void *ws, size_t ws_bytes,
                            cudaStream_t s, bool forward)
{
    nefct_status st = check_dd(g);
    if (st) return st;
    if (!src || !dst) return fail(NEFCT_ERR_INVALID, "input and output must be non-NULL");
    if (flags & ~NEFCT_FDK_NO_WEIGHT) return fail(NEFCT_ERR_INVALID, "unknown flag bits 0x%x", flags);
    const bool f32 = sizeof(T) == sizeof(float);
    const size_t nvox = (size_t)g->nx * g->ny * g->nz;
    const nefct_grid gr{g->nx, g->ny, g->nz, 0.f, 0.f, 0.f, (float)g->nx, (float)g->ny, (float)g->nz};
    DDParams<T> *p = new DDParams<T>();
    p->nx = g->nx; p->ny = g->ny; p->nz = g->nz; p->na = g->na; p->nb = g->nb;
    p->cyl = g->det_kind == NEFCT_DET_CYL;
    p->fdk = !(flags & NEFCT_FDK_NO_WEIGHT);
    p->sid = g->src_det; p->sad = g->src_iso;
    p->da = g->da; p->ai = g->a_offset; p->db = g->db; p->bi = g->b_offset;
    if (f32) {
        // float: a z-fastest volume copy [y][x][z] (forward source / backward
        // accumulator), so the 32 rows of a warp touch neighbouring z
        const size_t need = nefct_dd_workspace_bytes(g);
        if (!ws || ws_bytes < need) {
            delete p;
            return fail(NEFCT_ERR_WORKSPACE, "needs %zu workspace bytes, got %zu", need, ws_bytes);
        }
        p->sx = (unsigned long long)g->nz;
        p->sy = (unsigned long long)g->nx * g->nz;
        p->sz = 1;
        if (forward) {
            st = zmajor_copy((const float *)src, (float *)ws, gr, s);
            if (st) { delete p; return st; }
            p->src = (const T *)ws;
            p->dst = dst;
        } else {
            const cudaError_t e = cudaMemsetAsync(ws, 0, need, s);
            if (e != cudaSuccess) { delete p; return cuda_fail(e, "cudaMemsetAsync"); }
            p->src = src;
            p->dst = (T *)ws;
        }
    } else {
        // double (checks and tests): the x-fastest volume in place, no workspace
        p->sx = 1;
        p->sy = (unsigned long long)g->nx;
        p->sz = (unsigned long long)g->nx * g->ny;
        p->src = src;
        p->dst = dst;
        if (!forward) {
            const cudaError_t e = cudaMemsetAsync(dst, 0, nvox * sizeof(T), s);
            if (e != cudaSuccess) { delete p; return cuda_fail(e, "cudaMemsetAsync"); }
        }
    }
    const int cols = 4;
    const int kMax = ViewTable<T>::kMax;
    for (int v0 = 0; v0 < g->nv; v0 += kMax) {
        const int nvc = std::min(kMax, g->nv - v0);
        p->v0 = v0;
        p->nvc = nvc;
        for (int i = 0; i < nvc; ++i) {
            const double a = (double)g->angles[v0 + i];
            p->tab.cs[i] = (T)cos(a);
            p->tab.sn[i] = (T)sin(a);
            p->tab.off[i] = g->z_offsets ? (T)g->z_offsets[v0 + i] : (T)0;
        }
        const int rows = f32 ? 64 : 32 * kDDRows;
        dim3 grid((g->na + cols - 1) / cols, (g->nb + rows - 1) / rows, nvc), block(32, cols);
        if constexpr (std::is_same<T, float>::value) {
            if (forward) dd_colwarp_kernel<true><<<grid, block, 0, s>>>(*p);
            else dd_colwarp_kernel<false><<<grid, block, 0, s>>>(*p);
        } else {
            if (forward) dd_kernel<true><<<grid, block, 0, s>>>(*p);
            else dd_kernel<false><<<grid, block, 0, s>>>(*p);
        }
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) { delete p; return cuda_fail(e, forward ? "dd_kernel<forward>" : "dd_kernel<backward>"); }
    }
    delete p;
    if (f32 && !forward) return zfold((const float *)ws, (float *)dst, gr, s);
    return NEFCT_OK;
}

}  // namespace nefct

using namespace nefct;

extern "C" {

size_t nefct_dd_workspace_bytes(const nefct_dd_geom *g)
{
    if (!g || g->nx < 1 || g->ny < 1 || g->nz < 1) return 0;
    return (size_t)g->nx * g->ny * g->nz * sizeof(float);
}

nefct_status nefct_dd_backproject(const nefct_dd_geom *g, const float *proj, float *vol, void *ws, size_t ws_bytes,
                                  void *stream)
{
    return dd_impl<float>(g, proj, vol, 0, ws, ws_bytes, (cudaStream_t)stream, false);
}

nefct_status nefct_dd_forward(const nefct_dd_geom *g, const float *vol, float *proj, uint32_t flags, void *ws,
                              size_t ws_bytes, void *stream)
{
    return dd_impl<float>(g, vol, proj, flags, ws, ws_bytes, (cudaStream_t)stream, true);
}

nefct_status nefct_dd_backward(const nefct_dd_geom *g, const float *proj, float *vol, uint32_t flags, void *ws,
                               size_t ws_bytes, void *stream)
{
    return dd_impl<float>(g, proj, vol, flags, ws, ws_bytes, (cudaStream_t)stream, false);
}

nefct_status nefct_dd_forward_f64(const nefct_dd_geom *g, const double *vol, double *proj, uint32_t flags,
                                  void *stream)
{
    return dd_impl<double>(g, vol, proj, flags, nullptr, 0, (cudaStream_t)stream, true);
}

nefct_status nefct_dd_backward_f64(const nefct_dd_geom *g, const double *proj, double *vol, uint32_t flags,
                                   void *stream)
{
    return dd_impl<double>(g, proj, vol, flags, nullptr, 0, (cudaStream_t)stream, false);
}

}  // extern "C"
