// Column-warp cone-beam walk (FP32, sm_100a).
//
// The rays of one detector column at one view share their x and y end
// points (the generator's x1, y1, x2, y2 do not depend on the row: the
// source and the column's detector points lie in one vertical plane), so the
// drive axis, pu, pv, kv and every transverse (v) plane position, floor and
// crossing ratio are bit-identical across the rows of a column; only the z
// part (pw, kw, W) differs.
//
// One warp walks 32 R rows of one column, R per lane, in lockstep over the
// union of their slab ranges:
//  * the v part of each slab is computed once per warp: lane j builds the
//    entry of slab kc + j of a 32-slab chunk into the warp's table in shared
//    memory, and every lane reads each slab's entry with broadcast loads, once
//    for its R rays; whether the slab crosses a v plane is the same for the
//    whole warp;
//  * the volume (forward) and the accumulator (transpose) are z-fastest
//    copies [y][x][z]: the rows of a warp sit at neighbouring z of the same
//    (u, v) voxel column, and a ray's two z voxels are adjacent in memory.
// A slab's v columns are in the grid or not for the whole warp, so the table
// drops the ones that are not; the z voxels need range checks only in the
// chunks of slabs where some ray of the warp can leave the grid in z (also
// slabs before or after a ray's own range).
//
// The z split of a slab.  With q1, q2 the positions at the slab's lower and
// upper plane (in z) and c = floor(q1) + 1, the share of the low voxel is
// rw = min(1, (c - q1) / (q2 - q1)): 1 without a crossing, so no crossing test
// is needed while |kz| (z voxels per slab) stays below 1; steeper rays take
// the general split.
//  * By default q1 = fma(kz, d, z0) and q2 - q1 = |kz| exactly: one fused
//    multiply-add, a floor and one saturating multiply-add per ray and slab, the
//    same in the forward and its transpose.  Positions count from the source's
//    row, so that z0 is a fraction held to 2^-25: rounded at the size of a row
//    number its error, constant along the ray, would go into every share divided
//    by |kz| (rel-L2 of the forward against FP64, 600 slices of 0.1 voxel, nearly
//    level rays: 1.5e-5, so 3.3e-6, the reference's operations in float 8.7e-6; 24
//    cubic ones: 1.00e-6, 9.4e-7, 9.8e-7).
//  * REF (calls with NEFCT_TIE_GT, the switches of the reference's own
//    backprojection): q1 and q2 with the reference's operations in its order.
//    A nearly level ray (|kz| ~ 1e-3) divides rounding errors of ~1e-5 voxel
//    by |kz|, and a voxel that few views reach shows them: there the result
//    follows the reference's rounding.
#pragma once

#include <limits.h>

#include "siddon.cuh"

namespace nefct {

// Transverse (v) part of a column's walk: the same for every row.
struct ColWalk {
    float pu, pv, kv, dv, nv2, nu2;
    int nv;
    unsigned su, sv;
    bool vdiv;
};

// v part of one slab of a column warp: biased bases of the low/high v voxel
// columns (index of (k, v, z) = b + floor bits of z), which of them are in the
// grid, and the v crossing ratio.
struct ColEntry {
    unsigned b1, b2;    // k*su + c*sv - 0x4B400000 for the low/high v floor c
    unsigned in;        // bit 0, 1: the low, high column is in the grid
    float rv;           // crossing ratio, 1 without a v crossing
    bool vx;            // the slab crosses a v plane
};

__device__ __forceinline__ ColWalk col_walk_of(const GridDev<float> &g, const Walk<float> &w, unsigned su, unsigned sv)
{
    ColWalk c;
    c.pu = w.pu; c.pv = w.pv; c.kv = w.kv;
    c.dv = w.dv; c.vdiv = w.vdiv;
    c.nv2 = w.nv2; c.nu2 = w.nu2; c.nv = w.nv;
    c.su = su; c.sv = sv;
    return c;
}

// Offset t - pu of plane k (t = k - nu2 is exact: nu2 is a multiple of 1/2
// and |k| < 2^22).
__device__ __forceinline__ float col_plane(const ColWalk &c, int k)
{
    return __fsub_rn(__fsub_rn((float)k, c.nu2), c.pu);
}

// v position at plane offset d in the reference's operations and order.
// DIV: 1 (0) divides by dv (not); -1: as c says.
template <int DIV = -1> __device__ __forceinline__ float col_vpos(const ColWalk &c, float d)
{
    float q = __fadd_rn(c.pv, __fmul_rn(c.kv, d));
    if (DIV < 0 ? c.vdiv : DIV != 0) q = __fdiv_rn(q, c.dv);
    return __fadd_rn(q, c.nv2);
}

// Crossing ratio of a slab with v positions q1 <= q2 and biased floors m1, m2; at
// most 1 (the approximate reciprocal can pass it by an ulp, and would give a
// share to a voxel that the ray does not touch, outside the grid at its faces).
__device__ __forceinline__ float col_ratio(float q1, float q2, float m1, float m2)
{
    const float num = __fadd_rn(__fadd_rn(m2, -kFloorMagic), -q1);
    return m1 != m2 ? __saturatef(__fmul_rn(num, rcp_approx(__fadd_rn(q2, -q1)))) : 1.f;
}

// Whether a voxel of biased floor m, and the one above it, are among n.
struct Inside {
    float lo, hi;           // biased floors 0 and n
    // first: what floor 0 stands for
    __device__ __forceinline__ Inside(int n, int first = 0)
        : lo(kFloorMagic - (float)first), hi(kFloorMagic + (float)(n - first)) {}
    __device__ __forceinline__ Inside(float lo_, float hi_) : lo(lo_), hi(hi_) {}
    __device__ __forceinline__ bool low(float m) const { return m >= lo && m < hi; }
    __device__ __forceinline__ bool high(float m) const { return m >= lo - 1.f && m < hi - 1.f; }
    // the high one of a slab with floors m < mh, admitted from m = -1 on
    // (the reference's slab admission, siddon.cu.cc:80, :92, :112, :116, :132)
    __device__ __forceinline__ bool far(float m, float mh) const { return m >= lo - 1.f && mh >= lo && mh < hi; }
};

// Entry of slab k: planes t = k - nu2 and t + 1.
__device__ __forceinline__ ColEntry col_entry(const ColWalk &c, int k)
{
    const float qa = col_vpos(c, col_plane(c, k)), qb = col_vpos(c, col_plane(c, k + 1));
    const float ma = magic_floor<true>(qa), mb = magic_floor<true>(qb);
    const float m1 = fminf(ma, mb), m2 = fmaxf(ma, mb);
    const Inside in(c.nv);
    ColEntry e;
    e.rv = col_ratio(fminf(qa, qb), fmaxf(qa, qb), m1, m2);
    e.vx = m1 != m2;
    e.in = (unsigned)in.low(m1) | (unsigned)(e.vx && in.far(m1, m2)) << 1;
    const unsigned base = (unsigned)k * c.su - (unsigned)kFloorMagicBits * (c.sv + 1u);
    e.b1 = base + (unsigned)__float_as_int(m1) * c.sv;
    e.b2 = base + (unsigned)__float_as_int(m2) * c.sv;
    return e;
}

// z part of a ray, in voxel rows from row zi on (the source's row; REF: row 0).
struct ZRay {
    float kz, z0, ikz;      // position kz * d + z0 at plane offset d; ikz = 1 / |kz| (at most 1e30)
    float kw, pw;           // REF: position ((pw + kw * d) * rdz) + nz2
    int zi;
    int down;               // kz < 0: the slab's lower z plane is its exit plane
    bool live, steep;
};

// Rays from this slope on take the general split (below 1 by more than the
// rounding of the positions).
constexpr float kSteep = 0.999f;

// Grid constants of the z positions.
struct ZGrid {
    float dz, rdz, nz2;     // dz, 1 / dz, nz / 2
    bool div;               // dz != 1
    int nz;
};
__device__ __forceinline__ ZGrid z_grid(const GridDev<float> &g)
{
    return ZGrid{g.dz, __fdiv_rn(1.f, g.dz), g.nz2, g.dz != 1.f, g.nz};
}

// The source's row zi (within 2^20 rows of the grid, so positions stay below
// 2^21) and its height above it: pw / dz + nz / 2 - zi, exact but for the
// division's remainder, which is added back.  The same for every ray of a view.
struct ZSource {
    int zi;
    float row, z0;
};
template <bool REF> __device__ __forceinline__ ZSource z_source(const Walk<float> &w, const ZGrid &zg)
{
    if (REF) return ZSource{0, 0.f, 0.f};
    ZSource s;
    s.row = rintf(fminf(fmaxf(w.z0, -1048576.f), 1048576.f));
    s.zi = (int)s.row;
    const float q = zg.div ? __fdiv_rn(w.pw, zg.dz) : w.pw;
    s.z0 = __fsub_rn(q, __fsub_rn(s.row, zg.nz2));
    if (zg.div) s.z0 = __fmaf_rn(__fmaf_rn(-q, zg.dz, w.pw), zg.rdz, s.z0);
    return s;
}

// (a lane without a ray walks row 0: its indices stay in the grid)
template <bool REF>
__device__ __forceinline__ ZRay z_ray(const Walk<float> &w, const ZGrid &zg, const ZSource &s, bool live)
{
    ZRay z;
    z.live = live;
    z.kz = live ? w.kz : 0.f;
    z.kw = live ? w.kw : 0.f;
    z.pw = live ? w.pw : __fmul_rn(__fsub_rn(0.5f, zg.nz2), zg.dz);
    z.zi = s.zi;
    z.z0 = 0.f;
    if (!REF) {
        // (a level ray has its height as rounded: along a plane of the grid that
        // decides which slice it lies in, as in the reference)
        z.z0 = !live ? __fsub_rn(0.5f, s.row) : z.kz == 0.f ? __fsub_rn(w.z0, s.row) : s.z0;
        // (the slope's rounding, added back at the grid's middle plane)
        if (zg.div && live) z.z0 = __fmaf_rn(-w.pu * zg.rdz, __fmaf_rn(-w.kz, zg.dz, w.kw), z.z0);
    }
    z.ikz = fminf(__fdiv_rn(1.f, fabsf(z.kz)), 1e30f);
    z.down = z.kz < 0.f;
    z.steep = fabsf(z.kz) > kSteep;
    return z;
}

// Position at plane offset d in the reference's order of operations (its
// division by dz as a multiplication by 1 / dz).
__device__ __forceinline__ float z_pos(const ZRay &z, const ZGrid &zg, float d)
{
    float q = __fadd_rn(z.pw, __fmul_rn(z.kw, d));
    if (zg.div) q = __fmul_rn(q, zg.rdz);
    return __fadd_rn(q, zg.nz2);
}

// Position at plane offset d.
template <bool REF> __device__ __forceinline__ float z_at(const ZRay &z, const ZGrid &zg, float d)
{
    return REF ? z_pos(z, zg, d) : __fmaf_rn(z.kz, d, z.z0);
}

// z split of a slab of a ray that is not steep: biased floor and low share.  q,
// qh: positions at its lower and upper plane (qh: REF only).
// (The grid has at most 2^20 rows and slabs, and such a ray moves at most one
// row per slab: positions stay below 2^22, no clamp is needed for the floor.)
template <bool REF> __device__ __forceinline__ void z_share(const ZRay &z, float q, float qh, float &m, float &r)
{
    m = __fadd_rd(q, kFloorMagic);
    if (REF) {
        const float c = __fadd_rn(m, 1.f - kFloorMagic);
        r = __saturatef(__fmul_rn(__fadd_rn(c, -q), rcp_approx(__fadd_rn(qh, -q))));
    } else {
        r = __saturatef(__fmaf_rn(__fadd_rn(__fadd_rn(m, -kFloorMagic), -q), z.ikz, z.ikz));
    }
}

// The same from the offsets of the lower and upper plane.
template <bool REF>
__device__ __forceinline__ void z_inner(const ZRay &z, const ZGrid &zg, float lo, float hi, float &m, float &r)
{
    z_share<REF>(z, z_at<REF>(z, zg, lo), REF ? z_pos(z, zg, hi) : 0.f, m, r);
}

// z split of any ray's slab: biased floors of its low and high voxel and the low
// share.  q, qh: positions at the lower and upper plane (qh: REF or steep only).
template <bool REF>
__device__ __forceinline__ void z_split(const ZRay &z, float q, float qh, float &m, float &mh, float &r)
{
    if (!z.steep) {
        z_share<REF>(z, q, qh, m, r);
        mh = __fadd_rn(m, 1.f);
        return;
    }
    m = magic_floor<true>(q);
    mh = magic_floor<true>(qh);
    q = fminf(fmaxf(q, -kFloorClamp), kFloorClamp);
    qh = fminf(fmaxf(qh, -kFloorClamp), kFloorClamp);
    const float iden = REF ? rcp_approx(__fadd_rn(qh, -q)) : z.ikz;
    r = mh != m ? __fmul_rn(__fadd_rn(__fadd_rn(mh, -kFloorMagic), -q), iden) : 1.f;
}

// ---- sinks: what one ray does with a slab's voxels ----
//
// The shares of a slab are the overlaps of the ray's v intervals [0, rv], [rv,
// 1] and z intervals [0, r], [r, 1] (the reference's pairing, Q1): (v1, z1),
// (v1, z2) or (v2, z1), (v2, z2).  f.inner(vx, p, w): these three voxels, all in
// the grid; f.edge(kind, p, ok, w): bit i of ok: voxel i is in the grid (a
// voxel without a share is not touched).

// Slabs without a v crossing; with one and both columns in the grid; with one
// and a single column in the grid.
enum SlabKind { kPlain, kCross, kHalf };

// The voxels of a slab of one ray, their shares, and whether it crosses a v plane.
struct RaySlab {
    unsigned p[3];
    float w[3];
    bool vx;
};

// Forward: sums of value * share, by kind of slab and by aligned block of 32
// slabs (close() ends a block), so that the total does not depend on which
// rays walk together; sums of partial sums also round less than one running
// sum.
struct GatherSink {
    static constexpr bool kGather = true;
    const float *__restrict__ vol;
    float sum[3], whole;

    __device__ __forceinline__ GatherSink() {}
    __device__ __forceinline__ GatherSink(const float *v) : vol(v), sum{0.f, 0.f, 0.f}, whole(0.f) {}
    __device__ __forceinline__ void edge(SlabKind kind, const unsigned (&p)[3], unsigned ok, const float (&w)[3])
    {
        float s = kind == kPlain ? sum[0] : kind == kCross ? sum[1] : sum[2];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float v = (ok >> i & 1u) && w[i] != 0.f ? __ldg(vol + p[i]) : 0.f;
            s = __fmaf_rn(v, w[i], s);
        }
        if (kind == kPlain) sum[0] = s;
        else if (kind == kCross) sum[1] = s;
        else sum[2] = s;
    }
    // G slabs: all loads first, so that they overlap (of the last two voxels of a
    // slab, those without a share, most of them, are not read)
    template <int G> __device__ __forceinline__ void inner(const RaySlab (&s)[G])
    {
        float v[G][3];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            v[g][0] = __ldg(vol + s[g].p[0]);
            v[g][1] = s[g].w[1] != 0.f ? __ldg(vol + s[g].p[1]) : 0.f;
            v[g][2] = s[g].w[2] != 0.f ? __ldg(vol + s[g].p[2]) : 0.f;
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float *const w = s[g].w;
            if (s[g].vx) sum[1] = __fmaf_rn(v[g][2], w[2], __fmaf_rn(v[g][1], w[1], __fmaf_rn(v[g][0], w[0], sum[1])));
            else sum[0] = __fmaf_rn(v[g][1], w[1], __fmaf_rn(v[g][0], w[0], sum[0]));
        }
    }
    __device__ __forceinline__ void close()
    {
        whole = __fadd_rn(whole, __fadd_rn(__fadd_rn(sum[0], sum[1]), sum[2]));
        sum[0] = sum[1] = sum[2] = 0.f;
    }
};

// Transpose: one reduction of yw * share per voxel with a share.
struct ScatterSink {
    static constexpr bool kGather = false;
    float *acc;
    float yw;

    __device__ __forceinline__ void edge(SlabKind, const unsigned (&p)[3], unsigned ok, const float (&w)[3]) const
    {
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if ((ok >> i & 1u) && w[i] != 0.f) atomicAdd(acc + p[i], yw * w[i]);
    }
    template <int G> __device__ __forceinline__ void inner(const RaySlab (&s)[G]) const
    {
#pragma unroll
        for (int g = 0; g < G; ++g) edge(kPlain, s[g].p, 7u, s[g].w);
    }
    __device__ __forceinline__ void close() const {}
};

// Deterministic transpose: each contribution yw * share, scaled by a power of
// two (exact) and rounded to a 64-bit integer (siddon.cuh, to_fixed).
struct FixedSink {
    static constexpr bool kGather = false;
    unsigned long long *acc;
    float yw, scale;

    __device__ __forceinline__ void edge(SlabKind, const unsigned (&p)[3], unsigned ok, const float (&w)[3]) const
    {
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if ((ok >> i & 1u) && w[i] != 0.f)
                atomicAdd(acc + p[i], (unsigned long long)to_fixed((yw * w[i]) * scale));
    }
    template <int G> __device__ __forceinline__ void inner(const RaySlab (&s)[G]) const
    {
#pragma unroll
        for (int g = 0; g < G; ++g) edge(kPlain, s[g].p, 7u, s[g].w);
    }
    __device__ __forceinline__ void close() const {}
};

// Slabs k..end of one ray alone (any strides), with a column warp's operations
// per slab, so with its bits; v positions and floors are carried from plane to
// plane.  CHECK: range checks, any slope; else every voxel is in the grid, and the
// ray is STEEP or DOWN says whether v falls along the walk.  A slab without a v
// crossing is taken as one with rv = 1 (its third voxel has no share).  The
// high column is the one at the slab's far plane: where dv < 1 it need not be
// the low one's neighbour.  ALIGN: the lanes of a warp close their blocks of 32
// slabs together; where the gathers stride along v (x-driven rays without the
// y-fastest copy) lanes in step read one x column of rows 4 nx bytes apart, whose
// sectors share banks, so there each keeps its own phase.
// Bound by issue (82 % with the copy) and the gathers' latency; 256^3, 48 views of
// 512 x 384: forward 3.56 ms with the y-fastest copy (one slab at a time 3.85), 4.19
// without (in step 4.83), transpose 3.98 and 8.02; with the reference's rounding
// 3.86, 4.39, 4.30 and 8.04.
template <bool REF, bool CHECK, bool DOWN, int DIV, bool ALIGN, bool STEEP, class Sink>
__device__ __forceinline__ void ray_slabs(const ColWalk &c, const ZRay &z, const ZGrid &zg, int k, int end, unsigned sw,
                                          Sink &f)
{
    constexpr bool ANY = CHECK || STEEP;
    const Inside vin(c.nv), zin(zg.nz, z.zi);
    float t = __fsub_rn((float)k, c.nu2), da = __fsub_rn(t, c.pu);
    float qa = col_vpos<DIV>(c, da), ma = magic_floor<CHECK>(qa), za = z_at<REF>(z, zg, da);
    unsigned base = (unsigned)k * c.su - (unsigned)kFloorMagicBits * (c.sv + sw) + (unsigned)z.zi * sw;
    auto slab = [&](RaySlab &s) {
        t = __fadd_rn(t, 1.f);
        const float db = __fsub_rn(t, c.pu), qb = col_vpos<DIV>(c, db), mb = magic_floor<CHECK>(qb);
        const float q1 = ANY ? fminf(qa, qb) : DOWN ? qb : qa, q2 = ANY ? fmaxf(qa, qb) : DOWN ? qa : qb;
        const float m1 = ANY ? fminf(ma, mb) : DOWN ? mb : ma, m2 = ANY ? fmaxf(ma, mb) : DOWN ? ma : mb;
        const bool vx = m1 != m2;
        const float rv = col_ratio(q1, q2, m1, m2);
        const float zb = z_at<REF>(z, zg, db), zl = z.down ? zb : za, zh = z.down ? za : zb;
        float m, mh, r;
        if constexpr (ANY) z_split<REF>(z, zl, zh, m, mh, r);
        else z_share<REF>(z, zl, zh, m, r);
        const unsigned z1 = base + (unsigned)__float_as_int(m) * sw;
        const unsigned up = ANY ? (unsigned)(__float_as_int(mh) - __float_as_int(m)) * sw : sw;
        const unsigned v1 = z1 + (unsigned)__float_as_int(m1) * c.sv, v2 = z1 + (unsigned)__float_as_int(m2) * c.sv;
        const bool vfirst = rv > r;             // the middle voxel is (v1, z2), else (v2, z1)
        const float both = fminf(rv, r), over = __fsub_rn(r, both);      // r's share in the high column
        s.p[0] = v1;
        s.p[1] = vfirst ? v1 + up : v2;
        s.p[2] = v2 + up;
        s.w[0] = both;
        s.w[1] = fabsf(__fsub_rn(rv, r));
        s.w[2] = __fsub_rn(__fsub_rn(1.f, rv), over);
        s.vx = vx;
        if constexpr (CHECK) {
            const bool a = vin.low(m1), b = vx && vin.far(m1, m2), l = zin.low(m), h = zin.far(m, mh);
            f.edge(!vx ? kPlain : a && b ? kCross : kHalf, s.p,
                   (unsigned)(a && l) | (unsigned)(vfirst ? a && h : b && l) << 1 | (unsigned)(b && h) << 2, s.w);
        }
        base += c.su;
        da = db;
        qa = qb;
        ma = mb;
        za = zb;
    };
    RaySlab one[1];
    auto single = [&]() {
        slab(one[0]);
        if constexpr (!CHECK) f.inner(one);
    };
    if constexpr (CHECK) {
#pragma unroll 1
        for (; k <= end; ++k) {
            single();
            if ((k & 31) == 31) f.close();
        }
    } else if constexpr (ALIGN) {
        while (k <= end) {
            const int last = min(k | 31, end);
            if constexpr (Sink::kGather) {
#pragma unroll 2
                for (; k < last; k += 2) {
                    RaySlab s[2];
                    slab(s[0]);
                    slab(s[1]);
                    f.inner(s);
                }
                if (k <= last) { single(); ++k; }
            } else {
#pragma unroll 4
                for (; k <= last; ++k) single();
            }
            if ((last & 31) == 31) f.close();
        }
    } else {
        // a single slab up to an even one, then pairs
        if (k <= end && (k & 1)) {
            single();
            if ((k++ & 31) == 31) f.close();
        }
#pragma unroll 4
        for (; k < end; k += 2) {
            RaySlab s[2];
            slab(s[0]);
            slab(s[1]);
            f.inner(s);
            if ((k & 31) == 30) f.close();
        }
        if (k <= end) {
            single();
            if ((k & 31) == 31) f.close();
        }
    }
}

// Slabs k..end, all in the grid, of a ray that is not steep.
template <bool REF, bool ALIGN, class Sink>
__device__ __forceinline__ void ray_inner(const ColWalk &c, const ZRay &z, const ZGrid &zg, int k, int end,
                                             unsigned sw, Sink &f)
{
    if (c.vdiv) {
        if (c.kv < 0.f) ray_slabs<REF, false, true, 1, ALIGN, false>(c, z, zg, k, end, sw, f);
        else ray_slabs<REF, false, false, 1, ALIGN, false>(c, z, zg, k, end, sw, f);
    } else {
        if (c.kv < 0.f) ray_slabs<REF, false, true, 0, ALIGN, false>(c, z, zg, k, end, sw, f);
        else ray_slabs<REF, false, false, 0, ALIGN, false>(c, z, zg, k, end, sw, f);
    }
}
// The thread walk: the slabs k0..k1 of a ray, of them ki0..ki1 without range checks.
template <bool REF, bool COPY, class Sink>
__device__ __forceinline__ void ray_walk(const GridDev<float> &g, const Walk<float> &w, unsigned su, unsigned sv,
                                         unsigned sw, Sink &f)
{
    const ColWalk c = col_walk_of(g, w, su, sv);
    const ZGrid zg = z_grid(g);
    const ZRay z = z_ray<REF>(w, zg, z_source<REF>(w, zg), true);
    const bool interior = w.ki0 <= w.ki1;
    int k = w.k0, end = interior ? w.ki0 - 1 : w.k1;
#pragma unroll 1
    for (;;) {
        ray_slabs<REF, true, false, -1, true, false>(c, z, zg, k, end, sw, f);
        if (end == w.k1) break;
        if (z.steep) ray_slabs<REF, false, false, -1, true, true>(c, z, zg, w.ki0, w.ki1, sw, f);
        else if (!COPY && sv != 1u) ray_inner<REF, COPY>(c, z, zg, w.ki0, w.ki1, sw, f);
        else ray_inner<REF, true>(c, z, zg, w.ki0, w.ki1, sw, f);
        if (w.ki1 == w.k1) break;
        k = w.ki1 + 1;
        end = w.k1;
    }
    f.close();
}

// ---- column warps ----

// Warp's table of one 32-slab chunk, its slabs grouped by kind (slabs without
// a v column in the grid are dropped): rows [0, cross) plain, [cross, half)
// cross, [half, n) half.  a = (address of the low v column -- of the one
// column in the grid for a half slab -- less one element per floor bias,
// offsets of the lower and the upper z plane), c = (address of the high v column, or
// 1 in c.x when a half slab's column is the high one; rv; 1 - rv).  d: the
// offsets of the slab's entry and exit planes.
// base, z0, z1: the volume's address, from the row on that the rays' z positions
// count from, less one element per floor bias, and the biased floors of its
// first row and of the one past its last (here, not in registers).
struct ColTable {
    uint4 a[32], c[32];
    float2 d[32];
    unsigned long long base;
    float z0, z1;
};

// Column warps are blocks of 32 x (at most 8) threads: one table per warp.
__device__ __forceinline__ ColTable &col_table()
{
    __shared__ ColTable tables[8];
    return tables[threadIdx.y];
}

// A column's walk for one warp: the shared v part, the R rays of the lane and
// the warp's slab ranges.
template <int R> struct ColRays {
    ColWalk c;
    ZGrid zg;
    ZRay z[R];
    float W[R];
    int K0, K1;                     // slabs that some ray of the warp can touch
    int ZI0, ZI1;                   // slabs where no ray of the warp needs a z range check
    bool rising, falling, steep;    // the warp has rays of this kind
};

// Rays r (the whole warp calls it; has: the lane has the ray and it takes
// part); false when no ray of the warp contributes.  UPPER: slabs without range
// checks touch a low voxel's upper neighbour whether it has a share or not (the
// forward's loads; the transpose's reductions skip it).
template <int R, bool REF, bool UPPER>
__device__ __forceinline__ bool col_rays(const GridDev<float> &g, const float (&r)[R][6], const bool (&has)[R],
                                         uint32_t flags, ColRays<R> &q)
{
    int k0 = INT_MAX, k1 = INT_MIN, zi0 = INT_MIN, zi1 = INT_MAX;
    bool any = false, up = false, down = false, steep = false;
    ZSource source;
    q.zg = z_grid(g);
#pragma unroll
    for (int i = 0; i < R; ++i) {
        Walk<float> w;
        const bool live = setup_walk(g, r[i], flags, w) && has[i];
        if (i == 0) {
            // x and y do not depend on the row: every lane has the same v part
            const unsigned xs = (unsigned)g.nz, ys = (unsigned)g.nx * (unsigned)g.nz;
            q.c = col_walk_of(g, w, w.xdrive ? xs : ys, w.xdrive ? ys : xs);
            source = z_source<REF>(w, q.zg);
        }
        q.z[i] = z_ray<REF>(w, q.zg, source, live);
        q.W[i] = w.W;
        if (live) {
            any = true;
            k0 = min(k0, w.k0);
            k1 = max(k1, w.k1);
            zi0 = max(zi0, UPPER ? w.zu0 : w.zi0);
            zi1 = min(zi1, UPPER ? w.zu1 : w.zi1);
            up = up || !q.z[i].down;
            down = down || q.z[i].down;
            steep = steep || q.z[i].steep;
        }
    }
    if (!__any_sync(0xffffffffu, any)) return false;
    q.K0 = __reduce_min_sync(0xffffffffu, k0);
    q.K1 = __reduce_max_sync(0xffffffffu, k1);
    q.ZI0 = __reduce_max_sync(0xffffffffu, zi0);
    q.ZI1 = __reduce_min_sync(0xffffffffu, zi1);
    q.rising = __any_sync(0xffffffffu, up);
    q.falling = __any_sync(0xffffffffu, down);
    q.steep = __any_sync(0xffffffffu, steep);
    return true;
}

struct ColChunk {
    int cross, half, n;
};

// The table's view-wide part (before the first chunk; whole warps come from
// collectives, so the last walk's reads are done).
template <typename T>
__device__ __forceinline__ void col_table_start(ColTable &tab, const T *vol, int zi, int nz)
{
    if ((threadIdx.x & 31) == 0) {
        tab.base = (unsigned long long)(vol + zi) - sizeof(T) * (unsigned)kFloorMagicBits;
        tab.z0 = kFloorMagic - (float)zi;
        tab.z1 = kFloorMagic + (float)(nz - zi);
    }
}

// Lane j evaluates slab kc + j, if it is one of K0..K1.  T: the volume's elements.
template <typename T>
__device__ __forceinline__ ColChunk col_chunk(const ColWalk &cw, int kc, int K0, int K1, bool falling, ColTable &tab)
{
    const int lane = threadIdx.x & 31, k = kc + lane;
    const ColEntry e = col_entry(cw, k);
    const float da = col_plane(cw, k), db = col_plane(cw, k + 1);
    const bool vx = e.vx;
    const unsigned in = k >= K0 && k <= K1 ? e.in : 0u;
    const bool is_plain = !vx && in != 0u, is_cross = vx && in == 3u, is_half = vx && (in == 1u || in == 2u);
    const unsigned plain = __ballot_sync(0xffffffffu, is_plain), cross = __ballot_sync(0xffffffffu, is_cross);
    const unsigned half = __ballot_sync(0xffffffffu, is_half), below = (1u << lane) - 1u;
    ColChunk h;
    h.cross = __popc(plain);
    h.half = h.cross + __popc(cross);
    h.n = h.half + __popc(half);
    const int row = is_plain ? __popc(plain & below) : is_cross ? h.cross + __popc(cross & below)
                                                                 : h.half + __popc(half & below);
    __syncwarp();                       // the previous chunk's reads are done
    if (is_plain || is_cross || is_half) {
        const unsigned long long base = tab.base;
        const unsigned i1 = is_half && in == 2u ? e.b2 : e.b1;
        const unsigned long long p1 = base + sizeof(T) * (i1 + (unsigned)kFloorMagicBits);
        const unsigned long long p2 = base + sizeof(T) * (e.b2 + (unsigned)kFloorMagicBits);
        tab.a[row] = make_uint4((unsigned)p1, (unsigned)(p1 >> 32), __float_as_uint(falling ? db : da),
                                __float_as_uint(falling ? da : db));
        tab.c[row] = make_uint4(is_half ? in - 1u : (unsigned)p2, (unsigned)(p2 >> 32), __float_as_uint(e.rv),
                                __float_as_uint(__fsub_rn(1.f, e.rv)));
        tab.d[row] = make_float2(da, db);
    }
    __syncwarp();
    return h;
}

// Voxel of biased floor m in the column at the table's address (lo, hi).
template <typename T = float> __device__ __forceinline__ T *col_voxel(unsigned lo, unsigned hi, float m)
{
    return reinterpret_cast<T *>(((unsigned long long)hi << 32 | lo) + sizeof(T) * (unsigned)__float_as_int(m));
}

// The transpose's accumulators: floats, or 64-bit integers of yw * share times
// a power of two (exact), rounded (the deterministic transpose: integer sums
// do not depend on the order of the reductions).  red() reduces v != 0 without
// returning the old value (the address is global: a plain atomicAdd on an
// address rebuilt from integers compiles to a generic atomic, half as fast).
struct FloatAcc {
    using T = float;
    float *vol;
    __device__ __forceinline__ float value(float v) const { return v; }
    // y times the share 1 - r, rounded once
    __device__ __forceinline__ float rest(float y, float r) const { return __fmaf_rn(-y, r, y); }
    static __device__ __forceinline__ void red(float *p, float v)
    {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.neu.f32 p, %1, 0f00000000;\n\t@p red.global.add.f32 [%0], %1;\n\t}" ::"l"(p),
                     "f"(v)
                     : "memory");
    }
};
struct FixedAcc {
    using T = long long;
    unsigned long long *vol;
    float scale;
    __device__ __forceinline__ long long value(float v) const { return to_fixed(v * scale); }
    __device__ __forceinline__ long long rest(float y, float r) const { return value(y * __fsub_rn(1.f, r)); }
    static __device__ __forceinline__ void red(long long *p, long long v)
    {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s64 p, %1, 0;\n\t@p red.global.add.u64 [%0], %1;\n\t}" ::"l"(p), "l"(v)
                     : "memory");
    }
};

// Plane offsets of ray z at a table row: the warp's, or (MIXED: the warp has
// rising and falling rays) the ray's own.
template <bool MIXED>
__device__ __forceinline__ void col_planes(const ColTable &tab, int j, const uint4 &te, const ZRay &z, float &lo, float &hi)
{
    if (MIXED) {
        const float2 d = tab.d[j];
        lo = z.down ? d.y : d.x;
        hi = z.down ? d.x : d.y;
    } else {
        lo = __uint_as_float(te.z);
        hi = __uint_as_float(te.w);
    }
}

// z split of ray z at a table row (z_split; only STEEP warps have steep rays,
// the others' high voxel is the low one's upper neighbour: no mh).
template <bool REF, bool MIXED, bool STEEP>
__device__ __forceinline__ void col_split(const ColTable &tab, int j, const uint4 &te, const ZRay &z, const ZGrid &zg,
                                          float &m, float &mh, float &r)
{
    float lo, hi;
    col_planes<MIXED>(tab, j, te, z, lo, hi);
    if constexpr (STEEP) z_split<REF>(z, z_at<REF>(z, zg, lo), z_at<REF>(z, zg, hi), m, mh, r);
    else z_inner<REF>(z, zg, lo, hi, m, r);
}

// Forward of one chunk's table rows.  Each kind of slab is walked in a loop of
// its own: no branch stands between the loads of consecutive slabs, so they
// overlap.  ZCHK: z range checks.
template <int R, bool REF, bool MIXED, bool STEEP, bool ZCHK>
__device__ __forceinline__ void col_gather_rows(const ColRays<R> &q, const ColTable &tab, const ColChunk &h,
                                                GatherSink (&f)[R])
{
    const Inside in = REF ? Inside(q.zg.nz) : ZCHK ? Inside(tab.z0, tab.z1) : Inside(0);
    auto load = [&](unsigned lo, unsigned hi, float m, float mh, float &a, float &b) {
        const float *const p = col_voxel(lo, hi, m);
        a = !ZCHK || in.low(m) ? __ldg(p) : 0.f;
        if constexpr (STEEP) b = !ZCHK || in.far(m, mh) ? __ldg(col_voxel(lo, hi, mh)) : 0.f;
        else b = !ZCHK || in.high(m) ? __ldg(p + 1) : 0.f;
    };
#pragma unroll 4
    for (int j = 0; j < h.cross; ++j) {
        const uint4 te = tab.a[j];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            float m, mh, r, a, b;
            col_split<REF, MIXED, STEEP>(tab, j, te, q.z[i], q.zg, m, mh, r);
            load(te.x, te.y, m, mh, a, b);
            f[i].sum[0] = __fmaf_rn(b, __fsub_rn(1.f, r), __fmaf_rn(a, r, f[i].sum[0]));
        }
    }
#pragma unroll 2
    for (int j = h.cross; j < h.half; ++j) {
        const uint4 te = tab.a[j], tc = tab.c[j];
        const float rv = __uint_as_float(tc.z), ov = __uint_as_float(tc.w);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            float m, mh, r, a, b, c, d;
            col_split<REF, MIXED, STEEP>(tab, j, te, q.z[i], q.zg, m, mh, r);
            load(te.x, te.y, m, mh, a, b);
            load(tc.x, tc.y, m, mh, c, d);
            const float w11 = fminf(rv, r), w21 = __fsub_rn(r, w11);
            const float acc = __fmaf_rn(b, __fsub_rn(rv, w11), __fmaf_rn(a, w11, f[i].sum[1]));
            f[i].sum[1] = __fmaf_rn(d, __fsub_rn(ov, w21), __fmaf_rn(c, w21, acc));
        }
    }
#pragma unroll 1
    for (int j = h.half; j < h.n; ++j) {
        const uint4 te = tab.a[j], tc = tab.c[j];
        const float rv = __uint_as_float(tc.z), ov = __uint_as_float(tc.w);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            float m, mh, r, a, b;
            col_split<REF, MIXED, STEEP>(tab, j, te, q.z[i], q.zg, m, mh, r);
            load(te.x, te.y, m, mh, a, b);
            const float w11 = fminf(rv, r), w21 = __fsub_rn(r, w11);
            const float wl = tc.x ? w21 : w11, wh = tc.x ? __fsub_rn(ov, w21) : __fsub_rn(rv, w11);
            f[i].sum[2] = __fmaf_rn(b, wh, __fmaf_rn(a, wl, f[i].sum[2]));
        }
    }
}

// Forward of the lane's R rays: sums into f.
template <int R, bool REF, bool MIXED, bool STEEP>
__device__ __forceinline__ void col_gather(const ColRays<R> &q, const float *__restrict__ vol, GatherSink (&f)[R])
{
    ColTable &tab = col_table();
    col_table_start(tab, vol, q.z[0].zi, q.zg.nz);
    for (int kc = q.K0 & ~31; kc <= q.K1; kc += 32) {
        const ColChunk h = col_chunk<float>(q.c, kc, q.K0, q.K1, q.falling, tab);
        if (max(kc, q.K0) >= q.ZI0 && min(kc + 31, q.K1) <= q.ZI1)
            col_gather_rows<R, REF, MIXED, STEEP, false>(q, tab, h, f);
        else
            col_gather_rows<R, REF, MIXED, STEEP, true>(q, tab, h, f);
#pragma unroll
        for (int i = 0; i < R; ++i) f[i].close();
    }
}

// How the transpose's R rays of a lane share reductions: not at all; as
// neighbours, in z order and all within less than a voxel of the first one in
// every slab; as two neighbours at any distance.
enum Merge { kSingle, kNear, kAny };

// Transpose of one chunk's table rows.  Neighbouring rays' shares of a voxel
// column are summed in registers over the voxels w, w + 1, w + 2 of the first
// one's low voxel w, so a slab takes at most three reductions per column
// instead of two per ray, and the lanes of a warp, R rows apart, rarely hit
// the same voxel.
// STEEP rays do not merge.
template <int R, bool REF, bool MIXED, bool STEEP, Merge MERGE, bool ZCHK, class Acc>
__device__ __forceinline__ void col_scatter_rows(const ColRays<R> &q, const ColTable &tab, const ColChunk &h,
                                                 const Acc &acc, const float (&y)[R])
{
    using T = typename Acc::T;
    const Inside in = REF ? Inside(q.zg.nz) : ZCHK ? Inside(tab.z0, tab.z1) : Inside(0);
    // values l, u of the low and high voxels of rays i.. in one voxel column
    constexpr int S = MERGE == kSingle ? 1 : R;
    static_assert(!STEEP || MERGE == kSingle, "");
    auto reduce = [&](unsigned lo, unsigned hi, const float (&m)[S], const float (&mh)[S], T (&l)[S], T (&u)[S]) {
        if (ZCHK) {
#pragma unroll
            for (int k = 0; k < S; ++k) {
                if (!in.low(m[k])) l[k] = (T)0;
                if (STEEP ? !in.far(m[k], mh[k]) : !in.high(m[k])) u[k] = (T)0;
            }
        }
        T *const p = col_voxel<T>(lo, hi, m[0]);
        if constexpr (MERGE == kNear) {
            T top = (T)0;
#pragma unroll
            for (int k = 1; k < S; ++k) {
                const bool same = m[0] == m[k];
                l[0] += same ? l[k] : (T)0;
                u[0] += same ? u[k] : l[k];
                top += same ? (T)0 : u[k];
            }
            Acc::red(p + 2, top);
        } else if constexpr (MERGE == kAny) {
            const bool same = m[0] == m[1], next = m[1] == m[0] + 1.f;
            T *const s = col_voxel<T>(lo, hi, m[1]);
            l[0] += same ? l[1] : (T)0;
            u[0] += same ? u[1] : next ? l[1] : (T)0;
            Acc::red(s, same || next ? (T)0 : l[1]);
            Acc::red(s + 1, same ? (T)0 : u[1]);
        }
        Acc::red(p, l[0]);
        Acc::red(STEEP ? col_voxel<T>(lo, hi, mh[0]) : p + 1, u[0]);
    };
#pragma unroll 1
    for (int j = h.cross; j < h.n; ++j) {
        const uint4 te = tab.a[j], tc = tab.c[j];
        const float rv = __uint_as_float(tc.z), ov = __uint_as_float(tc.w);
#pragma unroll
        for (int i = 0; i < R; i += S) {
            float m[S], mh[S];
            T l1[S], u1[S], l2[S], u2[S];
#pragma unroll
            for (int k = 0; k < S; ++k) {
                float r;
                col_split<REF, MIXED, STEEP>(tab, j, te, q.z[i + k], q.zg, m[k], mh[k], r);
                const float w11 = fminf(rv, r), w21 = __fsub_rn(r, w11), yk = y[i + k];
                l1[k] = acc.value(yk * w11);
                u1[k] = acc.value(yk * __fsub_rn(rv, w11));
                l2[k] = acc.value(yk * w21);
                u2[k] = acc.value(yk * __fsub_rn(ov, w21));
            }
            if (j < h.half) {
                reduce(te.x, te.y, m, mh, l1, u1);
                reduce(tc.x, tc.y, m, mh, l2, u2);
            } else if (tc.x == 0u) {
                reduce(te.x, te.y, m, mh, l1, u1);
            } else {
                reduce(te.x, te.y, m, mh, l2, u2);
            }
        }
    }
#pragma unroll 2
    for (int j = 0; j < h.cross; ++j) {
        const uint4 te = tab.a[j];
#pragma unroll
        for (int i = 0; i < R; i += S) {
            float m[S], mh[S];
            T l[S], u[S];
#pragma unroll
            for (int k = 0; k < S; ++k) {
                float r;
                col_split<REF, MIXED, STEEP>(tab, j, te, q.z[i + k], q.zg, m[k], mh[k], r);
                l[k] = acc.value(y[i + k] * r);
                u[k] = acc.rest(y[i + k], r);
            }
            reduce(te.x, te.y, m, mh, l, u);
        }
    }
}

// Transpose of the lane's R rays (y finite, 0 for a ray that takes no part).
template <int R, bool REF, bool MIXED, bool STEEP, Merge MERGE, class Acc>
__device__ __forceinline__ void col_scatter(const ColRays<R> &q, const Acc &acc, const float (&y)[R])
{
    ColTable &tab = col_table();
    col_table_start(tab, acc.vol, q.z[0].zi, q.zg.nz);
    for (int kc = q.K0 & ~31; kc <= q.K1; kc += 32) {
        const ColChunk h = col_chunk<typename Acc::T>(q.c, kc, q.K0, q.K1, q.falling, tab);
        if (max(kc, q.K0) >= q.ZI0 && min(kc + 31, q.K1) <= q.ZI1)
            col_scatter_rows<R, REF, MIXED, STEEP, MERGE, false>(q, tab, h, acc, y);
        else
            col_scatter_rows<R, REF, MIXED, STEEP, MERGE, true>(q, tab, h, acc, y);
    }
}

}  // namespace nefct
