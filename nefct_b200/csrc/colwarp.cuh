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
//    multiply-add, a floor and one saturating multiply-add per ray and slab,
//    with fewer roundings than the reference's (the error against FP64 is no
//    larger), the same in the forward and its transpose.
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

// v part of one slab: biased bases of the low/high v voxel columns (index of
// (k, v, z) = b + sw * floor bits of z), the clamped v floors for the
// boundary checks, and the v crossing ratio.
struct ColEntry {
    unsigned b1, b2;    // k*su + c*sv - sw*0x4B400000 for the low/high v floor c
    unsigned cv;        // (c1 + 2) | (c2 + 2) << 16, c clamped to [-2, nv + 1]
    float rv;           // crossing ratio, 1 without a v crossing
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

// Entry of slab k: planes t = k - nu2 and t + 1, positions and floors in the
// reference's operations and order.  Clamping a floor to [-2, nv + 1] keeps
// every admission decision of the boundary checks.  sw: z stride.
__device__ __forceinline__ ColEntry col_entry(const ColWalk &c, int k, unsigned sw)
{
    auto vpos = [&](float d) {
        float q = __fadd_rn(c.pv, __fmul_rn(c.kv, d));
        if (c.vdiv) q = __fdiv_rn(q, c.dv);
        return __fadd_rn(q, c.nv2);
    };
    const float qa = vpos(col_plane(c, k)), qb = vpos(col_plane(c, k + 1));
    const float ma = magic_floor<true>(qa), mb = magic_floor<true>(qb);
    const float q1 = fminf(qa, qb), q2 = fmaxf(qa, qb);
    const float m1 = fminf(ma, mb), m2 = fmaxf(ma, mb);
    ColEntry e;
    e.rv = m1 != m2 ? FP<float>::ratio(__fadd_rn(__fadd_rn(m2, -kFloorMagic), -q1), __fadd_rn(q2, -q1)) : 1.f;
    const int c1 = min(max(__float_as_int(m1) - kFloorMagicBits, -2), c.nv + 1);
    const int c2 = min(max(__float_as_int(m2) - kFloorMagicBits, -2), c.nv + 1);
    const unsigned base = (unsigned)k * c.su - (unsigned)kFloorMagicBits * sw;
    e.b1 = base + (unsigned)c1 * c.sv;
    e.b2 = base + (unsigned)c2 * c.sv;
    e.cv = (unsigned)(c1 + 2) | ((unsigned)(c2 + 2) << 16);
    return e;
}

// z part of a ray, in voxel rows.
struct ZRay {
    float kz, z0, ikz;      // position kz * d + z0 at plane offset d; ikz = 1 / |kz| (at most 1e30)
    float kw, pw;           // REF: position ((pw + kw * d) * rdz) + nz2
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

// (a lane without a ray walks row 0 under either rounding: its indices stay in
// the grid)
__device__ __forceinline__ ZRay z_ray(const Walk<float> &w, const ZGrid &zg, bool live)
{
    ZRay z;
    z.live = live;
    z.kz = live ? w.kz : 0.f;
    z.z0 = live ? w.z0 : 0.5f;
    z.kw = live ? w.kw : 0.f;
    z.pw = live ? w.pw : __fmul_rn(__fsub_rn(0.5f, zg.nz2), zg.dz);
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

// The z split of one slab: biased floors of its low and high voxel and the
// share rw of the low one.  d, dh: offsets of the lower and upper plane.
struct ZSplit {
    unsigned i1, i2;
    float rw;
};

// z split of a slab of a ray that is not steep: biased floor and low share.
// (The grid has at most 2^20 rows and slabs, and such a ray moves at most one
// row per slab: positions stay below 2^22, no clamp is needed for the floor.)
template <bool REF>
__device__ __forceinline__ void z_inner(const ZRay &z, const ZGrid &zg, float lo, float hi, float &m, float &r)
{
    const float q = REF ? z_pos(z, zg, lo) : __fmaf_rn(z.kz, lo, z.z0);
    m = __fadd_rd(q, kFloorMagic);
    if (REF) {
        const float c = __fadd_rn(m, 1.f - kFloorMagic);
        r = __saturatef(__fmul_rn(__fadd_rn(c, -q), rcp_approx(__fadd_rn(z_pos(z, zg, hi), -q))));
    } else {
        r = __saturatef(__fmaf_rn(__fadd_rn(__fadd_rn(m, -kFloorMagic), -q), z.ikz, z.ikz));
    }
}

template <bool REF>
__device__ __forceinline__ ZSplit z_split(const ZRay &z, const ZGrid &zg, float d, float dh)
{
    ZSplit s;
    float m;
    if (!z.steep) {
        z_inner<REF>(z, zg, d, dh, m, s.rw);
        s.i1 = (unsigned)__float_as_int(m);
        s.i2 = s.i1 + 1u;
        return s;
    }
    float q = REF ? z_pos(z, zg, d) : __fmaf_rn(z.kz, d, z.z0);
    float qh = REF ? z_pos(z, zg, dh) : __fmaf_rn(z.kz, dh, z.z0);
    m = magic_floor<true>(q);
    const float mh = magic_floor<true>(qh);
    q = fminf(fmaxf(q, -kFloorClamp), kFloorClamp);
    qh = fminf(fmaxf(qh, -kFloorClamp), kFloorClamp);
    const float iden = REF ? rcp_approx(__fadd_rn(qh, -q)) : z.ikz;
    s.rw = mh != m ? __fmul_rn(__fadd_rn(__fadd_rn(mh, -kFloorMagic), -q), iden) : 1.f;
    s.i1 = (unsigned)__float_as_int(m);
    s.i2 = (unsigned)__float_as_int(mh);
    return s;
}

// Shares of a slab with a v crossing: the overlap of the ray's v intervals
// [0, rv], [rv, 1] and z intervals [0, rw], [rw, 1] (the reference's pairing,
// Q1): (v1, w1), (v1, w2), (v2, w1), (v2, w2); one of the middle two is 0.
struct Shares {
    float w11, w12, w21, w22;
};
__device__ __forceinline__ Shares slab_shares(float rv, float rw)
{
    Shares s;
    s.w11 = fminf(rv, rw);
    s.w12 = __fsub_rn(rv, s.w11);
    s.w21 = __fsub_rn(rw, s.w11);
    s.w22 = __fsub_rn(__fsub_rn(1.f, rv), s.w21);
    return s;
}

// Which of a slab's v columns are in the grid (bits v1, v2), with the
// reference's slab admission (siddon.cu.cc:80, :92, :112, :116, :132).
__device__ __forceinline__ unsigned v_columns(bool vx, unsigned cv, int nv)
{
    const int cv1 = (int)(cv & 0xffffu) - 2, cv2 = (int)(cv >> 16) - 2;
    const bool adm = (unsigned)(cv1 + (int)vx) < (unsigned)(nv + (int)vx);
    return (unsigned)(adm && cv1 >= 0) | (unsigned)(adm && cv2 < nv) << 1;
}

// Which of a slab's voxels are in the grid: bits v1w1, v1w2, v2w1, v2w2.
__device__ __forceinline__ unsigned slab_inside(const ZRay &z, const ZSplit &s, bool vx, unsigned cv, int nv, int nz)
{
    const int cw1 = (int)s.i1 - kFloorMagicBits, cw2 = (int)s.i2 - kFloorMagicBits;
    bool adm = z.live;
    if (z.steep) {
        const bool wx = s.i1 != s.i2;
        adm = adm && (unsigned)(cw1 + (int)wx) < (unsigned)(nz + (int)wx);
    }
    const unsigned w = (unsigned)(adm && (unsigned)cw1 < (unsigned)nz) | (unsigned)(adm && (unsigned)cw2 < (unsigned)nz) << 1;
    const unsigned v = v_columns(vx, cv, nv);
    return (v & 1u ? w : 0u) | (v & 2u ? w << 2 : 0u);
}

// ---- sinks: what one ray does with a slab's voxels ----
//
// f.pair(kind, b, s, ok, wl, wh): voxels (v, w1) with share wl and (v, w2)
// with share wh of the voxel column at b; ok: bit 0 and 1, whether they are in
// the grid.

// Slabs without a v crossing; with one and both columns in the grid; with one
// and a single column in the grid.
enum SlabKind { kPlain, kCross, kHalf };

// Forward: sums of value * share, by kind of slab and by aligned block of 32
// slabs (close() ends a block), so that the total does not depend on which
// rays walk together; sums of partial sums also round less than one running
// sum.  SKIP0: voxels of share 0 are not read.
template <bool SKIP0 = false> struct GatherSink {
    const float *__restrict__ vol;
    unsigned sw;
    float sum[3], whole;

    __device__ __forceinline__ GatherSink() {}
    __device__ __forceinline__ GatherSink(const float *v, unsigned sw_) : vol(v), sw(sw_), sum{0.f, 0.f, 0.f}, whole(0.f) {}
    __device__ __forceinline__ void pair(SlabKind kind, unsigned b, const ZSplit &s, unsigned ok, float wl, float wh)
    {
        const float lo = (ok & 1u) && (!SKIP0 || wl != 0.f) ? __ldg(vol + (b + s.i1 * sw)) : 0.f;
        const float hi = (ok & 2u) && (!SKIP0 || wh != 0.f) ? __ldg(vol + (b + s.i2 * sw)) : 0.f;
        const float acc = kind == kPlain ? sum[0] : kind == kCross ? sum[1] : sum[2];
        const float v = __fmaf_rn(hi, wh, __fmaf_rn(lo, wl, acc));
        if (kind == kPlain) sum[0] = v;
        else if (kind == kCross) sum[1] = v;
        else sum[2] = v;
    }
    // Interior slab: voxels p0, pm and p2 with their shares (of the last two,
    // those without a share, most of them, are not read).
    __device__ __forceinline__ void inner(bool vx, unsigned p0, unsigned pm, unsigned p2, float w0, float wm, float w2)
    {
        const float v0 = __ldg(vol + p0);
        const float vm = wm != 0.f ? __ldg(vol + pm) : 0.f;
        const float v2 = w2 != 0.f ? __ldg(vol + p2) : 0.f;
        const float v = __fmaf_rn(v2, w2, __fmaf_rn(vm, wm, __fmaf_rn(v0, w0, vx ? sum[1] : sum[0])));
        if (vx) sum[1] = v;
        else sum[0] = v;
    }
    __device__ __forceinline__ void close()
    {
        whole = __fadd_rn(whole, __fadd_rn(__fadd_rn(sum[0], sum[1]), sum[2]));
        sum[0] = sum[1] = sum[2] = 0.f;
    }
};

// Transpose: one reduction of yw * share per voxel with a share.
struct ScatterSink {
    float *acc;
    unsigned sw;
    float yw;

    __device__ __forceinline__ void pair(SlabKind, unsigned b, const ZSplit &s, unsigned ok, float wl, float wh) const
    {
        if ((ok & 1u) && wl != 0.f) atomicAdd(acc + (b + s.i1 * sw), yw * wl);
        if ((ok & 2u) && wh != 0.f) atomicAdd(acc + (b + s.i2 * sw), yw * wh);
    }
    __device__ __forceinline__ void inner(bool, unsigned p0, unsigned pm, unsigned p2, float w0, float wm, float w2) const
    {
        if (w0 != 0.f) atomicAdd(acc + p0, yw * w0);
        if (wm != 0.f) atomicAdd(acc + pm, yw * wm);
        if (w2 != 0.f) atomicAdd(acc + p2, yw * w2);
    }
    __device__ __forceinline__ void close() const {}
};

// Deterministic transpose: each contribution yw * share, scaled by a power of
// two (exact) and rounded to a 64-bit integer (siddon.cuh, to_fixed).
struct FixedSink {
    unsigned long long *acc;
    unsigned sw;
    float yw, scale;

    __device__ __forceinline__ void pair(SlabKind, unsigned b, const ZSplit &s, unsigned ok, float wl, float wh) const
    {
        if ((ok & 1u) && wl != 0.f) atomicAdd(acc + (b + s.i1 * sw), (unsigned long long)to_fixed((yw * wl) * scale));
        if ((ok & 2u) && wh != 0.f) atomicAdd(acc + (b + s.i2 * sw), (unsigned long long)to_fixed((yw * wh) * scale));
    }
    __device__ __forceinline__ void inner(bool, unsigned p0, unsigned pm, unsigned p2, float w0, float wm, float w2) const
    {
        if (w0 != 0.f) atomicAdd(acc + p0, (unsigned long long)to_fixed((yw * w0) * scale));
        if (wm != 0.f) atomicAdd(acc + pm, (unsigned long long)to_fixed((yw * wm) * scale));
        if (w2 != 0.f) atomicAdd(acc + p2, (unsigned long long)to_fixed((yw * w2) * scale));
    }
    __device__ __forceinline__ void close() const {}
};

// One slab of one ray, range checked (also right for interior slabs).
template <bool REF, class Sink>
__device__ __forceinline__ void ray_slab(const ZRay &z, const ZGrid &zg, float d, float dh, unsigned b1, unsigned b2,
                                         float rv, unsigned cv, int nv, Sink &f)
{
    const ZSplit s = z_split<REF>(z, zg, d, dh);
    const bool four = b1 != b2;
    const unsigned ok = slab_inside(z, s, four, cv, nv, zg.nz);
    if (!four) {
        f.pair(kPlain, b1, s, ok, s.rw, __fsub_rn(1.f, s.rw));
    } else {
        const Shares h = slab_shares(rv, s.rw);
        const SlabKind kind = v_columns(true, cv, nv) == 3u ? kCross : kHalf;
        if (ok & 3u) f.pair(kind, b1, s, ok, h.w11, h.w12);
        if (ok & 12u) f.pair(kind, b2, s, ok >> 2, h.w21, h.w22);
    }
}

// Slabs k..end of one ray alone (any strides): every slab's v part evaluated by
// the thread, with a column warp's operations per slab, so with its bits.
template <bool REF, class Sink>
__device__ __forceinline__ void ray_each(const ColWalk &c, const ZRay &z, const ZGrid &zg, unsigned sw, Sink &f, int k,
                                         int end)
{
#pragma unroll 1
    for (; k <= end; ++k) {
        const ColEntry e = col_entry(c, k, sw);
        const float a = col_plane(c, k), b = col_plane(c, k + 1);
        ray_slab<REF>(z, zg, z.down ? b : a, z.down ? a : b, e.b1, e.b2, e.rv, e.cv, c.nv, f);
        if ((k & 31) == 31) f.close();
    }
}

// The thread walk's interior slabs (ki0..ki1): no range checks, v positions and
// floors carried from plane to plane, a slab without a v crossing taken as one
// with rv = 1 (its third voxel has no share).  DOWN: v falls along the walk.
// Bound by issue and the gathers' latency; 256^3, 72 views of 512 x 384: forward
// 6.2 ms with the y-fastest copy and 7.5 without, transpose 6.6 and 12.3 (every
// slab range checked and evaluated anew: 17.0, 17.5, 15.2 and 15.1; the walk that
// evaluates the z position as the reference does, and sums in one pass: 5.6,
// 6.5, 8.1 and 12.1, with other bits than the column warps).
template <bool REF, bool DOWN, class Sink>
__device__ __forceinline__ void ray_inner(const ColWalk &c, const ZRay &z, const ZGrid &zg, int k, int end, unsigned sw,
                                          Sink &f)
{
    auto vpos = [&](float d) {
        float q = __fadd_rn(c.pv, __fmul_rn(c.kv, d));
        if (c.vdiv) q = __fdiv_rn(q, c.dv);
        return __fadd_rn(q, c.nv2);
    };
    float t = __fsub_rn((float)k, c.nu2), da = __fsub_rn(t, c.pu);
    float qa = vpos(da), ma = magic_floor<false>(qa);
    unsigned base = (unsigned)k * c.su - (unsigned)kFloorMagicBits * (c.sv + sw);
    while (k <= end) {
        const int last = min(k | 31, end);
#pragma unroll 4
        for (; k <= last; ++k) {
            t = __fadd_rn(t, 1.f);
            const float db = __fsub_rn(t, c.pu), qb = vpos(db), mb = magic_floor<false>(qb);
            const float q1 = DOWN ? qb : qa, q2 = DOWN ? qa : qb, m1 = DOWN ? mb : ma, m2 = DOWN ? ma : mb;
            const bool vx = m1 != m2;
            const float rv = vx ? FP<float>::ratio(__fadd_rn(__fadd_rn(m2, -kFloorMagic), -q1), __fadd_rn(q2, -q1)) : 1.f;
            float m, r;
            z_inner<REF>(z, zg, z.down ? db : da, z.down ? da : db, m, r);
            const float both = fminf(rv, r), over = __fsub_rn(r, both);      // r's share in the high column
            // (the high column is the one at the slab's far plane: where dv < 1 it
            // need not be the low one's neighbour)
            const unsigned row = base + (unsigned)__float_as_int(m) * sw;
            const unsigned p0 = row + (unsigned)__float_as_int(m1) * c.sv, ph = row + (unsigned)__float_as_int(m2) * c.sv;
            f.inner(vx, p0, rv > r ? p0 + sw : ph, ph + sw, both, fabsf(__fsub_rn(rv, r)),
                    __fsub_rn(__fsub_rn(1.f, rv), over));
            base += c.su;
            da = db;
            qa = qb;
            ma = mb;
        }
        if ((last & 31) == 31) f.close();
    }
}

// The thread walk.
template <bool REF, class Sink>
__device__ __forceinline__ void ray_walk(const GridDev<float> &g, const Walk<float> &w, unsigned su, unsigned sv,
                                         unsigned sw, Sink &f)
{
    const ColWalk c = col_walk_of(g, w, su, sv);
    const ZGrid zg = z_grid(g);
    const ZRay z = z_ray(w, zg, true);
    const bool interior = !z.steep && w.ki0 <= w.ki1;
    ray_each<REF>(c, z, zg, sw, f, w.k0, interior ? w.ki0 - 1 : w.k1);
    if (interior) {
        if (c.kv < 0.f) ray_inner<REF, true>(c, z, zg, w.ki0, w.ki1, sw, f);
        else ray_inner<REF, false>(c, z, zg, w.ki0, w.ki1, sw, f);
        ray_each<REF>(c, z, zg, sw, f, w.ki1 + 1, w.k1);
    }
    f.close();
}

// ---- column warps ----

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
// part); false when no ray of the warp contributes.
template <int R>
__device__ __forceinline__ bool col_rays(const GridDev<float> &g, const float (&r)[R][6], const bool (&has)[R],
                                         uint32_t flags, ColRays<R> &q)
{
    int k0 = INT_MAX, k1 = INT_MIN, zi0 = INT_MIN, zi1 = INT_MAX;
    bool any = false, up = false, down = false, steep = false;
    q.zg = z_grid(g);
#pragma unroll
    for (int i = 0; i < R; ++i) {
        Walk<float> w;
        const bool live = setup_walk(g, r[i], flags, w) && has[i];
        if (i == 0) {
            // x and y do not depend on the row: every lane has the same v part
            const unsigned xs = (unsigned)g.nz, ys = (unsigned)g.nx * (unsigned)g.nz;
            q.c = col_walk_of(g, w, w.xdrive ? xs : ys, w.xdrive ? ys : xs);
        }
        q.z[i] = z_ray(w, q.zg, live);
        q.W[i] = w.W;
        if (live) {
            any = true;
            k0 = min(k0, w.k0);
            k1 = max(k1, w.k1);
            zi0 = max(zi0, w.zi0);
            zi1 = min(zi1, w.zi1);
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

// Warp's table of one 32-slab chunk, its slabs grouped by kind (slabs without
// a v column in the grid are dropped): rows [0, cross) plain, [cross, half)
// cross, [half, n) half.  a = (address of the low v column -- of the one
// column in the grid for a half slab -- less one element per floor bias,
// offsets of the lower and the upper z plane), c = (address of the high v column, or
// 1 in c.x when a half slab's column is the high one; rv; 1 - rv).  d: the
// offsets of the slab's entry and exit planes.
struct ColTable {
    uint4 a[32], c[32];
    float2 d[32];
};

struct ColChunk {
    int cross, half, n;
};

// Column warps are blocks of 32 x (at most 8) threads: one table per warp.
__device__ __forceinline__ ColTable &col_table()
{
    __shared__ ColTable tables[8];
    return tables[threadIdx.y];
}

// Lane j evaluates slab kc + j, if it is one of K0..K1.  T: the volume's elements.
template <typename T>
__device__ __forceinline__ ColChunk col_chunk(const ColWalk &cw, int kc, int K0, int K1, bool falling, const T *vol,
                                              ColTable &tab)
{
    const int lane = threadIdx.x & 31, k = kc + lane;
    const ColEntry e = col_entry(cw, k, 1u);
    const float da = col_plane(cw, k), db = col_plane(cw, k + 1);
    const bool vx = e.b1 != e.b2;
    const unsigned in = k >= K0 && k <= K1 ? v_columns(vx, e.cv, cw.nv) : 0u;
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
        const char *const base = reinterpret_cast<const char *>(vol) - sizeof(T) * (unsigned)kFloorMagicBits;
        const unsigned i1 = is_half && in == 2u ? e.b2 : e.b1;
        const unsigned long long p1 = (unsigned long long)(base + sizeof(T) * (i1 + (unsigned)kFloorMagicBits));
        const unsigned long long p2 = (unsigned long long)(base + sizeof(T) * (e.b2 + (unsigned)kFloorMagicBits));
        tab.a[row] = make_uint4((unsigned)p1, (unsigned)(p1 >> 32), __float_as_uint(falling ? db : da),
                                __float_as_uint(falling ? da : db));
        tab.c[row] = make_uint4(is_half ? in - 1u : (unsigned)p2, (unsigned)(p2 >> 32), __float_as_uint(e.rv),
                                __float_as_uint(__fsub_rn(1.f, e.rv)));
        tab.d[row] = make_float2(da, db);
    }
    __syncwarp();
    return h;
}

// Every slab of one ray per lane, range checked: warps that the walks below
// do not take (steep rays), and the deterministic transpose.
template <bool REF, class Sink>
__device__ __forceinline__ void col_each(const ColWalk &cw, int K0, int K1, const ZRay &z, const ZGrid &zg, Sink &f)
{
    ColTable &tab = col_table();
    const int lane = threadIdx.x & 31;
    for (int kc = K0 & ~31; kc <= K1; kc += 32) {
        const ColEntry e = col_entry(cw, kc + lane, 1u);
        __syncwarp();
        tab.a[lane] = make_uint4(e.b1, e.b2, __float_as_uint(e.rv), e.cv);
        tab.d[lane] = make_float2(col_plane(cw, kc + lane), col_plane(cw, kc + lane + 1));
        __syncwarp();
        const int n = min(K1 - kc + 1, 32);
#pragma unroll 1
        for (int j = max(K0 - kc, 0); j < n; ++j) {
            const uint4 te = tab.a[j];
            const float2 d = tab.d[j];
            ray_slab<REF>(z, zg, z.down ? d.y : d.x, z.down ? d.x : d.y, te.x, te.y, __uint_as_float(te.z), te.w, cw.nv,
                          f);
        }
        f.close();
    }
}

// Voxel of biased floor m in the column at the table's address (lo, hi).
template <typename T = float> __device__ __forceinline__ T *col_voxel(unsigned lo, unsigned hi, float m)
{
    return reinterpret_cast<T *>(((unsigned long long)hi << 32 | lo) + sizeof(T) * (unsigned)__float_as_int(m));
}

// Whether the voxel of biased floor m, and the one above it, are in the grid.
struct ZInside {
    float lo, hi;           // biased floors 0 and nz
    __device__ __forceinline__ ZInside(int nz) : lo(kFloorMagic), hi(kFloorMagic + (float)nz) {}
    __device__ __forceinline__ bool low(float m) const { return m >= lo && m < hi; }
    __device__ __forceinline__ bool high(float m) const { return m >= lo - 1.f && m < hi - 1.f; }
};

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

// Forward of one chunk's table rows.  Each kind of slab is walked in a loop of
// its own: no branch stands between the loads of consecutive slabs, so they
// overlap.  ZCHK: z range checks.
template <int R, bool REF, bool MIXED, bool ZCHK>
__device__ __forceinline__ void col_gather_rows(const ColRays<R> &q, const ColTable &tab, const ColChunk &h,
                                                GatherSink<> (&f)[R])
{
    const ZInside in(q.zg.nz);
    auto load = [&](const float *p, float m, float &a, float &b) {
        a = !ZCHK || in.low(m) ? __ldg(p) : 0.f;
        b = !ZCHK || in.high(m) ? __ldg(p + 1) : 0.f;
    };
#pragma unroll 4
    for (int j = 0; j < h.cross; ++j) {
        const uint4 te = tab.a[j];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            float lo, hi, m, r, a, b;
            col_planes<MIXED>(tab, j, te, q.z[i], lo, hi);
            z_inner<REF>(q.z[i], q.zg, lo, hi, m, r);
            load(col_voxel(te.x, te.y, m), m, a, b);
            f[i].sum[0] = __fmaf_rn(b, __fsub_rn(1.f, r), __fmaf_rn(a, r, f[i].sum[0]));
        }
    }
#pragma unroll 2
    for (int j = h.cross; j < h.half; ++j) {
        const uint4 te = tab.a[j], tc = tab.c[j];
        const float rv = __uint_as_float(tc.z), ov = __uint_as_float(tc.w);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            float lo, hi, m, r, a, b, c, d;
            col_planes<MIXED>(tab, j, te, q.z[i], lo, hi);
            z_inner<REF>(q.z[i], q.zg, lo, hi, m, r);
            load(col_voxel(te.x, te.y, m), m, a, b);
            load(col_voxel(tc.x, tc.y, m), m, c, d);
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
            float lo, hi, m, r, a, b;
            col_planes<MIXED>(tab, j, te, q.z[i], lo, hi);
            z_inner<REF>(q.z[i], q.zg, lo, hi, m, r);
            load(col_voxel(te.x, te.y, m), m, a, b);
            const float w11 = fminf(rv, r), w21 = __fsub_rn(r, w11);
            const float wl = tc.x ? w21 : w11, wh = tc.x ? __fsub_rn(ov, w21) : __fsub_rn(rv, w11);
            f[i].sum[2] = __fmaf_rn(b, wh, __fmaf_rn(a, wl, f[i].sum[2]));
        }
    }
}

// Forward of the lane's R rays (not steep): sums into f.
template <int R, bool REF, bool MIXED>
__device__ __forceinline__ void col_gather(const ColRays<R> &q, const float *__restrict__ vol, GatherSink<> (&f)[R])
{
    ColTable &tab = col_table();
    for (int kc = q.K0 & ~31; kc <= q.K1; kc += 32) {
        const ColChunk h = col_chunk(q.c, kc, q.K0, q.K1, q.falling, vol, tab);
        if (max(kc, q.K0) >= q.ZI0 && min(kc + 31, q.K1) <= q.ZI1) col_gather_rows<R, REF, MIXED, false>(q, tab, h, f);
        else col_gather_rows<R, REF, MIXED, true>(q, tab, h, f);
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
template <int R, bool REF, bool MIXED, Merge MERGE, bool ZCHK, class Acc>
__device__ __forceinline__ void col_scatter_rows(const ColRays<R> &q, const ColTable &tab, const ColChunk &h,
                                                 const Acc &acc, const float (&y)[R])
{
    using T = typename Acc::T;
    const ZInside in(q.zg.nz);
    // values l, u of the low and high voxels of rays i.. in one voxel column
    constexpr int S = MERGE == kSingle ? 1 : R;
    auto reduce = [&](unsigned lo, unsigned hi, const float (&m)[S], T (&l)[S], T (&u)[S]) {
        if (ZCHK) {
#pragma unroll
            for (int k = 0; k < S; ++k) {
                if (!in.low(m[k])) l[k] = (T)0;
                if (!in.high(m[k])) u[k] = (T)0;
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
        Acc::red(p + 1, u[0]);
    };
#pragma unroll 1
    for (int j = h.cross; j < h.n; ++j) {
        const uint4 te = tab.a[j], tc = tab.c[j];
        const float rv = __uint_as_float(tc.z), ov = __uint_as_float(tc.w);
#pragma unroll
        for (int i = 0; i < R; i += S) {
            float lo, hi, m[S];
            T l1[S], u1[S], l2[S], u2[S];
#pragma unroll
            for (int k = 0; k < S; ++k) {
                float r;
                col_planes<MIXED>(tab, j, te, q.z[i + k], lo, hi);
                z_inner<REF>(q.z[i + k], q.zg, lo, hi, m[k], r);
                const float w11 = fminf(rv, r), w21 = __fsub_rn(r, w11), yk = y[i + k];
                l1[k] = acc.value(yk * w11);
                u1[k] = acc.value(yk * __fsub_rn(rv, w11));
                l2[k] = acc.value(yk * w21);
                u2[k] = acc.value(yk * __fsub_rn(ov, w21));
            }
            if (j < h.half) {
                reduce(te.x, te.y, m, l1, u1);
                reduce(tc.x, tc.y, m, l2, u2);
            } else if (tc.x == 0u) {
                reduce(te.x, te.y, m, l1, u1);
            } else {
                reduce(te.x, te.y, m, l2, u2);
            }
        }
    }
#pragma unroll 2
    for (int j = 0; j < h.cross; ++j) {
        const uint4 te = tab.a[j];
#pragma unroll
        for (int i = 0; i < R; i += S) {
            float lo, hi, m[S];
            T l[S], u[S];
#pragma unroll
            for (int k = 0; k < S; ++k) {
                float r;
                col_planes<MIXED>(tab, j, te, q.z[i + k], lo, hi);
                z_inner<REF>(q.z[i + k], q.zg, lo, hi, m[k], r);
                l[k] = acc.value(y[i + k] * r);
                u[k] = acc.rest(y[i + k], r);
            }
            reduce(te.x, te.y, m, l, u);
        }
    }
}

// Transpose of the lane's R rays (not steep; y finite, 0 for a ray that takes
// no part).
template <int R, bool REF, bool MIXED, Merge MERGE, class Acc>
__device__ __forceinline__ void col_scatter(const ColRays<R> &q, const Acc &acc, const float (&y)[R])
{
    ColTable &tab = col_table();
    for (int kc = q.K0 & ~31; kc <= q.K1; kc += 32) {
        const ColChunk h = col_chunk(q.c, kc, q.K0, q.K1, q.falling, acc.vol, tab);
        if (max(kc, q.K0) >= q.ZI0 && min(kc + 31, q.K1) <= q.ZI1)
            col_scatter_rows<R, REF, MIXED, MERGE, false>(q, tab, h, acc, y);
        else
            col_scatter_rows<R, REF, MIXED, MERGE, true>(q, tab, h, acc, y);
    }
}

}  // namespace nefct
