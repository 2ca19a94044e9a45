// Cone-beam and LOR Siddon projectors on sm_100a: host side of the cone-beam
// projector (validation, per-view tables, workspace, transposes, the
// deterministic transpose), the intersection count, the LOR pair and the
// C-ABI entry points (declared in include/nefct_b200.h).  The cone-beam
// kernels themselves are in cb_kernels.cuh.
//
// Neighbouring rays of a warp cross a driving slab at neighbouring
// transverse positions; with the transverse axis contiguous in memory a
// warp's gather touches one or two 128-byte lines.  That holds for y-driven
// rays in the x-fastest volume; x-driven rays read a y-fastest copy of the
// volume (one transpose per call, in the caller's workspace).
#include <math.h>
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "cb_kernels.cuh"

namespace nefct {

template <bool DIV>
__global__ void __launch_bounds__(256) cb_count_kernel(const __grid_constant__ CBParams<float> p)
{
    int ia, ib, iv;
    cb_cell(p, ia, ib, iv);
    unsigned n = 0;
    if (ia < p.na && ib < p.nb) {
        float r[6];
        cb_ray(p, ia, ib, iv, r);
        Walk<float> w;
        if (setup_walk(p.g, r, p.flags, w)) n = count_walk<float, DIV>(w, p.g);
    }
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(p.count, (unsigned long long)n);
}

// ---------------- deterministic transpose (fixed point) ----------------

template <bool REF>
__global__ void __launch_bounds__(256) cb_backward_fixed_kernel(const __grid_constant__ CBParams<float> p)
{
    int ia, ib, iv;
    cb_cell(p, ia, ib, iv);
    if (ia >= p.na || ib >= p.nb) return;
    const float y = cb_sino_value(p, ia, ib, iv);
    if (y == 0.f) return;
    float r[6];
    cb_ray(p, ia, ib, iv, r);
    Walk<float> w;
    if (!setup_walk(p.g, r, p.flags, w)) return;
    const unsigned sw = (unsigned)(p.g.nx * p.g.ny);
    unsigned su, sv;
    thread_strides(p.g.nx, p.g.ny, w.xdrive, p.fixT != nullptr, su, sv);
    FixedSink f{w.xdrive && p.fixT ? p.fixT : p.fix, y * w.W, *p.fix_scale};
    ray_walk<REF, true>(p.g, w, su, sv, sw, f);
}

// vol[z][y][x] = accZ[y][x][z] / scale (the integer sums of the column warps)
__global__ void __launch_bounds__(256) fixed_zfold_kernel(const unsigned long long *__restrict__ acc, int nx, int ny,
                                                          int nz, const float *scale, float *__restrict__ vol)
{
    __shared__ unsigned long long tile[32][33];
    const int y = blockIdx.z, x0 = blockIdx.x * 32, z0 = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int x = x0 + j, z = z0 + threadIdx.x;
        if (x < nx && z < nz) tile[j][threadIdx.x] = acc[((size_t)y * nx + x) * nz + z];
    }
    __syncthreads();
    const double inv = 1.0 / (double)*scale;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int x = x0 + threadIdx.x, z = z0 + j;
        if (x < nx && z < nz) vol[((size_t)z * ny + y) * nx + x] = (float)((double)(long long)tile[threadIdx.x][j] * inv);
    }
}

// max |x| as float bits (non-negative floats order like their bit patterns)
__global__ void __launch_bounds__(256) maxabs_kernel(const float *__restrict__ x, size_t n, unsigned *out)
{
    unsigned m = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        m = max(m, __float_as_uint(fabsf(x[i])));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// scale = 2^k with k the largest integer such that bound * max|y| * 2^k <= 2^61,
// where bound >= (rays) * (largest weight); then no per-voxel sum of
// |contribution| * scale can exceed 2^61.
__global__ void fixed_scale_kernel(const unsigned *maxbits, double bound, float *scale)
{
    const double B = bound * (double)__uint_as_float(*maxbits);
    int k = 0;
    if (B > 0.0 && B < 1e300) k = (int)floor(61.0 - log2(B));
    k = max(-126, min(127, k));
    *scale = ldexpf(1.0f, k);
}

// vol[z][y][x] = (accN[z][y][x] + accT[z][x][y]) / scale, integer sum first
__global__ void __launch_bounds__(256) fixed_fold_kernel(const unsigned long long *__restrict__ accN,
                                                         const unsigned long long *__restrict__ accT, int nx, int ny,
                                                         const float *scale, float *__restrict__ vol)
{
    __shared__ unsigned long long tile[32][33];
    const size_t plane = (size_t)nx * ny * blockIdx.z;
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
    if (accT) {
        for (int j = threadIdx.y; j < 32; j += 8) {
            const int y = y0 + threadIdx.x, x = x0 + j;
            if (x < nx && y < ny) tile[j][threadIdx.x] = accT[plane + (size_t)x * ny + y];
        }
    }
    __syncthreads();
    const double inv = 1.0 / (double)*scale;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int x = x0 + threadIdx.x, y = y0 + j;
        if (x < nx && y < ny) {
            unsigned long long v = accN[plane + (size_t)y * nx + x];
            if (accT) v += tile[threadIdx.x][j];
            vol[plane + (size_t)y * nx + x] = (float)((double)(long long)v * inv);
        }
    }
}

// ---------------- LOR projector pair (cpp/siddon) ----------------

struct LorParams {
    GridDev<float> g;
    const float *lors;
    long long n;
    uint32_t flags;
    const float *vol;
    const float *vals;
    float *out;
    const int32_t *order;     // walk order (a permutation of 0..n-1), or nullptr
};

// A line's walk: the general walk's operations (siddon.cuh) with the slope
// signs as run-time selects instead of template variants, which keeps the
// kernels under 64 registers and a warp's lines of different signs together
// (the variants took 100 to 116 registers, so half the warps to hide the
// gathers' latency with, and ran one after the other).  256^3, 4 Mi ring lines
// in walk order: forward 4.11 -> 2.99 ms, bound by the gathers' requests (19
// sectors each), backward 4.64 -> 4.68 ms, by the L2's rate of scattered
// reductions (1.9e11/s); in list order 22.8 -> 2.95 and 15.8 -> 4.47 ms.  A
// y-fastest copy for one of the driving axes, either way round, is slower:
// 3.5 and 7 to 9 ms (neighbouring lines then reduce into the same sectors).
// Index of voxel (k, v, z): base + k su + v sv + z sw, floors biased.
struct LineWalk {
    float pv, kv, dv, nv2, pw, kw, dz, nz2, pu, t, qv, mv, qz, mz;
    unsigned su, sv, sw, base;
    int nv, nz;
    bool vdown, zdown, vdiv, zdiv;

    __device__ __forceinline__ void plane(float tt, float &v, float &z) const
    {
        const float d = __fsub_rn(tt, pu);
        v = __fadd_rn(pv, __fmul_rn(kv, d));
        z = __fadd_rn(pw, __fmul_rn(kw, d));
        if (vdiv) v = __fdiv_rn(v, dv);
        if (zdiv) z = __fdiv_rn(z, dz);
        v = __fadd_rn(v, nv2);
        z = __fadd_rn(z, nz2);
    }

    __device__ __forceinline__ LineWalk(const GridDev<float> &g, const Walk<float> &w)
        : pv(w.pv), kv(w.kv), dv(w.dv), nv2(w.nv2), pw(w.pw), kw(w.kw), dz(g.dz), nz2(g.nz2), pu(w.pu),
          su(w.xdrive ? 1u : (unsigned)g.nx), sv(w.xdrive ? (unsigned)g.nx : 1u), sw((unsigned)g.nx * (unsigned)g.ny),
          nv(w.nv), nz(g.nz), vdown(w.kv < 0.f), zdown(w.kw < 0.f), vdiv(w.vdiv), zdiv(g.dz != 1.f)
    {
        t = __fsub_rn((float)w.k0, w.nu2);
        base = (unsigned)w.k0 * su - (unsigned)kFloorMagicBits * (sv + sw);
        plane(t, qv, qz);
        mv = magic_floor<true>(qv);
        mz = magic_floor<true>(qz);
    }

    template <bool CHECK> __device__ __forceinline__ SlabSlots<float> next()
    {
        t = __fadd_rn(t, 1.f);
        float bv, bz;
        plane(t, bv, bz);
        const float nv_ = magic_floor<CHECK>(bv), nz_ = magic_floor<CHECK>(bz);
        const float q1v = vdown ? bv : qv, q2v = vdown ? qv : bv, m1v = vdown ? nv_ : mv, m2v = vdown ? mv : nv_;
        const float q1z = zdown ? bz : qz, q2z = zdown ? qz : bz, m1z = zdown ? nz_ : mz, m2z = zdown ? mz : nz_;
        qv = bv; qz = bz; mv = nv_; mz = nz_;
        const bool vx = m1v != m2v, wx = m1z != m2z;
        const float rv = vx ? FP<float>::ratio(__fadd_rn(__fadd_rn(m2v, -kFloorMagic), -q1v), __fadd_rn(q2v, -q1v)) : 1.f;
        const float rw = wx ? FP<float>::ratio(__fadd_rn(__fadd_rn(m2z, -kFloorMagic), -q1z), __fadd_rn(q2z, -q1z)) : 1.f;
        const bool vfirst = rv > rw;
        const unsigned i1 = base + (unsigned)__float_as_int(m1v) * sv, i2 = base + (unsigned)__float_as_int(m2v) * sv;
        const unsigned j1 = (unsigned)__float_as_int(m1z) * sw, j2 = (unsigned)__float_as_int(m2z) * sw;
        base += su;
        SlabSlots<float> s;
        s.r[0] = fminf(rv, rw);
        s.r[1] = fabsf(__fsub_rn(rv, rw));
        s.r[2] = __fsub_rn(1.f, fmaxf(rv, rw));
        s.idx[0] = i1 + j1;
        s.idx[1] = vfirst ? i1 + j2 : i2 + j1;
        s.idx[2] = i2 + j2;
        s.mid3 = vx && wx;
        s.ok[0] = true;
        s.ok[1] = vx || wx;
        s.ok[2] = vx && wx;
        if (CHECK) {
            const int cv1 = __float_as_int(m1v) - kFloorMagicBits, cv2 = __float_as_int(m2v) - kFloorMagicBits;
            const int cw1 = __float_as_int(m1z) - kFloorMagicBits, cw2 = __float_as_int(m2z) - kFloorMagicBits;
            const bool adm = (unsigned)(cv1 + (int)vx) < (unsigned)(nv + (int)vx) &&
                             (unsigned)(cw1 + (int)wx) < (unsigned)(nz + (int)wx);
            const int v = vfirst ? cv1 : cv2, z = vfirst ? cw2 : cw1;
            s.ok[0] = adm && (cv1 | cw1) >= 0;
            s.ok[1] = adm && s.ok[1] && (unsigned)v < (unsigned)nv && (unsigned)z < (unsigned)nz;
            s.ok[2] = adm && s.ok[2] && cv2 < nv && cw2 < nz;
        }
        return s;
    }
};

// Calls f(slots) for the slabs k0..k1 of the line, those outside [ki0, ki1]
// range checked.
template <class Fn> __device__ __forceinline__ void line_walk(LineWalk &l, const Walk<float> &w, Fn &f)
{
    const int a = w.ki0 <= w.ki1 ? w.ki0 : w.k1 + 1, b = w.ki0 <= w.ki1 ? w.ki1 : w.k1;
    int k = w.k0;
#pragma unroll 1
    for (; k < a; ++k) f(l.next<true>());
#pragma unroll 2
    for (; k <= b; ++k) f(l.next<false>());
#pragma unroll 1
    for (; k <= w.k1; ++k) f(l.next<true>());
}

// The walk visits lines in `order` so that a warp's 32 lines are nearly
// parallel neighbours (similar trip counts, nearby voxels); results stay at
// each line's own index.
template <bool Q5>
__global__ void __launch_bounds__(256, 4) lor_forward_kernel(const __grid_constant__ LorParams p)
{
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < p.n;
         t += (long long)gridDim.x * blockDim.x) {
        const long long i = p.order ? (long long)p.order[t] : t;
        float r[6];
        for (int j = 0; j < 6; ++j) r[j] = p.lors[j * p.n + i];
        Walk<float> w;
        float sum = 0.f;
        if (setup_walk(p.g, r, p.flags, w)) {
            LineWalk l(p.g, w);
            float acc = 0.f, mid = 0.f;
            auto f = [&](const SlabSlots<float> &s) {
                const float v0 = s.ok[0] ? __ldg(p.vol + s.idx[0]) : 0.f;
                const float v1 = s.ok[1] ? __ldg(p.vol + s.idx[1]) : 0.f;
                const float v2 = s.ok[2] ? __ldg(p.vol + s.idx[2]) : 0.f;
                acc += v0 * s.r[0];
                if (Q5 && s.mid3) mid += v1 * s.r[1];
                else acc += v1 * s.r[1];
                acc += v2 * s.r[2];
            };
            line_walk(l, w, f);
            sum = Q5 ? acc * w.W + mid * w.Wmid : acc * w.W;
        }
        p.out[i] = sum;
    }
}

template <bool Q5>
__global__ void __launch_bounds__(256, 4) lor_backward_kernel(const __grid_constant__ LorParams p)
{
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < p.n;
         t += (long long)gridDim.x * blockDim.x) {
        const long long i = p.order ? (long long)p.order[t] : t;
        const float y = p.vals[i];
        if (y == 0.f) continue;
        float r[6];
        for (int j = 0; j < 6; ++j) r[j] = p.lors[j * p.n + i];
        Walk<float> w;
        if (!setup_walk(p.g, r, p.flags, w)) continue;
        LineWalk l(p.g, w);
        const float yw = y * w.W, ym = y * w.Wmid;
        auto f = [&](const SlabSlots<float> &s) {
            if (s.ok[0]) atomicAdd(p.out + s.idx[0], yw * s.r[0]);
            if (s.ok[1]) atomicAdd(p.out + s.idx[1], ((Q5 && s.mid3) ? ym : yw) * s.r[1]);
            if (s.ok[2]) atomicAdd(p.out + s.idx[2], yw * s.r[2]);
        };
        line_walk(l, w, f);
    }
}

// Ordering key of a line (31 bits, larger = later): driving axis, in-plane
// direction folded to [0, pi), signed distance of the in-plane line from the
// grid centre, z where the line passes the centre, and z slope.  Lines with
// equal keys are nearly parallel neighbours.
__global__ void __launch_bounds__(256) lor_key_kernel(const __grid_constant__ LorParams p, int32_t *keys)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < p.n;
         i += (long long)gridDim.x * blockDim.x) {
        const float x1 = p.lors[i] - p.g.cx, y1 = p.lors[p.n + i] - p.g.cy, z1 = p.lors[2 * p.n + i] - p.g.cz;
        const float dx = p.lors[3 * p.n + i] - p.g.cx - x1, dy = p.lors[4 * p.n + i] - p.g.cy - y1;
        const float dz = p.lors[5 * p.n + i] - p.g.cz - z1;
        const float sx = (float)p.g.nx * p.g.dx_, sy = p.g.dy * (float)p.g.ny * p.g.dx_;
        const float sz = p.g.dz * (float)p.g.nz * p.g.dx_;
        const float lxy = sqrtf(dx * dx + dy * dy);
        const unsigned xdrive = fabsf(dx) >= fabsf(dy);
        float th = atan2f(dy, dx);
        if (th < 0.f) th += 3.14159265f;
        if (th >= 3.14159265f) th -= 3.14159265f;
        const float ux = lxy > 0.f ? dx / lxy : 1.f, uy = lxy > 0.f ? dy / lxy : 0.f;
        const float rad = 0.5f * sqrtf(sx * sx + sy * sy) + 1e-6f;
        const float perp = (x1 * uy - y1 * ux) / rad;                 // [-1, 1] for lines through the grid
        const float along = -(x1 * ux + y1 * uy);                     // parameter (in-plane length) of the centre
        const float slope = lxy > 0.f ? dz / lxy : 0.f;
        const float zc = (z1 + slope * along) / (sz + 1e-6f);         // about [-0.5, 0.5] inside
        auto q = [](float v, float lo, float hi, int bits) {
            const float f = fminf(fmaxf((v - lo) / (hi - lo), 0.f), 1.f);
            return (unsigned)fminf(f * (float)(1 << bits), (float)((1 << bits) - 1));
        };
        // z centre and slope interleaved bit by bit (a Z-order curve): the
        // lines of one direction and offset bin fall into warps of similar
        // z entry and exit, so the walks of a warp have similar lengths
        const unsigned zq = q(zc, -1.f, 1.f, 7), sq = q(atanf(slope), -1.5708f, 1.5708f, 7);
        unsigned zs = 0;
#pragma unroll
        for (int b = 0; b < 7; ++b) zs |= ((zq >> b) & 1u) << (2 * b + 1) | ((sq >> b) & 1u) << (2 * b);
        const unsigned k = (xdrive << 30) | (q(th, 0.f, 3.14159265f, 8) << 22) | (q(perp, -1.f, 1.f, 8) << 14) | zs;
        keys[i] = (int32_t)k;
    }
}

// ---------------- host side ----------------

static const uint32_t kWalkFlags = NEFCT_TIE_GT | NEFCT_SKIP_SHORT | NEFCT_NO_INV_L2 | NEFCT_Q5 |
                                   NEFCT_Q8_INDEX | NEFCT_NO_TRANSPOSE | NEFCT_DETERMINISTIC | NEFCT_EXACT;

// Flags of the cone-beam calls: the walk switches except NEFCT_Q5, a quirk of
// the LOR projector (cpp/siddon) that no cone-beam walk applies.
static nefct_status check_cb_flags(uint32_t flags)
{
    if (flags & ~kWalkFlags) return fail(NEFCT_ERR_INVALID, "unknown flag bits 0x%x", flags & ~kWalkFlags);
    if (flags & NEFCT_Q5)
        return fail(NEFCT_ERR_UNSUPPORTED, "NEFCT_Q5 belongs to the LOR projector; the cone-beam walks do not take it");
    return NEFCT_OK;
}

static nefct_status check_grid(const nefct_grid &g)
{
    if (g.nx < 1 || g.ny < 1 || g.nz < 1)
        return fail(NEFCT_ERR_INVALID, "grid dimensions must be >= 1 (got %d x %d x %d)", g.nx, g.ny, g.nz);
    if (g.nx > (1 << 20) || g.ny > (1 << 20) || g.nz > (1 << 20))
        return fail(NEFCT_ERR_INVALID, "grid dimensions must be <= 2^20 (got %d x %d x %d)", g.nx, g.ny, g.nz);
    if ((long long)g.nx * g.ny * g.nz >= (1ll << 31))
        return fail(NEFCT_ERR_INVALID, "grid has %lld voxels; at most 2^31-1 are supported",
                    (long long)g.nx * g.ny * g.nz);
    const float v[6] = {g.cx, g.cy, g.cz, g.sx, g.sy, g.sz};
    for (int i = 0; i < 6; ++i)
        if (!std::isfinite(v[i])) return fail(NEFCT_ERR_INVALID, "grid centre/size must be finite");
    if (!(g.sx > 0.f && g.sy > 0.f && g.sz > 0.f)) return fail(NEFCT_ERR_INVALID, "grid size must be > 0");
    return NEFCT_OK;
}

nefct_status check_cb_geom(const nefct_cb_geom *g)
{
    if (!g) return fail(NEFCT_ERR_INVALID, "geometry is NULL");
    nefct_status st = check_grid(g->grid);
    if (st) return st;
    if (g->nv < 1 || !g->angles) return fail(NEFCT_ERR_INVALID, "need nv >= 1 view angles (nv=%d)", g->nv);
    if (g->na < 1 || g->nb < 1) return fail(NEFCT_ERR_INVALID, "detector must be >= 1 x 1 (got %d x %d)", g->na, g->nb);
    if ((long long)g->na * g->nb * g->nv >= (1ll << 40))
        return fail(NEFCT_ERR_INVALID, "sinogram too large");
    if ((long long)g->na * g->nb >= (1ll << 31)) return fail(NEFCT_ERR_INVALID, "detector too large");
    if (g->nb > 65535 || g->grid.nz > 65535)
        return fail(NEFCT_ERR_INVALID, "detector rows and nz must be <= 65535 (got %d, %d)", g->nb, g->grid.nz);
    if (g->det_kind != NEFCT_DET_FLAT && g->det_kind != NEFCT_DET_CYL)
        return fail(NEFCT_ERR_INVALID, "det_kind must be NEFCT_DET_FLAT or NEFCT_DET_CYL (got %d)", g->det_kind);
    const float v[6] = {g->src_iso, g->src_det, g->da, g->a_shift, g->db, g->b_shift};
    for (int i = 0; i < 6; ++i)
        if (!std::isfinite(v[i])) return fail(NEFCT_ERR_INVALID, "scanner geometry must be finite");
    if (g->da == 0.f || g->db == 0.f) return fail(NEFCT_ERR_INVALID, "detector pitch must be non-zero");
    for (int i = 0; i < g->nv; ++i) {
        if (!std::isfinite(g->angles[i])) return fail(NEFCT_ERR_INVALID, "angle %d is not finite", i);
        if (g->z_offsets && !std::isfinite(g->z_offsets[i]))
            return fail(NEFCT_ERR_INVALID, "z offset %d is not finite", i);
    }
    return NEFCT_OK;
}

template <typename T> static void fill_cb_params(CBParams<T> &p, const nefct_cb_geom *g, uint32_t flags)
{
    p.g = make_grid_dev<T>(g->grid);
    p.na = g->na; p.nb = g->nb; p.nv_total = g->nv;
    p.rg = make_ray_geom<T>(*g);
    p.flags = flags;
}

// cos/sin of the view angles from the double-precision functions, rounded.
template <typename T> static void fill_views(CBParams<T> &p, const nefct_cb_geom *g, int v0, int nvc)
{
    p.v0 = v0; p.nvc = nvc;
    for (int i = 0; i < nvc; ++i) {
        const double a = (double)g->angles[v0 + i];
        p.tab.cs[i] = (T)cos(a);
        p.tab.sn[i] = (T)sin(a);
        p.tab.off[i] = g->z_offsets ? (T)g->z_offsets[v0 + i] : (T)0;
    }
}

// volZ[y][x][z] = vol[z][y][x]  (32x32 tiles of each y plane)
__global__ void __launch_bounds__(256) zmajor_kernel(const float *__restrict__ in, float *__restrict__ out, int nx,
                                                     int ny, int nz)
{
    __shared__ float tile[32][33];
    const int y = blockIdx.z, x0 = blockIdx.x * 32, z0 = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int x = x0 + threadIdx.x, z = z0 + j;
        if (x < nx && z < nz) tile[j][threadIdx.x] = in[((size_t)z * ny + y) * nx + x];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int x = x0 + j, z = z0 + threadIdx.x;
        if (x < nx && z < nz) out[((size_t)y * nx + x) * nz + z] = tile[threadIdx.x][j];
    }
}

// vol[z][y][x] = accZ[y][x][z]
__global__ void __launch_bounds__(256) zfold_kernel(const float *__restrict__ acc, float *__restrict__ vol, int nx,
                                                    int ny, int nz)
{
    __shared__ float tile[32][33];
    const int y = blockIdx.z, x0 = blockIdx.x * 32, z0 = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int x = x0 + j, z = z0 + threadIdx.x;
        if (x < nx && z < nz) tile[j][threadIdx.x] = acc[((size_t)y * nx + x) * nz + z];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int x = x0 + threadIdx.x, z = z0 + j;
        if (x < nx && z < nz) vol[((size_t)z * ny + y) * nx + x] = tile[threadIdx.x][j];
    }
}

// z-fastest copy [y][x][z] of an x-fastest volume (column-warp forward)
nefct_status zmajor_copy(const float *in, float *out, const nefct_grid &g, cudaStream_t s)
{
    dim3 grid((g.nx + 31) / 32, (g.nz + 31) / 32, g.ny);
    zmajor_kernel<<<grid, dim3(32, 8), 0, s>>>(in, out, g.nx, g.ny, g.nz);
    NEFCT_CHECK_LAUNCH("zmajor_kernel");
    return NEFCT_OK;
}

// vol = the x-fastest layout of the z-fastest accumulator (column-warp transpose)
nefct_status zfold(const float *acc, float *vol, const nefct_grid &g, cudaStream_t s)
{
    dim3 grid((g.nx + 31) / 32, (g.nz + 31) / 32, g.ny);
    zfold_kernel<<<grid, dim3(32, 8), 0, s>>>(acc, vol, g.nx, g.ny, g.nz);
    NEFCT_CHECK_LAUNCH("zfold_kernel");
    return NEFCT_OK;
}

template <typename T>
static nefct_status transpose_xy(const T *in, T *out, const nefct_grid &g, cudaStream_t s)
{
    dim3 grid((g.nx + 31) / 32, (g.ny + 31) / 32, g.nz);
    transpose_xy_kernel<T><<<grid, dim3(32, 8), 0, s>>>(in, out, g.nx, g.ny);
    NEFCT_CHECK_LAUNCH("transpose_xy_kernel");
    return NEFCT_OK;
}

// Launches of the forward / transpose kernels for one problem whose volume
// copy (forward) or accumulator (transpose) is given -- y-fastest for the
// thread walk, z-fastest for column warps (colwarp); no transpose, memset or
// fold.  Used by the batch's per-problem strategy.
nefct_status cb_forward_launches(const nefct_cb_geom *g, const float *vol, const float *volT, float *sino,
                                 uint32_t flags, cudaStream_t s, bool colwarp)
{
    CBParams<float> p;
    fill_cb_params(p, g, flags);
    p.vol = vol;
    p.volT = volT;
    p.out = sino;
    for (int v0 = 0; v0 < g->nv; v0 += ViewTable<float>::kMax) {
        const int nvc = std::min(ViewTable<float>::kMax, g->nv - v0);
        fill_views(p, g, v0, nvc);
        const cudaError_t e = cb_launch_forward<float>(p, g->na, g->nb, nvc, flags, s, colwarp);
        if (e != cudaSuccess) return cuda_fail(e, "cb_forward_kernel");
    }
    return NEFCT_OK;
}

nefct_status cb_backward_launches(const nefct_cb_geom *g, const float *sino, float *out, float *outT,
                                  uint32_t flags, cudaStream_t s, bool colwarp)
{
    CBParams<float> p;
    fill_cb_params(p, g, flags);
    p.sino = sino;
    p.out = out;
    p.outT = outT;
    for (int v0 = 0; v0 < g->nv; v0 += ViewTable<float>::kMax) {
        const int nvc = std::min(ViewTable<float>::kMax, g->nv - v0);
        fill_views(p, g, v0, nvc);
        const cudaError_t e = cb_launch_backward<float>(p, g->na, g->nb, nvc, flags, s, colwarp);
        if (e != cudaSuccess) return cuda_fail(e, "cb_backward_kernel");
    }
    return NEFCT_OK;
}

template <typename T>
static nefct_status cb_forward_impl(const nefct_cb_geom *g, const T *vol, T *sino, uint32_t flags, void *ws,
                                    size_t wsb, cudaStream_t s)
{
    nefct_status st = check_cb_geom(g);
    if (st) return st;
    if (!vol || !sino) return fail(NEFCT_ERR_INVALID, "vol and sino must be non-NULL");
    if ((st = check_cb_flags(flags))) return st;
    CBParams<T> *p = new CBParams<T>();
    fill_cb_params(*p, g, flags);
    p->vol = vol;
    p->out = sino;
    const size_t nvox = (size_t)g->grid.nx * g->grid.ny * g->grid.nz;
    const bool cw = cb_use_colwarp<T>(g->grid, flags, true, g->nb);
    if (!(flags & NEFCT_NO_TRANSPOSE)) {
        if (!ws || wsb < nvox * sizeof(T)) {
            delete p;
            return fail(NEFCT_ERR_WORKSPACE, "forward needs %zu workspace bytes, got %zu", nvox * sizeof(T), wsb);
        }
        if constexpr (std::is_same<T, float>::value) {
            if (cw) st = zmajor_copy(vol, (float *)ws, g->grid, s);
            else st = transpose_xy(vol, (T *)ws, g->grid, s);
        } else {
            st = transpose_xy(vol, (T *)ws, g->grid, s);
        }
        if (st) { delete p; return st; }
        p->volT = (const T *)ws;
    }
    const int kMax = ViewTable<T>::kMax;
    for (int v0 = 0; v0 < g->nv; v0 += kMax) {
        const int nvc = std::min(kMax, g->nv - v0);
        fill_views(*p, g, v0, nvc);
        cudaError_t e = cb_launch_forward<T>(*p, g->na, g->nb, nvc, flags, s, cw);
        if (e != cudaSuccess) { delete p; return cuda_fail(e, "cb_forward_kernel"); }
    }
    delete p;
    return NEFCT_OK;
}

// Upper bound of (rays) x (largest contribution weight) for the fixed-point
// scale: |kv| <= 1 by the choice of driving axis; the transverse
// source-detector distance is >= src_det (flat: sqrt(src_det^2 + a^2);
// cylindrical: exactly src_det), so |kw| <= sqrt(2) max|b| / src_det and
// L >= src_det / dx in voxel units.
static double fixed_bound(const nefct_cb_geom *g, uint32_t flags)
{
    const double dx = (double)g->grid.sx / g->grid.nx;
    const double half = g->nb * (double)g->db / 2.0;
    const double b0 = fabs((0.0 + g->b_shift) * g->db - half);
    const double b1 = fabs((g->nb - 1.0 + g->b_shift) * g->db - half);
    const double kw = sqrt(2.0) * std::max(b0, b1) / g->src_det;
    double W = sqrt(2.0 + kw * kw) * dx;
    if (!(flags & NEFCT_NO_INV_L2)) W *= (dx / g->src_det) * (dx / g->src_det);
    return (double)g->na * g->nb * g->nv * W * 1.001;
}

size_t cb_fixed_workspace(const nefct_cb_geom *g, uint32_t flags)
{
    const size_t nvox = (size_t)g->grid.nx * g->grid.ny * g->grid.nz;
    return 256 + nvox * sizeof(unsigned long long) * ((flags & NEFCT_NO_TRANSPOSE) ? 1 : 2);
}

static nefct_status cb_backward_fixed_impl(const nefct_cb_geom *g, const float *sino, float *vol, uint32_t flags,
                                           void *ws, size_t wsb, cudaStream_t s)
{
    if (flags & NEFCT_EXACT)
        return fail(NEFCT_ERR_UNSUPPORTED, "NEFCT_EXACT is not available with NEFCT_DETERMINISTIC");
    if (!(g->src_det > 0.f)) return fail(NEFCT_ERR_INVALID, "deterministic transpose needs src_det > 0");
    const size_t nvox = (size_t)g->grid.nx * g->grid.ny * g->grid.nz;
    const bool tr = !(flags & NEFCT_NO_TRANSPOSE);
    const size_t need = cb_fixed_workspace(g, flags);
    if (!ws || wsb < need)
        return fail(NEFCT_ERR_WORKSPACE, "deterministic backward needs %zu workspace bytes, got %zu", need, wsb);
    unsigned char *w = (unsigned char *)ws;
    unsigned *maxbits = (unsigned *)w;
    float *scale = (float *)(w + 16);
    unsigned long long *accN = (unsigned long long *)(w + 256);
    unsigned long long *accT = tr ? accN + nvox : nullptr;
    // column warps reduce everything into accN in z-fastest order
    const bool cw = tr && cb_use_colwarp<float>(g->grid, flags & ~NEFCT_DETERMINISTIC, false, g->nb);
    NEFCT_CHECK_CUDA(cudaMemsetAsync(w, 0, cw ? 256 + nvox * sizeof(unsigned long long) : need, s));
    const size_t ns = (size_t)g->na * g->nb * g->nv;
    maxabs_kernel<<<(unsigned)std::min<size_t>((ns + 255) / 256, 148 * 16), 256, 0, s>>>(sino, ns, maxbits);
    NEFCT_CHECK_LAUNCH("maxabs_kernel");
    fixed_scale_kernel<<<1, 1, 0, s>>>(maxbits, fixed_bound(g, flags), scale);
    NEFCT_CHECK_LAUNCH("fixed_scale_kernel");
    CBParams<float> p;
    fill_cb_params(p, g, flags);
    p.sino = sino;
    p.fix = accN;
    p.fixT = accT;
    p.fix_scale = scale;
    for (int v0 = 0; v0 < g->nv; v0 += ViewTable<float>::kMax) {
        const int nvc = std::min(ViewTable<float>::kMax, g->nv - v0);
        fill_views(p, g, v0, nvc);
        if (cw) {
            // the same per-contribution integers as the thread walk's, so the
            // sums and the result are bitwise the same
            const cudaError_t e = cb_launch_backward_fixed(p, g->na, g->nb, nvc, flags, s);
            if (e != cudaSuccess) return cuda_fail(e, "cb_colwarp_backward_kernel (fixed)");
            continue;
        }
        dim3 grid, block;
        cb_shape(p, g->na, g->nb, nvc, grid, block);
        if (ref_rounding(flags)) cb_backward_fixed_kernel<true><<<grid, block, 0, s>>>(p);
        else cb_backward_fixed_kernel<false><<<grid, block, 0, s>>>(p);
        NEFCT_CHECK_LAUNCH("cb_backward_fixed_kernel");
    }
    if (cw) {
        dim3 grid((g->grid.nx + 31) / 32, (g->grid.nz + 31) / 32, g->grid.ny);
        fixed_zfold_kernel<<<grid, dim3(32, 8), 0, s>>>(accN, g->grid.nx, g->grid.ny, g->grid.nz, scale, vol);
        NEFCT_CHECK_LAUNCH("fixed_zfold_kernel");
        return NEFCT_OK;
    }
    dim3 grid((g->grid.nx + 31) / 32, (g->grid.ny + 31) / 32, g->grid.nz);
    fixed_fold_kernel<<<grid, dim3(32, 8), 0, s>>>(accN, accT, g->grid.nx, g->grid.ny, scale, vol);
    NEFCT_CHECK_LAUNCH("fixed_fold_kernel");
    return NEFCT_OK;
}

template <typename T>
static nefct_status cb_backward_impl(const nefct_cb_geom *g, const T *sino, T *vol, uint32_t flags, void *ws,
                                     size_t wsb, cudaStream_t s)
{
    nefct_status st = check_cb_geom(g);
    if (st) return st;
    if (!vol || !sino) return fail(NEFCT_ERR_INVALID, "vol and sino must be non-NULL");
    if ((st = check_cb_flags(flags))) return st;
    if (flags & NEFCT_DETERMINISTIC) {
        if (sizeof(T) != sizeof(float))
            return fail(NEFCT_ERR_UNSUPPORTED, "NEFCT_DETERMINISTIC is available for float32 only");
        return cb_backward_fixed_impl(g, (const float *)sino, (float *)vol, flags, ws, wsb, s);
    }
    const size_t nvox = (size_t)g->grid.nx * g->grid.ny * g->grid.nz;
    const bool tr = !(flags & NEFCT_NO_TRANSPOSE);
    if (tr && (!ws || wsb < nvox * sizeof(T)))
        return fail(NEFCT_ERR_WORKSPACE, "backward needs %zu workspace bytes, got %zu", nvox * sizeof(T), wsb);
    CBParams<T> *p = new CBParams<T>();
    fill_cb_params(*p, g, flags);
    p->sino = sino;
    p->out = vol;
    p->outT = tr ? (T *)ws : nullptr;
    // column warps reduce into the z-fastest workspace only; the fold then
    // writes every voxel of vol
    const bool cw = cb_use_colwarp<T>(g->grid, flags, false, g->nb);
    cudaError_t e = cw ? cudaSuccess : cudaMemsetAsync(vol, 0, nvox * sizeof(T), s);
    if (e == cudaSuccess && tr) e = cudaMemsetAsync(ws, 0, nvox * sizeof(T), s);
    if (e != cudaSuccess) { delete p; return cuda_fail(e, "cudaMemsetAsync"); }
    const int kMax = ViewTable<T>::kMax;
    for (int v0 = 0; v0 < g->nv; v0 += kMax) {
        const int nvc = std::min(kMax, g->nv - v0);
        fill_views(*p, g, v0, nvc);
        e = cb_launch_backward<T>(*p, g->na, g->nb, nvc, flags, s, cw);
        if (e != cudaSuccess) { delete p; return cuda_fail(e, "cb_backward_kernel"); }
    }
    delete p;
    if constexpr (std::is_same<T, float>::value) {
        if (cw) return zfold(ws ? (const float *)ws : nullptr, vol, g->grid, s);
    }
    if (tr) {
        dim3 grid((g->grid.nx + 31) / 32, (g->grid.ny + 31) / 32, g->grid.nz);
        fold_add_kernel<T><<<grid, dim3(32, 8), 0, s>>>((const T *)ws, vol, g->grid.nx, g->grid.ny);
        NEFCT_CHECK_LAUNCH("fold_add_kernel");
    }
    return NEFCT_OK;
}

static nefct_status lor_impl(const nefct_grid *grid, const float *lors, int64_t n, const float *src, float *dst,
                             uint32_t flags, cudaStream_t s, bool forward, const int32_t *order = nullptr)
{
    if (!grid) return fail(NEFCT_ERR_INVALID, "grid is NULL");
    nefct_status st = check_grid(*grid);
    if (st) return st;
    if (n < 0) return fail(NEFCT_ERR_INVALID, "negative LOR count");
    if (flags & (NEFCT_EXACT | NEFCT_DETERMINISTIC | NEFCT_Q8_INDEX))
        return fail(NEFCT_ERR_UNSUPPORTED, "the LOR projector takes the walk flags of cpp/siddon only");
    if ((!lors || !src || !dst) && n > 0) return fail(NEFCT_ERR_INVALID, "NULL buffer");
    if (flags & ~kWalkFlags) return fail(NEFCT_ERR_INVALID, "unknown flag bits 0x%x", flags & ~kWalkFlags);
    if (forward && n == 0) return NEFCT_OK;          // no lines: nothing to write
    if (!dst) return fail(NEFCT_ERR_INVALID, "NULL output");
    const size_t bytes = (size_t)grid->nx * grid->ny * grid->nz * sizeof(float);
    LorParams p{};
    p.g = make_grid_dev<float>(*grid);
    p.lors = lors; p.n = n; p.flags = flags; p.order = order;
    if (n >= (1ll << 31) && order) return fail(NEFCT_ERR_INVALID, "ordered walks take fewer than 2^31 lines");
    p.out = dst;
    if (!forward) {
        NEFCT_CHECK_CUDA(cudaMemsetAsync(dst, 0, bytes, s));
        p.vals = src;
    } else {
        p.vol = src;
    }
    if (n == 0) return NEFCT_OK;
    const unsigned blocks = (unsigned)std::min<long long>((n + 255) / 256, 148ll * 64);
    const bool q5 = (flags & NEFCT_Q5) != 0;
    if (forward && q5) lor_forward_kernel<true><<<blocks, 256, 0, s>>>(p);
    else if (forward) lor_forward_kernel<false><<<blocks, 256, 0, s>>>(p);
    else if (q5) lor_backward_kernel<true><<<blocks, 256, 0, s>>>(p);
    else lor_backward_kernel<false><<<blocks, 256, 0, s>>>(p);
    NEFCT_CHECK_LAUNCH(forward ? "lor_forward_kernel" : "lor_backward_kernel");
    return NEFCT_OK;
}

// ---------------- forward projection for callers that cannot allocate ----------------
//
// Some callers of this library are not allowed to allocate device memory:
// reconstruction services that reserve all GPU memory at start-up and forbid
// later allocations (fixed memory budget, predictable latency), host
// frameworks that own the device memory pool and only hand out the tensors a
// plugin reads and writes, and bindings that receive bare device pointers
// with no access to an allocator.  nefct_cb_forward needs a volume-sized
// scratch buffer that such callers cannot provide.  For them the scratch
// lives in this fixed array, part of the library's device image: every GPU
// that loads the library holds it (32 MiB) until the process exits.
static constexpr size_t kStaticScratchFloats = size_t(8) << 20;   // 8 Mi voxels
static __device__ __align__(256) float g_static_scratch[kStaticScratchFloats];

// Host code cannot use g_static_scratch's name as a device address.  The
// address belongs to the CUDA context the library's device code is loaded
// in, so it is cached per context, keyed by the context's unique ID
// (cuCtxGetId: never reused within a process), and looked up again
// (cudaGetSymbolAddress) for a context not seen before: the first call in a
// process, on another device, under a caller's own driver-API context, or
// after cudaDeviceReset replaced the device's primary context.  The driver
// calls are reached through cudaGetDriverEntryPoint (no link to libcuda).
using CtxGetCurrentFn = int (*)(void **ctx);
using CtxGetIdFn = int (*)(void *ctx, unsigned long long *id);
static constexpr int kMaxContexts = 64;
static std::mutex g_static_mu;
static CtxGetCurrentFn g_ctx_get_current = nullptr;
static CtxGetIdFn g_ctx_get_id = nullptr;
static unsigned long long g_static_ctx[kMaxContexts];
static float *g_static_addr[kMaxContexts];
static int g_static_n = 0, g_static_next = 0;

// ID of the context current on this thread (have = false: none is current).
// Call with g_static_mu held.
static nefct_status current_context_id(bool &have, unsigned long long &id)
{
    if (!g_ctx_get_current || !g_ctx_get_id) {
        void *f1 = nullptr, *f2 = nullptr;
        cudaDriverEntryPointQueryResult q1 = cudaDriverEntryPointSymbolNotFound, q2 = q1;
        cudaError_t e = cudaGetDriverEntryPoint("cuCtxGetCurrent", &f1, cudaEnableDefault, &q1);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetDriverEntryPoint(cuCtxGetCurrent)");
        e = cudaGetDriverEntryPoint("cuCtxGetId", &f2, cudaEnableDefault, &q2);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetDriverEntryPoint(cuCtxGetId)");
        if (q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess || !f1 || !f2)
            return fail(NEFCT_ERR_UNSUPPORTED, "the driver lacks cuCtxGetCurrent / cuCtxGetId (CUDA 12.0+ needed)");
        g_ctx_get_current = (CtxGetCurrentFn)f1;
        g_ctx_get_id = (CtxGetIdFn)f2;
    }
    void *ctx = nullptr;
    if (g_ctx_get_current(&ctx) != 0) return fail(NEFCT_ERR_CUDA, "cuCtxGetCurrent failed");
    have = ctx != nullptr;
    if (have && g_ctx_get_id(ctx, &id) != 0) return fail(NEFCT_ERR_CUDA, "cuCtxGetId failed");
    return NEFCT_OK;
}

static nefct_status static_scratch_address(float **addr)
{
    std::lock_guard<std::mutex> lock(g_static_mu);
    bool have = false;
    unsigned long long id = 0;
    nefct_status st = current_context_id(have, id);
    if (st) return st;
    if (have) {
        for (int i = 0; i < g_static_n; ++i)
            if (g_static_ctx[i] == id) {
                *addr = g_static_addr[i];
                return NEFCT_OK;
            }
    }
    // a context not seen yet (or none current: the lookup initialises the
    // device's primary context and makes it current)
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_static_scratch)");
    if (!have) {
        st = current_context_id(have, id);
        if (st) return st;
        if (!have) return fail(NEFCT_ERR_CUDA, "no CUDA context is current after cudaGetSymbolAddress");
    }
    int slot = -1;
    for (int i = 0; i < g_static_n; ++i)
        if (g_static_ctx[i] == id) slot = i;
    if (slot < 0) {
        slot = g_static_n < kMaxContexts ? g_static_n++ : g_static_next;
        g_static_next = (g_static_next + 1) % kMaxContexts;
    }
    g_static_ctx[slot] = id;
    g_static_addr[slot] = (float *)p;
    *addr = (float *)p;
    return NEFCT_OK;
}

static nefct_status cb_forward_static_impl(const nefct_cb_geom *g, const float *vol, float *sino, uint32_t flags,
                                           cudaStream_t s)
{
    nefct_status st = check_cb_geom(g);
    if (st) return st;
    if (!vol || !sino) return fail(NEFCT_ERR_INVALID, "vol and sino must be non-NULL");
    if ((st = check_cb_flags(flags))) return st;
    const size_t nvox = (size_t)g->grid.nx * g->grid.ny * g->grid.nz;
    const bool tr = !(flags & NEFCT_NO_TRANSPOSE);
    if (tr && nvox > kStaticScratchFloats)
        return fail(NEFCT_ERR_INVALID,
                    "nefct_cb_forward_noalloc handles at most %zu voxels (its fixed scratch is %zu MiB); this grid "
                    "has %zu -- use nefct_cb_forward with a workspace",
                    kStaticScratchFloats, kStaticScratchFloats * sizeof(float) >> 20, nvox);
    // the walk nefct_cb_forward takes for these flags and the current
    // launch tuning, over the same kind of volume copy, so the two give the
    // same bits
    const bool cw = cb_use_colwarp<float>(g->grid, flags, true, g->nb);
    float *scratch = nullptr;
    if (tr) {
        st = static_scratch_address(&scratch);
        if (st) return st;
        // the copy overwrites every scratch element this call reads
        st = cw ? zmajor_copy(vol, scratch, g->grid, s) : transpose_xy(vol, scratch, g->grid, s);
        if (st) return st;
    }
    CBParams<float> p;            // on the host stack: no allocation of any kind
    fill_cb_params(p, g, flags);
    p.vol = vol;
    p.volT = scratch;
    p.out = sino;
    for (int v0 = 0; v0 < g->nv; v0 += ViewTable<float>::kMax) {
        const int nvc = std::min(ViewTable<float>::kMax, g->nv - v0);
        fill_views(p, g, v0, nvc);
        const cudaError_t e = cb_launch_forward<float>(p, g->na, g->nb, nvc, flags, s, cw);
        if (e != cudaSuccess) return cuda_fail(e, "cb_forward_kernel (noalloc)");
    }
    return NEFCT_OK;
}

}  // namespace nefct

using namespace nefct;

extern "C" {

size_t nefct_cb_workspace_bytes(const nefct_cb_geom *g, uint32_t flags)
{
    if (!g || g->grid.nx < 1 || g->grid.ny < 1 || g->grid.nz < 1) return 0;
    if (flags & NEFCT_DETERMINISTIC) return cb_fixed_workspace(g, flags);
    if (flags & NEFCT_NO_TRANSPOSE) return 0;
    return (size_t)(g->grid.nx > 0 ? g->grid.nx : 0) * (size_t)(g->grid.ny > 0 ? g->grid.ny : 0) *
           (size_t)(g->grid.nz > 0 ? g->grid.nz : 0) * sizeof(float);
}

nefct_status nefct_cb_forward(const nefct_cb_geom *g, const float *vol, float *sino, uint32_t flags,
                              void *ws, size_t wsb, void *stream)
{
    return cb_forward_impl<float>(g, vol, sino, flags, ws, wsb, (cudaStream_t)stream);
}

nefct_status nefct_cb_backward(const nefct_cb_geom *g, const float *sino, float *vol, uint32_t flags,
                               void *ws, size_t wsb, void *stream)
{
    return cb_backward_impl<float>(g, sino, vol, flags, ws, wsb, (cudaStream_t)stream);
}

nefct_status nefct_cb_forward_f64(const nefct_cb_geom *g, const double *vol, double *sino, uint32_t flags,
                                  void *ws, size_t wsb, void *stream)
{
    return cb_forward_impl<double>(g, vol, sino, flags, ws, wsb, (cudaStream_t)stream);
}

nefct_status nefct_cb_backward_f64(const nefct_cb_geom *g, const double *sino, double *vol, uint32_t flags,
                                   void *ws, size_t wsb, void *stream)
{
    return cb_backward_impl<double>(g, sino, vol, flags, ws, wsb, (cudaStream_t)stream);
}

nefct_status nefct_cb_count_intersections(const nefct_cb_geom *g, uint32_t flags, unsigned long long *count,
                                          void *stream)
{
    nefct_status st = check_cb_geom(g);
    if (st) return st;
    if (!count) return fail(NEFCT_ERR_INVALID, "count is NULL");
    if (flags & ~kWalkFlags) return fail(NEFCT_ERR_INVALID, "unknown flag bits 0x%x", flags & ~kWalkFlags);
    CBParams<float> *p = new CBParams<float>();
    fill_cb_params(*p, g, flags);
    p->count = count;
    const int kMax = ViewTable<float>::kMax;
    for (int v0 = 0; v0 < g->nv; v0 += kMax) {
        const int nvc = std::min(kMax, g->nv - v0);
        fill_views(*p, g, v0, nvc);
        dim3 grid, block;
        cb_shape(*p, g->na, g->nb, nvc, grid, block);
        if (cubic(p->g)) cb_count_kernel<false><<<grid, block, 0, (cudaStream_t)stream>>>(*p);
        else cb_count_kernel<true><<<grid, block, 0, (cudaStream_t)stream>>>(*p);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) { delete p; return cuda_fail(e, "cb_count_kernel"); }
    }
    delete p;
    return NEFCT_OK;
}

nefct_status nefct_lor_forward(const nefct_grid *grid, const float *lors, int64_t n, const float *vol,
                               float *out, uint32_t flags, void *stream)
{
    return lor_impl(grid, lors, n, vol, out, flags, (cudaStream_t)stream, true);
}

nefct_status nefct_lor_backward(const nefct_grid *grid, const float *lors, int64_t n, const float *vals,
                                float *vol, uint32_t flags, void *stream)
{
    return lor_impl(grid, lors, n, vals, vol, flags, (cudaStream_t)stream, false);
}

nefct_status nefct_lor_order_keys(const nefct_grid *grid, const float *lors, int64_t n, int32_t *keys, void *stream)
{
    if (!grid) return fail(NEFCT_ERR_INVALID, "grid is NULL");
    nefct_status st = check_grid(*grid);
    if (st) return st;
    if (n < 0 || n >= (1ll << 31)) return fail(NEFCT_ERR_INVALID, "line count must be in [0, 2^31)");
    if (n == 0) return NEFCT_OK;
    if (!lors || !keys) return fail(NEFCT_ERR_INVALID, "NULL buffer");
    LorParams p{};
    p.g = make_grid_dev<float>(*grid);
    p.lors = lors;
    p.n = n;
    const long long blocks = std::min<long long>((n + 255) / 256, 148ll * 64);
    lor_key_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(p, keys);
    NEFCT_CHECK_LAUNCH("lor_key_kernel");
    return NEFCT_OK;
}

nefct_status nefct_lor_forward_ordered(const nefct_grid *grid, const float *lors, int64_t n, const int32_t *order,
                                       const float *vol, float *out, uint32_t flags, void *stream)
{
    if (!order && n > 0) return fail(NEFCT_ERR_INVALID, "order is NULL");
    return lor_impl(grid, lors, n, vol, out, flags, (cudaStream_t)stream, true, order);
}

nefct_status nefct_lor_backward_ordered(const nefct_grid *grid, const float *lors, int64_t n, const int32_t *order,
                                        const float *vals, float *vol, uint32_t flags, void *stream)
{
    if (!order && n > 0) return fail(NEFCT_ERR_INVALID, "order is NULL");
    return lor_impl(grid, lors, n, vals, vol, flags, (cudaStream_t)stream, false, order);
}

// See cb_forward_static_impl: the same kernels and result as
// nefct_cb_forward, with the scratch in the library's fixed device array
// instead of a caller workspace.
nefct_status nefct_cb_forward_noalloc(const nefct_cb_geom *g, const float *vol, float *sino, uint32_t flags,
                                      void *stream)
{
    return cb_forward_static_impl(g, vol, sino, flags, (cudaStream_t)stream);
}

}  // extern "C"
