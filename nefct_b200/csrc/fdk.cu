// FDK on sm_100a: cosine + Parker weighting with ramp filtering, and the
// voxel-driven bilinear backprojection with the FDK distance weight.
//
// Filter (mat_codes/filtering.m:5-48, ParkerWeight.m:5-27): the MATLAB code
// zero-pads each detector row to L = max(64, 2^nextpow2(2*nu)), multiplies
// its FFT by the windowed |FFT(ramp)|*2 and crops.  The device does the same
// with its own FFT: two weighted rows travel as the real and imaginary parts
// of one complex signal (the filter response H is real and even, so the two
// filtered rows come back as the real and imaginary parts of the inverse
// transform), forward transform, multiply by H/L, inverse transform as the
// conjugate of a forward transform of the conjugate.  The transforms are
// Stockham autosort FFTs of 16 elements per thread: two or three passes of
// radix 16 (the first of the forward and the last of the inverse of radix 2
// to 16, whichever makes up L) in registers, with the elements exchanged
// through shared memory between passes; the first pass reads the weighted rows
// from global memory and the last writes the filtered rows.  H is built on the
// host in FP64 (radix-2 FFT below) with the MATLAB scale folded in.
//
// Backprojection (nefct/cc/pixel_3d/pixel.cu.cc:12-146 geometry and index
// rules, Q9-Q11, times (src_iso/(src_iso + x'))^2 from
// mat_codes/backprojection.m:12): one thread owns a column of kZ voxels
// along z; per view it computes the column's rotated position, detector
// column and magnification once and then the kZ row taps (one fused
// multiply-add, an exact floor and four gathers per voxel and view).  Views are
// processed in chunks so a chunk's filtered projections stay in L2.  A
// warp covers an 8 x 4 tile of (x, y) voxel columns.
#include <limits.h>
#include <math.h>
#include <algorithm>
#include <complex>
#include <vector>

#include "common.cuh"

namespace nefct {

nefct_status check_cb_geom(const nefct_cb_geom *g);

// ---------------- host: spatial ramp kernel ----------------

static void fft_inplace(std::vector<std::complex<double>> &a, bool inverse)
{
    const size_t n = a.size();
    for (size_t i = 1, j = 0; i < n; ++i) {
        size_t bit = n >> 1;
        for (; j & bit; bit >>= 1) j ^= bit;
        j ^= bit;
        if (i < j) std::swap(a[i], a[j]);
    }
    for (size_t len = 2; len <= n; len <<= 1) {
        const double ang = 2.0 * M_PI / (double)len * (inverse ? 1.0 : -1.0);
        const std::complex<double> wl(cos(ang), sin(ang));
        for (size_t i = 0; i < n; i += len) {
            std::complex<double> w(1.0, 0.0);
            for (size_t k = 0; k < len / 2; ++k) {
                const std::complex<double> u = a[i + k], v = a[i + k + len / 2] * w;
                a[i + k] = u + v;
                a[i + k + len / 2] = u - v;
                w *= wl;
            }
        }
    }
    if (inverse)
        for (auto &x : a) x /= (double)n;
}

// Transform length of filtering.m: L = max(64, 2^nextpow2(2*nu)).
static int ramp_length(int na)
{
    int p = 0;
    while ((1 << p) < 2 * na) ++p;
    return std::max(64, 1 << p);
}

// H[k] * scale / L for k = 0..L/2 (H[L - k] = H[k]): the windowed filter
// response of filtering.m:54-88 with its scale and the inverse transform's
// 1/L folded in.
static std::vector<float> ramp_response(int na, int window, double scale)
{
    const int L = ramp_length(na);
    // ramp_flat (filtering.m:54-60): nn = -L/2..L/2-1, 1/4 at 0, -1/(pi nn)^2 at odd nn
    std::vector<std::complex<double>> r(L);
    for (int i = 0; i < L; ++i) {
        const int nn = i - L / 2;
        double v = 0.0;
        if (nn == 0) v = 0.25;
        else if (nn & 1) v = -1.0 / ((M_PI * nn) * (M_PI * nn));
        r[i] = v;
    }
    fft_inplace(r, false);
    // Filter (:63-88): 2|FFT|, window on bins 1..L/2 (mirrored to length L)
    std::vector<float> h(L / 2 + 1);
    for (int k = 0; k <= L / 2; ++k) {
        double f = 2.0 * std::abs(r[k]);
        const double w = 2.0 * M_PI * k / L;
        if (k >= 1) {
            switch (window) {
            case NEFCT_WIN_SHEPP_LOGAN: f *= sin(w / 2.0) / (w / 2.0); break;
            case NEFCT_WIN_COSINE: f *= cos(w / 2.0); break;
            case NEFCT_WIN_HAMMING: f *= 0.54 + 0.46 * cos(w); break;
            case NEFCT_WIN_HANN: f *= (1.0 + cos(w)) / 2.0; break;
            default: break;
            }
        }
        if (w > M_PI) f = 0.0;
        h[k] = (float)(f * scale / L);
    }
    return h;
}

// ---------------- device: weighting + FFT filtering ----------------

static constexpr int kMaxCols = 2048;            // detector columns the filter supports
static constexpr int kMaxL = 4096;               // ramp_length(kMaxCols)

struct FilterParams {
    int na, nb, nv, L, log2L, pairs_per_view, pairs;
    float src_det, da, a_shift, db, b_shift;    // cosine weight (FP32)
    double src_det_d, da_d, a_shift_d;          // Parker weight (FP64, as ParkerWeight.m)
    int parker;                                 // 0 off, +1/-1 = ParkerWeight dir
    double dang;                                // view step, degrees
    double fanang;                              // ParkerWeight's fanang (half the fan angle), degrees
    float h[kMaxL / 2 + 1];                     // H[k] * scale / L, k = 0..L/2
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// (-i) * a
__device__ __forceinline__ float2 cmul_mi(float2 a) { return make_float2(a.y, -a.x); }

// Cosine weight of filtering.m:10, DSD / sqrt(DSD^2 + v^2 + u^2), from the
// row's part c = DSD^2 + v^2 (cos_row) and the column (FP32 with rsqrt: a
// few ulp, against the FP64 of the MATLAB code).
__device__ __forceinline__ float cos_row(const FilterParams &p, int row)
{
    const float v = __fsub_rn(__fmul_rn((float)row + p.b_shift, p.db), __fmul_rn((float)p.nb, p.db) * 0.5f);
    return __fadd_rn(__fmul_rn(p.src_det, p.src_det), __fmul_rn(v, v));
}
__device__ __forceinline__ float cos_weight(const FilterParams &p, float c, int col)
{
    const float u = __fsub_rn(__fmul_rn((float)col + p.a_shift, p.da), __fmul_rn((float)p.na, p.da) * 0.5f);
    return p.src_det * rsqrtf(__fadd_rn(c, __fmul_rn(u, u)));
}

// Parker weight of detector column col at view iv, ParkerWeight.m:5-25
// (1-based views there), in FP64 as the MATLAB code.
__device__ __forceinline__ float parker_weight(const FilterParams &p, int iv, int col)
{
    const double ud = ((double)col + p.a_shift_d) * p.da_d - (double)p.na * p.da_d / 2.0;
    const double as = atan(ud / p.src_det_d) / M_PI * 180.0;
    const double f = p.fanang;
    const double n180 = 180.0 / p.dang;
    const double pw = ((n180 - p.nv) / 2.0 + (iv + 1)) / n180 * 180.0 + p.parker * as;
    double pk = 1.0;
    if (pw <= f / 2 && pw > -f / 2) {
        const double sn = fmax(sin(M_PI / 2 * (f / 2 + pw) / f), 0.0);
        pk = sn * sn;
    }
    if (pw >= 180 - f / 2 && pw < 180 + f / 2) {
        const double c = fmax(cos(M_PI / 2 * (f / 2 + pw - 180) / f), 0.0);
        pk *= c * c;
    }
    if (pw < -f / 2 || pw > 180 + f / 2) pk = 0.0;
    return (float)pk;
}

// exp(-2 pi i n / 16), n = 0..9 (the powers that the radix-16 butterfly uses).
static __constant__ float2 kRoot16[10] = {
    {1.f, 0.f}, {0.923879532511286756f, -0.382683432365089772f}, {0.707106781186547524f, -0.707106781186547524f},
    {0.382683432365089772f, -0.923879532511286756f}, {0.f, -1.f}, {-0.382683432365089772f, -0.923879532511286756f},
    {-0.707106781186547524f, -0.707106781186547524f}, {-0.923879532511286756f, -0.382683432365089772f}, {-1.f, 0.f},
    {-0.923879532511286756f, 0.382683432365089772f}};

template <int N> __device__ __forceinline__ float2 mul_root16(float2 a)
{
    constexpr float h = 0.707106781186547524f;
    if constexpr (N == 0) return a;
    else if constexpr (N == 2) return make_float2((a.x + a.y) * h, (a.y - a.x) * h);
    else if constexpr (N == 4) return cmul_mi(a);
    else if constexpr (N == 6) return make_float2((a.y - a.x) * h, (a.x + a.y) * -h);
    else return cmul(a, kRoot16[N]);
}

// DFT of four values in place.  ZIN: c and d are zero; LOW: only the outputs a
// and b are wanted.
template <bool ZIN, bool LOW> __device__ __forceinline__ void dft4(float2 &a, float2 &b, float2 &c, float2 &d)
{
    const float2 t0 = ZIN ? a : cadd(a, c), t1 = ZIN ? a : csub(a, c);
    const float2 t2 = ZIN ? b : cadd(b, d), t3 = cmul_mi(ZIN ? b : csub(b, d));
    a = cadd(t0, t2);
    b = cadd(t1, t3);
    if (!LOW) {
        c = csub(t0, t2);
        d = csub(t1, t3);
    }
}

// DFT of the R values x[m] = a[I + m S], S = 16 / R, in place.  ZIN: the upper
// half of the inputs is zero; LOW: only the lower half of the outputs is wanted.
template <int R, int I, bool ZIN, bool LOW> __device__ __forceinline__ void dft(float2 (&a)[16])
{
    constexpr int S = 16 / R;
    if constexpr (R == 2) {
        const float2 x = a[I], y = a[I + S];
        a[I] = ZIN ? x : cadd(x, y);
        if (!LOW) a[I + S] = ZIN ? x : csub(x, y);
    } else if constexpr (R == 4) {
        dft4<ZIN, LOW>(a[I], a[I + S], a[I + 2 * S], a[I + 3 * S]);
    } else if constexpr (R == 8) {
        // x[q + 2 s]: radix 4 over s, then radix 2 over q; output k1 + 4 k2
        dft4<ZIN, false>(a[I], a[I + 2 * S], a[I + 4 * S], a[I + 6 * S]);
        dft4<ZIN, false>(a[I + S], a[I + 3 * S], a[I + 5 * S], a[I + 7 * S]);
        const float2 y[4] = {a[I], a[I + 2 * S], a[I + 4 * S], a[I + 6 * S]};
        const float2 z[4] = {a[I + S], mul_root16<2>(a[I + 3 * S]), mul_root16<4>(a[I + 5 * S]),
                             mul_root16<6>(a[I + 7 * S])};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            a[I + k * S] = cadd(y[k], z[k]);
            if (!LOW) a[I + (k + 4) * S] = csub(y[k], z[k]);
        }
    } else {
        // x[q + 4 s]: radix 4 over s, then radix 4 over q; output k1 + 4 k2
        dft4<ZIN, false>(a[0], a[4], a[8], a[12]);
        dft4<ZIN, false>(a[1], a[5], a[9], a[13]);
        dft4<ZIN, false>(a[2], a[6], a[10], a[14]);
        dft4<ZIN, false>(a[3], a[7], a[11], a[15]);
        a[5] = mul_root16<1>(a[5]);
        a[9] = mul_root16<2>(a[9]);
        a[13] = mul_root16<3>(a[13]);
        a[6] = mul_root16<2>(a[6]);
        a[10] = mul_root16<4>(a[10]);
        a[14] = mul_root16<6>(a[14]);
        a[7] = mul_root16<3>(a[7]);
        a[11] = mul_root16<6>(a[11]);
        a[15] = mul_root16<9>(a[15]);
#pragma unroll
        for (int k = 0; k < 16; k += 4) dft4<false, LOW>(a[k], a[k + 1], a[k + 2], a[k + 3]);
        // a[4 k1 + k2] is output k1 + 4 k2
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
            for (int k2 = k1 + 1; k2 < 4; ++k2) {
                const float2 t = a[4 * k1 + k2];
                a[4 * k1 + k2] = a[4 * k2 + k1];
                a[4 * k2 + k1] = t;
            }
    }
}

// Every radix-R butterfly of a thread's 16 elements.
template <int R, bool ZIN, bool LOW, int I = 0> __device__ __forceinline__ void dft_all(float2 (&a)[16])
{
    dft<R, I, ZIN, LOW>(a);
    if constexpr (I + 1 < 16 / R) dft_all<R, ZIN, LOW, I + 1>(a);
}

// Twiddle factors of a radix-R pass with Ns points per finished sub-transform:
// W^(r k), W = exp(-2 pi i / (R Ns)), at [(r - 1) Ns + k], r = 1..R - 1, k < Ns.
// (Products of the powers 1, 2, 3, 4, 8 and 12 in place of the others took the
// same time, with 10 % more rounding error.)
template <int R, int Ns> __device__ __forceinline__ void tw_fill(float2 *tw)
{
    for (int i = threadIdx.x; i < (R - 1) * Ns; i += blockDim.x) {
        const int row = i / Ns, k = i - row * Ns;
        float sn, cs;
        sincospif((float)((row + 1) * k) / (float)(R * Ns / 2), &sn, &cs);    // exact argument (power-of-two denominator)
        tw[i] = make_float2(cs, -sn);
    }
}

// a[i + r S] (element j + r L / R, S = 16 / R, j = t + i T) times W^(r k),
// k = j mod Ns.
template <int R, int Ns, int T> __device__ __forceinline__ void tw_apply(const float2 *tw, int t, float2 (&a)[16])
{
    constexpr int S = 16 / R;
#pragma unroll
    for (int i = 0; i < S; ++i) {
        const int k = (t + i * T) & (Ns - 1);
#pragma unroll
        for (int r = 1; r < R; ++r) a[i + r * S] = cmul(a[i + r * S], tw[(r - 1) * Ns + k]);
    }
}

// The transforms of length L = 2^LOG2L: T threads of 16 elements each, thread t
// holding elements t + m T (m = 0..15) before and after every pass.  The
// forward's passes have the radices C, 16 (, 16), the inverse's 16 (, 16), C.
template <int LOG2L> struct Fft {
    static constexpr int L = 1 << LOG2L, T = L / 16;
    static constexpr bool three = LOG2L > 8;
    static constexpr int C = three ? L / 256 : L / 16;
    static constexpr int threads = 256, groups = threads / T;
    // one element of padding per 16: the strided writes of an exchange (16
    // elements 2 to 16 apart, or rows of Ns consecutive ones 16 Ns apart) and the
    // consecutive reads are free of bank conflicts
    static constexpr int buffer = L + L / 16;
    // twiddle tables: forward's second and third pass, inverse's second and third
    static constexpr int f2 = 0, f3 = f2 + 15 * C, i2 = three ? f3 + 15 * 16 * C : f3;
    static constexpr int i3 = three ? i2 + 15 * 16 : i2, tables = i3 + (C - 1) * (L / C);
    static constexpr size_t smem = (size_t)(groups * buffer + tables) * sizeof(float2) + (L / 2 + 4) * sizeof(float);

    static __device__ __forceinline__ int pad(int e) { return e + (e >> 4); }

    // Barrier of the T threads of a transform (T < 32: within a warp).
    static __device__ __forceinline__ void sync(int group)
    {
        if constexpr (T <= 32) __syncwarp();
        else if constexpr (T == threads) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(T) : "memory");
    }

    // Writes the outputs of a radix-R pass with Ns points per finished
    // sub-transform and reads the next pass's inputs.
    template <int R, int Ns> static __device__ __forceinline__ void exchange(float2 *buf, int t, int group, float2 (&a)[16])
    {
        constexpr int S = 16 / R;
        sync(group);                          // the last exchange's reads are done
#pragma unroll
        for (int i = 0; i < S; ++i) {
            const int j = t + i * T, k = j & (Ns - 1), o = (j - k) * R + k;
#pragma unroll
            for (int r = 0; r < R; ++r) buf[pad(o + r * Ns)] = a[i + r * S];
        }
        sync(group);
#pragma unroll
        for (int m = 0; m < 16; ++m) a[m] = buf[pad(t + m * T)];
    }

    // Elements m >= 8 are zero on entry.
    static __device__ __forceinline__ void forward(float2 *buf, const float2 *tw, int t, int group, float2 (&a)[16])
    {
        dft_all<C, true, false>(a);
        exchange<C, 1>(buf, t, group, a);
        tw_apply<16, C, T>(tw + f2, t, a);
        dft_all<16, false, false>(a);
        if constexpr (three) {
            exchange<16, C>(buf, t, group, a);
            tw_apply<16, 16 * C, T>(tw + f3, t, a);
            dft_all<16, false, false>(a);
        }
    }

    // A forward transform too; only the elements m < 8 are wanted.
    static __device__ __forceinline__ void inverse(float2 *buf, const float2 *tw, int t, int group, float2 (&a)[16])
    {
        dft_all<16, false, false>(a);
        exchange<16, 1>(buf, t, group, a);
        if constexpr (three) {
            tw_apply<16, 16, T>(tw + i2, t, a);
            dft_all<16, false, false>(a);
            exchange<16, 16>(buf, t, group, a);
        }
        tw_apply<C, L / C, T>(tw + i3, t, a);
        dft_all<C, false, true>(a);
    }
};

// Persistent CTAs; T threads take consecutive row pairs (view iv, rows b and
// b + 1), so the Parker weights of a thread's columns, FP64 with an arc tangent
// and a sine or cosine each, are evaluated once per view it meets instead of
// once per pair.
//
// What bounds it: the shared-memory pipe (about 70 % of its wavefronts: four
// exchanges and three passes of twiddle factors per pair; a radix-4 FFT exchanges
// nine times at L = 1024).  300 views of 500 x 300: 327 -> 195 us (the rows cross
// memory in 55); 200 views of 1000 x 300: 512 -> 270 us; 100 views of 2048 x 300:
// 1009 -> 312 us; 1000 views of 120 x 200: 323 -> 77 us; 211 views of 389 x 283
// with Parker weights: 275 -> 140 us.  At most 85 registers, three CTAs per SM:
// 0.304 ms for 360 views of 512 x 384, against 0.322 with two; CTAs of 64 or 128
// threads as fast.
template <int LOG2L, bool PARKER>
__global__ void __launch_bounds__(256, LOG2L < 12 ? 3 : 2) fdk_filter_kernel(const __grid_constant__ FilterParams p,
                                                            const float *__restrict__ sino, float *__restrict__ out)
{
    using F = Fft<LOG2L>;
    extern __shared__ __align__(16) float2 fsm[];
    float2 *const tw = fsm + F::groups * F::buffer;
    float *const hs = reinterpret_cast<float *>(tw + F::tables);
    tw_fill<16, F::C>(tw + F::f2);
    if constexpr (F::three) {
        tw_fill<16, 16 * F::C>(tw + F::f3);
        tw_fill<16, 16>(tw + F::i2);
    }
    tw_fill<F::C, F::L / F::C>(tw + F::i3);
    for (int k = threadIdx.x; k <= F::L / 2; k += blockDim.x) hs[k] = p.h[k];
    __syncthreads();
    const int na = p.na, group = threadIdx.x / F::T, t = threadIdx.x % F::T;
    float2 *const buf = fsm + group * F::buffer;
    const int gid = blockIdx.x * F::groups + group, ngroups = gridDim.x * F::groups;
    // every group takes as many steps as the longest (barriers): the last ones of some do nothing
    const int per = (p.pairs + ngroups - 1) / ngroups;
    float pk[PARKER ? 8 : 1];
    int pk_view = -1;
    for (int s = 0; s < per; ++s) {
        const long long pair = (long long)gid * per + s;
        const bool has = pair < p.pairs;
        const int pr = has ? (int)pair : 0;
        const int iv = pr / p.pairs_per_view;
        const int row = 2 * (pr - iv * p.pairs_per_view);
        const bool two = row + 1 < p.nb;
        const float *const x0 = sino + ((size_t)iv * p.nb + row) * na, *const x1 = x0 + na;
        // the weighted pair, zero beyond na (na <= L/2: m < 8)
        float2 a[16];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int e = t + m * F::T;
            const bool in = has && e < na;
            a[m] = make_float2(in ? __ldg(x0 + e) : 0.f, in && two ? __ldg(x1 + e) : 0.f);
        }
        if (PARKER && iv != pk_view) {
            pk_view = iv;
#pragma unroll 1
            for (int m = 0; m < 8; ++m) {
                const float w = parker_weight(p, iv, t + m * F::T);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (i == m) pk[PARKER ? i : 0] = w;
            }
        }
        const float c0 = cos_row(p, row), c1 = cos_row(p, row + 1);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int e = t + m * F::T;
            const float w0 = cos_weight(p, c0, e), w1 = cos_weight(p, c1, e);
            a[m].x *= PARKER ? w0 * pk[PARKER ? m : 0] : w0;
            a[m].y *= PARKER ? w1 * pk[PARKER ? m : 0] : w1;
        }
        F::forward(buf, tw, t, group, a);
        // conj(Z H / L): the real and imaginary parts of the conjugate of its
        // forward transform are the filtered rows
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const int e = t + m * F::T;
            const float h = hs[m < 8 ? e : F::L - e];
            a[m] = make_float2(a[m].x * h, -(a[m].y * h));
        }
        F::inverse(buf, tw, t, group, a);
        float *const y0 = out + ((size_t)iv * p.nb + row) * na, *const y1 = y0 + na;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int e = t + m * F::T;
            if (!has || e >= na) continue;
            y0[e] = a[m].x;
            if (two) y1[e] = -a[m].y;
        }
    }
}

// Launches the filter for transform length 2^LOG2L.
template <int LOG2L, bool PARKER>
static cudaError_t launch_filter(const FilterParams &p, const float *sino, float *out, cudaStream_t s)
{
    using F = Fft<LOG2L>;
    const auto kernel = fdk_filter_kernel<LOG2L, PARKER>;
    if (F::smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::smem);
        if (e != cudaSuccess) return e;
    }
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, F::threads, F::smem);
    const int blocks = std::min((p.pairs + F::groups - 1) / F::groups, sms * std::max(per_sm, 1));
    kernel<<<blocks, F::threads, F::smem, s>>>(p, sino, out);
    return cudaGetLastError();
}

template <int LOG2L>
static cudaError_t launch_filter(const FilterParams &p, const float *sino, float *out, cudaStream_t s)
{
    return p.parker ? launch_filter<LOG2L, true>(p, sino, out, s) : launch_filter<LOG2L, false>(p, sino, out, s);
}

// ---------------- device: voxel-driven backprojection ----------------

// Voxels along z per thread: the column part of a view is computed once per
// kZ voxels (measured at 256^3 x 360 views: 2 -> 11.1 ms, 4 -> 8.68 ms,
// 8 -> 8.27 ms, 12 -> 8.47 ms, 16 -> 10.4 ms; 8 fits the 64 registers that
// eight CTAs per SM leave, more spill or shrink the resident warps).
#ifndef NEFCT_FDK_KZ
#define NEFCT_FDK_KZ 8
#endif
static constexpr int kZ = NEFCT_FDK_KZ;
// Views per launch: as many as fit ~400 MB of a chunk (tap quads: 16 bytes
// per detector cell), 8 to 128.  Fewer launches mean fewer read-modify-write
// passes over the volume and fewer launch tails; that outweighs keeping the
// chunk L2-resident (256^3, 360 views of 512 x 384 with quads: 17 / 32 / 64
// / 128 views per launch take 7.56 / 7.26 / 7.07 / 6.98 ms).
static constexpr int kViewChunk = 128;
static inline int fdk_view_chunk(int na, int nb, size_t bytes_per_cell = sizeof(float))
{
    const double per_view = (double)na * nb * bytes_per_cell;
    return (int)std::min<double>(kViewChunk, std::max<double>(8.0, (double)(400 << 20) / per_view));
}

// Tap quads: for a chunk of views, quad[(v * nb + ib) * na + ia] holds the
// four bilinear taps of detector cell (ia, ib) -- (ia, ib), (ia + 1, ib),
// (ia, ib + 1), (ia + 1, ib + 1) -- so the backprojection reads them with one
// 16-byte load instead of four.  Cells of the last row / column (which the
// backprojection never reads as a quad's origin, Q11) hold zeros.  A thread
// takes kQuadRows cells of one column and reads each row once; bound by the
// memory (20 bytes per cell): 128 views of 512 x 384 in 80 us (6.3 TB/s); a cell
// per thread at a flat index, with its two divisions, took 114 us.
static constexpr int kQuadRows = 4;
__global__ void __launch_bounds__(256) fdk_quad_kernel(const float *__restrict__ sino, float4 *__restrict__ quad,
                                                       int na, int nb)
{
    const int tiles_a = (na + 63) / 64, tile = blockIdx.x / tiles_a;
    const int ia = (blockIdx.x - tile * tiles_a) * 64 + threadIdx.x, ib0 = (tile * 4 + threadIdx.y) * kQuadRows;
    if (ia >= na || ib0 >= nb) return;
    const size_t cell = ((size_t)blockIdx.y * nb + ib0) * na + ia;
    const float *const s = sino + cell;
    float lo[kQuadRows + 1], hi[kQuadRows + 1];
#pragma unroll
    for (int i = 0; i <= kQuadRows; ++i) {
        const bool in = ib0 + i < nb && ia + 1 < na;
        lo[i] = in ? __ldg(s + (size_t)i * na) : 0.f;
        hi[i] = in ? __ldg(s + (size_t)i * na + 1) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < kQuadRows; ++i) {
        if (ib0 + i >= nb) break;
        const bool in = ib0 + i + 1 < nb;
        quad[cell + (size_t)i * na] = in ? make_float4(lo[i], hi[i], lo[i + 1], hi[i + 1]) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// A warp owns an 8 x 4 (x, y) tile of voxel columns: at any view its
// voxels project onto fewer detector columns than a 32 x 1 row (whose
// detector footprint reaches ~50 columns), so its gathers touch fewer
// sectors (measured 7 % faster than 32 x 1 and 16 x 2, 1 % than 4 x 8).
// Eight lanes, which a 16-byte load serves at a time, own a 2 x 4 block of it
// (an 8 x 1 row: 6.29 against 6.06 ms at 256^3 x 360 views).
static constexpr int kTW = 8;

// Voxel centres held in the kernel parameters (x, then y, then z) when the
// three axes together have at most this many voxels.
static constexpr int kCtrMax = 6144;

struct BpParams {
    int nx, ny, nz, na, nb, nv0, nvc, first;
    float sx, sy, sz, corner_x, corner_y, corner_z;
    float src_iso, src_det, da, ai_p, db, bi_p;
    float inv_da, inv_db, cb;         // 1/da, 1/db and nb/2 - bi_p - 0.5, rounded to float
    int cyl, weight;
    float cs[kViewChunk], sn[kViewChunk];
    int has_ctr;                      // ctr holds every voxel centre (else computed per thread)
    float ctr[kCtrMax];
};

// What bounds it: the L1's data path (91 % of its wavefronts, eight per
// 16-byte gather of a warp instead of the four its bytes fill).  256^3, 360
// views of 512 x 384: 5.93 ms with the repacks and the edge pass (6.06 with the
// repacks at two thirds of their present rate), against 6.98 ms with the row test
// and the clamped row on every voxel and no bound on the registers.  Two 8-byte
// tap pairs in place of the quads: 6.10 against 6.06 ms.
//
// Per view the column part (rotation, magnification m, detector column a,
// its bilinear weights, the distance weight) follows the reference's
// operations with its divisions replaced by one approximate reciprocal of
// the source distance (a few ulp; every weight is continuous in it);
// (double)(t - ai) - 0.5 rounded to float equals the float subtraction
// t - ai - 0.5f exactly (the double difference is exact), so no FP64 is
// needed.  Per voxel the detector row is b = (m/db) * z + (nb/2 -
// bi - 0.5) by one fused multiply-add (the reference's (m*z)/db + nb/2 - bi
// - 0.5 rounds four times; the two differ by a few ulp of b, which moves the
// bilinear weights continuously) and floored exactly by the magic-constant
// sum (floor(b) + 1.5*2^23 = round-down(b + 1.5*2^23), valid for |b| < 2^22).
// When |m/db| * max|z| + |nb/2 - bi - 0.5| could reach 2^21 (a voxel at or
// near the source plane has an infinite or NaN b) the thread clamps b to
// [-2, nb + 1] first.  The distance weight is folded into the column
// weights (wa u, wa2 u) once per view.  Every operation is written with its
// rounding (no contraction left to the compiler), so fdk_edge_kernel
// recomputes the same values.
// QUAD: the taps come from the chunk's tap quads (fdk_quad_kernel) with one
// 16-byte load; the arithmetic is the same, so are the results, bit for bit.

// Column part of one view for the voxel column at (xc, yc): bp_column the
// detector column (a, ia) and the magnification, bp_weights (for a column
// that is kept) the row slope bm and the column weights.
struct BpColumn {
    float a, bm, wau, wa2u;
    float inv, m;
    int ia;
};

__device__ __forceinline__ void bp_column(const BpParams &p, float cphi, float sphi, float xc, float yc, BpColumn &c)
{
    const float xc0 = __fmaf_rn(xc, cphi, __fmul_rn(yc, sphi));
    const float yc0 = __fmaf_rn(-xc, sphi, __fmul_rn(yc, cphi));
    const float nah = (float)(p.na / 2);                   // integer half (Q9)
    // 1 / (xc0 - xs) = 1 / (src_iso + xc0): magnification and distance weight share it
    c.inv = rcp_approx(__fadd_rn(xc0, p.src_iso));
    c.m = __fmul_rn(p.src_det, c.inv);                     // SAD / (xc0 - xs)
    float t;
    if (p.cyl) t = __fmaf_rn(atan2f(yc0, __fadd_rn(xc0, p.src_iso)), p.inv_da, nah);
    else t = __fmaf_rn(__fmul_rn(c.m, yc0), p.inv_da, nah);
    c.a = __fsub_rn(__fsub_rn(t, p.ai_p), 0.5f);
    c.ia = __float2int_rd(c.a);
}

__device__ __forceinline__ void bp_weights(const BpParams &p, BpColumn &c)
{
    c.bm = __fmul_rn(c.m, p.inv_db);
    float u = 1.f;
    if (p.weight) {
        const float r = __fmul_rn(p.src_iso, c.inv);
        u = __fmul_rn(r, r);
    }
    const float wa2 = __fsub_rn(c.a, (float)c.ia), wa = __fsub_rn(1.f, wa2);
    c.wau = __fmul_rn(wa, u);
    c.wa2u = __fmul_rn(wa2, u);
}

// Voxel centre along one axis, pixel.cu.cc:116-118 ((i + 0.5) * s / n + c, in double).
__host__ __device__ __forceinline__ float bp_centre(int i, float s, int n, float c)
{
    return (float)((i + 0.5) * (double)s / n + (double)c);
}
// The same from the host-filled table (the host's double arithmetic gives
// the same values), saving each thread its double divisions per launch.
__device__ __forceinline__ float bp_cx(const BpParams &p, int i)
{
    return p.has_ctr ? p.ctr[i] : bp_centre(i, p.sx, p.nx, p.corner_x);
}
__device__ __forceinline__ float bp_cy(const BpParams &p, int i)
{
    return p.has_ctr ? p.ctr[p.nx + i] : bp_centre(i, p.sy, p.ny, p.corner_y);
}
__device__ __forceinline__ float bp_cz(const BpParams &p, int i)
{
    return p.has_ctr ? p.ctr[p.nx + p.ny + i] : bp_centre(i, p.sz, p.nz, p.corner_z);
}

// Contribution of one voxel at detector row b from the column's taps:
// false when Q11 drops it (ib < 0 || ib + 1 >= nb).
template <bool QUAD>
__device__ __forceinline__ bool bp_tap(const BpParams &p, const float *pv, const float4 *pq, const BpColumn &c, float b,
                                       float &r0, float &r1, float &wb, float &wb2)
{
    const float mb = __fadd_rd(b, 12582912.0f);
    const unsigned ib = (unsigned)(__float_as_int(mb) - 0x4B400000);
    if (ib >= (unsigned)(p.nb - 1)) return false;
    wb2 = __fsub_rn(b, __fsub_rn(mb, 12582912.0f));
    wb = __fsub_rn(1.f, wb2);
    float t00, t01, t10, t11;
    if (QUAD) {
        const float4 q4 = __ldg(pq + (size_t)ib * p.na);
        t00 = q4.x; t01 = q4.y; t10 = q4.z; t11 = q4.w;
    } else {
        const float *q = pv + (size_t)ib * p.na;
        t00 = __ldg(q); t01 = __ldg(q + 1); t10 = __ldg(q + p.na); t11 = __ldg(q + p.na + 1);
    }
    r0 = __fmaf_rn(t01, c.wa2u, __fmul_rn(t00, c.wau));
    r1 = __fmaf_rn(t11, c.wa2u, __fmul_rn(t10, c.wau));
    return true;
}

template <bool QUAD>
__global__ void __launch_bounds__(128, 8) fdk_bp_kernel(const __grid_constant__ BpParams p,
                                                        const float *__restrict__ sino,
                                                        const float4 *__restrict__ quad, float *__restrict__ vol)
{
    const int lane = threadIdx.x;
    const int ix = blockIdx.x * kTW + (lane & 1) + (lane >> 3) * 2;
    const int iy = (blockIdx.y * 4 + threadIdx.y) * (32 / kTW) + ((lane >> 1) & 3);
    const int z0 = blockIdx.z * kZ;
    if (ix >= p.nx || iy >= p.ny) return;
    const float xc = bp_cx(p, ix);
    const float yc = bp_cy(p, iy);
    float zc[kZ], acc[kZ];
    const size_t plane = (size_t)p.nx * p.ny;
    const size_t col = (size_t)iy * p.nx + ix;
#pragma unroll
    for (int k = 0; k < kZ; ++k) {
        const int iz = z0 + k;
        zc[k] = bp_cz(p, min(iz, p.nz - 1));
        acc[k] = (!p.first && iz < p.nz) ? vol[iz * plane + col] : 0.f;
    }
    float zabs = 0.f;
#pragma unroll
    for (int k = 0; k < kZ; ++k) zabs = fmaxf(zabs, fabsf(zc[k]));
    const float bhi = (float)(p.nb + 1), brow = (float)(p.nb - 1);
    const unsigned pitch = (unsigned)p.na * (unsigned)(QUAD ? sizeof(float4) : sizeof(float));   // bytes per row
    for (int v = 0; v < p.nvc; ++v) {
        BpColumn c;
        bp_column(p, p.cs[v], p.sn[v], xc, yc, c);
        if (c.ia < 0 || c.ia + 1 >= p.na) continue;             // Q11
        bp_weights(p, c);
        const float *pv = sino + (size_t)v * p.na * p.nb + c.ia;
        const float4 *pq = QUAD ? quad + (size_t)v * p.na * p.nb + c.ia : nullptr;
        float r0, r1, wb, wb2;
        if (fabsf(c.bm) * zabs + fabsf(p.cb) < 2097152.f) {
            // rows are monotone in z: with the first and last voxel's row inside
            // the detector none is dropped
            const float b0 = __fmaf_rn(c.bm, zc[0], p.cb), b1 = __fmaf_rn(c.bm, zc[kZ - 1], p.cb);
            if (fminf(b0, b1) >= 0.f && fmaxf(b0, b1) < brow) {
                const char *const base = (QUAD ? (const char *)pq : (const char *)pv) - (size_t)0x4B400000u * pitch;
#pragma unroll
                for (int k = 0; k < kZ; ++k) {
                    const float b = __fmaf_rn(c.bm, zc[k], p.cb);
                    const float mb = __fadd_rd(b, 12582912.0f);
                    const float w2 = __fsub_rn(b, __fsub_rn(mb, 12582912.0f)), w1 = __fsub_rn(1.f, w2);
                    const char *const q = base + (unsigned long long)(unsigned)__float_as_int(mb) * pitch;
                    float t00, t01, t10, t11;
                    if (QUAD) {
                        const float4 q4 = __ldg((const float4 *)q);
                        t00 = q4.x; t01 = q4.y; t10 = q4.z; t11 = q4.w;
                    } else {
                        const float *const f = (const float *)q;
                        t00 = __ldg(f); t01 = __ldg(f + 1); t10 = __ldg(f + p.na); t11 = __ldg(f + p.na + 1);
                    }
                    const float a0 = __fmaf_rn(t01, c.wa2u, __fmul_rn(t00, c.wau));
                    const float a1 = __fmaf_rn(t11, c.wa2u, __fmul_rn(t10, c.wau));
                    acc[k] = __fmaf_rn(a1, w2, __fmaf_rn(a0, w1, acc[k]));
                }
                continue;
            }
#pragma unroll
            for (int k = 0; k < kZ; ++k) {
                // branch-free: a dropped row (Q11) reads row nb - 2's taps with
                // zero weights (adds +0: measured 2.6 % faster than skipping)
                const float b = __fmaf_rn(c.bm, zc[k], p.cb);
                const float mb = __fadd_rd(b, 12582912.0f);
                const unsigned ib = (unsigned)(__float_as_int(mb) - 0x4B400000);
                const bool keep = ib < (unsigned)(p.nb - 1);
                const unsigned ibc = keep ? ib : (unsigned)(p.nb - 2);
                const float w2 = __fsub_rn(b, __fsub_rn(mb, 12582912.0f));
                const float wb2k = keep ? w2 : 0.f, wbk = keep ? __fsub_rn(1.f, w2) : 0.f;
                float t00, t01, t10, t11;
                if (QUAD) {
                    const float4 q4 = __ldg(pq + (size_t)ibc * p.na);
                    t00 = q4.x; t01 = q4.y; t10 = q4.z; t11 = q4.w;
                } else {
                    const float *q = pv + (size_t)ibc * p.na;
                    t00 = __ldg(q); t01 = __ldg(q + 1); t10 = __ldg(q + p.na); t11 = __ldg(q + p.na + 1);
                }
                const float a0 = __fmaf_rn(t01, c.wa2u, __fmul_rn(t00, c.wau));
                const float a1 = __fmaf_rn(t11, c.wa2u, __fmul_rn(t10, c.wau));
                acc[k] = __fmaf_rn(a1, wb2k, __fmaf_rn(a0, wbk, acc[k]));
            }
        } else {
#pragma unroll
            for (int k = 0; k < kZ; ++k)
                if (bp_tap<QUAD>(p, pv, pq, c, fminf(fmaxf(__fmaf_rn(c.bm, zc[k], p.cb), -2.f), bhi), r0, r1, wb, wb2))
                    acc[k] = __fmaf_rn(r1, wb2, __fmaf_rn(r0, wb, acc[k]));
        }
    }
#pragma unroll
    for (int k = 0; k < kZ; ++k)
        if (z0 + k < p.nz) vol[(z0 + k) * plane + col] = acc[k];
}

// ---- detector-edge decisions with the reference's own operations ----
//
// The few-ulp differences above move the bilinear weights continuously
// everywhere except at the detector's edges, where the reference drops a
// voxel whose tap pair reaches past the last column or row, or starts before
// the first (Q11): there a row or column within ulps of the edge can be kept
// by one evaluation and dropped by the other.  For a flat detector,
// fdk_edge_kernel revisits, after fdk_bp_kernel, every (column, view) of the
// chunk whose detector column lies within `edge` of column 0 or na - 1, and
// every voxel whose row lies within `edge` of row 0 or nb - 1; it decides
// each with the reference's operations in order (pixel.cu.cc:24-33, no
// contraction: exact_col, exact_row) and takes a voxel the kernel kept and
// the reference drops out of the sum, or puts one the reference keeps in.

// pixel.cu.cc:24-29: the rotated voxel centre and the magnification
// SAD / (x' - xs) (xs = -src_iso).
__device__ __forceinline__ float exact_mag(const BpParams &p, float cphi, float sphi, float xc, float yc, float &yr)
{
    const float xr = __fadd_rn(__fmul_rn(xc, cphi), __fmul_rn(yc, sphi));
    yr = __fadd_rn(__fmul_rn(-xc, sphi), __fmul_rn(yc, cphi));
    return __fdiv_rn(p.src_det, __fadd_rn(xr, p.src_iso));
}

// pixel.cu.cc:30-32: a = yd / da + na / 2 - ai - 0.5 (the last subtraction
// in double, rounded to float: the same as the float subtraction).
__device__ __forceinline__ float exact_col(const BpParams &p, float cphi, float sphi, float xc, float yc)
{
    float yr;
    const float m = exact_mag(p, cphi, sphi, xc, yc, yr);
    return __fsub_rn(__fsub_rn(__fadd_rn(__fdiv_rn(__fmul_rn(m, yr), p.da), (float)(p.na / 2)), p.ai_p), 0.5f);
}

// pixel.cu.cc:28,31: b = (SAD / (x' - xs)) * z / db + nb / 2 - bi - 0.5.
__device__ __forceinline__ float exact_row(const BpParams &p, float cphi, float sphi, float xc, float yc, float zc)
{
    float yr;
    const float m = exact_mag(p, cphi, sphi, xc, yc, yr);
    return __fsub_rn(__fsub_rn(__fadd_rn(__fdiv_rn(__fmul_rn(m, zc), p.db), (float)(p.nb / 2)), p.bi_p), 0.5f);
}

// Column (row) decisions: kept when 0 <= floor(x) and floor(x) + 1 < n.
__device__ __forceinline__ bool bp_keep(float x, int n)
{
    const int i = __float2int_rd(x);
    return i >= 0 && i + 1 < n;
}

// One warp per voxel column; lane l takes views l, l + 32, ... of one table
// (up to kViewChunk views, after every chunk's backprojection) and finds, in
// parallel, the voxels whose decisions differ and the corrections; the
// corrections are then applied by one lane at a time in view order, so the
// result stays deterministic (and the same with and without tap quads: the
// taps are read from the filtered sinogram, which the quads copy).
static constexpr int kEdgeSlots = 4;

__global__ void __launch_bounds__(256) fdk_edge_kernel(const __grid_constant__ BpParams p,
                                                       const float *__restrict__ sino, float *vol)
{
    // the view table in shared memory: lanes read different views, which the
    // parameter bank would serve one address at a time
    __shared__ float s_cs[kViewChunk], s_sn[kViewChunk];
    for (int i = threadIdx.x; i < p.nvc; i += blockDim.x) {
        s_cs[i] = p.cs[i];
        s_sn[i] = p.sn[i];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long colid = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (colid >= (long long)p.nx * p.ny) return;           // uniform across the warp
    const int ix = (int)(colid % p.nx), iy = (int)(colid / p.nx);
    const float xc = bp_cx(p, ix);
    const float yc = bp_cy(p, iy);
    const float naf = (float)p.na, nbf = (float)p.nb;
    // Width of the bands decided again: the kernel's detector coordinate
    // differs from the reference's by a few ulp of terms of about half the
    // detector (rcp_approx and the fused row: <= ~8 ulp of max(na, nb), i.e.
    // under max(na, nb) * 2^-20); the band is 16x that plus 1/1024.  A
    // wider band only adds work (every voxel in it is decided twice).
    const float edge = 1.f / 1024 + fmaxf(naf, nbf) * (1.f / 65536);
    const size_t plane = (size_t)p.nx * p.ny;
    float *const vcol = vol + (size_t)iy * p.nx + ix;
    const float idz = (float)p.nz / p.sz;
    const float z_first = bp_cz(p, 0), z_last = bp_cz(p, p.nz - 1);
    for (int v0 = 0; v0 < p.nvc; v0 += 32) {
        const int v = v0 + lane;
        const bool has = v < p.nvc;
        const int vt = min(v, p.nvc - 1);                  // lanes past the table read its last entry
        const float cphi = s_cs[vt], sphi = s_sn[vt];
        BpColumn c, cr;
        bool col_ours = false, col_ref = false;
        if (has) {
            bp_column(p, cphi, sphi, xc, yc, c);
            bp_weights(p, c);
            col_ours = c.ia >= 0 && c.ia + 1 < p.na;
            col_ref = col_ours;
            cr = c;                           // the column as the reference places it
            if (!p.cyl && (fabsf(c.a) < edge || fabsf(c.a - (naf - 1.f)) < edge)) {
                cr.a = exact_col(p, cphi, sphi, xc, yc);
                cr.ia = __float2int_rd(cr.a);
                col_ref = cr.ia >= 0 && cr.ia + 1 < p.na;
                const float wa2 = __fsub_rn(cr.a, (float)cr.ia);
                const float u = __fadd_rn(c.wau, c.wa2u);     // the distance weight (wa + wa2 = 1)
                cr.wau = __fmul_rn(__fsub_rn(1.f, wa2), u);
                cr.wa2u = __fmul_rn(wa2, u);
            }
        }
        const size_t off = (size_t)v * p.na * p.nb;
        auto contribution = [&](const BpColumn &cc, float b, float &out) -> bool {
            float r0, r1, wb, wb2;
            if (!bp_tap<false>(p, sino + off + cc.ia, nullptr, cc, b, r0, r1, wb, wb2)) return false;
            out = __fmaf_rn(r1, wb2, __fmul_rn(r0, wb));
            return true;
        };
        // correction of voxel iz (0 where the decisions agree)
        auto delta = [&](int iz, bool whole_column) -> float {
            const float zc = bp_cz(p, iz);
            const float b = __fmaf_rn(c.bm, zc, p.cb);
            const bool near_row = fabsf(b) < edge || fabsf(b - (nbf - 1.f)) < edge;
            if (!whole_column && !near_row) return 0.f;
            const float br = near_row ? exact_row(p, cphi, sphi, xc, yc, zc) : b;
            float co = 0.f, cref = 0.f;
            const bool ours = col_ours && bp_keep(b, p.nb) && contribution(c, b, co);
            const bool ref = col_ref && bp_keep(br, p.nb) && contribution(cr, br, cref);
            if (ours == ref && !whole_column) return 0.f;
            return __fsub_rn(ref ? cref : 0.f, ours ? co : 0.f);
        };
        // voxel range of the band of rows within `edge` of row 0 (e = 0) or
        // nb - 1 (e = 1): the rows are monotone in z (b = bm z + cb), so the
        // band is one z interval, mapped to voxel indices in float with a
        // margin of 1/1024 voxel (its rounding is ~1e-5 voxel); the band is
        // a few thousandths of a voxel wide, so few (column, view) pairs have
        // a candidate and few warps take the (divergent) candidate path
        float b_first = 0.f, b_last = 0.f, ibm = 0.f;
        auto band = [&](int e, int &i0, int &i1) {
            const float target = e ? nbf - 1.f : 0.f;
            const float za = (target - edge - p.cb) * ibm, zb = (target + edge - p.cb) * ibm;
            const float flo = (fminf(za, zb) - p.corner_z) * idz - 0.5f - 1.f / 1024;
            const float fhi = (fmaxf(za, zb) - p.corner_z) * idz - 0.5f + 1.f / 1024;
            i0 = max(0, __float2int_ru(fmaxf(flo, -1.f)));
            i1 = min(p.nz - 1, __float2int_rd(fminf(fhi, (float)p.nz)));
        };
        // rows of the column over the grid's z extent (a little wider): a
        // band outside it has no voxel
        auto reaches = [&](int e) {
            const float target = e ? nbf - 1.f : 0.f;
            return fminf(b_first, b_last) - 1.f < target && target < fmaxf(b_first, b_last) + 1.f;
        };
        int n = 0, slot_iz[kEdgeSlots];
        float slot_d[kEdgeSlots];
        bool serial = has && col_ours != col_ref;   // the whole column differs: done one lane at a time
        if (has && !serial && col_ours && c.bm != 0.f) {
            b_first = __fmaf_rn(c.bm, z_first, p.cb);
            b_last = __fmaf_rn(c.bm, z_last, p.cb);
            ibm = rcp_approx(c.bm);
            for (int e = 0; e < 2; ++e) {
                if (!reaches(e)) continue;
                int i0, i1;
                band(e, i0, i1);
                for (int iz = i0; iz <= i1; ++iz) {
                    const float d = delta(iz, false);
                    if (d == 0.f) continue;
                    if (n < kEdgeSlots) { slot_iz[n] = iz; slot_d[n] = d; ++n; }
                    else serial = true;
                }
            }
        }
        // apply in view order: lane by lane
        unsigned pending = __ballot_sync(0xffffffffu, n > 0 || serial);
        while (pending) {
            const int src = __ffs(pending) - 1;
            pending &= pending - 1;
            if (lane == src) {
                if (col_ours != col_ref) {
                    for (int iz = 0; iz < p.nz; ++iz) {
                        const float d = delta(iz, true);
                        if (d != 0.f) vcol[(size_t)iz * plane] = __fadd_rn(vcol[(size_t)iz * plane], d);
                    }
                } else if (serial) {                   // more corrections than slots (rare)
                    for (int e = 0; e < 2; ++e) {
                        int i0, i1;
                        band(e, i0, i1);
                        for (int iz = i0; iz <= i1; ++iz) {
                            const float d = delta(iz, false);
                            if (d != 0.f) vcol[(size_t)iz * plane] = __fadd_rn(vcol[(size_t)iz * plane], d);
                        }
                    }
                } else {
                    for (int k = 0; k < n; ++k)
                        vcol[(size_t)slot_iz[k] * plane] = __fadd_rn(vcol[(size_t)slot_iz[k] * plane], slot_d[k]);
                }
            }
            __syncwarp();
        }
    }
}
}  // namespace nefct

using namespace nefct;

extern "C" {

nefct_status nefct_fdk_filter(const nefct_cb_geom *g, const float *sino, float *out, int32_t window,
                              int32_t parker, void *stream)
{
    nefct_status st = check_cb_geom(g);
    if (st) return st;
    if (!sino || !out) return fail(NEFCT_ERR_INVALID, "sino and out must be non-NULL");
    if (sino == out) return fail(NEFCT_ERR_INVALID, "fdk filter output may not alias its input");
    if (g->det_kind != NEFCT_DET_FLAT)
        return fail(NEFCT_ERR_UNSUPPORTED, "FDK filtering is defined for flat detectors only (filtering.m)");
    if (window < NEFCT_WIN_RAM_LAK || window > NEFCT_WIN_HANN)
        return fail(NEFCT_ERR_INVALID, "unknown filter window %d", window);
    if (parker < -1 || parker > 1) return fail(NEFCT_ERR_INVALID, "parker must be -1, 0 or 1");
    if (g->na > kMaxCols) return fail(NEFCT_ERR_UNSUPPORTED, "FDK filter supports up to %d detector columns", kMaxCols);
    if (g->src_iso <= 0.f || g->src_det <= 0.f) return fail(NEFCT_ERR_INVALID, "distances must be > 0");
    FilterParams *pp = new FilterParams();
    FilterParams &p = *pp;
    p.na = g->na; p.nb = g->nb; p.nv = g->nv;
    p.L = ramp_length(g->na);
    p.log2L = 0;
    while ((1 << p.log2L) < p.L) ++p.log2L;
    p.pairs_per_view = (g->nb + 1) / 2;
    if ((long long)p.pairs_per_view * g->nv > INT_MAX) { delete pp; return fail(NEFCT_ERR_UNSUPPORTED, "too many detector rows x views"); }
    p.pairs = p.pairs_per_view * g->nv;
    p.src_det = g->src_det; p.da = g->da; p.a_shift = g->a_shift; p.db = g->db; p.b_shift = g->b_shift;
    p.src_det_d = g->src_det; p.da_d = g->da; p.a_shift_d = g->a_shift;
    p.parker = parker;
    // scale of filtering.m:43-47: /2/du * dbeta/2 * DSD/DSO
    double dbeta;
    if (parker) {
        if (g->nv < 2) { delete pp; return fail(NEFCT_ERR_INVALID, "Parker weighting needs >= 2 views"); }
        p.dang = fabs((double)g->angles[1] - (double)g->angles[0]) * 180.0 / M_PI;
        if (!(p.dang > 0.0)) { delete pp; return fail(NEFCT_ERR_INVALID, "Parker weighting needs a non-zero view step"); }
        dbeta = 2.0 * M_PI / (180.0 / p.dang);
        const double u0 = (0.0 + g->a_shift) * g->da - g->na * (double)g->da / 2.0;
        const double u1 = (g->na - 1 + (double)g->a_shift) * g->da - g->na * (double)g->da / 2.0;
        p.fanang = fabs(atan(u1 / g->src_det) - atan(u0 / g->src_det)) / M_PI * 180.0 / 2.0;
    } else {
        p.dang = 0.0;
        p.fanang = 0.0;
        dbeta = 2.0 * M_PI / g->nv;
    }
    const double scale = 1.0 / 2.0 / fabs((double)g->da) * dbeta / 2.0 * ((double)g->src_det / g->src_iso);
    const std::vector<float> h = ramp_response(g->na, window, scale);
    std::copy(h.begin(), h.end(), p.h);
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaSuccess;
    if (p.pairs > 0) {
        switch (p.log2L) {
        case 6: e = launch_filter<6>(p, sino, out, s); break;
        case 7: e = launch_filter<7>(p, sino, out, s); break;
        case 8: e = launch_filter<8>(p, sino, out, s); break;
        case 9: e = launch_filter<9>(p, sino, out, s); break;
        case 10: e = launch_filter<10>(p, sino, out, s); break;
        case 11: e = launch_filter<11>(p, sino, out, s); break;
        case 12: e = launch_filter<12>(p, sino, out, s); break;
        default: delete pp; return fail(NEFCT_ERR_UNSUPPORTED, "FFT length 2^%d outside 2^6..2^12", p.log2L);
        }
    }
    if (e != cudaSuccess) { delete pp; return cuda_fail(e, "fdk_filter_kernel"); }
    delete pp;
    NEFCT_CHECK_LAUNCH("fdk_filter_kernel");
    return NEFCT_OK;
}

size_t nefct_fdk_workspace_bytes(const nefct_cb_geom *g)
{
    if (!g || g->na < 1 || g->nb < 1) return 0;
    const int chunk = fdk_view_chunk(g->na, g->nb, sizeof(float4));
    return (size_t)std::min(chunk, std::max(g->nv, 1)) * g->na * g->nb * sizeof(float4);
}

nefct_status nefct_fdk_backproject_ws(const nefct_cb_geom *g, const float *filtered, float *vol, uint32_t flags,
                                      void *ws, size_t ws_bytes, void *stream)
{
    nefct_status st = check_cb_geom(g);
    if (st) return st;
    if (!filtered || !vol) return fail(NEFCT_ERR_INVALID, "filtered and vol must be non-NULL");
    if (flags & ~NEFCT_FDK_NO_WEIGHT) return fail(NEFCT_ERR_INVALID, "unknown flag bits 0x%x", flags);
    if (ws && ws_bytes < nefct_fdk_workspace_bytes(g))
        return fail(NEFCT_ERR_WORKSPACE, "needs %zu workspace bytes, got %zu", nefct_fdk_workspace_bytes(g), ws_bytes);
    if (ws && ((uintptr_t)ws & 15)) return fail(NEFCT_ERR_INVALID, "workspace must be 16-byte aligned");
    // (the kernel's row pitches are 32-bit numbers of bytes: longer rows of quads
    // are not made; rows of floats fit, with fewer than 2^31 cells)
    const bool quad = ws != nullptr && g->na < 1 << 28;
    // a detector of one row or column has no cell with four taps (Q11): every
    // voxel is dropped
    if (g->na < 2 || g->nb < 2) {
        const size_t voxels = (size_t)g->grid.nx * g->grid.ny * g->grid.nz;
        NEFCT_CHECK_CUDA(cudaMemsetAsync(vol, 0, voxels * sizeof(float), (cudaStream_t)stream));
        return NEFCT_OK;
    }
    BpParams *p = new BpParams();
    p->nx = g->grid.nx; p->ny = g->grid.ny; p->nz = g->grid.nz;
    p->na = g->na; p->nb = g->nb;
    p->sx = g->grid.sx; p->sy = g->grid.sy; p->sz = g->grid.sz;
    // the reference takes the grid's low corner (Q10)
    p->corner_x = g->grid.cx - g->grid.sx / 2.f;
    p->corner_y = g->grid.cy - g->grid.sy / 2.f;
    p->corner_z = g->grid.cz - g->grid.sz / 2.f;
    p->src_iso = g->src_iso; p->src_det = g->src_det;
    // pixel_3d's `ai` is the siddon_3d `ai` minus one half (Q9)
    p->da = g->da; p->ai_p = g->a_shift - 0.5f; p->db = g->db; p->bi_p = g->b_shift - 0.5f;
    p->inv_da = (float)(1.0 / (double)g->da);
    p->inv_db = (float)(1.0 / (double)g->db);
    p->cb = (float)((double)(g->nb / 2) - (double)p->bi_p - 0.5);
    p->cyl = g->det_kind == NEFCT_DET_CYL;
    p->weight = !(flags & NEFCT_FDK_NO_WEIGHT);
    p->has_ctr = (long long)g->grid.nx + g->grid.ny + g->grid.nz <= kCtrMax;
    if (p->has_ctr) {
        float *c = p->ctr;
        for (int i = 0; i < p->nx; ++i) *c++ = bp_centre(i, p->sx, p->nx, p->corner_x);
        for (int i = 0; i < p->ny; ++i) *c++ = bp_centre(i, p->sy, p->ny, p->corner_y);
        for (int i = 0; i < p->nz; ++i) *c++ = bp_centre(i, p->sz, p->nz, p->corner_z);
    }
    cudaStream_t s = (cudaStream_t)stream;
    dim3 grid((g->grid.nx + kTW - 1) / kTW, (g->grid.ny + 4 * (32 / kTW) - 1) / (4 * (32 / kTW)), (g->grid.nz + kZ - 1) / kZ);
    const int chunk = quad ? fdk_view_chunk(g->na, g->nb, sizeof(float4)) : fdk_view_chunk(g->na, g->nb);
    float4 *q4 = (float4 *)ws;
    for (int v0 = 0; v0 < g->nv; v0 += chunk) {
        p->nv0 = v0;
        p->nvc = std::min(chunk, g->nv - v0);
        p->first = v0 == 0;
        for (int i = 0; i < p->nvc; ++i) {
            p->cs[i] = (float)cos((double)g->angles[v0 + i]);
            p->sn[i] = (float)sin((double)g->angles[v0 + i]);
        }
        const float *chunk_sino = filtered + (size_t)v0 * g->na * g->nb;
        cudaError_t e;
        if (quad) {
            const unsigned tiles = (unsigned)((g->na + 63) / 64) * (unsigned)((g->nb + 4 * kQuadRows - 1) / (4 * kQuadRows));
            fdk_quad_kernel<<<dim3(tiles, p->nvc), dim3(64, 4), 0, s>>>(chunk_sino, q4, g->na, g->nb);
            e = cudaGetLastError();
            if (e != cudaSuccess) { delete p; return cuda_fail(e, "fdk_quad_kernel"); }
            fdk_bp_kernel<true><<<grid, dim3(32, 4), 0, s>>>(*p, chunk_sino, q4, vol);
        } else {
            fdk_bp_kernel<false><<<grid, dim3(32, 4), 0, s>>>(*p, chunk_sino, nullptr, vol);
        }
        e = cudaGetLastError();
        if (e != cudaSuccess) { delete p; return cuda_fail(e, "fdk_bp_kernel"); }
    }
    // detector-edge decisions, a warp per voxel column, kViewChunk views per launch
    const long long columns = (long long)g->grid.nx * g->grid.ny;
    const unsigned eblocks = (unsigned)((columns + 7) / 8);        // a warp per column
    for (int v0 = 0; v0 < g->nv; v0 += kViewChunk) {
        p->nv0 = v0;
        p->nvc = std::min(kViewChunk, g->nv - v0);
        for (int i = 0; i < p->nvc; ++i) {
            p->cs[i] = (float)cos((double)g->angles[v0 + i]);
            p->sn[i] = (float)sin((double)g->angles[v0 + i]);
        }
        fdk_edge_kernel<<<eblocks, 256, 0, s>>>(*p, filtered + (size_t)v0 * g->na * g->nb, vol);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) { delete p; return cuda_fail(e, "fdk_edge_kernel"); }
    }
    delete p;
    return NEFCT_OK;
}

nefct_status nefct_fdk_backproject(const nefct_cb_geom *g, const float *filtered, float *vol, uint32_t flags,
                                   void *stream)
{
    return nefct_fdk_backproject_ws(g, filtered, vol, flags, nullptr, 0, stream);
}

}  // extern "C"
