// Transpose cone-beam kernels (thread walk and column warps) for float and
// double: see cb_kernels.cuh.
#include "cb_kernels.cuh"

namespace nefct {

// Column warps: one warp per 32 R rows of column ia at view iv, from row
// p.row0 on, into the z-fastest accumulator p.outT (FIXED: the deterministic
// transpose's integers p.fix).
template <int R, bool REF, bool NEXT, bool FIXED, bool STEEP>
__global__ void __launch_bounds__(256, 4) cb_colwarp_backward_kernel(const __grid_constant__ CBParams<float> p)
{
    const int ia = blockIdx.x * blockDim.y + threadIdx.y;
    const int first = p.row0 + (int)(p.band_major ? blockIdx.z : blockIdx.y) * 32 * R;
    const int iv = p.band_major ? blockIdx.y : blockIdx.z;
    if (ia >= p.na) return;                       // uniform across the warp
    float r[R][6], y[R];
    bool has[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int ib = col_row<R, NEXT>(first, threadIdx.x, i, p.rg.db < 0.f);
        has[i] = ib < p.nb;
        y[i] = has[i] ? cb_sino_value(p, ia, ib, iv) : 0.f;
        cb_ray(p, ia, has[i] ? ib : 0, iv, r[i]);
    }
    if constexpr (FIXED) colwarp_backward<R, REF, NEXT, STEEP>(p.g, r, has, p.flags, y, FixedAcc{p.fix, *p.fix_scale});
    else colwarp_backward<R, REF, NEXT, STEEP>(p.g, r, has, p.flags, y, FloatAcc{p.outT});
}

template <bool REF, bool FIXED, bool STEEP>
static cudaError_t launch_colwarp(CBParams<float> &p, int na, int rows, int nvc, int R, cudaStream_t s)
{
    dim3 grid, block;
    cb_colwarp_shape(p, na, rows, nvc, grid, block, R);
    if (R == 1) cb_colwarp_backward_kernel<1, REF, false, FIXED, STEEP><<<grid, block, 0, s>>>(p);
    else if (R == 2) cb_colwarp_backward_kernel<2, REF, true, FIXED, STEEP><<<grid, block, 0, s>>>(p);
    else if (R == 3) cb_colwarp_backward_kernel<3, REF, true, FIXED, STEEP><<<grid, block, 0, s>>>(p);
    else cb_colwarp_backward_kernel<4, REF, true, FIXED, STEEP><<<grid, block, 0, s>>>(p);
    return cudaGetLastError();
}

template <bool FIXED, bool STEEP>
static cudaError_t launch_rows(CBParams<float> &p, int na, int nb, int nvc, uint32_t flags, cudaStream_t s)
{
    const bool ref = ref_rounding(flags);
    return cb_row_launches(p, nb, col_rows_next(p.g, p.rg, nb), [&](int rows, int R) {
        return ref ? launch_colwarp<true, FIXED, STEEP>(p, na, rows, nvc, R, s)
                   : launch_colwarp<false, FIXED, STEEP>(p, na, rows, nvc, R, s);
    });
}

template <bool FIXED>
static cudaError_t launch_rows(CBParams<float> &p, int na, int nb, int nvc, uint32_t flags, cudaStream_t s)
{
    return cb_may_be_steep(p.g, p.rg, nb) ? launch_rows<FIXED, true>(p, na, nb, nvc, flags, s)
                                          : launch_rows<FIXED, false>(p, na, nb, nvc, flags, s);
}

cudaError_t cb_launch_backward_fixed(CBParams<float> &p, int na, int nb, int nvc, uint32_t flags, cudaStream_t s)
{
    return launch_rows<true>(p, na, nb, nvc, flags, s);
}

template <typename T>
cudaError_t cb_launch_backward(CBParams<T> &p, int na, int nb, int nvc, uint32_t flags, cudaStream_t s, bool colwarp)
{
    if constexpr (std::is_same<T, float>::value) {
        if (colwarp) return launch_rows<false>(p, na, nb, nvc, flags, s);
    }
    return cb_launch<T, false>(p, na, nb, nvc, flags, s);
}

template cudaError_t cb_launch_backward<float>(CBParams<float> &, int, int, int, uint32_t, cudaStream_t, bool);
template cudaError_t cb_launch_backward<double>(CBParams<double> &, int, int, int, uint32_t, cudaStream_t, bool);

}  // namespace nefct
