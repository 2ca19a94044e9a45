// Forward cone-beam kernels (thread walk and column warps) for float and
// double: see cb_kernels.cuh.
#include "cb_kernels.cuh"

namespace nefct {

// Column warps: one warp per 32 R rows of column ia at view iv, over the
// z-fastest copy p.volT, into p.out.  TAIL: from row p.row0 on (else 0; the one
// more value costs R = 3 0.8 % in spills).
template <int R, bool REF, bool TAIL>
__global__ void __launch_bounds__(256, 4) cb_colwarp_forward_kernel(const __grid_constant__ CBParams<float> p)
{
    const int ia = blockIdx.x * blockDim.y + threadIdx.y;
    const int tile = p.band_major ? blockIdx.z : blockIdx.y;
    const int first = tile * 32 * R + (TAIL ? p.row0 : 0);
    const int iv = p.band_major ? blockIdx.y : blockIdx.z;
    if (ia >= p.na) return;                       // uniform across the warp
    auto row = [&](int i, float (&r)[6]) {
        const int ib = col_row<R, false>(first, threadIdx.x, i, false);
        cb_ray(p, ia, ib < p.nb ? ib : 0, iv, r);
        return ib < p.nb;
    };
    auto store = [&](int i, float v) {
        const int ib = col_row<R, false>(first, threadIdx.x, i, false);
        p.out[(size_t)(p.v0 + iv) * p.na * p.nb + (size_t)ib * p.na + ia] = v;
    };
    colwarp_forward<R, REF, kSteepInline>(p.g, p.flags, p.volT, row, store);
}

template <bool REF>
static cudaError_t launch_colwarp(CBParams<float> &p, int na, int rows, int nvc, int R, cudaStream_t s)
{
    dim3 grid, block;
    cb_colwarp_shape(p, na, rows, nvc, grid, block, R);
    if (p.row0) {                                 // fewer rows per lane than the launch before
        if (R == 1) cb_colwarp_forward_kernel<1, REF, true><<<grid, block, 0, s>>>(p);
        else if constexpr (!REF) cb_colwarp_forward_kernel<2, false, true><<<grid, block, 0, s>>>(p);
    } else if (R == 1) cb_colwarp_forward_kernel<1, REF, false><<<grid, block, 0, s>>>(p);
    else if (R == 2) cb_colwarp_forward_kernel<2, REF, false><<<grid, block, 0, s>>>(p);
    else if constexpr (!REF) cb_colwarp_forward_kernel<3, false, false><<<grid, block, 0, s>>>(p);
    return cudaGetLastError();
}

// Slab steps of a warp of 32 R rows, relative: 1, 1.76 or 2.57 with R = 1, 2,
// 3 (256^3, 24 views of 512 x 384: 1.00 / 0.88 / 0.86 ms; R = 4 spills: 0.92
// ms).
static constexpr int kForwardCost[4] = {0, 100, 176, 257};

template <typename T>
cudaError_t cb_launch_forward(CBParams<T> &p, int na, int nb, int nvc, uint32_t flags, cudaStream_t s, bool colwarp)
{
    if constexpr (std::is_same<T, float>::value) {
        if (colwarp) {
            const bool ref = ref_rounding(flags);
            return cb_row_launches(p, nb, cb_rows_per_lane(nb, 1, ref ? 2 : 3, kForwardCost), [&](int rows, int R) {
                return ref ? launch_colwarp<true>(p, na, rows, nvc, R, s) : launch_colwarp<false>(p, na, rows, nvc, R, s);
            });
        }
    }
    return cb_launch<T, true>(p, na, nb, nvc, flags, s);
}

template cudaError_t cb_launch_forward<float>(CBParams<float> &, int, int, int, uint32_t, cudaStream_t, bool);
template cudaError_t cb_launch_forward<double>(CBParams<double> &, int, int, int, uint32_t, cudaStream_t, bool);

}  // namespace nefct
