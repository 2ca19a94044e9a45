// Forward cone-beam kernels (thread walk and column warps) for float and
// double: see cb_kernels.cuh.
#include "cb_kernels.cuh"

namespace nefct {

// Column warps: one warp per 32 R rows of column ia at view iv, over the
// z-fastest copy p.volT, into p.out.
template <int R, bool REF>
__global__ void __launch_bounds__(256, 4) cb_colwarp_forward_kernel(const __grid_constant__ CBParams<float> p)
{
    const int ia = blockIdx.x * blockDim.y + threadIdx.y;
    const int tile = p.band_major ? blockIdx.z : blockIdx.y;
    const int iv = p.band_major ? blockIdx.y : blockIdx.z;
    if (ia >= p.na) return;                       // uniform across the warp
    auto row = [&](int i, float (&r)[6]) {
        const int ib = col_row<R, false>(tile, threadIdx.x, i, false);
        cb_ray(p, ia, ib < p.nb ? ib : 0, iv, r);
        return ib < p.nb;
    };
    auto store = [&](int i, float v) {
        const int ib = col_row<R, false>(tile, threadIdx.x, i, false);
        p.out[(size_t)(p.v0 + iv) * p.na * p.nb + (size_t)ib * p.na + ia] = v;
    };
    colwarp_forward<R, REF>(p.g, p.flags, p.volT, row, store);
}

template <int R, bool REF>
static cudaError_t launch_colwarp(CBParams<float> &p, int na, int nb, int nvc, cudaStream_t s)
{
    dim3 grid, block;
    cb_colwarp_shape(p, na, nb, nvc, grid, block, R);
    cb_colwarp_forward_kernel<R, REF><<<grid, block, 0, s>>>(p);
    return cudaGetLastError();
}

// Rows per lane: the fewest slab steps.  A warp of 32 R rows takes 1, 1.76 or
// 2.57 times as long with R = 1, 2, 3 (256^3, 24 views of 512 x 384: 1.00 /
// 0.88 / 0.86 ms; R = 4 spills: 0.92 ms), so nb rows take ceil(nb / 32 R) of
// those: three rows per lane unless the last tile would be mostly empty.
static int rows_per_lane(int nb)
{
    const int cost[3] = {100, 176, 257};
    int best = 0, least = INT_MAX;
    for (int r = 3; r >= 1; --r) {
        const int c = (nb + 32 * r - 1) / (32 * r) * cost[r - 1];
        if (c < least) { least = c; best = r; }
    }
    return best;
}

template <typename T>
cudaError_t cb_launch_forward(CBParams<T> &p, int na, int nb, int nvc, uint32_t flags, cudaStream_t s, bool colwarp)
{
    if constexpr (std::is_same<T, float>::value) {
        if (colwarp) {
            if (ref_rounding(flags)) return launch_colwarp<2, true>(p, na, nb, nvc, s);
            switch (rows_per_lane(nb)) {
            case 1: return launch_colwarp<1, false>(p, na, nb, nvc, s);
            case 2: return launch_colwarp<2, false>(p, na, nb, nvc, s);
            default: return launch_colwarp<3, false>(p, na, nb, nvc, s);
            }
        }
    }
    return cb_launch<T, true>(p, na, nb, nvc, flags, s);
}

template cudaError_t cb_launch_forward<float>(CBParams<float> &, int, int, int, uint32_t, cudaStream_t, bool);
template cudaError_t cb_launch_forward<double>(CBParams<double> &, int, int, int, uint32_t, cudaStream_t, bool);

}  // namespace nefct
