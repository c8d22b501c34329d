// Dense y = A_inv x of the direct coarse solve (dense_matvec.inl:109-117):
// every (row, right-hand side) accumulates over the columns in order.
#pragma once

#include "kernels.cuh"

namespace xg {
namespace k {

// The inverse is stored column by column (element (i, j) at j*n + i). A block
// takes RB consecutive rows: all its threads copy a chunk of columns of those
// rows (32 contiguous bytes a column) and the matching rows of x into shared
// memory, then RB*NV of them run their sums over the chunk. A sum is a chain of
// n additions (about 1,300 cycles at n = 305), so what counts is that the copy
// is one round trip and not one per 64 columns: with 64 threads and chunks of
// 64 columns the solve took 28 us at n = 305, nv = 8 in FP32.
constexpr int DT = 256;
template <typename F, int NV>
__host__ __device__ constexpr int dense_rows() {
    const int a = 32 / (int)sizeof(F), b = 32 / NV;
    return a > b ? a : b;
}
template <typename F, int NV>
__host__ __device__ constexpr uint32_t dense_chunk() {  // columns within 48 KB
    return (48u * 1024u) / (uint32_t)((NV + dense_rows<F, NV>()) * sizeof(F));
}
template <typename F, int NV>
__global__ void __launch_bounds__(DT)
    k_dense(const F *__restrict__ a, uint64_t n, const F *__restrict__ x, F *__restrict__ y,
            uint32_t chunk) {
    constexpr int RB = dense_rows<F, NV>();
    static_assert(RB * NV <= DT, "one thread a (row, right-hand side)");
    extern __shared__ __align__(16) unsigned char dense_smem[];
    F *xs = (F *)dense_smem, *as = xs + (size_t)chunk * NV;
    const int r = threadIdx.x / NV, k = threadIdx.x % NV;
    const uint64_t i0 = (uint64_t)blockIdx.x * RB;
    const bool on = r < RB && i0 + r < n;
    F acc = F(0);
    for (uint64_t j0 = 0; j0 < n; j0 += chunk) {
        const uint32_t jc = (uint32_t)(n - j0 < chunk ? n - j0 : chunk);
        if (j0) __syncthreads();  // the previous chunk is consumed
#pragma unroll 8
        for (uint32_t t = threadIdx.x; t < jc * RB; t += DT) {
            const uint32_t jj = t / RB, rr = t % RB;
            as[t] = i0 + rr < n ? __ldg(&a[(j0 + jj) * n + i0 + rr]) : F(0);
        }
#pragma unroll 8
        for (uint32_t t = threadIdx.x; t < jc * NV; t += DT) xs[t] = __ldg(&x[j0 * NV + t]);
        __syncthreads();
        if (on) {
#pragma unroll 8
            for (uint32_t jj = 0; jj < jc; ++jj)
                acc = add(acc, mul(as[jj * RB + r], xs[jj * NV + k]));
        }
    }
    if (on) y[(i0 + r) * NV + k] = acc;
}

}  // namespace k
}  // namespace xg
