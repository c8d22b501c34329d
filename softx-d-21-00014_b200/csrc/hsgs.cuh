// Hybrid symmetric Gauss-Seidel sweep from shared memory (csr_gs.inl:77-130,
// blas2.h:184-281): the forward then the backward sweep of every Gauss-Seidel
// block, one lane per (block, right-hand side).
//
// A sweep is a chain: a row's update needs the row before it, 2 x 40 rows one
// after the other for blocks of 40 rows, so the latency of what a row reads
// sets the time, not bytes. Read from global memory, each row waits for three
// dependent round trips (row pointer, column, x): 95-160 us a sweep whatever
// the level's size (one B200, 7-point 43x40x37 hierarchy, nv = 1). Here a
// thread block copies the rows of a few Gauss-Seidel blocks (entries, right-hand
// side, x, diagonal) into shared memory with coalesced loads, and a lane keeps
// the next row's operands in registers while the current one finishes: only
// the value just computed is forwarded, by register. Products and sums are
// formed in the same order as before, bit for bit.
#pragma once

#include "kernels.cuh"

namespace xg {
namespace k {

constexpr int HS_THREADS = 128;  // copy the block in and out; warp 0 sweeps
constexpr int HS_PF = 6;         // entries of the next row held in registers

// Where a sweep's operands lie: rows of Gauss-Seidel block g are
// [g * rows, (g + 1) * rows), the last one short.
struct HsgsShape {
    uint64_t n;
    uint32_t rows;    // rows of a Gauss-Seidel block
    uint32_t group;   // Gauss-Seidel blocks of a thread block (group * NV <= 32)
    uint32_t ent_max; // most entries a thread block copies
};

__host__ __device__ inline uint32_t hs_round16(uint32_t b) { return (b + 15u) & ~15u; }

// Shared memory of a thread block: t and x (one row of padding per
// Gauss-Seidel block, so that the lanes of different blocks hit different
// banks at nv = 1), the diagonal, the row pointers, the entries.
template <typename F, typename I, int NV>
__host__ __device__ inline uint32_t hs_smem_bytes(const HsgsShape &s) {
    const uint32_t rows = s.rows * s.group;
    return 2 * hs_round16((rows + s.group) * NV * (uint32_t)sizeof(F)) +
           hs_round16(rows * (uint32_t)sizeof(F)) + hs_round16((rows + 1) * 4) +
           hs_round16(s.ent_max * (uint32_t)sizeof(F)) + hs_round16(s.ent_max * (uint32_t)sizeof(I));
}

// A row's operands as a lane holds them one row ahead.
template <typename F>
struct HsgsRow {
    uint32_t j, len;
    F s, cf, xo;
    uint32_t c[HS_PF];
    F v[HS_PF], xv[HS_PF];
};

template <typename F, typename I, int NV>
__device__ __forceinline__ void hs_load(HsgsRow<F> &r, uint32_t i, const uint32_t *ptr,
                                        const F *t, const F *x, const F *d, const I *col,
                                        const F *val, F w) {
    r.j = ptr[i];
    r.len = ptr[i + 1] - r.j;
    r.s = t[i * NV];
    r.xo = x[i * NV];
    r.cf = mul(w, d[i]);
#pragma unroll
    for (int e = 0; e < HS_PF; ++e)
        if ((uint32_t)e < r.len) {
            r.c[e] = (uint32_t)col[r.j + e];
            r.v[e] = val[r.j + e];
            r.xv[e] = x[r.c[e] * NV];
        }
}

// x_i + (w d_i) (t_i - sum): entries in row order. ip, xp: the row updated
// last and its value, which the operands were loaded before.
template <typename F, typename I, int NV>
__device__ __forceinline__ F hs_row(const HsgsRow<F> &r, const F *x, const I *col, const F *val,
                                    uint32_t ip, F xp) {
    F s = r.s;
#pragma unroll
    for (int e = 0; e < HS_PF; ++e)
        if ((uint32_t)e < r.len) s = sub(s, mul(r.c[e] == ip ? xp : r.xv[e], r.v[e]));
    if (r.len > (uint32_t)HS_PF) {
#pragma unroll 4
        for (uint32_t e = HS_PF; e < r.len; ++e)
            s = sub(s, mul(x[(uint32_t)col[r.j + e] * NV], val[r.j + e]));
    }
    return add(r.xo, mul(r.cf, s));
}

// t: b - A_offblock x_old, or b itself where x starts from zero (xin null).
template <typename F, typename I, int NV>
__global__ void __launch_bounds__(HS_THREADS)
    k_hsgs_block(const uint32_t *__restrict__ row, const I *__restrict__ gcol,
                 const F *__restrict__ gval, HsgsShape sh, const F *__restrict__ gt,
                 const F *xin, F *xout, const F *__restrict__ gd,
                 const double *__restrict__ relax_sc) {
    extern __shared__ __align__(16) unsigned char hs_smem[];
    const uint32_t cap = sh.rows * sh.group;
    F *t = (F *)hs_smem;
    const uint32_t vecb = hs_round16((cap + sh.group) * NV * (uint32_t)sizeof(F));
    F *x = (F *)(hs_smem + vecb);
    F *d = (F *)(hs_smem + 2 * vecb);
    uint32_t *ptr = (uint32_t *)(hs_smem + 2 * vecb + hs_round16(cap * (uint32_t)sizeof(F)));
    F *val = (F *)((unsigned char *)ptr + hs_round16((cap + 1) * 4));
    I *col = (I *)((unsigned char *)val + hs_round16(sh.ent_max * (uint32_t)sizeof(F)));

    const uint64_t R0 = (uint64_t)blockIdx.x * cap;
    const uint32_t rows = (uint32_t)(sh.n - R0 < cap ? sh.n - R0 : cap);
    const uint32_t J0 = __ldg(&row[R0]), nj = __ldg(&row[R0 + rows]) - J0;
    for (uint32_t e = threadIdx.x; e < nj; e += HS_THREADS) {
        val[e] = __ldg(&gval[(uint64_t)J0 + e]);
        col[e] = __ldg(&gcol[(uint64_t)J0 + e]);
    }
    for (uint32_t e = threadIdx.x; e <= rows; e += HS_THREADS) ptr[e] = __ldg(&row[R0 + e]) - J0;
    for (uint32_t e = threadIdx.x; e < rows; e += HS_THREADS) d[e] = __ldg(&gd[R0 + e]);
    for (uint32_t e = threadIdx.x; e < rows * NV; e += HS_THREADS) {
        const uint32_t at = e + (e / NV / sh.rows) * NV;  // one padding row a Gauss-Seidel block
        t[at] = __ldg(&gt[R0 * NV + e]);
        x[at] = xin ? xin[R0 * NV + e] : F(0);
    }
    __syncthreads();
    const uint32_t g = threadIdx.x / NV, k = threadIdx.x % NV;
    if (g < sh.group && g * sh.rows < rows) {
        const uint32_t f = g * sh.rows;  // first row
        const uint32_t nr = rows - f < sh.rows ? rows - f : sh.rows;
        const F w = (F)relax_sc[k];
        const uint32_t *lp = ptr + f;
        const F *lt = t + (f + g) * NV + k, *ld = d + f;
        F *lx = x + (f + g) * NV + k;
        HsgsRow<F> cur, nxt;
        uint32_t ip = 0xFFFFFFFFu;
        F xp = F(0);
        hs_load<F, I, NV>(cur, 0, lp, lt, lx, ld, col, val, w);
        for (uint32_t i = 0; i < nr; ++i) {
            if (i + 1 < nr) hs_load<F, I, NV>(nxt, i + 1, lp, lt, lx, ld, col, val, w);
            xp = hs_row<F, I, NV>(cur, lx, col, val, ip, xp);
            lx[i * NV] = xp;
            ip = i;
            cur = nxt;
        }
        ip = 0xFFFFFFFFu;
        hs_load<F, I, NV>(cur, nr - 1, lp, lt, lx, ld, col, val, w);
        for (uint32_t i = nr; i-- > 0;) {
            if (i > 0) hs_load<F, I, NV>(nxt, i - 1, lp, lt, lx, ld, col, val, w);
            xp = hs_row<F, I, NV>(cur, lx, col, val, ip, xp);
            lx[i * NV] = xp;
            ip = i;
            cur = nxt;
        }
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < rows * NV; e += HS_THREADS)
        xout[R0 * NV + e] = x[e + (e / NV / sh.rows) * NV];
}

}  // namespace k
}  // namespace xg
