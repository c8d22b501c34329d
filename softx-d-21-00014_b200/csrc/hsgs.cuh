// Hybrid symmetric Gauss-Seidel sweep from shared memory (csr_gs.inl:77-130,
// blas2.h:184-281): the forward then the backward sweep of every Gauss-Seidel
// block, one lane per (block, right-hand side).
//
// A sweep is a chain: a row's update needs the row before it, 2 x 40 rows one
// after the other for blocks of 40 rows, so the latency of a row sets the time,
// not bytes. Read from global memory, each row waits for three dependent round
// trips (row pointer, column, x): 95-160 us a sweep whatever the level's size
// (one B200, 7-point 43x40x37 hierarchy, nv = 1). Whole solves with that sweep and
// with this one (ms): that system 36.6 and 6.6; on large levels with many right-hand
// sides, where a few sweeping warps an SM are the limit, 7-point 96^3 FP32 nv = 16
// 54.2 and 39.6, nv = 32 69.3 and 60.3, 64^3 FP64 nv = 32 32.1 and 29.7. Here a thread block copies the
// rows of a few Gauss-Seidel blocks into shared memory with coalesced loads, and
// a lane works from there with a few instructions an entry: a row's entries are
// padded to fours when the smoother is set up (what a padding entry adds is
// exactly nothing), and each is kept as the offset of its x and its value side
// by side. Products and sums are formed in the same order as before, bit for
// bit.
#pragma once

#include "kernels.cuh"

namespace xg {
namespace k {

constexpr int HS_THREADS = 128;  // copy the block in and out; warp 0 sweeps
constexpr int HS_PRODS = 6144;   // products of the lagged term held at a time
constexpr int HS_CHUNK = 4;      // a row's entries are padded to a multiple of this
// A padding entry has value 0 and the column one past the block's rows, where
// the lane's x is 0: its product is +0, and s - (+0) is s for every s.

// An entry in shared memory: the byte offset of its x and its value.
template <typename F>
struct HsPair;
template <>
struct __align__(8) HsPair<float> {
    uint32_t off;
    float v;
};
template <>
struct __align__(16) HsPair<double> {
    double v;
    uint32_t off, pad;
};

// Where a sweep's operands lie: rows of Gauss-Seidel block g are
// [g * rows, (g + 1) * rows), the last one short.
struct HsgsShape {
    uint64_t n;
    uint32_t rows;    // rows of a Gauss-Seidel block
    uint32_t group;   // Gauss-Seidel blocks of a thread block (group * NV <= 32)
    uint32_t ent_max; // most entries a thread block copies
};

// The lagged term b - A_offblock x_old formed by the sweep's own thread blocks:
// the off-block entries (row null: t is given).
template <typename F>
struct HsgsOff {
    const uint32_t *row = nullptr;
    const void *col = nullptr;
    const F *val = nullptr;
};

__host__ __device__ inline uint32_t hs_round16(uint32_t b) { return (b + 15u) & ~15u; }

// Shared memory of a thread block: the entries, t and x (one more row per
// Gauss-Seidel block: the padding entries' zero, which also puts the lanes of
// different blocks on different banks at nv = 1), the diagonal, each row's first
// chunk and chunk count; with the lagged term its row pointers and products too.
template <typename F, int NV>
__host__ __device__ inline uint32_t hs_smem_bytes(const HsgsShape &s, bool lagged) {
    const uint32_t rows = s.rows * s.group;
    const uint32_t more =
        lagged ? hs_round16((rows + 1) * 4) + (uint32_t)HS_PRODS * (uint32_t)sizeof(F) : 0u;
    return more + hs_round16(s.ent_max * (uint32_t)sizeof(HsPair<F>)) +
           2 * hs_round16((rows + s.group) * NV * (uint32_t)sizeof(F)) +
           hs_round16(rows * (uint32_t)sizeof(F)) + hs_round16(rows * 8);
}

// One sweep direction of a lane's Gauss-Seidel block: rows row_at(0), row_at(1),
// ..., row_at(nr - 1), each x_i + (w d_i) (t_i - sum of its entries in order).
// The lane works on three rows at once, one step apart: the row's chunk range
// three rows ahead, its first PC chunks two rows ahead, the x they meet one row
// ahead; so a step waits for shared memory only in rows of more than PC chunks,
// and is otherwise the chain of the row's own additions. An x read one row
// ahead is older than the row before it: that one comes from a register. The
// pipeline's slots are compile-time (three steps a turn), so they stay in
// registers.
template <typename F, int NV, int PC, class RowAt>
__device__ __forceinline__ void hs_direction(uint32_t nr, const RowAt &row_at, const uint2 *rows,
                                             const F *t, F *x, const F *d, const HsPair<F> *ent,
                                             F w) {
    constexpr int PE = PC * HS_CHUNK;
    uint2 R[3];
    HsPair<F> E[3][PE];
    F X[3][PE], S[3], D[3], O[3];
    uint32_t ip = 0xFFFFFFFFu;  // offset of the row updated last, its value in xp
    F xp = F(0);
    auto at = [&](uint32_t q) { return row_at(q < nr ? q : nr - 1); };  // past the end: reread
    auto x_at = [&](uint32_t off) { return *(const F *)((const char *)x + off); };
    auto chunk = [&](HsPair<F>(&e)[PE], int first, uint32_t c) {
        constexpr int V16 = HS_CHUNK * sizeof(HsPair<F>) / 16;
#pragma unroll
        for (int h = 0; h < V16; ++h)
            reinterpret_cast<uint4 *>(&e[first])[h] =
                reinterpret_cast<const uint4 *>(ent + c * HS_CHUNK)[h];
    };
    auto entries = [&](int k) {  // a short row rereads its first chunk (unused)
#pragma unroll
        for (int c = 0; c < PC; ++c)
            chunk(E[k], c * HS_CHUNK, R[k].x + ((uint32_t)c < R[k].y ? (uint32_t)c : 0u));
    };
    auto operands = [&](int k, uint32_t q) {
        const uint32_t i = at(q);
        S[k] = t[i * NV];
        O[k] = x[i * NV];
        D[k] = d[i];
#pragma unroll
        for (int e = 0; e < PE; ++e) X[k][e] = x_at(E[k][e].off);
    };
    auto step = [&](auto kc, uint32_t q) {
        constexpr int k = decltype(kc)::value, k1 = (k + 1) % 3, k2 = (k + 2) % 3;
        if (q >= nr) return;
        operands(k1, q + 1);
        entries(k2);
        const uint32_t i = at(q);
        F s = S[k];
#pragma unroll
        for (int c = 0; c < PC; ++c) {
            if (c > 0 && (uint32_t)c >= R[k].y) break;
#pragma unroll
            for (int f = 0; f < HS_CHUNK; ++f) {
                const HsPair<F> &e = E[k][c * HS_CHUNK + f];
                s = sub(s, mul(e.off == ip ? xp : X[k][c * HS_CHUNK + f], e.v));
            }
        }
        for (uint32_t c = PC; c < R[k].y; ++c) {
            HsPair<F> e[PE];
            F m[HS_CHUNK];
            chunk(e, 0, R[k].x + c);
#pragma unroll
            for (int f = 0; f < HS_CHUNK; ++f) m[f] = mul(x_at(e[f].off), e[f].v);
#pragma unroll
            for (int f = 0; f < HS_CHUNK; ++f) s = sub(s, m[f]);
        }
        xp = add(O[k], mul(mul(w, D[k]), s));
        x[i * NV] = xp;
        ip = i * (uint32_t)(NV * sizeof(F));
        R[k] = rows[at(q + 3)];
    };
    R[0] = rows[at(0)];
    R[1] = rows[at(1)];
    R[2] = rows[at(2)];
    entries(0);
    entries(1);
    operands(0, 0);
    using K0 = std::integral_constant<int, 0>;
    using K1 = std::integral_constant<int, 1>;
    using K2 = std::integral_constant<int, 2>;
    for (uint32_t q = 0; q < nr; q += 3) {
        step(K0(), q);
        step(K1(), q + 1);
        step(K2(), q + 2);
    }
}

// IO void: t is b - A_offblock x_old, or b itself where x starts from zero (xin
// null). Otherwise t is b, and the thread block forms the lagged term from xin
// and the off-block entries with columns IO; xout is then another vector than
// xin, since other blocks still read their neighbours' old values. Its products
// (thread = entry and right-hand side, coalesced, all gathers in flight) go to
// shared memory a window at a time, and every (row, right-hand side) adds its
// own in entry order: the same sums as the separate residual kernel, without
// its launch, its pass over t and its chain of gathers down a row.
template <typename F, typename I, int NV, int PC, typename IO = void>
__global__ void __launch_bounds__(HS_THREADS)
    k_hsgs_block(const uint32_t *__restrict__ row, const I *__restrict__ gcol,
                 const F *__restrict__ gval, HsgsShape sh, HsgsOff<F> off,
                 const F *__restrict__ gt, const F *xin, F *xout, const F *__restrict__ gd,
                 const double *__restrict__ relax_sc) {
    constexpr bool LAG = !std::is_same<IO, void>::value;
    extern __shared__ __align__(16) unsigned char hs_smem[];
    const uint32_t cap = sh.rows * sh.group;
    const uint32_t vecb = hs_round16((cap + sh.group) * NV * (uint32_t)sizeof(F));
    HsPair<F> *ent = (HsPair<F> *)hs_smem;
    unsigned char *at16 = hs_smem + hs_round16(sh.ent_max * (uint32_t)sizeof(HsPair<F>));
    F *t = (F *)at16, *x = (F *)(at16 + vecb), *d = (F *)(at16 + 2 * vecb);
    at16 += 2 * vecb + hs_round16(cap * (uint32_t)sizeof(F));
    uint2 *chunks = (uint2 *)at16;  // a row's first chunk and its chunk count
    at16 += hs_round16(cap * 8);

    const uint64_t R0 = (uint64_t)blockIdx.x * cap;
    const uint32_t rows = (uint32_t)(sh.n - R0 < cap ? sh.n - R0 : cap);
    const uint32_t J0 = __ldg(&row[R0]), nj = __ldg(&row[R0 + rows]) - J0;
#pragma unroll 4
    for (uint32_t e = threadIdx.x; e < nj; e += HS_THREADS) {
        HsPair<F> p;
        p.off = (uint32_t)__ldg(&gcol[(uint64_t)J0 + e]) * (uint32_t)(NV * sizeof(F));
        p.v = __ldg(&gval[(uint64_t)J0 + e]);
        ent[e] = p;
    }
    for (uint32_t e = threadIdx.x; e < rows; e += HS_THREADS) {
        const uint32_t a = __ldg(&row[R0 + e]) - J0, b = __ldg(&row[R0 + e + 1]) - J0;
        chunks[e] = make_uint2(a / HS_CHUNK, (b - a) / HS_CHUNK);
    }
    for (uint32_t e = threadIdx.x; e < sh.group * NV; e += HS_THREADS)  // the padding's zeros
        x[((e / NV + 1) * (sh.rows + 1) - 1) * NV + e % NV] = F(0);
    for (uint32_t e = threadIdx.x; e < rows; e += HS_THREADS) d[e] = __ldg(&gd[R0 + e]);
    for (uint32_t e = threadIdx.x; e < rows * NV; e += HS_THREADS) {
        const uint32_t at = e + (e / NV / sh.rows) * NV;  // one padding row a Gauss-Seidel block
        t[at] = LAG ? F(0) : __ldg(&gt[R0 * NV + e]);
        x[at] = xin ? xin[R0 * NV + e] : F(0);
    }
    if constexpr (LAG) {
        F *prod = (F *)at16;
        uint32_t *optr = (uint32_t *)(prod + HS_PRODS);
        const uint32_t O0 = __ldg(&off.row[R0]), no = __ldg(&off.row[R0 + rows]) - O0;
        const IO *__restrict__ ocol = (const IO *)off.col + O0;
        const F *__restrict__ oval = off.val + O0;
        for (uint32_t e = threadIdx.x; e <= rows; e += HS_THREADS)
            optr[e] = __ldg(&off.row[R0 + e]) - O0;
        constexpr uint32_t W = HS_PRODS / NV;  // entries of a window
        for (uint32_t w0 = 0; w0 < no; w0 += W) {
            const uint32_t w1 = no - w0 < W ? no : w0 + W;
#pragma unroll 8
            for (uint32_t q = threadIdx.x; q < (w1 - w0) * NV; q += HS_THREADS)
                prod[q] = mul(__ldg(&xin[(uint32_t)__ldg(&ocol[w0 + q / NV]) * (uint32_t)NV +
                                         q % NV]),
                              __ldg(&oval[w0 + q / NV]));
            __syncthreads();
            for (uint32_t e = threadIdx.x; e < rows * NV; e += HS_THREADS) {
                const uint32_t r = e / NV, at = e + (r / sh.rows) * NV;
                const uint32_t lo = optr[r] > w0 ? optr[r] : w0;
                const uint32_t hi = optr[r + 1] < w1 ? optr[r + 1] : w1;
                F s = t[at];
#pragma unroll 8
                for (uint32_t j = lo; j < hi; ++j) s = add(s, prod[(j - w0) * NV + e % NV]);
                t[at] = s;
            }
            __syncthreads();
        }
        for (uint32_t e = threadIdx.x; e < rows * NV; e += HS_THREADS) {
            const uint32_t at = e + (e / NV / sh.rows) * NV;
            t[at] = add(mul(F(1), __ldg(&gt[R0 * NV + e])), mul(F(-1), t[at]));
        }
    }
    __syncthreads();
    const uint32_t g = threadIdx.x / NV, k = threadIdx.x % NV;
    if (g < sh.group && g * sh.rows < rows) {
        const uint32_t f = g * sh.rows;  // first row
        const uint32_t nr = rows - f < sh.rows ? rows - f : sh.rows;
        const F w = (F)relax_sc[k];
        const F *lt = t + (f + g) * NV + k;
        F *lx = x + (f + g) * NV + k;
        hs_direction<F, NV, PC>(nr, [](uint32_t q) { return q; }, chunks + f, lt, lx, d + f, ent, w);
        hs_direction<F, NV, PC>(nr, [nr](uint32_t q) { return nr - 1 - q; }, chunks + f, lt, lx,
                                d + f, ent, w);
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < rows * NV; e += HS_THREADS)
        xout[R0 * NV + e] = x[e + (e / NV / sh.rows) * NV];
}

}  // namespace k
}  // namespace xg
