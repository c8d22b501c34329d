// Device kernels of the solve phase (sm_100a).
//
// Layout: every n-vector with nv right-hand sides is stored row-major
// interleaved, element (i, k) at i*NV + k, as XAMG stores it
// (src/primitives/vector/vector.h:509-525). CSR blocks keep 32-bit row
// pointers, XAMG-narrowed column indices (u8/u16/u32) and float or double
// values.
//
// Arithmetic: products and sums use the round-to-nearest intrinsics
// (__dmul_rn, __dadd_rn, ...), which the compiler never contracts into FMA,
// and each row is accumulated in the reference's order (entry by entry, from
// 0 for y = Ax, from y for y += Ax). Every element a kernel writes therefore
// equals, bit for bit, what the reference's -ffp-contract=off CPU loop
// computes.
//
// Row schedule ("canonical order"): a block has 256 threads; thread t works on
// row slot t/NV and right-hand side t%NV, so a tile covers 256/NV consecutive
// rows and consecutive threads read consecutive x entries of a row. (The SpMV
// runs these 256 canonical threads on 256/VK physical ones, each carrying VK
// consecutive right-hand sides; see canon_partial.) Tiles are
// dealt round-robin to B = min(ntiles, 1184) blocks (8 per SM on 148 SMs).
// Dot products are accumulated per thread in tile order, combined within a
// warp by an xor butterfly (offsets 16..NV), across the 8 warps in warp
// order, and across blocks in 32 groups: group l sums blocks l, l+32, ... (its
// last block to finish), and a full butterfly over the groups finishes (the
// last group's). The order depends only on
// (n, NV), so results are reproducible run to run and the CPU oracle can
// replay it exactly.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

namespace xg {
namespace k {

constexpr int CT = 256;     // threads per block
constexpr int BMAX = 1184;  // block cap of the canonical schedule

// ---------------------------------------------------------------------------
// Separately rounded arithmetic
// ---------------------------------------------------------------------------
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double dvd(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float dvd(float a, float b) { return __fdiv_rn(a, b); }

template <typename T>
__device__ __forceinline__ T shfl_xor(T v, int off) {
    return __shfl_xor_sync(0xffffffffu, v, off);
}

template <typename T>
__device__ __forceinline__ T ld_cg(const T *p) {
    return __ldcg(p);
}

// ---------------------------------------------------------------------------
// Per-solver scalar block: NV-wide FP64 scalars of the Krylov recurrences,
// kept in device memory so that no kernel waits on the host for them.
// ---------------------------------------------------------------------------
enum Sc : int {
    SC_RHO = 0,
    SC_RHO0,
    SC_RES,
    SC_ALPHA,
    SC_OMEGA,
    SC_BETA,
    SC_PHI,
    SC_PSI,
    SC_THETA,
    SC_SCAL1,
    SC_SCAL2,
    SC_SCAL3,
    SC_SCAL4,
    SC_ICONV,
    SC_ALPHA_C,
    SC_OMEGA_C,
    SC_NSCAL,  // -(omega*beta), the v coefficient of the p update
    SC_RELAX,
    SC_ETA,    // (r, r) of the reordered BiCGStab
    SC_COUNT
};
constexpr int SC_STRIDE = 32;

__host__ __device__ inline int canon_rows_per_tile(int nv) { return CT / nv; }

inline int canon_blocks(uint64_t n, int nv) {
    const uint64_t R = CT / nv;
    const uint64_t nt = (n + R - 1) / R;
    return (int)(nt < (uint64_t)BMAX ? (nt == 0 ? 1 : nt) : (uint64_t)BMAX);
}

// ---------------------------------------------------------------------------
// Canonical reduction: block partials, then the last block finishes.
// ---------------------------------------------------------------------------
struct RedArgs {
    void *part;              // [BMAX][32][4] partial sums (element type of the kernel)
    unsigned *ticket;        // [0] groups done, [RED_GROUP + l] blocks of group l done;
                             // zero between launches
    unsigned *flag = nullptr;  // bit 0: a bounded wait ran out (read by the host)
    void *groups = nullptr;    // [32][32][4] sums of the groups
};
constexpr int RED_GROUPS = 32, RED_GROUP = 32;
constexpr int RED_TICKETS = RED_GROUP + RED_GROUPS;

// A block may run the 256 canonical threads with CT/VK physical threads:
// physical thread p plays canonical threads p*VK .. p*VK+VK-1 (right-hand
// sides k0 .. k0+VK-1 of one row slot) and keeps one accumulator per
// canonical thread. Canonical warp w is then physical threads
// [w*32/VK, (w+1)*32/VK), and a canonical butterfly offset `off` (a multiple
// of VK, since off >= NV >= VK) is the physical offset off/VK, so every sum is
// formed from the same operands in the same order as with VK = 1.
//
// canon_partial: the block's sum of canonical block cb's accumulators into
// part[cb] (called by every thread; zeroes acc). A physical block may run
// several canonical blocks one after the other.
template <typename T, int NV, int NRED, int VK>
__device__ __forceinline__ void canon_partial(T (&acc)[VK][NRED], const RedArgs &ra, uint32_t cb) {
    constexpr int NT = CT / VK;   // physical threads of the block
    constexpr int SUB = 32 / VK;  // physical threads of one canonical warp
    constexpr int G = NV / VK;    // physical threads of one row slot
    __shared__ T wsum[8 * NV * NRED];
    T *part = (T *)ra.part;
    const int cw = threadIdx.x / SUB, cl = threadIdx.x % SUB;  // canonical lane = cl*VK + v
#pragma unroll
    for (int v = 0; v < VK; ++v) {
#pragma unroll
        for (int r = 0; r < NRED; ++r) {
            T s = acc[v][r];
#pragma unroll
            for (int off = 16; off >= NV; off >>= 1) s = add(s, shfl_xor(s, off / VK));
            if (cl < G) wsum[(cw * NV + cl * VK + v) * NRED + r] = s;
            acc[v][r] = T(0);
        }
    }
    __syncthreads();
    for (int o = threadIdx.x; o < NV * NRED; o += NT) {  // o = k*NRED + r
        T s = wsum[o];
#pragma unroll
        for (int w = 1; w < 8; ++w) s = add(s, wsum[w * NV * NRED + o]);
        part[(size_t)cb * NV * NRED + o] = s;
    }
    __syncthreads();  // wsum is free for the next canonical block
}

// The sums of a launch from its blocks' partials: canonical blocks l, l+32, ... are
// group l; its sum is formed in block order, and the groups are added by a full
// butterfly: fin(k, sums of k). Two forms of the same sums:
//
// Few sums (canon_few: at most six): canon_final, called by every
// thread at the end of the launch block. The last block to finish forms them all, a
// warp each, lane l group l.
//
// Many: canon_group, called by every thread after each of the block's canonical
// blocks. The last canonical block of each group has its group summed, one thread a
// sum, while other blocks still run, and the last group adds the groups; one block
// forming them all kept the launch waiting for NV*NRED*B loads from one SM (the
// three dot products of 32 right-hand sides took 142 us with the SpMV's 70). Drawn
// at the end of the launch block instead, the tickets made y = A x with one dot
// product 7 to 15 % slower at nv = 16 and 32 (27-point 80^3, nv = 32: 249 against
// 271 us).
//
// The second round of fences, tickets and loads is 5 to 10 us, which few sums do not
// win back: one dot product, 512,000 rows of one entry, nv = 1, 20.9 us in groups,
// 13.1 without (27,000 rows: 10.8 and 8.0). With eight they do: a dot product at nv =
// 8, 27,000 and 512,000 rows, 9.4 and 15.0 against 10.5 and 16.3.
template <int NO>
__host__ __device__ constexpr bool canon_few() { return NO <= 6; }

template <typename T, int NV, int NRED, int NT, class Fin>
__device__ __forceinline__ void canon_final(const RedArgs &ra, uint32_t B, const Fin &fin) {
    constexpr int NW = NT / 32, NO = NV * NRED;
    __shared__ T sums[NO];
    __shared__ int is_last;
    const T *part = (const T *)ra.part;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(&ra.ticket[0], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (int o = warp; o < NO; o += NW) {
        T a = T(0);
        for (uint32_t bb = lane; bb < B; bb += RED_GROUPS)
            a = add(a, ld_cg(&part[(size_t)bb * NO + o]));
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) a = add(a, shfl_xor(a, off));
        if (lane == 0) sums[o] = a;
    }
    __syncthreads();
    if (threadIdx.x == 0) ra.ticket[0] = 0u;
    for (int kk = threadIdx.x; kk < NV; kk += NT) fin(kk, &sums[kk * NRED]);
}

template <typename T, int NV, int NRED, int NT, class Fin>
__device__ __forceinline__ void canon_group(const RedArgs &ra, uint32_t cb, uint32_t B,
                                            const Fin &fin) {
    constexpr int NW = NT / 32, NO = NV * NRED;
    __shared__ T sums[NO];
    __shared__ int is_last;
    const T *part = (const T *)ra.part;
    T *group = (T *)ra.groups;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t l = cb % RED_GROUPS, members = (B - l + RED_GROUPS - 1) / RED_GROUPS;
    const uint32_t ngroups = B < (uint32_t)RED_GROUPS ? B : (uint32_t)RED_GROUPS;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(&ra.ticket[RED_GROUP + l], 1u) == members - 1;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (int o = threadIdx.x; o < NO; o += NT) {
        T a = T(0);
#pragma unroll 8
        for (uint32_t bb = l; bb < B; bb += RED_GROUPS)
            a = add(a, ld_cg(&part[(size_t)bb * NO + o]));
        group[l * NO + o] = a;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        ra.ticket[RED_GROUP + l] = 0u;
        is_last = atomicAdd(&ra.ticket[0], 1u) == ngroups - 1;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
#pragma unroll 4
    for (int o = warp; o < NO; o += NW) {
        T a = (uint32_t)lane < ngroups ? ld_cg(&group[lane * NO + o]) : T(0);
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) a = add(a, shfl_xor(a, off));
        if (lane == 0) sums[o] = a;
    }
    __syncthreads();
    if (threadIdx.x == 0) ra.ticket[0] = 0u;
    for (int kk = threadIdx.x; kk < NV; kk += NT) fin(kk, &sums[kk * NRED]);
}

// ---------------------------------------------------------------------------
// CSR SpMV with a compile-time epilogue.
//   p = epi.pre<VK>(i, k0): the operands the row's epilogue needs
//   y = epi.init(p); for j in row i: y = y + x[col[j]*NV+k] * val[j]
//   epi.fin(i, k0, y, p, terms[VK][NRED])
// for the VK right-hand sides a thread carries; init(i, k) and
// store(i, k, y, terms) are the same for one right-hand side.
// FX is the element type x is stored in; it is converted to F on load (the
// fused form of vector::convert before a reduced-precision restriction).
// ---------------------------------------------------------------------------
template <typename F>
struct CsrArgs {
    const uint32_t *row;
    const void *col;
    const F *val;
    uint64_t n;
    float vscale = 1.0f;  // FP16-stored values: the level's power-of-two scale
};

// Shared-memory staging: a tile's entries [row[r0], row[r0+R]) (values and
// columns in their stored types) are copied into shared memory by the bulk
// copy engine (cp.async.bulk, completion on an mbarrier), double-buffered so
// that the copy of a block's next tile overlaps the work on the current one;
// every thread then walks its own row from shared memory. The copy takes the
// 16-byte-aligned part of each array range; the few entries outside it (at an
// array's unaligned start or end) are copied with plain loads by the issuing
// thread before it arrives on the barrier. Tiles with more entries than the
// staging capacity read global memory directly.

// Column index of entry j: narrowed absolute index (I unsigned) or, for
// I = int16_t, a signed offset from the row index (the 2-byte relative form
// used where every |col - row| < 32768).
template <typename I>
__device__ __forceinline__ uint64_t col_at(I c, uint64_t i) {
    if constexpr (std::is_same<I, int16_t>::value)
        return (uint64_t)((int64_t)i + (int64_t)c);
    else
        return (uint64_t)c;
}

// Right-hand sides one SpMV thread carries: x[c*NV + k0 .. k0+VK-1] is
// loaded with one vector load of up to 32 bytes, so a warp issues 1/VK of the
// shared-memory reads of (column, value) and of the gather instructions that
// a thread per right-hand side would. The canonical order does not change
// (canon_partial).
#ifndef XG_SPMV_VK64
#define XG_SPMV_VK64 2  // FP64 x
#endif
#ifndef XG_SPMV_VK32
#define XG_SPMV_VK32 4  // FP32 x
#endif
// (The launcher may also pick 4 for FP64 x on short rows.)
template <typename FX, int NV>
__host__ __device__ constexpr int spmv_vk() {
    constexpr int w = sizeof(FX) == 8 ? XG_SPMV_VK64 : XG_SPMV_VK32;
    return NV < w ? NV : w;
}

template <typename FX, int VK>
__device__ __forceinline__ void ld_x(const FX *p, FX (&o)[VK]) {
    if constexpr (VK == 1) {
        o[0] = __ldg(p);
    } else if constexpr (std::is_same<FX, double>::value && VK == 4) {
        asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
            : "=d"(o[0]), "=d"(o[1]), "=d"(o[2]), "=d"(o[3])
            : "l"(p));
    } else if constexpr (std::is_same<FX, float>::value && VK == 8) {
        asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]), "=f"(o[4]), "=f"(o[5]), "=f"(o[6]),
              "=f"(o[7])
            : "l"(p));
    } else if constexpr (std::is_same<FX, double>::value) {
#pragma unroll
        for (int h = 0; h < VK; h += 2) {
            const double2 t = __ldg(reinterpret_cast<const double2 *>(p + h));
            o[h] = t.x;
            o[h + 1] = t.y;
        }
    } else if constexpr (VK == 2) {
        const float2 t = __ldg(reinterpret_cast<const float2 *>(p));
        o[0] = t.x;
        o[1] = t.y;
    } else {
#pragma unroll
        for (int h = 0; h < VK; h += 4) {
            const float4 t = __ldg(reinterpret_cast<const float4 *>(p + h));
            o[h] = t.x;
            o[h + 1] = t.y;
            o[h + 2] = t.z;
            o[h + 3] = t.w;
        }
    }
}

// VK consecutive values of a vector as one operand: 16-byte accesses where they
// make up whole ones (the launcher checks the pointers' alignment).
template <typename T, int VK>
struct Vec {
    T v[VK];
};
template <int VK, typename T>
__device__ __forceinline__ Vec<T, VK> ldv(const T *p) {
    Vec<T, VK> o;
    if constexpr (VK * sizeof(T) % 16 == 0) {
#pragma unroll
        for (int h = 0; h < (int)(VK * sizeof(T) / 16); ++h)
            reinterpret_cast<uint4 *>(o.v)[h] = reinterpret_cast<const uint4 *>(p)[h];
    } else if constexpr (VK * sizeof(T) == 8) {
        *reinterpret_cast<uint2 *>(o.v) = *reinterpret_cast<const uint2 *>(p);
    } else {
#pragma unroll
        for (int v = 0; v < VK; ++v) o.v[v] = p[v];
    }
    return o;
}
template <int VK, typename T>
__device__ __forceinline__ void stv(T *p, const Vec<T, VK> &o) {
    if constexpr (VK * sizeof(T) % 16 == 0) {
#pragma unroll
        for (int h = 0; h < (int)(VK * sizeof(T) / 16); ++h)
            reinterpret_cast<uint4 *>(p)[h] = reinterpret_cast<const uint4 *>(o.v)[h];
    } else if constexpr (VK * sizeof(T) == 8) {
        *reinterpret_cast<uint2 *>(p) = *reinterpret_cast<const uint2 *>(o.v);
    } else {
#pragma unroll
        for (int v = 0; v < VK; ++v) p[v] = o.v[v];
    }
}
// Whether p allows ldv and stv of VK values: 16 bytes where those make up whole 16,
// 8 where they are 8 (two floats), else the value's own size.
template <int VK, typename T>
inline bool aligned_for(const T *p) {
    constexpr size_t B = VK * sizeof(T);
    return (uintptr_t)p % (B % 16 == 0 ? 16 : B == 8 ? 8 : sizeof(T)) == 0;
}

// Register budget and gathers in flight, measured on the 27-point 128^3 matrix,
// nv = 8 (us; gathers of up to 16 bytes, 1024 threads an SM and four entries at
// a time with the leftover ones one by one, before):
// * No dot products: 1024 threads an SM at 64 registers, four gathers of up to
//   16 bytes at a time; with 32-byte gathers 640 threads at 102 registers, which
//   hold four of them beside the epilogue's operands (at 64 registers the
//   Chebyshev step spills). FP64 y = A x 272 -> 226, Chebyshev step 340 -> 248;
//   BF16 values 150 -> 109 and 185 -> 137.
// * Dot products: the canonical 1,184 blocks are eight an SM, so with four
//   right-hand sides a thread 512 threads have 128 registers: eight 16-byte or
//   six 32-byte gathers in flight. Three dots 340 -> 263 (FP32 x), 340 -> 269
//   (FP64 x); one dot 285 -> 246. Two right-hand sides a thread keep four gathers:
//   six took 75 us for one dot of the 27-point 80^3 matrix at nv = 2 against 70, and
//   more on short rows, whose leftover entries are a group of their own.
// * Short rows (SHORT): a row's few gathers end before more of them could be in
//   flight, so what counts is the threads: 1,024 an SM at 64 registers, although
//   some kernels then spill a few words. y = A x of a 7-point 80^3 matrix in FP64
//   at nv = 16 and 32: 60 and 117 us with 640 threads an SM, 48 and 89 with 1,024.
//   Not where all tiles run at once anyway: 12^3 to 30^3, nv = 4, 4.3 and 5.2 us
//   against 6.2.
template <typename FX, int VK, int NRED, int SHORT>
constexpr int spmv_min_blocks() {
    if (NRED > 0) return VK > 1 ? 8 : 4;
    return VK * sizeof(FX) >= 32 && !SHORT ? 5 * VK / 2 : 4 * VK;
}
template <typename FX, int VK, int NRED>
constexpr int spmv_unroll() {
    return NRED > 0 && VK == 4 ? (sizeof(FX) == 8 ? 6 : 8) : 4;
}

// A stored matrix value in the arithmetic type F: the value itself, or a
// BF16 value widened exactly to float.
template <typename F, typename V>
__device__ __forceinline__ F val_as(V v) {
    if constexpr (std::is_same<V, __nv_bfloat16>::value)
        return (F)__bfloat162float(v);
    else
        return (F)v;
}
// The same with a scale: an FP16-stored value times its level's power-of-two
// scale (an exact product), every other storage type as above.
template <typename F, typename V>
__device__ __forceinline__ F val_as(V v, float sc) {
    if constexpr (std::is_same<V, __half>::value)
        return (F)__fmul_rn(__half2float(v), sc);
    else
        return val_as<F, V>(v);
}

// Column index in 32 bits (the launcher checks that every x offset c*NV + k
// fits): the gather address is one 32-bit multiply-add and one widening add.
template <typename I>
__device__ __forceinline__ uint32_t col_at32(I c, uint32_t i) {
    if constexpr (std::is_same<I, int16_t>::value)
        return (uint32_t)((int32_t)i + (int32_t)c);
    else
        return (uint32_t)c;
}

// Row accumulation, entry by entry in row order: U gathers issue before the
// sums that use them, and a row's last few entries (27 = 6 x 4 + 3) issue
// together too instead of one by one; the additions stay in order. cl/vl point at
// the row's first entry.
template <typename F, typename FX, typename I, int NV, int VK, int NRED, typename V = F>
__device__ __forceinline__ void row_sum(F (&y)[VK], uint32_t len, uint64_t i, int k0, const I *cl,
                                        const V *vl, const FX *x, float vsc = 1.0f) {
    const uint32_t i32 = (uint32_t)i;
    constexpr int U = spmv_unroll<FX, VK, NRED>();
    uint32_t j = 0;
    for (; j + U <= len; j += U) {
        F a[U];
        FX xv[U][VK];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const uint32_t c = col_at32<I>(cl[j + q], i32);
            a[q] = val_as<F, V>(vl[j + q], vsc);
            ld_x<FX, VK>(x + (c * (uint32_t)NV + (uint32_t)k0), xv[q]);
        }
#pragma unroll
        for (int q = 0; q < U; ++q)
#pragma unroll
            for (int v = 0; v < VK; ++v) y[v] = add(y[v], mul((F)xv[q][v], a[q]));
    }
    if (j < len) {  // fewer than U left: the last entry stands in for the missing ones
        F a[U];
        FX xv[U][VK];
#pragma unroll
        for (int q = 0; q < U - 1; ++q) {
            const uint32_t e = j + q < len ? j + q : len - 1;
            const uint32_t c = col_at32<I>(cl[e], i32);
            a[q] = val_as<F, V>(vl[e], vsc);
            ld_x<FX, VK>(x + (c * (uint32_t)NV + (uint32_t)k0), xv[q]);
        }
#pragma unroll
        for (int q = 0; q < U - 1; ++q)
            if (j + q < len)
#pragma unroll
                for (int v = 0; v < VK; ++v) y[v] = add(y[v], mul((F)xv[q][v], a[q]));
    }
}

// --- mbarrier and bulk-copy primitives (PTX) -------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *m, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(m)), "r"(count)
                 : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect(uint64_t *m, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(m)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *m, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(m)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Waits for phase `parity` of the barrier for at most limit_ns nanoseconds
// of the global timer (and a bounded number of polls); false if the limit ran
// out.
constexpr uint64_t WAIT_LIMIT_NS = 2000000000ull;
__device__ __forceinline__ bool mbar_wait(uint64_t *m, uint32_t parity,
                                          uint64_t limit_ns = WAIT_LIMIT_NS) {
    if (mbar_try_wait(m, parity)) return true;
    const uint64_t t0 = global_ns();
    for (uint32_t it = 0; it < (1u << 30); ++it) {
        if (mbar_try_wait(m, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
    return false;
}
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes,
                                         uint64_t *m) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
        "[%3];" ::"r"(smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(m))
        : "memory");
}

// Staging plan of entries [j0, j1) of an array of n elements of T: the
// 16-byte-aligned global range [c0, c1) goes by bulk copy (src/dst/return
// value: its source, destination and byte count) and entry j lands at
// sbuf[j - j0 + stage_shift(arr, j0)]; entries outside [c0, c1) are copied
// here with plain loads.
template <typename T>
__device__ __forceinline__ uint32_t stage_range(T *sbuf, const T *arr, uint64_t n, uint32_t j0,
                                                uint32_t j1, const T *&src, T *&dst) {
    constexpr uintptr_t A16 = 15;
    const uintptr_t base = (uintptr_t)arr, end = (uintptr_t)(arr + n);
    const uintptr_t lo = (uintptr_t)(arr + j0), hi = (uintptr_t)(arr + j1);
    const uintptr_t g0 = lo & ~A16;
    const uintptr_t b16 = (base + A16) & ~A16, e16 = end & ~A16, h16 = (hi + A16) & ~A16;
    uintptr_t c0 = g0 > b16 ? g0 : b16;
    uintptr_t c1 = h16 < e16 ? h16 : e16;
    if (c1 <= c0) c0 = c1 = lo;  // nothing aligned to copy in bulk
    T *s0 = sbuf + (lo - g0) / sizeof(T);  // s0[j - j0] is entry j's slot
    const uint32_t cnt = j1 - j0;
    uint32_t head = c0 > lo ? (uint32_t)((c0 - lo) / sizeof(T)) : 0u;  // entries before c0
    if (head > cnt) head = cnt;
    for (uint32_t e = 0; e < head; ++e) s0[e] = arr[j0 + e];
    uint32_t tail = c1 > lo ? (uint32_t)((c1 - lo) / sizeof(T)) : 0u;  // first entry at/after c1
    if (tail < head) tail = head;
    for (uint32_t e = tail; e < cnt; ++e) s0[e] = arr[j0 + e];
    src = (const T *)c0;
    dst = sbuf + (c0 - g0) / sizeof(T);
    return (uint32_t)(c1 - c0);
}

template <typename T>
__device__ __forceinline__ uint32_t stage_shift(const T *arr, uint32_t j0) {
    return (uint32_t)(((uintptr_t)(arr + j0) & 15) / sizeof(T));
}

// Kernel with dynamic shared memory: nbuf (1 or 2) buffers, each of cap
// entries of values and columns plus 32 bytes of alignment slack per array;
// tiles with more entries read global memory directly. V is the type the
// values are stored in: F, or BF16 for an FP32 level stored in BF16 (the
// arithmetic stays in F).
// CT/VK threads; thread p carries row slot p/(NV/VK) and right-hand sides
// k0 = (p % (NV/VK))*VK .. k0+VK-1 (x aligned to VK elements).
// Tiles are dealt round-robin to B canonical blocks (tile t to block t % B);
// physical block p runs canonical blocks p, p + gridDim.x, ... in turn, so a
// grid of the blocks that fit the GPU at once covers any B. Without dot
// products B is simply the grid size, and the tiles may be dealt in runs of
// `run` consecutive tiles (run q to block q % gridDim.x), so that a block's
// successive tiles share columns in its SM's L1.
template <typename F, typename FX, typename I, int NV, int VK, int NRED, class Epi,
          typename V = F, int SHORT = 0>
__global__ void __launch_bounds__(CT / VK, spmv_min_blocks<FX, VK, NRED, SHORT>())
    k_spmv(CsrArgs<F> A, const FX *__restrict__ x, Epi epi, RedArgs ra, uint32_t cap,
           uint32_t nbuf, uint32_t B, uint32_t run = 1, uint32_t stride = 0) {
    constexpr int G = NV / VK;
    constexpr int R = CT / NV;
    constexpr int NR = NRED > 0 ? NRED : 1;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t mbar[2];
    const uint32_t VB = ((cap * (uint32_t)sizeof(V) + 32u) + 15u) & ~15u;
    const uint32_t BB = VB + (((cap * (uint32_t)sizeof(I) + 32u) + 15u) & ~15u);
    const uint32_t CAP = cap;
    const int rt = threadIdx.x / G, k0 = (threadIdx.x % G) * VK;
    const uint32_t *__restrict__ row = A.row;
    const I *__restrict__ col = (const I *)A.col;
    const V *__restrict__ val = (const V *)A.val;
    const uint32_t n = (uint32_t)A.n;  // rows, tiles and elements fit in 32 bits (launcher)
    const uint32_t ntiles = n / R + (n % R != 0);
    // A position in this physical block's sequence of tiles (END: past it);
    // positions are tiles except in the plane walk below. NRED == 0: `left`
    // positions of the current run remain, this one included; NRED > 0: `left`
    // is the canonical block.
    constexpr uint32_t END = 0xFFFFFFFFu;
    struct Pos {
        uint32_t t, left;
    };
    auto after = [&](Pos p) -> Pos {
        uint64_t t;
        if constexpr (NRED == 0) {
            t = (uint64_t)p.t + 1;
            if (p.left > 1) {
                --p.left;
            } else {
                t += (uint64_t)(gridDim.x - 1) * run;
                p.left = run;
            }
        } else {
            t = (uint64_t)p.t + B;
            if (t >= ntiles) {
                p.left += gridDim.x;
                t = p.left < B ? p.left : ntiles;
            }
        }
        p.t = t < ntiles ? (uint32_t)t : END;
        return p;
    };
    // Plane walk (no dot products, stride > 0): the blocks run through walk
    // positions u as above, position u being tile (u % M) * stride + u / M for
    // u < M * stride (M = ntiles / stride) and tile u after that: a
    // bijection, under which consecutive positions are tiles stride apart.
    auto first_row = [&](uint32_t u) -> uint32_t {
        if constexpr (NRED == 0)
            if (stride) {
                const uint32_t wM = ntiles / stride;
                if (u < wM * stride) u = (u % wM) * stride + u / wM;
            }
        return u * R;
    };
    // This thread's row of a tile: its index (n or more: none) and its entries.
    // The row pointers are read a tile ahead of their use, so that neither
    // the copy of the next tile nor the row sum waits for them.
    struct Row {
        uint32_t r0, j0, j1;
    };
    auto row_of = [&](uint32_t u) -> Row {
        Row r;
        r.r0 = first_row(u);
        const uint32_t i = r.r0 + rt;
        r.j0 = __ldg(&row[i < n ? i : n]);
        r.j1 = __ldg(&row[i < n ? i + 1 : n]);
        return r;
    };
    F acc[VK][NR];
#pragma unroll
    for (int v = 0; v < VK; ++v)
#pragma unroll
        for (int r = 0; r < NR; ++r) acc[v][r] = F(0);

    if (threadIdx.x == 0) {
        mbar_init(&mbar[0], 1);
        mbar_init(&mbar[1], 1);
        mbar_init_fence();
    }
    __syncthreads();
    uint32_t n_issued = 0, n_used = 0;  // staged tiles issued (thread 0) / consumed
    bool timed_out = false;
    // first entry past a tile that starts at row r0
    auto tile_end = [&](uint32_t r0) { return __ldg(&row[n - r0 > (uint32_t)R ? r0 + R : n]); };
    // thread 0: copy a tile's entries into the next buffer if they fit
    auto issue = [&](uint32_t j0, uint32_t j1) {
        if (j1 - j0 > CAP) return;
        unsigned char *buf = smem_raw + (size_t)(n_issued % nbuf) * BB;
        uint64_t *m = &mbar[n_issued % nbuf];
        ++n_issued;
        const V *vsrc;
        V *vdst;
        const I *csrc;
        I *cdst;
        const uint64_t nnz = __ldg(&row[n]);
        const uint32_t vb = stage_range<V>((V *)buf, val, nnz, j0, j1, vsrc, vdst);
        const uint32_t cb = stage_range<I>((I *)(buf + VB), col, nnz, j0, j1, csrc, cdst);
        mbar_arrive_expect(m, vb + cb);  // releases the plain-load writes above
        fence_proxy_async_smem();
        if (vb) bulk_g2s(vdst, vsrc, vb, m);
        if (cb) bulk_g2s(cdst, csrc, cb, m);
    };
    Pos at{NRED == 0 ? blockIdx.x * run : blockIdx.x, NRED == 0 ? run : blockIdx.x};
    if (at.t >= ntiles) at.t = END;
    Pos an = at;
    Row cur{}, nxt{};
    if (at.t != END) {
        cur = row_of(at.t);
        if (threadIdx.x == 0) issue(cur.j0, tile_end(cur.r0));  // thread 0 has the first row
        an = after(at);
        if (an.t != END) nxt = row_of(an.t);
    }
    while (at.t != END) {
        const bool more = an.t != END;
        if (nbuf == 2 && threadIdx.x == 0 && more) issue(nxt.j0, tile_end(nxt.r0));
        Pos ann = an;
        Row nn{};
        if (more) {
            ann = after(an);
            if (ann.t != END) nn = row_of(ann.t);
        }
        const uint32_t i = cur.r0 + rt;
        // the epilogue's operands are on their way while the row is summed
        typename Epi::template Pre<VK> pre;
        if (i < n) pre = epi.template pre<VK>(i, k0);
        const uint32_t tj0 = __ldg(&row[cur.r0]);
        bool staged = tile_end(cur.r0) - tj0 <= CAP;
        const V *sv = nullptr;
        const I *sc = nullptr;
        if (staged) {
            const uint32_t b = n_used % nbuf;
            // a copy that never landed: raise the flag, read global memory
            if (!mbar_wait(&mbar[b], (n_used / nbuf) & 1u)) timed_out = true;
            ++n_used;
            const unsigned char *buf = smem_raw + (size_t)b * BB;
            sv = (const V *)buf + stage_shift<V>(val, tj0);
            sc = (const I *)(buf + VB) + stage_shift<I>(col, tj0);
            staged = !timed_out;
        }
        if (i < n) {
            F y[VK];
            epi.template init<VK>(y, pre);
            const uint32_t len = cur.j1 - cur.j0, o = cur.j0 - tj0;
            if (staged)
                row_sum<F, FX, I, NV, VK, NRED, V>(y, len, i, k0, sc + o, sv + o, x, A.vscale);
            else
                row_sum<F, FX, I, NV, VK, NRED, V>(y, len, i, k0, col + cur.j0, val + cur.j0, x,
                                             A.vscale);
            epi.template fin<VK>(i, k0, y, pre, acc);
        }
        __syncthreads();  // every reader is done with this tile's buffer
        if (nbuf == 1 && threadIdx.x == 0 && more) issue(nxt.j0, tile_end(nxt.r0));
        if constexpr (NRED > 0)
            if (!more || an.left != at.left) {
                canon_partial<F, NV, NRED, VK>(acc, ra, at.left);
                if constexpr (!canon_few<NV * NRED>())
                    canon_group<F, NV, NRED, CT / VK>(ra, at.left, B, epi);
            }
        at = an;
        an = ann;
        cur = nxt;
        nxt = nn;
    }
    if (timed_out) {
        atomicOr(ra.flag, 1u);
        // no block exits with a copy into its shared memory still in flight
        if (threadIdx.x == 0)
            for (uint32_t u = n_used; u < n_issued; ++u) mbar_wait(&mbar[u % nbuf], (u / nbuf) & 1u);
    }
    if constexpr (NRED > 0 && canon_few<NV * NRED>())
        canon_final<F, NV, NRED, CT / VK>(ra, B, epi);
}

// Warp-per-row SpMV for matrices with few rows (the coarse levels and their
// transfers), where k_spmv's time is one thread's chain of gathers down a
// whole row. A warp takes one row at a time: its lanes read up to 32 entries
// (one each, coalesced), then gather the products of 32/NV entries at once
// (lane = entry slot * NV + right-hand side, the entry by shuffle), each
// product rounded on its own (mul(x, a), as row_sum rounds it), into a
// shared-memory chunk of WCH entries; then lane k < NV adds the chunk's
// products to its sum in entry order. So every output element is the same
// sequence of separately rounded products and sums as in k_spmv, while a
// row's gathers are in flight together. The next entries, the next row's
// pointers and the epilogue's operands are on their way meanwhile.
constexpr int WT = 256;  // threads per block (8 warps)
template <int NV>
constexpr int wide_chunk() { return 512 / NV; }  // entries per warp-chunk
template <typename F, typename FX, typename I, int NV, class Epi, typename V = F>
__global__ void __launch_bounds__(WT) k_spmv_wide(CsrArgs<F> A, const FX *__restrict__ x, Epi epi) {
    constexpr int E = 32 / NV;  // entries a warp gathers per round
    constexpr int CH = wide_chunk<NV>();
    constexpr int GE = CH < 32 ? CH : 32;  // entries read at once, one a lane
    __shared__ F prod[WT / 32][CH * NV];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = lane % NV, es = lane / NV;
    const uint32_t *__restrict__ row = A.row;
    const I *__restrict__ col = (const I *)A.col;
    const V *__restrict__ val = (const V *)A.val;
    F *pw = prod[warp];
    const uint64_t nw = (uint64_t)gridDim.x * (WT / 32);
    uint64_t i = (uint64_t)blockIdx.x * (WT / 32) + warp;
    uint32_t j0 = 0, j1 = 0;
    if (i < A.n) {
        j0 = __ldg(&row[i]);
        j1 = __ldg(&row[i + 1]);
    }
    for (; i < A.n; i += nw) {
        const uint32_t i32 = (uint32_t)i;
        typename Epi::template Pre<1> pre;
        F y[1] = {F(0)};
        uint32_t nj0 = 0, nj1 = 0;
        uint32_t cn = 0;  // entry j0 + lane of the group to come
        F vn = F(0);
        if (lane < GE && j0 + lane < j1) {
            cn = col_at32<I>(__ldg(&col[j0 + lane]), i32);
            vn = val_as<F, V>(__ldg(&val[j0 + lane]), A.vscale);
        }
        if (lane < NV) pre = epi.template pre<1>(i32, lane);
        if (i + nw < A.n) {
            nj0 = __ldg(&row[i + nw]);
            nj1 = __ldg(&row[i + nw + 1]);
        }
        if (lane < NV) epi.template init<1>(y, pre);
        for (uint32_t c0 = j0; c0 < j1; c0 += CH) {
            const uint32_t len = j1 - c0 < (uint32_t)CH ? j1 - c0 : (uint32_t)CH;
            for (uint32_t g0 = 0; g0 < len; g0 += GE) {
                const uint32_t c = cn;
                const F av = vn;
                const uint32_t jn = c0 + g0 + GE + lane;
                if (lane < GE && jn < j1) {
                    cn = col_at32<I>(__ldg(&col[jn]), i32);
                    vn = val_as<F, V>(__ldg(&val[jn]), A.vscale);
                }
#pragma unroll 8
                for (int r = 0; r < GE / E; ++r) {
                    const int e = r * E + es;
                    const uint32_t ce = __shfl_sync(0xffffffffu, c, e);
                    const F ae = __shfl_sync(0xffffffffu, av, e);
                    if (g0 + e < len)
                        pw[(g0 + e) * NV + k] =
                            mul((F)__ldg(&x[ce * (uint32_t)NV + (uint32_t)k]), ae);
                }
            }
            __syncwarp();
            if (lane < NV) {
#pragma unroll 8
                for (uint32_t e = 0; e < len; ++e) y[0] = add(y[0], pw[e * NV + lane]);
            }
            __syncwarp();
        }
        F none[1][1] = {{F(0)}};
        if (lane < NV) epi.template fin<1>(i32, lane, y, pre, none);
        j0 = nj0;
        j1 = nj1;
    }
}

// Bounded-wait check: one block waits on an mbarrier that nothing arrives
// at, gives up after limit_ns and raises the timeout flag, as a staging wait
// of k_spmv does when its copy never lands. Nothing is in flight when it
// returns.
static __global__ void k_wait_selftest(uint64_t limit_ns, unsigned *flag) {
    __shared__ __align__(8) uint64_t m;
    if (threadIdx.x == 0) {
        mbar_init(&m, 1);
        mbar_init_fence();
    }
    __syncthreads();
    if (!mbar_wait(&m, 0, limit_ns) && threadIdx.x == 0) atomicOr(flag, 1u);
}

// Largest entry count of a tile of R rows (for matrices whose row pointers
// live only on the device).
static __global__ void k_tile_max(const uint32_t *__restrict__ row, uint64_t n, uint64_t R,
                                  unsigned *out) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t r0 = t * R;
    if (r0 < n) {
        const uint64_t r1 = r0 + R < n ? r0 + R : n;
        atomicMax(out, row[r1] - row[r0]);
    }
}

// Element-wise canonical kernel (same schedule, no matrix). At most 64
// registers a thread, so that four 256-thread blocks share an SM (the merged
// group kernels with nv <= 8 take 76 registers left alone, three blocks);
// these streaming kernels are bound by the loads in flight. With VK > 1 a
// thread plays VK canonical threads of a row with 16-byte accesses (elemv): as
// many threads an SM in blocks of CT/VK, VK times the bytes in flight.
template <typename F, int NV, int NRED, class Epi, int VK = 1>
__global__ void __launch_bounds__(CT / VK, 4 * VK) k_rows(uint64_t n, Epi epi, RedArgs ra) {
    constexpr int R = CT / NV, G = NV / VK;
    constexpr int NR = NRED > 0 ? NRED : 1;
    const int rt = threadIdx.x / G, k0 = (threadIdx.x % G) * VK;
    const uint64_t ntiles = (n + R - 1) / R;
    F acc[VK][NR];
#pragma unroll
    for (int v = 0; v < VK; ++v)
#pragma unroll
        for (int r = 0; r < NR; ++r) acc[v][r] = F(0);
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint64_t i = tile * R + rt;
        if (i < n) {
            if constexpr (VK == 1)
                epi.elem(i, k0, acc[0]);
            else
                epi.template elemv<VK>(i, k0, acc);
        }
    }
    if constexpr (NRED > 0) {
        canon_partial<F, NV, NRED, VK>(acc, ra, blockIdx.x);
        if constexpr (canon_few<NV * NRED>())
            canon_final<F, NV, NRED, CT / VK>(ra, gridDim.x, epi);
        else
            canon_group<F, NV, NRED, CT / VK>(ra, blockIdx.x, gridDim.x, epi);
    }
}

// Scalar-only kernel: one thread per right-hand side.
template <class Op>
__global__ void k_scalar(int nv, Op op) {
    if ((int)threadIdx.x < nv) op(threadIdx.x);
}

// ---------------------------------------------------------------------------
// Epilogues. `NoFin` is used when the epilogue has no reduction.
// ---------------------------------------------------------------------------
struct NoFin {
    template <typename T>
    __device__ void operator()(int, const T *) const {}
};

// The epilogues of SpMVs without dot products, as the autotuner tells them apart:
// plain products, which read at most y beside the sum, and the smoothers' steps and
// residuals with their vectors. Each kind has a launch shape of its own in the
// matrix (DCsr::tuned, DCsr::st_choice), so that a product that somebody asks for
// does not decide the smoother's.
enum TuneKind : int { TK_PLAIN = 0, TK_SMOOTH, TK_COUNT };

// What every SpMV epilogue shares: a row sum that starts from zero, and the
// one-right-hand-side forms written with the vector ones. (redirect, where there
// are no dot products: the outputs go to scratch vectors a and b; the autotuner
// times the very kernel that the solve launches.) D is the epilogue,
// F its arithmetic type. Elements are indexed in 32 bits (the launchers check
// that they fit).
template <class D, typename F>
struct EpiBase {
    // bytes per value of the scratch vectors redirect() takes
    static constexpr size_t SCRATCH_A = sizeof(F), SCRATCH_B = 0;
    __device__ F init(uint64_t, int) const { return F(0); }
    template <int VK, class P>
    __device__ void init(F (&y)[VK], const P &) const {
#pragma unroll
        for (int v = 0; v < VK; ++v) y[v] = F(0);
    }
    template <int NR>
    __device__ void store(uint64_t i, int k, F v, F (&acc)[NR]) const {
        const D &d = static_cast<const D &>(*this);
        F y[1] = {v};
        d.template fin<1>((uint32_t)i, k, y, d.template pre<1>((uint32_t)i, k), reinterpret_cast<F(&)[1][NR]>(acc));
    }
};

// y = A x  (csr_matvec.inl:213-231)
template <typename F, int NV>
struct EStore : EpiBase<EStore<F, NV>, F>, NoFin {
    static constexpr int KIND = TK_PLAIN;
    F *y;
    __host__ __device__ explicit EStore(F *y_) : y(y_) {}
    template <int VK>
    bool aligned() const { return aligned_for<VK>(y); }
    void redirect(void *a, void *) { y = (F *)a; }
    template <int VK>
    struct Pre {};
    template <int VK>
    __device__ Pre<VK> pre(uint32_t, int) const { return {}; }
    template <int VK, int NR>
    __device__ void fin(uint32_t i, int k0, const F (&s)[VK], const Pre<VK> &,
                        F (&)[VK][NR]) const {
        Vec<F, VK> o;
#pragma unroll
        for (int v = 0; v < VK; ++v) o.v[v] = s[v];
        stv<VK>(y + (i * NV + k0), o);
    }
};

// y += A x  (csr_matvec.inl:106-120: accumulate directly into y)
template <typename F, int NV>
struct EAxpy : NoFin {
    static constexpr int KIND = TK_PLAIN;
    static constexpr size_t SCRATCH_A = sizeof(F), SCRATCH_B = 0;
    F *y;
    __host__ __device__ explicit EAxpy(F *y_) : y(y_) {}
    template <int VK>
    bool aligned() const { return aligned_for<VK>(y); }
    void redirect(void *a, void *) { y = (F *)a; }
    template <int VK>
    struct Pre {
        Vec<F, VK> y;
    };
    template <int VK>
    __device__ Pre<VK> pre(uint32_t i, int k0) const { return {ldv<VK>(y + (i * NV + k0))}; }
    __device__ F init(uint64_t i, int k) const { return y[i * NV + k]; }
    template <int VK>
    __device__ void init(F (&s)[VK], const Pre<VK> &p) const {
#pragma unroll
        for (int v = 0; v < VK; ++v) s[v] = p.y.v[v];
    }
    template <int NR>
    __device__ void store(uint64_t i, int k, F v, F (&)[NR]) const { y[i * NV + k] = v; }
    template <int VK, int NR>
    __device__ void fin(uint32_t i, int k0, const F (&s)[VK], const Pre<VK> &,
                        F (&)[VK][NR]) const {
        Vec<F, VK> o;
#pragma unroll
        for (int v = 0; v < VK; ++v) o.v[v] = s[v];
        stv<VK>(y + (i * NV + k0), o);
    }
};

// r = 1*b + (-1)*(A x)  (solver.h:249-250: Ax_y then axpby(1, b, -1, r)),
// optionally with (r, r) (vector_norm, blas.inl:537-555).
template <typename F, int NV, bool NORM>
struct EResid : EpiBase<EResid<F, NV, NORM>, F> {
    static constexpr int KIND = TK_SMOOTH;
    F *r;
    const F *b;
    double *out;  // NORM: sums land here (nv values)
    EResid(F *r_, const F *b_, double *out_) : r(r_), b(b_), out(out_) {}
    template <int VK>
    bool aligned() const { return aligned_for<VK>(r) && aligned_for<VK>(b); }
    void redirect(void *a, void *) { r = (F *)a; }
    template <int VK>
    struct Pre {
        Vec<F, VK> b;
    };
    template <int VK>
    __device__ Pre<VK> pre(uint32_t i, int k0) const { return {ldv<VK>(b + (i * NV + k0))}; }
    template <int VK, int NR>
    __device__ void fin(uint32_t i, int k0, const F (&s)[VK], const Pre<VK> &p,
                        F (&acc)[VK][NR]) const {
        Vec<F, VK> o;
#pragma unroll
        for (int v = 0; v < VK; ++v) {
            const F rv = add(mul(F(1), p.b.v[v]), mul(F(-1), s[v]));
            o.v[v] = rv;
            if constexpr (NORM) acc[v][0] = add(acc[v][0], mul(rv, rv));
        }
        stv<VK>(r + (i * NV + k0), o);
    }
    __device__ void operator()(int k, const F *s) const {
        if constexpr (NORM) out[k] = (double)s[0];
    }
};

// merged_bicgstab_group1 after r0 = A x (blas_merged_bicgstab.inl:60-72):
// r0 = b - r0; rho0 += r0*r0; p = r = r0. The finaliser also copies
// rho0 into rho (merged_bicgstab.inl:119). Element by element: the kernel-level
// entry point passes a caller's vectors, whatever their alignment.
template <int NV>
struct EGroup1 : EpiBase<EGroup1<NV>, double> {
    double *r0, *p, *r;
    const double *b;
    double *sc;
    EGroup1(double *r0_, double *p_, double *r_, const double *b_, double *sc_)
        : r0(r0_), p(p_), r(r_), b(b_), sc(sc_) {}
    template <int VK>
    bool aligned() const { return true; }
    template <int VK>
    struct Pre {
        double b[VK];
    };
    template <int VK>
    __device__ Pre<VK> pre(uint32_t i, int k0) const {
        Pre<VK> o;
#pragma unroll
        for (int v = 0; v < VK; ++v) o.b[v] = b[i * NV + k0 + v];
        return o;
    }
    template <int VK, int NR>
    __device__ void fin(uint32_t i, int k0, const double (&s)[VK], const Pre<VK> &q,
                        double (&acc)[VK][NR]) const {
#pragma unroll
        for (int v = 0; v < VK; ++v) {
            const uint32_t e = i * NV + k0 + v;
            const double rv = sub(q.b[v], s[v]);
            r0[e] = rv;
            p[e] = rv;
            r[e] = rv;
            acc[v][0] = add(acc[v][0], mul(rv, rv));
        }
    }
    __device__ void operator()(int k, const double *s) const {
        sc[SC_RHO0 * SC_STRIDE + k] = s[0];
        sc[SC_RHO * SC_STRIDE + k] = s[0];
    }
};

// v = A p_ ; scal1 = (v, r0) ; alpha = rho / scal1
// (merged_pbicgstab.inl:140-155)
template <int NV>
struct EDotAlpha : EpiBase<EDotAlpha<NV>, double> {
    double *v;
    const double *r0;
    double *sc;
    __host__ __device__ EDotAlpha(double *v_, const double *r0_, double *sc_)
        : v(v_), r0(r0_), sc(sc_) {}
    template <int VK>
    bool aligned() const { return aligned_for<VK>(v) && aligned_for<VK>(r0); }
    template <int VK>
    struct Pre {
        Vec<double, VK> r0;
    };
    template <int VK>
    __device__ Pre<VK> pre(uint32_t i, int k0) const { return {ldv<VK>(r0 + (i * NV + k0))}; }
    template <int VK, int NR>
    __device__ void fin(uint32_t i, int k0, const double (&s)[VK], const Pre<VK> &p,
                        double (&acc)[VK][NR]) const {
        Vec<double, VK> o;
#pragma unroll
        for (int w = 0; w < VK; ++w) {
            o.v[w] = s[w];
            acc[w][0] = add(acc[w][0], mul(s[w], p.r0.v[w]));
        }
        stv<VK>(v + (i * NV + k0), o);
    }
    __device__ void operator()(int k, const double *s) const {
        sc[SC_SCAL1 * SC_STRIDE + k] = s[0];
        sc[SC_ALPHA * SC_STRIDE + k] = dvd(sc[SC_RHO * SC_STRIDE + k], s[0]);
    }
};

// t = A s_ ; phi = (t,s), psi = (t,t), theta = (s,s); omega = phi/psi;
// res = theta - omega*phi; alpha_c = iconv*alpha; omega_c = iconv*omega
// (merged_pbicgstab.inl:168-192)
template <int NV>
struct EDot3 : EpiBase<EDot3<NV>, double> {
    double *t;
    const double *s;
    double *sc;
    __host__ __device__ EDot3(double *t_, const double *s_, double *sc_) : t(t_), s(s_), sc(sc_) {}
    template <int VK>
    bool aligned() const { return aligned_for<VK>(t) && aligned_for<VK>(s); }
    template <int VK>
    struct Pre {
        Vec<double, VK> s;
    };
    template <int VK>
    __device__ Pre<VK> pre(uint32_t i, int k0) const { return {ldv<VK>(s + (i * NV + k0))}; }
    template <int VK, int NR>
    __device__ void fin(uint32_t i, int k0, const double (&y)[VK], const Pre<VK> &p,
                        double (&acc)[VK][NR]) const {
        Vec<double, VK> o;
#pragma unroll
        for (int w = 0; w < VK; ++w) {
            const double sv = p.s.v[w];
            o.v[w] = y[w];
            acc[w][0] = add(acc[w][0], mul(y[w], sv));
            acc[w][1] = add(acc[w][1], mul(y[w], y[w]));
            acc[w][2] = add(acc[w][2], mul(sv, sv));
        }
        stv<VK>(t + (i * NV + k0), o);
    }
    __device__ void operator()(int k, const double *s3) const {
        double *S = sc;
        const double phi = s3[0], psi = s3[1], theta = s3[2];
        S[SC_PHI * SC_STRIDE + k] = phi;
        S[SC_PSI * SC_STRIDE + k] = psi;
        S[SC_THETA * SC_STRIDE + k] = theta;
        const double omega = dvd(phi, psi);
        S[SC_OMEGA * SC_STRIDE + k] = omega;
        double res = mul(omega, phi);
        res = add(mul(1.0, theta), mul(-1.0, res));
        S[SC_RES * SC_STRIDE + k] = res;
        const double ic = S[SC_ICONV * SC_STRIDE + k];
        S[SC_ALPHA_C * SC_STRIDE + k] = mul(ic, S[SC_ALPHA * SC_STRIDE + k]);
        S[SC_OMEGA_C * SC_STRIDE + k] = mul(ic, omega);
    }
};

// One Jacobi sweep with x not zero (blas_merged_jacobi.inl:74-80):
// x_out = x_in + relax*d*(b - A x_in)
template <typename F, int NV>
struct EJacobi : EpiBase<EJacobi<F, NV>, F>, NoFin {
    static constexpr int KIND = TK_SMOOTH;
    F *xout;
    const F *xin, *b, *d;
    F relax;
    __host__ __device__ EJacobi(F *xout_, const F *xin_, const F *b_, const F *d_, F relax_)
        : xout(xout_), xin(xin_), b(b_), d(d_), relax(relax_) {}
    template <int VK>
    bool aligned() const { return aligned_for<VK>(xout) && aligned_for<VK>(xin) && aligned_for<VK>(b); }
    void redirect(void *a, void *) { xout = (F *)a; }
    template <int VK>
    struct Pre {
        Vec<F, VK> x, b;
        F d;
    };
    template <int VK>
    __device__ Pre<VK> pre(uint32_t i, int k0) const {
        return {ldv<VK>(xin + (i * NV + k0)), ldv<VK>(b + (i * NV + k0)), d[i]};
    }
    template <int VK, int NR>
    __device__ void fin(uint32_t i, int k0, const F (&s)[VK], const Pre<VK> &p,
                        F (&)[VK][NR]) const {
        Vec<F, VK> o;
#pragma unroll
        for (int v = 0; v < VK; ++v)
            o.v[v] = add(p.x.v[v], mul(mul(relax, p.d), sub(p.b.v[v], s[v])));
        stv<VK>(xout + (i * NV + k0), o);
    }
};

// Chebyshev, first polynomial step (chebyshev.inl:179-190):
// r = b - A x; r := r*isd; t1 = c_top * r; t1 := t1*isd (input of the next
// SpMV). x_zero: r = 1*b without the SpMV (used by k_rows through elem()).
template <typename F, int NV>
struct ECheby0 : EpiBase<ECheby0<F, NV>, F>, NoFin {
    static constexpr int KIND = TK_SMOOTH;
    static constexpr size_t SCRATCH_B = sizeof(F);
    F *rs, *t1s;
    const F *b, *isd;
    F c;
    ECheby0(F *rs_, F *t1s_, const F *b_, const F *isd_, F c_)
        : rs(rs_), t1s(t1s_), b(b_), isd(isd_), c(c_) {}
    template <int VK>
    bool aligned() const { return aligned_for<VK>(rs) && aligned_for<VK>(t1s) && aligned_for<VK>(b); }
    void redirect(void *a, void *c2) {
        rs = (F *)a;
        t1s = (F *)c2;
    }
    template <int VK>
    struct Pre {
        Vec<F, VK> b;
        F d;
    };
    template <int VK>
    __device__ Pre<VK> pre(uint32_t i, int k0) const {
        return {ldv<VK>(b + (i * NV + k0)), isd[i]};
    }
    template <int VK, int NR>
    __device__ void fin(uint32_t i, int k0, const F (&s)[VK], const Pre<VK> &p,
                        F (&)[VK][NR]) const {
        Vec<F, VK> rr, t1;
#pragma unroll
        for (int v = 0; v < VK; ++v) {
            rr.v[v] = mul(add(mul(F(1), p.b.v[v]), mul(F(-1), s[v])), p.d);
            t1.v[v] = mul(mul(c, rr.v[v]), p.d);
        }
        stv<VK>(rs + (i * NV + k0), rr);
        stv<VK>(t1s + (i * NV + k0), t1);
    }
    template <int NR>
    __device__ void elem(uint64_t i, int k, F (&)[NR]) const {
        const uint64_t e = i * NV + k;
        const F d = isd[i];
        const F rr = mul(mul(F(1), b[e]), d);
        rs[e] = rr;
        t1s[e] = mul(mul(c, rr), d);
    }
    template <int VK, int NR>
    __device__ void elemv(uint64_t i, int k0, F (&)[VK][NR]) const {
        const uint64_t e = i * NV + k0;
        const F d = isd[i];
        const Vec<F, VK> bv = ldv<VK>(b + e);
        Vec<F, VK> rr, t1;
#pragma unroll
        for (int v = 0; v < VK; ++v) {
            rr.v[v] = mul(mul(F(1), bv.v[v]), d);
            t1.v[v] = mul(mul(c, rr.v[v]), d);
        }
        stv<VK>(rs + e, rr);
        stv<VK>(t1s + e, t1);
    }
};

// The same step from x = 0 with b still in double (the input of an FP32
// multigrid preconditioner): b is rounded to float, kept in b32 for the rest
// of the cycle, and the step is taken from the rounded value, in one pass
// instead of a conversion and the step.
template <int NV>
struct ECheby0From64 : NoFin {
    float *b32, *rs, *t1s;
    const double *b;
    const float *isd;
    float c;
    ECheby0From64(float *b32_, float *rs_, float *t1s_, const double *b_, const float *isd_,
                  float c_)
        : b32(b32_), rs(rs_), t1s(t1s_), b(b_), isd(isd_), c(c_) {}
    template <int VK, int NR>
    __device__ void elemv(uint64_t i, int k0, float (&)[VK][NR]) const {
        const uint64_t e = i * NV + k0;
        const float d = isd[i];
        const Vec<double, VK> bv = ldv<VK>(b + e);
        Vec<float, VK> bf, rr, t1;
#pragma unroll
        for (int v = 0; v < VK; ++v) {
            bf.v[v] = (float)bv.v[v];
            rr.v[v] = mul(mul(1.0f, bf.v[v]), d);
            t1.v[v] = mul(mul(c, rr.v[v]), d);
        }
        stv<VK>(b32 + e, bf);
        stv<VK>(rs + e, rr);
        stv<VK>(t1s + e, t1);
    }
    template <int NR>
    __device__ void elem(uint64_t i, int k, float (&acc)[NR]) const {
        elemv<1>(i, k, reinterpret_cast<float(&)[1][NR]>(acc));
    }
};

// Chebyshev inner step i (chebyshev.inl:189-199):
// t2 = A t1s; t2 := t2*isd; t1 = c_i*rs + 1*t2; then either t1s_out = t1*isd
// (more steps) or x = 1*(t1*isd) + 1*x (last step; x_zero: x = 1*(t1*isd)).
template <typename F, int NV>
struct ECheby1 : EpiBase<ECheby1<F, NV>, F>, NoFin {
    static constexpr int KIND = TK_SMOOTH;
    F *out;  // next t1s, or x on the last step
    const F *rs, *isd;
    F c;
    int last, x_zero;
    ECheby1(F *out_, const F *rs_, const F *isd_, F c_, int last_, int x_zero_)
        : out(out_), rs(rs_), isd(isd_), c(c_), last(last_), x_zero(x_zero_) {}
    template <int VK>
    bool aligned() const { return aligned_for<VK>(out) && aligned_for<VK>(rs); }
    void redirect(void *a, void *) { out = (F *)a; }
    template <int VK>
    struct Pre {
        Vec<F, VK> rs, x;
        F d;
    };
    template <int VK>
    __device__ Pre<VK> pre(uint32_t i, int k0) const {
        Pre<VK> p;
        p.rs = ldv<VK>(rs + (i * NV + k0));
        if (last && !x_zero) p.x = ldv<VK>(out + (i * NV + k0));
        p.d = isd[i];
        return p;
    }
    template <int VK, int NR>
    __device__ void fin(uint32_t i, int k0, const F (&s)[VK], const Pre<VK> &p,
                        F (&)[VK][NR]) const {
        Vec<F, VK> o;
#pragma unroll
        for (int v = 0; v < VK; ++v) {
            const F t2 = mul(s[v], p.d);
            const F t1 = add(mul(c, p.rs.v[v]), mul(F(1), t2));
            const F t1d = mul(t1, p.d);
            if (!last)
                o.v[v] = t1d;
            else if (x_zero)
                o.v[v] = mul(F(1), t1d);
            else
                o.v[v] = add(mul(F(1), t1d), mul(F(1), p.x.v[v]));
        }
        stv<VK>(out + (i * NV + k0), o);
    }
};

// Prolongation with a reduced-precision P (mg.inl:241-249): the product is
// accumulated in float, converted to double, then x = 1*t + 1*x
// (x_zero: x = 1*t, the ax_y branch of axpby).
template <int NV>
struct EProlongMixed : EpiBase<EProlongMixed<NV>, float>, NoFin {
    static constexpr int KIND = TK_PLAIN;
    static constexpr size_t SCRATCH_A = sizeof(double);
    double *x;
    int x_zero;
    EProlongMixed(double *x_, int x_zero_) : x(x_), x_zero(x_zero_) {}
    template <int VK>
    bool aligned() const { return aligned_for<VK>(x); }
    void redirect(void *a, void *) { x = (double *)a; }
    template <int VK>
    struct Pre {
        Vec<double, VK> x;
    };
    template <int VK>
    __device__ Pre<VK> pre(uint32_t i, int k0) const {
        Pre<VK> p;
        if (!x_zero) p.x = ldv<VK>(x + (i * NV + k0));
        return p;
    }
    template <int VK, int NR>
    __device__ void fin(uint32_t i, int k0, const float (&s)[VK], const Pre<VK> &p,
                        float (&)[VK][NR]) const {
        Vec<double, VK> o;
#pragma unroll
        for (int v = 0; v < VK; ++v) {
            const double t = (double)s[v];
            o.v[v] = x_zero ? mul(1.0, t) : add(mul(1.0, t), mul(1.0, p.x.v[v]));
        }
        stv<VK>(x + (i * NV + k0), o);
    }
};

// ---------------------------------------------------------------------------
// Element-wise epilogues for k_rows
// ---------------------------------------------------------------------------

// dot[k] = (x, y)_k  (blas.inl:504-519)
template <typename F, int NV>
struct EDot {
    const F *x, *y;
    double *out;
    template <int NR>
    __device__ void elem(uint64_t i, int k, F (&acc)[NR]) const {
        const uint64_t e = i * NV + k;
        acc[0] = add(acc[0], mul(x[e], y[e]));
    }
    __device__ void operator()(int k, const F *s) const { out[k] = (double)s[0]; }
};

// merged_bicgstab_group2 (blas_merged_bicgstab.inl:127-134)
template <int NV>
struct EGroup2 {
    const double *t, *s;
    double *out;  // phi, psi, theta at out[0..nv), out[32..), out[64..)
    template <int NR>
    __device__ void elem(uint64_t i, int k, double (&acc)[NR]) const {
        const uint64_t e = i * NV + k;
        const double tv = t[e], sv = s[e];
        acc[0] = add(acc[0], mul(tv, sv));
        acc[1] = add(acc[1], mul(tv, tv));
        acc[2] = add(acc[2], mul(sv, sv));
    }
    __device__ void operator()(int k, const double *s3) const {
        out[k] = s3[0];
        out[32 + k] = s3[1];
        out[64 + k] = s3[2];
    }
};

// group4 (blas_merged_bicgstab.inl:179-185): r = s - omega*t; rho += r*r0,
// optionally preceded by the x update of merged_pbicgstab.inl:193
// (x = alpha_c*p_ + omega_c*s_ + 1*x). The finaliser does lines 207-217:
// beta = (scal1/rho)*(alpha/omega); rho = scal1; nscal = -(omega*beta);
// and, for the unpreconditioned form, alpha_c/omega_c from the current iconv
// (merged_bicgstab.inl:192-199).
// PT: the type the preconditioned vectors pa, sa are stored in (float when
// an FP32 preconditioner leaves its result in float; widened exactly).
template <int NV, bool XUPD, typename PT = double>
struct EGroup4 {
    const double *s, *t, *r0;
    double *r;
    double *x;
    const PT *pa, *sa;
    double *sc;
    template <int NR>
    __device__ void elem(uint64_t i, int k, double (&acc)[NR]) const {
        const uint64_t e = i * NV + k;
        if constexpr (XUPD) {
            const double ac = sc[SC_ALPHA_C * SC_STRIDE + k], oc = sc[SC_OMEGA_C * SC_STRIDE + k];
            x[e] = add(add(mul(ac, (double)pa[e]), mul(oc, (double)sa[e])), mul(1.0, x[e]));
        }
        const double om = sc[SC_OMEGA * SC_STRIDE + k];
        const double rv = sub(s[e], mul(om, t[e]));
        r[e] = rv;
        acc[0] = add(acc[0], mul(rv, r0[e]));
    }
    template <int VK, int NR>
    __device__ void elemv(uint64_t i, int k0, double (&acc)[VK][NR]) const {
        const uint64_t e = i * NV + k0;
        const Vec<double, VK> sv = ldv<VK>(s + e), tv = ldv<VK>(t + e), r0v = ldv<VK>(r0 + e);
        if constexpr (XUPD) {
            Vec<double, VK> xv = ldv<VK>(x + e);
            const Vec<PT, VK> pv = ldv<VK>(pa + e), qv = ldv<VK>(sa + e);
#pragma unroll
            for (int v = 0; v < VK; ++v) {
                const double ac = sc[SC_ALPHA_C * SC_STRIDE + k0 + v];
                const double oc = sc[SC_OMEGA_C * SC_STRIDE + k0 + v];
                xv.v[v] = add(add(mul(ac, (double)pv.v[v]), mul(oc, (double)qv.v[v])),
                              mul(1.0, xv.v[v]));
            }
            stv<VK>(x + e, xv);
        }
        Vec<double, VK> rv;
#pragma unroll
        for (int v = 0; v < VK; ++v) {
            rv.v[v] = sub(sv.v[v], mul(sc[SC_OMEGA * SC_STRIDE + k0 + v], tv.v[v]));
            acc[v][0] = add(acc[v][0], mul(rv.v[v], r0v.v[v]));
        }
        stv<VK>(r + e, rv);
    }
    template <int VK>
    bool aligned() const {
        return aligned_for<VK>(s) && aligned_for<VK>(t) && aligned_for<VK>(r0) && aligned_for<VK>(r) &&
               (!XUPD || (aligned_for<VK>(x) && aligned_for<VK>(pa) && aligned_for<VK>(sa)));
    }
    __device__ void operator()(int k, const double *s1) const {
        double *S = sc;
        const double scal1 = s1[0];
        S[SC_SCAL1 * SC_STRIDE + k] = scal1;
        const double scal2 = dvd(scal1, S[SC_RHO * SC_STRIDE + k]);
        const double scal3 = dvd(S[SC_ALPHA * SC_STRIDE + k], S[SC_OMEGA * SC_STRIDE + k]);
        const double beta = mul(scal2, scal3);
        S[SC_SCAL2 * SC_STRIDE + k] = scal2;
        S[SC_SCAL3 * SC_STRIDE + k] = scal3;
        S[SC_BETA * SC_STRIDE + k] = beta;
        S[SC_RHO * SC_STRIDE + k] = scal1;
        S[SC_NSCAL * SC_STRIDE + k] = mul(mul(S[SC_OMEGA * SC_STRIDE + k], beta), -1.0);
        const double ic = S[SC_ICONV * SC_STRIDE + k];
        S[SC_ALPHA_C * SC_STRIDE + k] = mul(ic, S[SC_ALPHA * SC_STRIDE + k]);
        S[SC_OMEGA_C * SC_STRIDE + k] = mul(ic, S[SC_OMEGA * SC_STRIDE + k]);
    }
};

// ---------------------------------------------------------------------------
// Flat element-wise kernels (no reduction): one thread per element e of the
// [n][NV] array, grid-stride.
// ---------------------------------------------------------------------------
template <class Op>
__global__ void __launch_bounds__(CT) k_flat(uint64_t m, Op op) {
    for (uint64_t e = (uint64_t)blockIdx.x * CT + threadIdx.x; e < m;
         e += (uint64_t)gridDim.x * CT)
        op(e);
}

// s = 1*r + (-alpha)*v  (merged_pbicgstab.inl:159-161)
struct OpSUpdate {
    double *s;
    const double *r, *v, *sc;
    int nv;
    __device__ void operator()(uint64_t e) const {
        const int k = (int)(e % nv);
        const double na = mul(sc[SC_ALPHA * SC_STRIDE + k], -1.0);
        s[e] = add(mul(1.0, r[e]), mul(na, v[e]));
    }
};

// x = alpha_c*pa + omega_c*sa + 1*x  (merged_pbicgstab.inl:193, blas_ext.inl:173-177)
template <typename PT = double>
struct OpXUpdateT {
    double *x;
    const PT *pa, *sa;
    const double *sc;
    int nv;
    __device__ void operator()(uint64_t e) const {
        const int k = (int)(e % nv);
        const double ac = sc[SC_ALPHA_C * SC_STRIDE + k], oc = sc[SC_OMEGA_C * SC_STRIDE + k];
        x[e] = add(add(mul(ac, (double)pa[e]), mul(oc, (double)sa[e])), mul(1.0, x[e]));
    }
};
using OpXUpdate = OpXUpdateT<double>;

// PCG (pcg.inl:103-150). Ap = A p with scal2 = (p, Ap); finaliser:
// alpha = scal1 / scal2, alpha_conv = iconv * alpha, then alpha = -1 * alpha
// (kept in SC_NSCAL). scal1 = (r, z) is the previous (r, z) (EPcgDots).
template <int NV>
struct EPcgAp : EpiBase<EPcgAp<NV>, double> {
    double *Ap;
    const double *p;
    double *sc;
    EPcgAp(double *Ap_, const double *p_, double *sc_) : Ap(Ap_), p(p_), sc(sc_) {}
    template <int VK>
    bool aligned() const { return aligned_for<VK>(Ap) && aligned_for<VK>(p); }
    template <int VK>
    struct Pre {
        Vec<double, VK> p;
    };
    template <int VK>
    __device__ Pre<VK> pre(uint32_t i, int k0) const { return {ldv<VK>(p + (i * NV + k0))}; }
    template <int VK, int NR>
    __device__ void fin(uint32_t i, int k0, const double (&y)[VK], const Pre<VK> &q,
                        double (&acc)[VK][NR]) const {
        Vec<double, VK> o;
#pragma unroll
        for (int w = 0; w < VK; ++w) {
            o.v[w] = y[w];
            acc[w][0] = add(acc[w][0], mul(q.p.v[w], y[w]));
        }
        stv<VK>(Ap + (i * NV + k0), o);
    }
    __device__ void operator()(int k, const double *s) const {
        double *S = sc;
        S[SC_SCAL2 * SC_STRIDE + k] = s[0];
        const double alpha = dvd(S[SC_SCAL1 * SC_STRIDE + k], s[0]);
        S[SC_ALPHA * SC_STRIDE + k] = alpha;
        S[SC_ALPHA_C * SC_STRIDE + k] = mul(S[SC_ICONV * SC_STRIDE + k], alpha);
        S[SC_NSCAL * SC_STRIDE + k] = mul(-1.0, alpha);
    }
};

// (r, z) and (r, r) in one pass; finaliser: first call scal1 = (r, z);
// afterwards scal3 = (r, z), beta = scal3 / scal1, res = (r, r), and
// scal1 = scal3 for the next iteration (XAMG recomputes dot(r, z) there from
// the same vectors, pcg.inl:105).
template <int NV>
struct EPcgDots {
    const double *r, *z;
    double *sc;
    bool first;
    template <int NR>
    __device__ void elem(uint64_t i, int k, double (&acc)[NR]) const {
        const uint64_t e = i * NV + k;
        const double rv = r[e];
        acc[0] = add(acc[0], mul(rv, z[e]));
        acc[1] = add(acc[1], mul(rv, rv));
    }
    __device__ void operator()(int k, const double *s) const {
        double *S = sc;
        if (first) {
            S[SC_SCAL1 * SC_STRIDE + k] = s[0];
            return;
        }
        S[SC_SCAL3 * SC_STRIDE + k] = s[0];
        S[SC_BETA * SC_STRIDE + k] = dvd(s[0], S[SC_SCAL1 * SC_STRIDE + k]);
        S[SC_SCAL1 * SC_STRIDE + k] = s[0];
        S[SC_RES * SC_STRIDE + k] = s[1];
    }
};

// x = alpha_conv*p + 1*x (x = alpha_conv*p while x is zero-flagged);
// r = (-alpha)*Ap + 1*r  (pcg.inl:123-127, axpby blas.inl:89-151)
struct OpPcgXR {
    double *x, *r;
    const double *p, *Ap, *sc;
    int nv;
    bool x_zero;
    __device__ void operator()(uint64_t e) const {
        const int k = (int)(e % nv);
        const double ac = sc[SC_ALPHA_C * SC_STRIDE + k], na = sc[SC_NSCAL * SC_STRIDE + k];
        x[e] = x_zero ? mul(ac, p[e]) : add(mul(ac, p[e]), mul(1.0, x[e]));
        r[e] = add(mul(na, Ap[e]), mul(1.0, r[e]));
    }
};

// p = 1*z + beta*p  (pcg.inl:142)
struct OpPcgP {
    double *p;
    const double *z, *sc;
    int nv;
    __device__ void operator()(uint64_t e) const {
        const int k = (int)(e % nv);
        p[e] = add(mul(1.0, z[e]), mul(sc[SC_BETA * SC_STRIDE + k], p[e]));
    }
};

// Reordered BiCGStab (rbicgstab.inl:44-243, merged_rbicgstab.inl:44-230).
// merged_rbicgstab_group1 (blas_merged_rbicgstab.inl:33-116): r = r - alpha v,
// then theta = (t, r), phi = (t, t), psi = (t, r0), eta = (r, r). The
// unmerged form's r = (-alpha) v + 1 r is the same value bit for bit.
// Finaliser: omega = theta / phi; res = 1 eta + (-1)(omega theta);
// alpha_conv, omega_conv; rho = -(omega psi); beta = rho / (delta omega),
// delta = (v, r0) in SC_SCAL1.
template <int NV>
struct ERbGroup1 {
    double *r;
    const double *v, *t, *r0;
    double *sc;
    template <int NR>
    __device__ void elem(uint64_t i, int k, double (&acc)[NR]) const {
        const uint64_t e = i * NV + k;
        const double rv = sub(r[e], mul(sc[SC_ALPHA * SC_STRIDE + k], v[e]));
        r[e] = rv;
        const double tv = t[e];
        acc[0] = add(acc[0], mul(tv, rv));
        acc[1] = add(acc[1], mul(tv, tv));
        acc[2] = add(acc[2], mul(tv, r0[e]));
        acc[3] = add(acc[3], mul(rv, rv));
    }
    __device__ void operator()(int k, const double *s4) const {
        double *S = sc;
        const double theta = s4[0], phi = s4[1], psi = s4[2], eta = s4[3];
        S[SC_THETA * SC_STRIDE + k] = theta;
        S[SC_PHI * SC_STRIDE + k] = phi;
        S[SC_PSI * SC_STRIDE + k] = psi;
        S[SC_ETA * SC_STRIDE + k] = eta;
        const double omega = dvd(theta, phi);
        S[SC_OMEGA * SC_STRIDE + k] = omega;
        S[SC_RES * SC_STRIDE + k] = add(mul(1.0, eta), mul(-1.0, mul(omega, theta)));
        const double ic = S[SC_ICONV * SC_STRIDE + k];
        S[SC_ALPHA_C * SC_STRIDE + k] = mul(ic, S[SC_ALPHA * SC_STRIDE + k]);
        S[SC_OMEGA_C * SC_STRIDE + k] = mul(ic, omega);
        const double rho = mul(-1.0, mul(omega, psi));
        S[SC_RHO * SC_STRIDE + k] = rho;
        S[SC_BETA * SC_STRIDE + k] = dvd(rho, mul(S[SC_SCAL1 * SC_STRIDE + k], omega));
    }
};

// t_ = 1 z + (-alpha) s  (axpby_z, blas_ext.inl:193-239, with its zero-flag
// branches)
struct OpRbT {
    double *t_;
    const double *z, *s, *sc;
    int nv;
    bool z_zero, s_zero;
    __device__ void operator()(uint64_t e) const {
        const int k = (int)(e % nv);
        const double na = mul(-1.0, sc[SC_ALPHA * SC_STRIDE + k]);
        t_[e] = z_zero ? mul(na, s[e]) : s_zero ? mul(1.0, z[e]) : add(mul(1.0, z[e]), mul(na, s[e]));
    }
};

// x = alpha_conv v_ + omega_conv t_ + 1 x (axpbypcz; x zero-flagged: without
// the x term)
__device__ __forceinline__ double rb_x(double ac, double v, double oc, double t, double x,
                                       bool x_zero) {
    return x_zero ? add(mul(ac, v), mul(oc, t)) : add(add(mul(ac, v), mul(oc, t)), mul(1.0, x));
}

// r = (-omega) t + 1 r; with x: the unmerged form's x update before the
// convergence test (rbicgstab.inl:200-205)
struct OpRbR {
    double *r, *x;
    const double *t, *v_, *t_, *sc;
    int nv;
    bool x_zero;
    __device__ void operator()(uint64_t e) const {
        const int k = (int)(e % nv);
        r[e] = add(mul(mul(-1.0, sc[SC_OMEGA * SC_STRIDE + k]), t[e]), mul(1.0, r[e]));
        if (x)
            x[e] = rb_x(sc[SC_ALPHA_C * SC_STRIDE + k], v_[e], sc[SC_OMEGA_C * SC_STRIDE + k],
                        t_[e], x[e], x_zero);
    }
};

// the merged form's x update on convergence (merged_rbicgstab.inl:199-203)
struct OpRbX {
    double *x;
    const double *v_, *t_, *sc;
    int nv;
    bool x_zero;
    __device__ void operator()(uint64_t e) const {
        const int k = (int)(e % nv);
        x[e] = rb_x(sc[SC_ALPHA_C * SC_STRIDE + k], v_[e], sc[SC_OMEGA_C * SC_STRIDE + k], t_[e],
                    x[e], x_zero);
    }
};

// Merged: merged_rbicgstab_group2 (blas_merged_rbicgstab.inl:120-193) with
// alpha_conv, omega_conv taken with the updated iconv:
//   x = x + (ac v_ + oc t_); z = t_ - omega z; v_ = (z + beta v_) - (beta omega) s.
// Unmerged (rbicgstab.inl:226-236): z = 1 t_ + (-omega) z;
//   v_ = (1 z + ((-omega) beta) s) + beta v_.
struct OpRbG2 {
    double *x, *v_, *z;
    const double *t_, *s, *sc;
    int nv;
    bool merged, x_zero;
    __device__ void operator()(uint64_t e) const {
        const int k = (int)(e % nv);
        const double om = sc[SC_OMEGA * SC_STRIDE + k], be = sc[SC_BETA * SC_STRIDE + k];
        const double tv = t_[e];
        if (merged) {
            const double ic = sc[SC_ICONV * SC_STRIDE + k];
            const double ac = mul(ic, sc[SC_ALPHA * SC_STRIDE + k]), oc = mul(ic, om);
            const double xo = x_zero ? 0.0 : x[e];
            x[e] = add(xo, add(mul(ac, v_[e]), mul(oc, tv)));
            const double zn = sub(tv, mul(om, z[e]));
            z[e] = zn;
            v_[e] = sub(add(zn, mul(be, v_[e])), mul(mul(be, om), s[e]));
        } else {
            const double nom = mul(-1.0, om);
            const double zn = add(mul(1.0, tv), mul(nom, z[e]));
            z[e] = zn;
            v_[e] = add(add(mul(1.0, zn), mul(mul(nom, be), s[e])), mul(be, v_[e]));
        }
    }
};

// p = 1*r + nscal*v + beta*p  (merged_pbicgstab.inl:216-218)
struct OpPUpdate {
    double *p;
    const double *r, *v, *sc;
    int nv;
    __device__ void operator()(uint64_t e) const {
        const int k = (int)(e % nv);
        const double ns = sc[SC_NSCAL * SC_STRIDE + k], be = sc[SC_BETA * SC_STRIDE + k];
        p[e] = add(add(mul(1.0, r[e]), mul(ns, v[e])), mul(be, p[e]));
    }
};

// merged_bicgstab_group5 (blas_merged_bicgstab.inl:241-248)
struct OpGroup5 {
    double *x, *p;
    const double *s, *r, *v, *sc;
    int nv;
    __device__ void operator()(uint64_t e) const {
        const int k = (int)(e % nv);
        const double ac = sc[SC_ALPHA_C * SC_STRIDE + k], oc = sc[SC_OMEGA_C * SC_STRIDE + k];
        const double be = sc[SC_BETA * SC_STRIDE + k];
        const double val = mul(be, sc[SC_OMEGA * SC_STRIDE + k]);
        x[e] = add(x[e], add(mul(ac, p[e]), mul(oc, s[e])));
        p[e] = sub(add(r[e], mul(be, p[e])), mul(val, v[e]));
    }
};

// First Jacobi sweep from x = 0 with r = 0 (blas_merged_jacobi.inl:61-67):
// x = relax*d*b
template <typename F>
struct OpJacobiZero {
    F *x;
    const F *b, *d;
    F relax;
    int nv;
    __device__ void operator()(uint64_t e) const {
        x[e] = mul(mul(relax, d[e / nv]), b[e]);
    }
};

template <typename T>
struct OpFill {
    T *x;
    T v;
    __device__ void operator()(uint64_t e) const { x[e] = v; }
};

template <typename TD, typename TS>
struct OpConvert {
    TD *d;
    const TS *s;
    __device__ void operator()(uint64_t e) const { d[e] = (TD)s[e]; }
};

// y = 1*x + 1*y, or y = 1*x when y is zero-flagged (axpby(a1, x, a1, y))
template <typename T>
struct OpAddInto {
    T *y;
    const T *x;
    int y_zero;
    __device__ void operator()(uint64_t e) const {
        y[e] = y_zero ? mul(T(1), x[e]) : add(mul(T(1), x[e]), mul(T(1), y[e]));
    }
};

// y[i][k] *= d[i]  (blas::scal with an nv = 1 vector, blas.inl:189-193)
template <typename F>
struct OpScaleRows {
    F *y;
    const F *d;
    int nv;
    __device__ void operator()(uint64_t e) const { y[e] = mul(y[e], d[e / nv]); }
};

// y = a_k*x + 1*y with a_k = coef[k] (axpby(relax, r, a1, x), jacobi.inl:103);
// y_zero: y = a_k*x (the ax_y branch)
template <typename F>
struct OpAxpyK {
    F *y;
    const F *x;
    const double *coef;
    int nv, y_zero;
    __device__ void operator()(uint64_t e) const {
        const F a = (F)coef[e % nv];
        y[e] = y_zero ? mul(a, x[e]) : add(mul(a, x[e]), mul(F(1), y[e]));
    }
};

// ---------------------------------------------------------------------------
// Hybrid symmetric Gauss-Seidel sweep (csr_gs.inl:77-130) over GS blocks:
// thread (block g, component k) runs the forward then the backward sweep of
// rows [off_g, off_g + size_g) with the block-local entries; t already holds
// b - A_offblock x_old. Blocks are independent, so no thread reads another
// thread's writes.
// ---------------------------------------------------------------------------
template <typename F, typename I, int NV>
__global__ void __launch_bounds__(CT)
    k_hsgs_sweep(const uint32_t *__restrict__ row, const I *__restrict__ col,
                 const F *__restrict__ val, const uint64_t *__restrict__ boff, int nblocks,
                 const F *__restrict__ t, F *__restrict__ x, const F *__restrict__ d,
                 const double *__restrict__ relax_sc) {
    const uint64_t gt = (uint64_t)blockIdx.x * CT + threadIdx.x;
    const int g = (int)(gt / NV), k = (int)(gt % NV);
    if (g >= nblocks) return;
    const uint64_t r0 = boff[g], r1 = boff[g + 1];
    if (r0 >= r1) return;
    const F w = (F)relax_sc[k];
    auto upd = [&](uint64_t i) {
        const uint64_t e = i * NV + k;
        F sum = t[e];
        for (uint32_t j = row[i]; j < row[i + 1]; ++j) {
            const uint64_t c = (uint64_t)col[j] + r0;
            sum = sub(sum, mul(x[c * NV + k], val[j]));
        }
        const F coeff = mul(w, d[i]);
        x[e] = add(x[e], mul(coeff, sum));
    };
    for (uint64_t i = r0; i < r1; ++i) upd(i);
    for (uint64_t i = r1; i-- > r0;) upd(i);
}

// --- persistent preconditioned BiCGStab ----------------------------------------
// Grid barrier with a bounded wait: every block of a cooperative launch
// arrives on one 64-bit counter (zero at the launch's start; round r ends when
// it reaches (r + 1) * expected). Thread 0 of a block arrives with a
// release-ordered atomic add and polls the counter with acquire-ordered loads;
// __syncthreads() on both sides extends that ordering to the whole block (the
// writes of every thread before the barrier are visible to every thread of
// every block after it). A monotonic counter needs no reset by the last
// arriver, so the round ends with its own arrival. A block whose wait passes
// limit_ns raises the timeout flag (read by the host as XAMG_ERR_TIMEOUT) and
// returns false, and the kernel then ends; the other blocks' next waits run
// out the same way, so no block waits without bound.
struct GridSync {
    unsigned long long *arrivals;  // zero at the launch's start
    unsigned *flag;                // bit 0: a wait ran out
    uint64_t limit_ns;
};
__device__ __forceinline__ bool grid_sync(const GridSync &g, unsigned expected) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        unsigned long long old;
        asm volatile("atom.add.release.gpu.global.u64 %0, [%1], 1;"
                     : "=l"(old)
                     : "l"(g.arrivals)
                     : "memory");
        const unsigned long long target = (old / expected + 1ull) * expected;
        uint64_t t0 = 0;
        for (uint32_t it = 0;; ++it) {
            unsigned long long cur;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];"
                         : "=l"(cur)
                         : "l"(g.arrivals)
                         : "memory");
            if (cur >= target) break;
            if ((it & 63u) == 0) {  // the clock is read every 64 polls
                const uint64_t t = global_ns();
                if (it == 0) {
                    t0 = t;
                } else if (t - t0 > g.limit_ns || it >= 0xffffff00u) {
                    atomicOr(g.flag, 1u);
                    ok = 0;
                    break;
                }
            }
        }
    }
    __syncthreads();
    return ok != 0;
}

// The last step of the canonical reduction run by every block for itself
// (the same sums, in the same order, as canon_final's), with the
// finaliser writing the block's own copy of the scalar block: no block
// depends on another's finaliser.
template <int NV, int NRED, class Fin>
__device__ __forceinline__ void canon_final_local(const double *part, uint32_t B, const Fin &fin) {
    __shared__ double sums[NV * NRED];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = warp; o < NV * NRED; o += CT / 32) {
        double a = 0.0;
        for (unsigned bb = lane; bb < B; bb += 32) a = add(a, ld_cg(&part[(size_t)bb * NV * NRED + o]));
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) a = add(a, shfl_xor(a, off));
        if (lane == 0) sums[o] = a;
    }
    __syncthreads();
    for (int kk = threadIdx.x; kk < NV; kk += CT) fin(kk, &sums[kk * NRED]);
    __syncthreads();
}

struct PersistArgs {
    double *x, *r0, *r, *p, *v, *s, *t, *pa, *sa, *tmp;
    const double *d;   // Jacobi inverse diagonal; null: no Jacobi preconditioner
    int ident;         // with d null: 1 the Identity preconditioner (pa, sa copies of p, s),
                       // 0 none (pa = p, sa = s)
    double relax;
    int sweeps;        // Jacobi sweeps (max_iters of the preconditioner list)
    double *sc;        // the solver's scalar block: read at the start, written at the end
    double *out;       // [3][32]: abs_res, rel_res, conv (0/1); [96]: iterations
    int max_iters, check;
    float abs_tol, rel_tol;
    RedArgs ra;        // partial sums: two halves used in turn
    GridSync gs;
    uint32_t B;        // canonical blocks (canon_blocks(n, NV)); the grid may be smaller
};

// A BiCGStab solve recorded as one graph (csrc/loop.cu): the convergence
// test's settings and the conditional handles it sets: loop (iterate again),
// rest (the rest of a non-converged iteration), last (the final x update).
struct LoopCtl {
    int nv, max_iters, check;
    float abs_tol, rel_tol;
    cudaGraphConditionalHandle loop, rest, last;
};
// The statistics the loop leaves in device memory (doubles): abs_res,
// rel_res and conv (0/1) per right-hand side, the iterations, and whether
// the last test passed.
constexpr int LOOP_ABS = 0, LOOP_REL = 32, LOOP_CONV = 64, LOOP_ITERS = 96, LOOP_DONE = 97,
              LOOP_COUNT = 98;

// merged_pbicgstab.inl:44-225 after its start (r0, rho0, p = r = r0 and the
// first test, done by Krylov::begin/started): every iteration, its
// convergence test (solver.h:173-241 with float32 tolerances) and the final
// x update in one cooperative launch of 256-thread blocks (grid barriers
// between the steps). Physical block p plays canonical blocks p, p + grid,
// ... of the B = canon_blocks(n, NV) (a grid smaller than B has fewer
// blocks at each barrier); every reduction is summed per canonical block in
// tile order. Each step applies the same element operations, row sums and
// canonical reductions as the separate kernels of Krylov::step_tail,
// step_body and stepped, so the iterates are the same bit for bit. Two right-hand
// sides are held to 64 registers, four blocks an SM (persist.cu: fits_nv).
template <int NV, typename I>
__global__ void __launch_bounds__(CT, NV == 2 ? 4 : 1) k_pbicgstab_persist(CsrArgs<double> A, PersistArgs P) {
    constexpr int R = CT / NV;
    __shared__ double SCS[SC_COUNT * SC_STRIDE];
    __shared__ double st_abs[NV], st_rel[NV];
    __shared__ int st_conv[NV];
    __shared__ int go;
    const uint32_t B = P.B;
    const uint64_t n = A.n;
    const uint64_t ntiles = (n + R - 1) / R;
    const int rt = threadIdx.x / NV, kk = threadIdx.x % NV;
    const uint32_t *__restrict__ row = A.row;
    const I *__restrict__ col = (const I *)A.col;
    const double *__restrict__ val = A.val;
    for (int o = threadIdx.x; o < SC_COUNT * SC_STRIDE; o += CT) SCS[o] = P.sc[o];
    for (int o = threadIdx.x; o < NV; o += CT) {
        st_abs[o] = 0.0;
        st_rel[o] = 0.0;
        st_conv[o] = 0;
    }
    __syncthreads();
    uint32_t half = 0;  // which half of the partial-sum buffer this reduction writes
    const size_t HALF = (size_t)B * NV * 4;
    auto part = [&]() { return (double *)P.ra.part + (size_t)half * HALF; };
    // every (row, right-hand side) this thread owns: canonical thread
    // threadIdx.x of the canonical blocks this block plays, tiles in order
    auto each_of = [&](uint64_t cb, auto &&fn) {
        for (uint64_t tile = cb; tile < ntiles; tile += B) {
            const uint64_t i = tile * R + rt;
            if (i < n) fn(i, (uint64_t)i * NV + kk);
        }
    };
    auto each = [&](auto &&fn) {
        for (uint64_t cb = blockIdx.x; cb < B; cb += gridDim.x) each_of(cb, fn);
    };
    // x written by other blocks in this launch: read through L2 (ld.cg), not
    // from a possibly stale L1 line
    auto rowsum = [&](const double *xv, uint64_t i) {
        double y = 0.0;
        for (uint32_t j = __ldg(&row[i]); j < __ldg(&row[i + 1]); ++j)
            y = add(y, mul(ld_cg(&xv[col_at<I>(__ldg(&col[j]), i) * NV + kk]), __ldg(&val[j])));
        return y;
    };
    auto sync = [&]() { return grid_sync(P.gs, gridDim.x); };
    // elem(i, e, acc) over every (row, right-hand side) this block owns,
    // summed per canonical block in tile order; then the grid's partials
    // summed in canonical order by every block (fin writes the scalars)
    auto reduce_each = [&](auto &acc, auto &&elem, auto &&fin) {
        constexpr int NR = sizeof(acc[0]) / sizeof(double);
        for (uint64_t cb = blockIdx.x; cb < B; cb += gridDim.x) {
#pragma unroll
            for (int r = 0; r < NR; ++r) acc[0][r] = 0.0;
            each_of(cb, [&](uint64_t i, uint64_t e) { elem(i, e, acc[0]); });
            canon_partial<double, NV, NR, 1>(acc, RedArgs{part(), nullptr, nullptr},
                                             (uint32_t)cb);
        }
        if (!sync()) return false;
        canon_final_local<NV, NR>(part(), B, fin);
        half ^= 1u;
        return true;
    };
    // out = M^-1 in: Jacobi sweeps from zero (jacobi.inl:113-119,
    // blas_merged_jacobi.inl), the last landing in out; the Identity copies;
    // without a preconditioner pa/sa are p/s themselves
    auto precond = [&](double *out, const double *in) {
        if (!P.d) {
            if (P.ident) {  // Identity::solve: x = b (ops::convert)
                const OpConvert<double, double> cp{out, in};
                each([&](uint64_t, uint64_t e) { cp(e); });
            }
            return true;
        }
        const int m = P.sweeps < 1 ? 1 : P.sweeps;
        auto tgt = [&](int j) { return ((m - j) % 2 == 0) ? out : P.tmp; };
        double *cur = tgt(1);
        const OpJacobiZero<double> jz{cur, in, P.d, P.relax, NV};
        each([&](uint64_t, uint64_t e) { jz(e); });
        for (int j = 2; j <= m; ++j) {
            if (!sync()) return false;
            double *o = tgt(j);
            const EJacobi<double, NV> ej(o, cur, in, P.d, P.relax);
            double none[1];
            each([&](uint64_t i, uint64_t) { ej.store(i, kk, rowsum(cur, i), none); });
            cur = o;
        }
        return true;
    };
    int it = 0;
    bool tail = false, done = false, ok = true;
    const EGroup4<NV, true> g4{P.s, P.t, P.r0, P.r, P.x, P.pa, P.sa, SCS};
    const OpPUpdate pu{P.p, P.r, P.v, SCS, NV};
    auto do_tail = [&]() {
        double acc[1][1] = {{0.0}};
        if (!reduce_each(acc, [&](uint64_t i, uint64_t, double(&a)[1]) { g4.elem(i, kk, a); },
                         g4))
            return false;
        each([&](uint64_t, uint64_t e) { pu(e); });
        return true;
    };
    while (ok) {
        ++it;
        if (tail && !(ok = do_tail())) break;
        if (!(ok = precond(P.pa, P.p))) break;
        if (!(ok = sync())) break;
        {   // v = A p_; alpha = rho / (v, r0)
            const EDotAlpha<NV> ea(P.v, P.r0, SCS);
            double acc[1][1] = {{0.0}};
            if (!(ok = reduce_each(
                      acc,
                      [&](uint64_t i, uint64_t, double(&a)[1]) {
                          ea.store(i, kk, rowsum(P.pa, i), a);
                      },
                      ea)))
                break;
        }
        {   // s = r - alpha v
            const OpSUpdate su{P.s, P.r, P.v, SCS, NV};
            each([&](uint64_t, uint64_t e) { su(e); });
        }
        if (!(ok = precond(P.sa, P.s))) break;
        if (!(ok = sync())) break;
        {   // t = A s_; omega, res
            const EDot3<NV> e3(P.t, P.s, SCS);
            double acc[1][3] = {{0.0, 0.0, 0.0}};
            if (!(ok = reduce_each(
                      acc,
                      [&](uint64_t i, uint64_t, double(&a)[3]) {
                          e3.store(i, kk, rowsum(P.sa, i), a);
                      },
                      e3)))
                break;
        }
        // convergence test (host_converged): every block decides alike
        if (threadIdx.x == 0) {
            bool flag = P.check != 0;
            if (flag) {
                for (int k2 = 0; k2 < NV; ++k2) {
                    if (SCS[SC_ICONV * SC_STRIDE + k2] != 0.0) {
                        const double a = sqrt(SCS[SC_RES * SC_STRIDE + k2]);
                        const double rr = a / sqrt(SCS[SC_RHO0 * SC_STRIDE + k2]);
                        if ((a > (double)P.abs_tol) && (rr > (double)P.rel_tol)) {
                            flag = false;
                        } else if (!st_conv[k2]) {
                            st_abs[k2] = a;
                            st_rel[k2] = rr;
                            st_conv[k2] = 1;
                        }
                    }
                }
                if (!flag)
                    for (int k2 = 0; k2 < NV; ++k2)
                        SCS[SC_ICONV * SC_STRIDE + k2] =
                            mul(SCS[SC_ICONV * SC_STRIDE + k2], (double)(!st_conv[k2]));
            }
            go = flag ? 0 : (it >= P.max_iters ? 1 : 2);
        }
        __syncthreads();
        if (go == 0) {   // converged: x = alpha_c p_ + omega_c s_ + x
            const OpXUpdate xu{P.x, P.pa, P.sa, SCS, NV};
            each([&](uint64_t, uint64_t e) { xu(e); });
            done = true;
            break;
        }
        tail = true;
        if (go == 1) {   // max_iters reached: the pending rest of the iteration
            ok = do_tail();
            done = ok;
            break;
        }
    }
    if (blockIdx.x == 0 && done) {
        for (int o = threadIdx.x; o < SC_COUNT * SC_STRIDE; o += CT) P.sc[o] = SCS[o];
        for (int o = threadIdx.x; o < NV; o += CT) {
            P.out[o] = st_abs[o];
            P.out[32 + o] = st_rel[o];
            P.out[64 + o] = (double)st_conv[o];
        }
        if (threadIdx.x == 0) P.out[96] = (double)it;
    }
}

// Waits at a grid barrier that one more block than the grid must reach:
// every wait runs out after limit_ns and raises the timeout flag (the
// barrier's bounded wait, exercised without a fault).
static __global__ void k_grid_selftest(GridSync g) { (void)grid_sync(g, gridDim.x + 1); }

}  // namespace k
}  // namespace xg
