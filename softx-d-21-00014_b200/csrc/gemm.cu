// BF16 GEMM on the fifth-generation tensor cores (tcgen05), FP32 accumulate:
//   C[M][N] = A[M][K] * B[N][K]^T
// with a fused epilogue (bias, ReLU, ReLU-derivative mask, loss gradient, BF16
// or FP32 output). It carries the dense layers of the learned coarse initial
// guess, the only tensor-core work of the solve phase. Either operand may also
// be given transposed (stored [K][M] or [K][N]): the MLP's weight and input
// gradients read activations and weights as the forward pass left them.
//
// One CTA computes a 128 x BN tile (BN 64, 128 or 256) over a share of K: warp 0
// streams 64-deep k-blocks of A and B into a ring of 128-byte-swizzled
// shared-memory stages with TMA (cp.async.bulk.tensor, completion on an
// mbarrier per stage), warp 1 issues tcgen05.mma (M = 128, N = BN, K = 16 per
// instruction) into a TMEM accumulator and releases each stage with
// tcgen05.commit, and warps 2-9 read the accumulator back with tcgen05.ld (each
// warp its 32-lane quarter and half of the columns) into the stages' shared
// memory, from where all threads apply the epilogue row by row: a TMEM lane is a
// row, so storing from the registers would touch 32 rows with every access.
// With few tiles the CTAs of a cluster may split K: after a cluster barrier
// every CTA sums its share of the rows over the cluster's partial tiles in rank
// order (a fixed order, no workspace) and applies the epilogue. Every wait is
// bounded (global timer); a wait that runs out raises the library's timeout flag
// and the CTA still frees its TMEM before it exits.
#include <algorithm>

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include "device.h"
#include "gemm_shape.h"
#include "ops.h"

namespace xg {
namespace ops {
namespace mm {

constexpr int MAX_STAGES = 8;
constexpr int THREADS = 320;
constexpr uint32_t BOX = 64 * BK * 2;  // one 64 x 64 TMA box of a transposed operand
// bytes of one stage: a 128 x 64 tile of A and a BN x 64 tile of B
__host__ __device__ constexpr uint32_t stage_bytes(int BN) { return (uint32_t)(BM + BN) * BK * 2; }
// pitch (floats) of a partial tile's row in shared memory: 16-byte stores of
// eight consecutive rows fall into distinct banks
__host__ __device__ constexpr uint32_t part_pitch(int BN) { return (uint32_t)BN + 4; }

enum Mode : int {
    F32 = 0,         // C = acc (+ bias)
    BF16 = 1,        // C = bf16(acc (+ bias))
    BF16_RELU = 2,   // C = bf16(max(acc + bias, 0))
    BF16_MASK = 3,   // C = bf16(acc) where aux > 0, else 0 (ReLU derivative)
    MSE_GRAD = 4,    // d = acc + bias - T; C = bf16(scale d), sum of d^2 per CTA
};

__device__ __forceinline__ uint32_t saddr(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// UMMA shared-memory matrix descriptor of an operand tile stored with the
// 128-byte swizzle. K-major: rows of 128 B (64 BF16 along K), 8-row groups
// 1024 B apart; 16 along K are 32 B. Transposed (MN-major): 64 x 64 boxes of
// 128 B rows (64 BF16 along M or N), one row per k: 8-k groups 1024 B apart,
// the next 64 of M or N one box further; 16 along K are 2048 B.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr, bool mn) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);  // start address, 16-byte units
    d |= (uint64_t)(mn ? BOX >> 4 : 1u) << 16;  // leading byte offset (unused when K-major)
    d |= (uint64_t)(1024 >> 4) << 32;         // stride byte offset: one 8-row group
    d |= (uint64_t)1 << 46;                   // descriptor version (sm_100)
    d |= (uint64_t)2 << 61;                   // layout: 128-byte swizzle
    return d;
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, N = BN,
// M = 128; bits 15 and 16 for a transposed A or B.
__device__ __forceinline__ uint32_t idesc(int BN, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
           ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y,
                                            uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
        "{%2, %3}], [%4];" ::"r"(saddr(dst)),
        "l"(map), "r"(x), "r"(y), "r"(saddr(bar))
        : "memory");
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t da, uint64_t db, uint32_t id,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(
            tmem),
        "l"(da), "l"(db), "r"(id), "r"(accumulate), "r"(0), "r"(0), "r"(0), "r"(0));
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     saddr(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// 32 consecutive FP32 accumulator columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
        "%11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, "
        "%28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Shared memory of another CTA of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct Epilogue {
    void *C;
    uint64_t ldc;
    const float *bias;   // null: none
    const void *aux;     // BF16_MASK: BF16 [M][ld_aux]; MSE_GRAD: FP32 targets [M][ld_aux]
    uint64_t ld_aux;
    float scale;         // MSE_GRAD
    double *sse;         // MSE_GRAD: one partial sum of squares per CTA
    bool aux_vec;        // four values of aux at once are aligned
};

// What the epilogue of four consecutive columns n.. of one row reads beside the
// bias.
struct Operands {
    float t[4];
};
template <int MODE>
__device__ __forceinline__ void operands(Operands &o, const Epilogue &ep, uint64_t row, int n) {
    if constexpr (MODE == MSE_GRAD) {
        const float *t = (const float *)ep.aux + row * ep.ld_aux + n;
        if (ep.aux_vec) {
            const float4 v = __ldg((const float4 *)t);
            o.t[0] = v.x, o.t[1] = v.y, o.t[2] = v.z, o.t[3] = v.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) o.t[i] = __ldg(&t[i]);
        }
    } else if constexpr (MODE == BF16_MASK) {
        const __nv_bfloat16 *m = (const __nv_bfloat16 *)ep.aux + row * ep.ld_aux + n;
        alignas(8) __nv_bfloat16 h[4];
        if (ep.aux_vec) {
            *reinterpret_cast<uint2 *>(h) = *reinterpret_cast<const uint2 *>(m);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) h[i] = m[i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) o.t[i] = __bfloat162float(h[i]);
    }
}
// Returns the squared errors of the four values (MSE_GRAD).
template <int MODE>
__device__ __forceinline__ double finish(const Operands &o, const float (&bias)[4],
                                         const Epilogue &ep, uint64_t row, int n, float4 acc) {
    float v[4] = {acc.x, acc.y, acc.z, acc.w};
    double sq = 0.0;
    if (MODE != BF16_MASK && ep.bias) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] += bias[i];
    }
    if constexpr (MODE == F32) {
        *(float4 *)((float *)ep.C + row * ep.ldc + n) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (MODE == BF16_RELU) v[i] = fmaxf(v[i], 0.f);
            if (MODE == BF16_MASK && !(o.t[i] > 0.f)) v[i] = 0.f;
            if (MODE == MSE_GRAD) {
                const float d = v[i] - o.t[i];
                sq += (double)d * d;
                v[i] = ep.scale * d;
            }
        }
        alignas(8) const __nv_bfloat162 h[2] = {__floats2bfloat162_rn(v[0], v[1]),
                                                __floats2bfloat162_rn(v[2], v[3])};
        *reinterpret_cast<uint2 *>((__nv_bfloat16 *)ep.C + row * ep.ldc + n) =
            *reinterpret_cast<const uint2 *>(h);
    }
    return sq;
}

// Grid: x = (N / BN) * split, y = M / 128; clusters of `split` CTAs along x
// share a tile, rank r taking k-blocks [KB r / split, KB (r + 1) / split).
template <int BN, int MODE>
__global__ void __launch_bounds__(THREADS, 2)
    k_gemm_bf16(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
                int K, int a_mn, int b_mn, int split, int stages, Epilogue ep, unsigned *flag) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[MAX_STAGES], empty[MAX_STAGES], acc_full;
    __shared__ uint32_t tmem_holder;
    __shared__ double sq_warp[THREADS / 32];
    constexpr uint32_t STAGE = stage_bytes(BN), TILE_A = BM * BK * 2;
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % split;
    const int m0 = blockIdx.y * BM, n0 = ((int)blockIdx.x / split) * BN;
    const int KB = K / BK;
    const int kb0 = (int)((int64_t)KB * rank / split), kb1 = (int)((int64_t)KB * (rank + 1) / split);
    const int nkb = kb1 - kb0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            k::mbar_init(&full[s], 1);
            k::mbar_init(&empty[s], 1);
        }
        k::mbar_init(&acc_full, 1);
        k::mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         saddr(&tmem_holder)),
                     "r"((uint32_t)BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_holder;
    bool ok = true;
    double sq = 0.0;
    // The epilogue's columns of this thread, the same in every row it takes, and
    // their bias, on its way during the main loop: read again for every row it took
    // 2 us of a BF16 tile of 128 columns.
    constexpr int Q = BN / 4;
    static_assert(THREADS % Q == 0, "a thread keeps its columns");
    const int col = (int)(threadIdx.x % Q) * 4, n = n0 + col;
    float bias[4];
    if (MODE != BF16_MASK && ep.bias) {
#pragma unroll
        for (int i = 0; i < 4; ++i) bias[i] = __ldg(&ep.bias[n + i]);
    }

    // The two threads of the main loop count stage, parity, addresses and descriptors
    // up: with a division by the number of stages and each descriptor formed anew, a
    // k-block took 0.385 us instead of 0.31 whatever the tile's width (one B200).
    if (warp == 0 && lane == 0) {
        // producer: TMA loads of the k-blocks into the stage ring
        int issued = 0, s = 0, kx = kb0 * BK;
        uint32_t parity = 1;  // of the stage's last release
        unsigned char *a = smem;
        for (; issued < nkb; ++issued) {
            if (issued >= stages && !k::mbar_wait(&empty[s], parity)) {
                ok = false;
                break;
            }
            k::mbar_arrive_expect(&full[s], STAGE);
            unsigned char *b = a + TILE_A;
            if (a_mn) {
                for (int j = 0; j < BM / 64; ++j)
                    tma_load_2d(a + j * BOX, &ta, m0 + j * 64, kx, &full[s]);
            } else {
                tma_load_2d(a, &ta, kx, m0, &full[s]);
            }
            if (b_mn) {
                for (int j = 0; j < BN / 64; ++j)
                    tma_load_2d(b + j * BOX, &tb, n0 + j * 64, kx, &full[s]);
            } else {
                tma_load_2d(b, &tb, kx, n0, &full[s]);
            }
            kx += BK;
            a += STAGE;
            if (++s == stages) {
                s = 0;
                a = smem;
                parity ^= 1u;
            }
        }
        if (!ok)  // no exit with a copy into this CTA's shared memory in flight
            for (int i = issued > stages ? issued - stages : 0; i < issued; ++i)
                k::mbar_wait(&full[i % stages], (uint32_t)(i / stages) & 1u);
    } else if (warp == 1 && lane == 0) {
        // MMA issuer: four K = 16 steps per stage, then release the stage. The
        // descriptors differ in their start address only, in 16-byte units.
        const uint32_t id = idesc(BN, a_mn, b_mn);
        const uint32_t sa = (a_mn ? 2048u : 32u) >> 4, sb = (b_mn ? 2048u : 32u) >> 4;
        const uint64_t a0 = sw128_desc(saddr(smem), a_mn), b0 = sw128_desc(saddr(smem) + TILE_A, b_mn);
        uint64_t da = a0, db = b0;
        int s = 0;
        uint32_t parity = 0;
        for (int i = 0; i < nkb; ++i) {
            if (!k::mbar_wait(&full[s], parity)) {
                ok = false;
                break;
            }
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk)
                mma_bf16(tmem, da + kk * sa, db + kk * sb, id, (i | kk) != 0);
            mma_commit(&empty[s]);
            da += STAGE >> 4;
            db += STAGE >> 4;
            if (++s == stages) {
                s = 0;
                da = a0;
                db = b0;
                parity ^= 1u;
            }
        }
        mma_commit(&acc_full);  // arrives once every MMA issued above has completed
    } else if (warp >= 2) {
        // this warp's 32 TMEM lanes are rows q*32 .. q*32+31 of the tile, its
        // columns the half `hf`
        const int q = warp & 3, hf = (warp - 2) >> 2;
        if (!k::mbar_wait(&acc_full, 0)) ok = false;
        tc_fence_after();
        if (ok) {
            float *part = (float *)smem;  // the stages are consumed by now
#pragma unroll 1
            for (int c0 = hf * (BN / 2); c0 < (hf + 1) * (BN / 2); c0 += 32) {
                float v[32];
                tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
                float4 *dst = (float4 *)(part + (q * 32 + lane) * part_pitch(BN) + c0);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            }
        }
    }
    if (!ok) atomicOr(flag, 1u);
    if (split == 1) {
        __syncthreads();  // the tile is written
        const float *part = (const float *)smem;
        constexpr int RT = THREADS / Q, STEPS = (BM + RT - 1) / RT;  // rows at a time
        const int r0 = (int)threadIdx.x / Q;
#pragma unroll 1
        for (int s0 = 0; s0 < STEPS; s0 += 4) {  // four rows' operands in flight
            Operands o[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int r = (s0 + u) * RT + r0;
                if (r < BM) operands<MODE>(o[u], ep, (uint64_t)m0 + r, n);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int r = (s0 + u) * RT + r0;
                if (r < BM)
                    sq += finish<MODE>(o[u], bias, ep, (uint64_t)m0 + r, n,
                                       *(const float4 *)(part + r * part_pitch(BN) + col));
            }
        }
    } else {
        __syncwarp();
        cluster_sync();  // every CTA's partial tile is written
        const int rows = BM / split;
        const uint32_t base = saddr(smem);
        for (int t = threadIdx.x; t < rows * Q; t += THREADS) {
            const int r = rank * rows + t / Q;
            const uint32_t off = (uint32_t)(r * part_pitch(BN) + col) * 4;
            Operands o;
            operands<MODE>(o, ep, (uint64_t)m0 + r, n);
            float4 p[8];
#pragma unroll
            for (int s = 0; s < 8; ++s)  // all in flight
                if (s < split) p[s] = ld_cluster(cluster_addr(base + off, (uint32_t)s));
            float4 v = p[0];
#pragma unroll
            for (int s = 1; s < 8; ++s)
                if (s < split) {
                    v.x += p[s].x;
                    v.y += p[s].y;
                    v.z += p[s].z;
                    v.w += p[s].w;
                }
            sq += finish<MODE>(o, bias, ep, (uint64_t)m0 + r, n, v);
        }
    }
    if constexpr (MODE == MSE_GRAD) {
        __syncwarp();
        for (int off = 16; off; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
        if (lane == 0) sq_warp[warp] = sq;
        __syncthreads();
        if (threadIdx.x == 0) {
            double a = sq_warp[0];
            for (int w = 1; w < THREADS / 32; ++w) a += sq_warp[w];
            ep.sse[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = a;
        }
    }
    __syncwarp();
    if (split > 1) cluster_sync();  // no CTA leaves while another reads its tile
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"((uint32_t)BN)
                     : "memory");
    }
}

namespace {

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        XG_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
        XG_REQUIRE(p && q == cudaDriverEntryPointSuccess, XAMG_ERR_CUDA,
                   "cuTensorMapEncodeTiled not available");
        fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

// Tensor map of a row-major [rows][cols] BF16 matrix read in 64 x box_rows
// boxes with the 128-byte swizzle.
CUtensorMap make_map(const void *ptr, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    CUtensorMap m;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr),
                                   dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    XG_REQUIRE(r == CUDA_SUCCESS, XAMG_ERR_CUDA, "tensor map encoding failed");
    return m;
}

template <int BN, int MODE>
void allow_smem() {
    static bool attr = false;  // one flag per instantiation
    if (!attr) {
        XG_CUDA(cudaFuncSetAttribute(k_gemm_bf16<BN, MODE>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     192 * 1024 + 1024));
        attr = true;
    }
}

// CTAs of clusters of `split` that the GPU holds at once (a cluster lies within
// one GPC, so this is fewer than one an SM); 0 where it holds none or the query
// fails.
template <int BN>
int query_cluster_ctas(int split) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)split * 64);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = stages_for(BN) * stage_bytes(BN) + 1024;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)split;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    allow_smem<BN, F32>();
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_gemm_bf16<BN, F32>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    return n * split;
}
int cluster_ctas(int bn, int split) {
    static int known[3][9] = {};  // 1 + the CTAs; 0: not asked yet
    int &n = known[bn == 256 ? 2 : bn == 128 ? 1 : 0][split];
    if (!n)
        n = 1 + (bn == 256   ? query_cluster_ctas<256>(split)
                 : bn == 128 ? query_cluster_ctas<128>(split)
                             : query_cluster_ctas<64>(split));
    return n - 1;
}

template <int BN, int MODE>
void launch_mode(const CUtensorMap &ta, const CUtensorMap &tb, uint64_t M, uint64_t N, int K,
                 bool a_mn, bool b_mn, const Shape &sh, const Epilogue &ep, cudaStream_t s) {
    static_assert(BM * part_pitch(BN) * 4 <= 3 * stage_bytes(BN), "a tile fits in the stages");
    const uint32_t smem = (uint32_t)sh.stages * stage_bytes(BN) + 1024;  // + alignment slack
    auto kern = k_gemm_bf16<BN, MODE>;
    allow_smem<BN, MODE>();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(N / BN) * (unsigned)sh.split, (unsigned)(M / BM));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)sh.split;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = sh.split > 1 ? 1 : 0;
    XG_CUDA(cudaLaunchKernelEx(&cfg, kern, ta, tb, K, (int)a_mn, (int)b_mn, sh.split, sh.stages,
                               ep, ctx().red().flag));
    ++g_kernel_launches;
}

template <int BN>
void launch(const CUtensorMap &ta, const CUtensorMap &tb, uint64_t M, uint64_t N, int K, bool a_mn,
            bool b_mn, const Shape &sh, int mode, const Epilogue &ep, cudaStream_t s) {
    switch (mode) {
    case F32: launch_mode<BN, F32>(ta, tb, M, N, K, a_mn, b_mn, sh, ep, s); break;
    case BF16: launch_mode<BN, BF16>(ta, tb, M, N, K, a_mn, b_mn, sh, ep, s); break;
    case BF16_RELU: launch_mode<BN, BF16_RELU>(ta, tb, M, N, K, a_mn, b_mn, sh, ep, s); break;
    case BF16_MASK: launch_mode<BN, BF16_MASK>(ta, tb, M, N, K, a_mn, b_mn, sh, ep, s); break;
    default: launch_mode<BN, MSE_GRAD>(ta, tb, M, N, K, a_mn, b_mn, sh, ep, s); break;
    }
}

uint64_t run(uint64_t M, uint64_t N, uint64_t K, const void *A, bool a_mn, const void *B, bool b_mn,
             int mode, const Epilogue &ep, bool may_split, cudaStream_t s) {
    XG_REQUIRE(M % BM == 0 && N % 128 == 0 && K % BK == 0 && K > 0, XAMG_ERR_INVALID_ARG,
               "gemm: M and N must be multiples of 128, K a positive multiple of 64");
    XG_REQUIRE(ep.ldc >= N && ep.ldc % 8 == 0, XAMG_ERR_INVALID_ARG,
               "gemm: ldc below N or not a multiple of 8");
    XG_REQUIRE(((uintptr_t)A | (uintptr_t)B | (uintptr_t)ep.C) % 16 == 0, XAMG_ERR_INVALID_ARG,
               "gemm: A, B and C must be 16-byte aligned");
    XG_REQUIRE(M / BM <= 65535, XAMG_ERR_INVALID_ARG, "gemm: M too large");
    const Shape sh = shape_for(M, N, K, ctx().sms, may_split, a_mn && b_mn, cluster_ctas);
    const CUtensorMap ta = a_mn ? make_map(A, K, M, BK) : make_map(A, M, K, BM);
    const CUtensorMap tb = b_mn ? make_map(B, K, N, BK) : make_map(B, N, K, (uint32_t)sh.bn);
    if (sh.bn == 256)
        launch<256>(ta, tb, M, N, (int)K, a_mn, b_mn, sh, mode, ep, s);
    else if (sh.bn == 128)
        launch<128>(ta, tb, M, N, (int)K, a_mn, b_mn, sh, mode, ep, s);
    else
        launch<64>(ta, tb, M, N, (int)K, a_mn, b_mn, sh, mode, ep, s);
    return (M / BM) * (N / sh.bn) * sh.split;
}

}  // namespace

Shape gemm_shape(uint64_t M, uint64_t N, uint64_t K, bool may_split, bool mn) {
    return shape_for(M, N, K, ctx().sms, may_split, mn, cluster_ctas);
}

void gemm_bf16(uint64_t M, uint64_t N, uint64_t K, const void *A, const void *B, void *C,
               uint64_t ldc, int mode, const float *bias, const void *aux, uint64_t ld_aux,
               cudaStream_t s, bool a_mn, bool b_mn, bool may_split) {
    XG_REQUIRE(mode >= F32 && mode <= BF16_MASK, XAMG_ERR_INVALID_ARG, "gemm: unknown mode");
    XG_REQUIRE(mode != BF16_MASK || (aux && ld_aux >= N), XAMG_ERR_INVALID_ARG,
               "gemm: the mask mode needs aux");
    const bool vec = (uintptr_t)aux % 8 == 0 && ld_aux % 4 == 0;
    run(M, N, K, A, a_mn, B, b_mn, mode, Epilogue{C, ldc, bias, aux, ld_aux, 0.f, nullptr, vec},
        may_split, s);
}

uint64_t gemm_mse_grad(uint64_t M, uint64_t N, uint64_t K, const void *A, const void *B, void *dY,
                       const float *bias, const float *T, float scale, double *sse,
                       cudaStream_t s) {
    return run(M, N, K, A, false, B, false, MSE_GRAD,
               Epilogue{dY, N, bias, T, N, scale, sse, (uintptr_t)T % 16 == 0}, false, s);
}

}  // namespace mm
}  // namespace ops
}  // namespace xg
