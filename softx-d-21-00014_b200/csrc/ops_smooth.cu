// Launchers of the block smoother (hybrid symmetric Gauss-Seidel) and the dense
// coarse solve.
#include "dense.cuh"
#include "hsgs.cuh"
#include "spmv_launch.cuh"

namespace xg {
namespace ops {

// Gauss-Seidel blocks a thread block takes (group): one warp of lanes at
// most (group * nv <= 32); fewer while the grid would not fill the GPU twice,
// since a block of rows is one serial chain and a lane waits for its warp's
// longest row. A block of rows that does not fit in shared memory
// (gpu_hsgs_rows of many hundreds) is swept from global memory.
constexpr uint32_t HS_SMEM_MAX = 96u * 1024u;

template <typename F, int NV>
static bool hsgs_shape(const HsgsPlan &p, bool lagged, k::HsgsShape &sh) {
    if (!p.padded) return false;
    int l = NV >= 32 ? 0 : NV >= 16 ? 1 : NV >= 8 ? 2 : NV >= 4 ? 3 : NV >= 2 ? 4 : 5;
    for (; l >= 0; --l) {
        sh = k::HsgsShape{p.n, p.rows, 1u << l, p.ent_max[l]};
        const uint64_t grid = (p.n + (uint64_t)p.rows * sh.group - 1) / ((uint64_t)p.rows * sh.group);
        const uint64_t values = (uint64_t)(p.rows + 1) * sh.group * NV + p.ent_max[l];
        if (values < HS_SMEM_MAX && k::hs_smem_bytes<F, NV>(sh, lagged) <= HS_SMEM_MAX &&
            (l == 0 || grid >= 2ull * (uint64_t)ctx().sms))
            return true;
    }
    return false;
}

template <typename F>
bool hsgs_can_pad(const HsgsPlan &plan, int nv) {
    HsgsPlan p = plan;
    p.padded = true;
    bool ok = false;
    dispatch_nv(nv, [&](auto nvc) {
        k::HsgsShape sh;
        ok = hsgs_shape<F, decltype(nvc)::value>(p, false, sh);
    });
    return ok;
}
template bool hsgs_can_pad<double>(const HsgsPlan &, int);
template bool hsgs_can_pad<float>(const HsgsPlan &, int);

// FP32 rows of more than one chunk of four on average keep two of them in
// registers ahead of their turn (in FP64 that takes 228 registers a thread).
template <typename F, typename I, int NV, int PC, typename IO>
static void hsgs_launch_pc(const DCsr &A, const k::HsgsShape &sh, const k::HsgsOff<F> &off,
                           const F *t, const F *xin, F *x, const F *d, const double *relax_sc,
                           cudaStream_t s) {
    auto kern = k::k_hsgs_block<F, I, NV, PC, IO>;
    static bool big_smem = false;  // one flag per instantiation
    if (!big_smem) {
        XG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)HS_SMEM_MAX));
        big_smem = true;
    }
    const uint64_t per = (uint64_t)sh.rows * sh.group;
    const uint32_t smem = k::hs_smem_bytes<F, NV>(sh, !std::is_same<IO, void>::value);
    kern<<<(unsigned)((A.nrows + per - 1) / per), k::HS_THREADS, smem, s>>>(
        A.row.as<uint32_t>(), (const I *)A.col.p, A.val.as<F>(), sh, off, t, xin, x, d, relax_sc);
    XG_CUDA(cudaGetLastError());
    ++g_kernel_launches;
}
template <typename F, typename I, int NV, typename IO>
static void hsgs_launch(const DCsr &A, const k::HsgsShape &sh, const k::HsgsOff<F> &off,
                        const F *t, const F *xin, F *x, const F *d, const double *relax_sc,
                        cudaStream_t s) {
    constexpr int PC = sizeof(F) == 4 ? 2 : 1;
    if (A.nnz > 5 * A.nrows)
        hsgs_launch_pc<F, I, NV, PC, IO>(A, sh, off, t, xin, x, d, relax_sc, s);
    else
        hsgs_launch_pc<F, I, NV, 1, IO>(A, sh, off, t, xin, x, d, relax_sc, s);
}

template <typename F>
void hsgs_sweep(const DCsr &A, const HsgsPlan &plan, const uint64_t *boff, int nblocks,
                const F *t, const F *xin, F *x, const F *d, const double *relax_sc, int nv,
                cudaStream_t s) {
    if (nblocks == 0 || A.nrows == 0) return;
    XG_DISPATCH(A, nv, {
        k::HsgsShape sh;
        if (hsgs_shape<F, NV>(plan, false, sh)) {
            hsgs_launch<F, I, NV, void>(A, sh, {}, t, xin, x, d, relax_sc, s);
        } else {
            if (!xin) fill<F>(x, A.nrows * (uint64_t)NV, F(0), s);
            const uint64_t threads = (uint64_t)nblocks * NV;
            const int B = (int)((threads + k::CT - 1) / k::CT);
            k::k_hsgs_sweep<F, I, NV><<<B, k::CT, 0, s>>>(A.row.as<uint32_t>(),
                                                          (const I *)A.col.p, A.val.as<F>(), boff,
                                                          nblocks, t, x, d, relax_sc);
            XG_CUDA(cudaGetLastError());
            ++g_kernel_launches;
        }
    });
}
template void hsgs_sweep<double>(const DCsr &, const HsgsPlan &, const uint64_t *, int,
                                 const double *, const double *, double *, const double *,
                                 const double *, int, cudaStream_t);
template void hsgs_sweep<float>(const DCsr &, const HsgsPlan &, const uint64_t *, int,
                                const float *, const float *, float *, const float *,
                                const double *, int, cudaStream_t);

// The fused form needs one-byte in-block columns (blocks of at most 254 rows,
// narrowed), absolute off-block columns and a block that fits beside the
// products; x offsets are formed in 32 bits. It saves a launch and the lagged
// term's way through memory (8-9 us on small levels), and costs 2-3 ns for each
// off-block product of a thread block, of which the sweep's registers let four
// share an SM. So it is taken where the thread blocks fit the GPU at once and
// form at most 4096 products each. Sweep, fused against SpMV + sweep (us, FP32):
// 56^3 nv = 1 second level (1.4 K products) 18 against 22; 88^3 nv = 4 third
// level (6.4 K) 35 against 27, finest level (2130 thread blocks) 94 against 59;
// 96^3 nv = 16 finest level 353 against 234, second level 284 against 117.
constexpr uint64_t HS_FUSE_PRODUCTS = 4096;
constexpr int HS_FUSE_BLOCKS = 4;
template <typename F>
bool hsgs_can_fuse(const DCsr &Adiag, uint64_t off_nnz, const HsgsPlan &plan, int nv) {
    if (Adiag.col_bytes != 1 || Adiag.nrows == 0) return false;
    if (Adiag.nrows * (uint64_t)nv >= (1ull << 32)) return false;
    bool ok = false;
    dispatch_nv(nv, [&](auto nvc) {
        k::HsgsShape sh;
        if (!hsgs_shape<F, decltype(nvc)::value>(plan, true, sh)) return;
        const uint64_t per = (uint64_t)plan.rows * sh.group;
        const uint64_t blocks = (Adiag.nrows + per - 1) / per;
        ok = blocks <= (uint64_t)HS_FUSE_BLOCKS * (uint64_t)ctx().sms &&
             off_nnz * (uint64_t)nv <= HS_FUSE_PRODUCTS * blocks;
    });
    return ok;
}
template bool hsgs_can_fuse<double>(const DCsr &, uint64_t, const HsgsPlan &, int);
template bool hsgs_can_fuse<float>(const DCsr &, uint64_t, const HsgsPlan &, int);

template <typename F>
void hsgs_fused_sweep(const DCsr &A, const DCsr &Aoff, const HsgsPlan &plan, const F *b,
                      const F *xin, F *xout, const F *d, const double *relax_sc, int nv,
                      cudaStream_t s) {
    XG_REQUIRE(xin != xout, XAMG_ERR_INTERNAL, "fused sweep in place");
    const k::HsgsOff<F> off{Aoff.row.as<uint32_t>(), Aoff.col.p, Aoff.val.as<F>()};
    dispatch_nv(nv, [&](auto nvc) {
        constexpr int NV = decltype(nvc)::value;
        k::HsgsShape sh;
        XG_REQUIRE((hsgs_shape<F, NV>(plan, true, sh)), XAMG_ERR_INTERNAL, "fused sweep");
        if (Aoff.col_bytes == 1)
            hsgs_launch<F, uint8_t, NV, uint8_t>(A, sh, off, b, xin, xout, d, relax_sc, s);
        else if (Aoff.col_bytes == 2)
            hsgs_launch<F, uint8_t, NV, uint16_t>(A, sh, off, b, xin, xout, d, relax_sc, s);
        else
            hsgs_launch<F, uint8_t, NV, uint32_t>(A, sh, off, b, xin, xout, d, relax_sc, s);
    });
}
template void hsgs_fused_sweep<double>(const DCsr &, const DCsr &, const HsgsPlan &,
                                       const double *, const double *, double *, const double *,
                                       const double *, int, cudaStream_t);
template void hsgs_fused_sweep<float>(const DCsr &, const DCsr &, const HsgsPlan &, const float *,
                                      const float *, float *, const float *, const double *, int,
                                      cudaStream_t);

template <typename F>
void dense_apply(const F *a, uint64_t n, const F *x, F *y, int nv, cudaStream_t s) {
    if (n == 0) return;
    dispatch_nv(nv, [&](auto nvc) {
        constexpr int NV = decltype(nvc)::value;
        constexpr uint64_t RB = k::dense_rows<F, NV>();
        const uint32_t chunk = (uint32_t)std::min<uint64_t>(n, k::dense_chunk<F, NV>());
        k::k_dense<F, NV><<<(unsigned)((n + RB - 1) / RB), k::DT, chunk * (NV + RB) * sizeof(F),
                            s>>>(a, n, x, y, chunk);
        XG_CUDA(cudaGetLastError());
        ++g_kernel_launches;
    });
}
template void dense_apply<double>(const double *, uint64_t, const double *, double *, int,
                                  cudaStream_t);
template void dense_apply<float>(const float *, uint64_t, const float *, float *, int,
                                 cudaStream_t);

}  // namespace ops
}  // namespace xg
