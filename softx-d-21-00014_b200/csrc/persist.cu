// Launchers of the persistent preconditioned BiCGStab (k_pbicgstab_reg,
// csrc/persist_reg.cuh, and k_pbicgstab_persist, csrc/kernels.cuh) and of its
// grid barrier's self-test.
#include "persist_reg.cuh"
#include "spmv_launch.cuh"

namespace xg {
namespace ops {

// The whole iteration runs as one cooperative launch: B = canon_blocks(n,
// nv) canonical blocks played by ceil(B / share) physical blocks (share =
// gpu_persistent: canonical blocks a physical block plays), which must be
// resident at once; the two halves of the partial-sum buffer must hold B x
// nv x 4 values each.
static int grid_of(int B, int share) { return (B + share - 1) / (share < 1 ? 1 : share); }

// By its registers an SM holds four blocks at nv = 1, 2 and 32, three at 4 and 8, two
// at 16. What the next block an SM would take is solved faster by the separate
// launches at nv = 4 and 16 (one launch against separate ones, ms, two Jacobi sweeps:
// 33^3 nv = 4 7-point 3.07 and 2.87, 27-point 3.51 and 2.62; 18^3 nv = 16 4.05 and
// 2.31, 3.05 and 1.68), and at nv = 2 on long rows (42^3 27-point 3.73 and 3.05), but
// not on short ones (39^3 and 42^3 7-point 2.36 and 3.11, 2.90 and 3.46).
template <int NV, typename I>
static bool fits_nv(const DCsr &A, int share) {
    const int B = k::canon_blocks(A.nrows, NV);
    if (NV == 2 && A.nnz >= 16 * A.nrows && grid_of(B, share) > 3 * ctx().sms) return false;
    if ((uint64_t)B * NV * 8 > (uint64_t)k::BMAX * 32 * 4) return false;
    const int res = occupancy(k::k_pbicgstab_persist<NV, I>, k::CT, 0);
    return (uint64_t)res * (uint64_t)ctx().sms >= (uint64_t)grid_of(B, share);
}

bool pbicgstab_persist_fits(const DCsr &A, int nv, int share) {
    bool ok = false;
    XG_DISPATCH(A, nv, { ok = fits_nv<NV, I>(A, share); });
    return ok;
}

// The register-resident form takes systems of at most one tile an SM (n * nv up
// to 148 * 256) with a tile's entries in shared memory, and at most four Jacobi
// sweeps; launches that share blocks (gpu_persistent > 1), larger systems and
// more sweeps keep their vectors in global memory.
constexpr uint32_t REG_SMEM_MAX = 200u * 1024u;

template <int NV, typename I>
static uint32_t reg_blocks(const DCsr &A, int sweeps, int share, uint32_t &smem, uint32_t &cap) {
    constexpr uint64_t R = k::CT / NV;
    const uint64_t ntiles = (A.nrows + R - 1) / R;
    if (share > 1 || sweeps > k::REG_MAX_SWEEPS) return 0;
    if (ntiles == 0 || ntiles > (uint64_t)ctx().sms) return 0;
    if (std::max(A.ncols, A.nrows) * (uint64_t)NV >= (1ull << 32)) return 0;
    cap = tile_max(A, NV, ctx().stream);
    if ((uint64_t)cap * 12 > REG_SMEM_MAX) return 0;
    smem = cap * 12;
    auto kern = k::k_pbicgstab_reg<NV, I>;
    static bool big_smem = false;  // one flag per instantiation
    if (!big_smem) {
        XG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)REG_SMEM_MAX));
        big_smem = true;
    }
    return occupancy(kern, k::CT, smem) >= 1 ? (uint32_t)ntiles : 0;
}

size_t pbicgstab_exchange_bytes(const DCsr &A, int nv, int sweeps, int share) {
    size_t bytes = 0;
    XG_DISPATCH(A, nv, {
        uint32_t smem;
        uint32_t cap;
        const uint32_t blocks = reg_blocks<NV, I>(A, sweeps, share, smem, cap);
        if (blocks) bytes = k::reg_exchange_values<NV>(A.nrows, blocks, sweeps) * sizeof(k::Tagged);
    });
    return bytes;
}

void pbicgstab_persist(const DCsr &A, const k::PersistArgs &P, int nv, int share, void *exchange,
                       uint64_t tag0, cudaStream_t s) {
    XG_DISPATCH(A, nv, {
        const int B = k::canon_blocks(A.nrows, NV);
        k::CsrArgs<double> a = A.args<double>();
        k::PersistArgs p = P;
        p.B = (uint32_t)B;
        if (exchange) {
            uint32_t smem = 0;
            uint32_t cap = 0;
            const uint32_t blocks = reg_blocks<NV, I>(A, P.sweeps, share, smem, cap);
            XG_REQUIRE(blocks == (uint32_t)B, XAMG_ERR_INTERNAL, "register-resident BiCGStab");
            k::Tagged *x = (k::Tagged *)exchange;
            unsigned long long t0 = tag0;
            void *args[] = {(void *)&a, (void *)&p, (void *)&x, (void *)&t0, (void *)&cap};
            XG_CUDA(cudaLaunchCooperativeKernel((const void *)k::k_pbicgstab_reg<NV, I>,
                                                dim3(blocks), dim3(k::CT), args, smem, s));
        } else {
            void *args[] = {(void *)&a, (void *)&p};
            XG_CUDA(cudaLaunchCooperativeKernel((const void *)k::k_pbicgstab_persist<NV, I>,
                                                dim3((unsigned)grid_of(B, share)), dim3(k::CT),
                                                args, 0, s));
        }
        ++g_kernel_launches;
    });
}

void grid_selftest(unsigned *count_gen, unsigned *flag, uint64_t limit_ns, cudaStream_t s) {
    XG_CUDA(cudaMemsetAsync(count_gen, 0, 2 * sizeof(unsigned), s));
    k::GridSync g{reinterpret_cast<unsigned long long *>(count_gen), flag, limit_ns};
    const int blocks = 4;  // resident together on any GPU this library runs on
    void *args[] = {(void *)&g};
    XG_CUDA(cudaLaunchCooperativeKernel((const void *)k::k_grid_selftest, dim3(blocks), dim3(32),
                                        args, 0, s));
    ++g_kernel_launches;
}

}  // namespace ops
}  // namespace xg
