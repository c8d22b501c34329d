// The persistent preconditioned BiCGStab for small systems: one thread per
// (row, right-hand side), every vector of the iteration in that thread's
// registers and the block's matrix entries in shared memory.
//
// An iteration of a small system is latency: five exchanges between all blocks
// (two products, three groups of dot products), one more for every Jacobi sweep
// after the first in each of the two preconditioner applications, and what lies
// between them. k_pbicgstab_persist keeps the vectors in global memory and puts a
// grid barrier (1.6 us) before every exchange's reads: 24.1 us an iteration on the
// 32^3 Poisson system with two sweeps, seven exchanges (128 blocks, nv = 1). Here every exchanged value carries
// the number of its exchange beside it, in one 16-byte access, and its readers
// poll the value itself: a product waits for the x of its own entries and a
// reduction for the blocks' partial sums, one store and one read through L2
// each, with no barrier, fence or reset between them.
#pragma once

#include "kernels.cuh"

namespace xg {
namespace k {

// A value with the number of the exchange it belongs to.
struct __align__(16) Tagged {
    double v;
    unsigned long long tag;
};
__device__ __forceinline__ void tagged_put(Tagged *p, double v, unsigned long long tag) {
    asm volatile(
        "{\n\t.reg .b128 t;\n\t"
        "mov.b128 t, {%1, %2};\n\t"
        "st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
        "l"((unsigned long long)__double_as_longlong(v)), "l"(tag)
        : "memory");
}
__device__ __forceinline__ Tagged tagged_get(const Tagged *p) {
    unsigned long long v, t;
    asm volatile(
        "{\n\t.reg .b128 t;\n\t"
        "ld.relaxed.gpu.global.b128 t, [%2];\n\t"
        "mov.b128 {%0, %1}, t;\n\t}"
        : "=l"(v), "=l"(t)
        : "l"(p)
        : "memory");
    return Tagged{__longlong_as_double((long long)v), t};
}

// Copies of a block's partial sums, each read by every REPth block only: with
// all blocks polling the same few lines, a reduction waited 2.3 us for them.
template <int NV>
__host__ __device__ constexpr int reg_copies() { return NV <= 2 ? 8 : NV <= 8 ? 4 : 2; }
// Vectors a preconditioner application publishes: one per Jacobi sweep, each in
// a buffer of its own.
constexpr int REG_MAX_SWEEPS = 4;
__host__ __device__ inline int reg_published(int sweeps) { return sweeps < 1 ? 1 : sweeps; }
// Values exchanged: the published vectors of both applications, and two sets
// (used in turn) of partial sums.
template <int NV>
inline size_t reg_exchange_values(uint64_t n, uint32_t blocks, int sweeps) {
    return 2 * (size_t)reg_published(sweeps) * n * NV +
           2 * (size_t)reg_copies<NV>() * NV * 3 * blocks;
}

// Grid: B = canon_blocks(n, NV) = tiles, one tile a block, all resident
// (cooperative launch). xch: reg_exchange_values values whose tags are all
// below tag0, the number of this launch's first exchange. cap: entries of the
// largest tile (shared memory: cap values and columns). No preconditioner, the
// Identity, or up to REG_MAX_SWEEPS Jacobi sweeps. Same element operations, row
// sums and canonical reductions, in the same order, as k_pbicgstab_persist: the
// same iterates bit for bit.
//
// A published vector is overwritten one iteration later, and a set of partial
// sums two reductions later. Between the two lies a whole reduction, which
// holds every block's partial sums, and a block gives its partial sum only after
// its reads of both: no block overwrites what another still waits for.
//
// One block an SM (at most 148): at two, 128 registers a thread spill.
template <int NV, typename I>
__global__ void __launch_bounds__(CT, 1)
    k_pbicgstab_reg(CsrArgs<double> A, PersistArgs P, Tagged *xch, unsigned long long tag0,
                    uint32_t cap) {
    constexpr int R = CT / NV, COPIES = reg_copies<NV>();
    extern __shared__ __align__(16) unsigned char reg_smem[];
    __shared__ double SCS[SC_COUNT * SC_STRIDE];
    __shared__ double st_abs[NV], st_rel[NV];
    __shared__ int st_conv[NV];
    __shared__ int go;
    __shared__ double wsum[8 * NV * 3];
    __shared__ double sums[NV * 3];
    double *val = (double *)reg_smem;
    uint32_t *col = (uint32_t *)(reg_smem + (size_t)cap * sizeof(double));
    const uint32_t B = gridDim.x;
    const uint32_t n = (uint32_t)A.n;
    const int rt = threadIdx.x / NV, kk = threadIdx.x % NV;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t r0row = blockIdx.x * R, i = r0row + rt;
    const bool on = i < n;
    const uint32_t e = on ? i * NV + kk : 0;

    // entries of the tile: values, and columns as element offsets of x
    const uint32_t t0 = __ldg(&A.row[r0row]), t1 = __ldg(&A.row[r0row + R < n ? r0row + R : n]);
    for (uint32_t j = threadIdx.x; j < t1 - t0; j += CT) val[j] = __ldg(&A.val[t0 + j]);
    const uint32_t j0 = on ? __ldg(&A.row[i]) - t0 : 0, j1 = on ? __ldg(&A.row[i + 1]) - t0 : 0;
    for (uint32_t j = j0 + kk; j < j1; j += NV)
        col[j] = col_at32<I>(__ldg(&((const I *)A.col)[t0 + j]), i) * NV;
    for (int o = threadIdx.x; o < SC_COUNT * SC_STRIDE; o += CT) SCS[o] = P.sc[o];
    for (int o = threadIdx.x; o < NV; o += CT) {
        st_abs[o] = 0.0;
        st_rel[o] = 0.0;
        st_conv[o] = 0;
    }
    // this thread's elements of the iteration's vectors
    double x = on ? P.x[e] : 0.0, r = on ? P.r[e] : 0.0, p = on ? P.p[e] : 0.0;
    const double rr0 = on ? P.r0[e] : 0.0;
    const double rd = P.d && on ? mul(P.relax, P.d[i]) : 0.0;  // relax * d
    double v = 0.0, s = 0.0, t = 0.0, pa = 0.0, sa = 0.0;
    __syncthreads();

    const int npub = reg_published(P.sweeps);
    const size_t vec = (size_t)n * NV;
    Tagged *sets = xch + 2 * npub * vec;
    unsigned long long tag = tag0;  // of the next exchange
    bool fine = true;               // no wait of this thread ran out
    // Whether a wait goes on: false past the limit, with the flag raised (the
    // clock is read every 64 polls).
    auto go_on = [&](uint32_t it, uint64_t &since) {
        if ((it & 63u) != 63u) return true;
        const uint64_t now = global_ns();
        if (!since) since = now;
        if (now - since <= P.gs.limit_ns && it < 0xffffff00u) return true;
        atomicOr(P.gs.flag, 1u);
        fine = false;
        return false;
    };
    // row sum over a published vector: the gathers of eight entries are in
    // flight together, and asked again until all have arrived
    auto rowsum = [&](const Tagged *xv, unsigned long long want) {
        double y = 0.0;
        for (uint32_t j = j0; j < j1; j += 8) {
            Tagged g[8];
            uint64_t since = 0;
            for (uint32_t it = 0;; ++it) {
                bool here = true;
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (j + q < j1) g[q] = tagged_get(&xv[col[j + q] + kk]);
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (j + q < j1) here = here && g[q].tag == want;
                if (here || !go_on(it, since)) break;
            }
            if (!fine) break;
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (j + q < j1) y = add(y, mul(g[q].v, val[j + q]));
        }
        return y;
    };

    // The canonical reduction of one value per thread and sum: the block's
    // partial sums go out, then every block adds all blocks' in canonical order
    // and runs the finaliser for itself. False when a wait ran out, here or in
    // a row sum before.
    uint32_t set = 0;
    auto slot = [&](int copy, int o, uint32_t b) {
        return sets + ((size_t)((set * COPIES + copy) * NV * 3 + o) * B + b);
    };
    auto reduce = [&](auto nrc, const double (&term)[3], auto &&fin) {
        constexpr int NR = decltype(nrc)::value;
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            double a = add(0.0, term[q]);
            if (!on) a = 0.0;
#pragma unroll
            for (int off = 16; off >= NV; off >>= 1) a = add(a, shfl_xor(a, off));
            if (lane < NV) wsum[(warp * NV + lane) * NR + q] = a;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < NV * NR * COPIES; q += CT) {
            const int o = q / COPIES;
            double a = wsum[o];
#pragma unroll
            for (int w = 1; w < 8; ++w) a = add(a, wsum[w * NV * NR + o]);
            tagged_put(slot(q % COPIES, o, blockIdx.x), a, tag);
        }
        for (int o = warp; o < NV * NR; o += CT / 32) {
            double a = 0.0;
            for (uint32_t b0 = lane; b0 < B; b0 += 128) {
                Tagged w[4];
                uint64_t since = 0;
                for (uint32_t it = 0; fine; ++it) {
                    bool here = true;
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (b0 + 32 * q < B)
                            w[q] = tagged_get(slot(blockIdx.x % COPIES, o, b0 + 32 * q));
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (b0 + 32 * q < B) here = here && w[q].tag == tag;
                    if (here || !go_on(it, since)) break;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (b0 + 32 * q < B) a = add(a, w[q].v);
            }
            __syncwarp();
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) a = add(a, shfl_xor(a, off));
            if (lane == 0) sums[o] = a;
        }
        if (__syncthreads_or(!fine)) return false;
        if (threadIdx.x < NV) fin((int)threadIdx.x, &sums[threadIdx.x * NR]);
        set ^= 1u;
        ++tag;
        __syncthreads();
        return true;
    };
    using One = std::integral_constant<int, 1>;
    using Three = std::integral_constant<int, 3>;

    // this thread's element of M^-1 in: Jacobi sweeps from zero, or a copy; each
    // sweep's vector is published for the other blocks' next one, the last for
    // their product (tagged `tag`)
    auto precond = [&](Tagged *to, double in) {
        double out = P.d ? mul(rd, in) : in;
        for (int j = 1; j < npub; ++j) {
            if (on) tagged_put(&to[e], out, tag);
            const double ax = rowsum(to, tag);
            out = add(out, mul(rd, sub(in, ax)));
            to += vec;
            ++tag;
        }
        if (on) tagged_put(&to[e], out, tag);
        return out;
    };
    int it = 0;
    bool tail = false, done = false, ok = true;
    const EGroup4<NV, true> g4{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, SCS};
    const EDotAlpha<NV> ea(nullptr, nullptr, SCS);
    const EDot3<NV> e3(nullptr, nullptr, SCS);
    auto xupd = [&]() {
        const double ac = SCS[SC_ALPHA_C * SC_STRIDE + kk], oc = SCS[SC_OMEGA_C * SC_STRIDE + kk];
        x = add(add(mul(ac, pa), mul(oc, sa)), mul(1.0, x));
    };
    auto do_tail = [&]() {
        xupd();
        r = sub(s, mul(SCS[SC_OMEGA * SC_STRIDE + kk], t));
        const double term[3] = {mul(r, rr0), 0.0, 0.0};
        if (!reduce(One(), term, g4)) return false;
        const double ns = SCS[SC_NSCAL * SC_STRIDE + kk], be = SCS[SC_BETA * SC_STRIDE + kk];
        p = add(add(mul(1.0, r), mul(ns, v)), mul(be, p));
        return true;
    };
    while (ok) {
        ++it;
        if (tail && !(ok = do_tail())) break;
        {   // v = A p_; alpha = rho / (v, r0)
            pa = precond(xch, p);
            v = rowsum(xch + (npub - 1) * vec, tag);
            const double term[3] = {mul(v, rr0), 0.0, 0.0};
            ++tag;
            if (!(ok = reduce(One(), term, ea))) break;
        }
        // s = r - alpha v
        s = add(mul(1.0, r), mul(mul(SCS[SC_ALPHA * SC_STRIDE + kk], -1.0), v));
        {   // t = A s_; omega, res
            sa = precond(xch + npub * vec, s);
            t = rowsum(xch + (2 * npub - 1) * vec, tag);
            const double term[3] = {mul(t, s), mul(t, t), mul(s, s)};
            ++tag;
            if (!(ok = reduce(Three(), term, e3))) break;
        }
        // convergence test (host_converged): every block decides alike
        if (threadIdx.x == 0) {
            bool flag = P.check != 0;
            if (flag) {
#pragma unroll 1
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
#pragma unroll 1
                    for (int k2 = 0; k2 < NV; ++k2)
                        SCS[SC_ICONV * SC_STRIDE + k2] =
                            mul(SCS[SC_ICONV * SC_STRIDE + k2], (double)(!st_conv[k2]));
            }
            go = flag ? 0 : (it >= P.max_iters ? 1 : 2);
        }
        __syncthreads();
        if (go == 0) {  // converged: x = alpha_c p_ + omega_c s_ + x
            xupd();
            done = true;
            break;
        }
        tail = true;
        if (go == 1) {  // max_iters reached: the pending rest of the iteration
            ok = do_tail();
            done = ok;
            break;
        }
    }
    if (done && on) P.x[e] = x;
    if (blockIdx.x == 0 && done) {
        __syncthreads();
        for (int o = threadIdx.x; o < SC_COUNT * SC_STRIDE; o += CT) P.sc[o] = SCS[o];
        for (int o = threadIdx.x; o < NV; o += CT) {
            P.out[o] = st_abs[o];
            P.out[32 + o] = st_rel[o];
            P.out[64 + o] = (double)st_conv[o];
        }
        if (threadIdx.x == 0) P.out[96] = (double)it;
    }
}

}  // namespace k
}  // namespace xg
