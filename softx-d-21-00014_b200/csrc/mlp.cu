// The small MLP of the learned coarse initial guess: three dense layers
// (n_in -> h -> h -> n_out, ReLU after the first two), BF16 weights and
// activations with FP32 accumulation on the tcgen05 GEMM (gemm.cu), FP32
// master weights trained with Adam on a mean-squared-error loss. Forward and
// backward passes are GEMMs with fused epilogues (the loss gradient in the last
// layer's), which read transposed operands where they lie, plus the bias
// gradients and Adam here.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <thread>

#include "device.h"
#include "mlp.h"
#include "ops.h"

namespace xg {

namespace {

__global__ void k_f32_to_bf16(const float *__restrict__ in, __nv_bfloat16 *__restrict__ out,
                              uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = __float2bfloat16_rn(in[i]);
}

// Bias gradients of the three layers in one launch: db[c] = sum over rows of
// G[r][c] in row order (BF16 in, FP32 out). A block copies 64 columns of up to
// CS_ROWS rows at a time into shared memory (128 contiguous bytes a row, all
// loads in flight) and 64 threads add their column from there. One thread
// walking a whole column in global memory took 14 us a layer at 512 rows.
struct ColSum {
    const __nv_bfloat16 *g;
    float *db;
    uint32_t cols, block0;  // first block of this layer
};
struct ColSums {
    ColSum l[3];
};
constexpr int CS_ROWS = 256, CS_THREADS = 256;
__global__ void __launch_bounds__(CS_THREADS) k_colsum_bf16(ColSums a, uint32_t rows) {
    __shared__ __align__(16) __nv_bfloat16 t[CS_ROWS][64];
    const ColSum L = blockIdx.x >= a.l[2].block0   ? a.l[2]
                     : blockIdx.x >= a.l[1].block0 ? a.l[1]
                                                   : a.l[0];
    const uint32_t c0 = (blockIdx.x - L.block0) * 64;
    float s = 0.f;
    for (uint32_t r0 = 0; r0 < rows; r0 += CS_ROWS) {
        const uint32_t nr = rows - r0 < CS_ROWS ? rows - r0 : CS_ROWS;
        if (r0) __syncthreads();
#pragma unroll
        for (int u = 0; u < CS_ROWS * 8 / CS_THREADS; ++u) {  // 16 bytes each
            const uint32_t q = u * CS_THREADS + threadIdx.x, r = q / 8, p = q % 8;
            if (r < nr)
                reinterpret_cast<uint4 *>(t[r])[p] = __ldg(
                    reinterpret_cast<const uint4 *>(L.g + (uint64_t)(r0 + r) * L.cols + c0) + p);
        }
        __syncthreads();
        if (threadIdx.x < 64) {
#pragma unroll 16
            for (uint32_t r = 0; r < nr; ++r) s += __bfloat162float(t[r][threadIdx.x]);
        }
    }
    if (threadIdx.x < 64) L.db[c0 + threadIdx.x] = s;
}

// Adam (Kingma & Ba 2015) on FP32 master parameters, every layer's weights and
// biases in one launch, four values a thread; bf16 receives the rounded
// weights. Bound by the 30 bytes a weight moves.
struct AdamSeg {
    float *p;
    const float *g;
    float *m, *v;
    __nv_bfloat16 *bf16;  // null: none
    uint64_t n4;          // values / 4
};
struct AdamSegs {
    AdamSeg s[6];
};
__global__ void __launch_bounds__(256)
    k_adam(AdamSegs a, float lr, float b1, float b2, float eps, float c1, float c2) {
#pragma unroll 1
    for (int q = 0; q < 6; ++q) {
        const AdamSeg s = a.s[q];
        for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < s.n4;
             i += (uint64_t)gridDim.x * blockDim.x) {
            float4 p4 = ((float4 *)s.p)[i], m4 = ((float4 *)s.m)[i], v4 = ((float4 *)s.v)[i];
            const float4 g4 = ((const float4 *)s.g)[i];
            float *p = &p4.x, *m = &m4.x, *v = &v4.x;
            const float *g = &g4.x;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float gi = g[j];
                const float mi = b1 * m[j] + (1.f - b1) * gi;
                const float vi = b2 * v[j] + (1.f - b2) * gi * gi;
                m[j] = mi;
                v[j] = vi;
                p[j] = p[j] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
            }
            ((float4 *)s.p)[i] = p4;
            ((float4 *)s.m)[i] = m4;
            ((float4 *)s.v)[i] = v4;
            if (s.bf16) {
                alignas(8) const __nv_bfloat162 h[2] = {
                    __floats2bfloat162_rn(p4.x, p4.y), __floats2bfloat162_rn(p4.z, p4.w)};
                ((uint2 *)s.bf16)[i] = *reinterpret_cast<const uint2 *>(h);
            }
        }
    }
}

unsigned grid_for(uint64_t n) { return (unsigned)std::min<uint64_t>((n + 255) / 256, 148 * 16); }

}  // namespace

void Mlp::init(uint32_t n_in_, uint32_t n_hidden, uint32_t n_out_, uint64_t seed) {
    XG_REQUIRE(n_in_ % 128 == 0 && n_hidden % 128 == 0 && n_out_ % 128 == 0 && n_in_ && n_hidden &&
                   n_out_,
               XAMG_ERR_INVALID_ARG, "mlp: layer widths must be positive multiples of 128");
    n_in = n_in_;
    h = n_hidden;
    n_out = n_out_;
    const uint32_t fan_in[3] = {n_in, h, h}, fan_out[3] = {h, h, n_out};
    std::mt19937_64 rng(seed);
    for (int l = 0; l < 3; ++l) {
        Layer &L = layer[l];
        L.in = fan_in[l];
        L.out = fan_out[l];
        // uniform(-1/sqrt(in), 1/sqrt(in)) weights, zero biases
        const float a = 1.0f / std::sqrt((float)L.in);
        std::uniform_real_distribution<float> U(-a, a);
        std::vector<float> w((size_t)L.out * L.in);
        for (auto &x : w) x = U(rng);
        upload(L.w, w, S());
        upload(L.b, std::vector<float>(L.out, 0.f), S());
        const size_t nw = w.size();
        L.gw.alloc(nw * 4);
        L.gb.alloc(L.out * 4);
        L.mw.alloc(nw * 4);
        L.vw.alloc(nw * 4);
        L.mb.alloc(L.out * 4);
        L.vb.alloc(L.out * 4);
        for (DevBuf *z : {&L.mw, &L.vw, &L.mb, &L.vb})
            XG_CUDA(cudaMemsetAsync(z->p, 0, z->bytes, S()));
        L.wt_bf.alloc(nw * 2);
    }
    refresh_bf16();
    step = 0;
}

// BF16 copy of the weights, W^T as [out][in]: the forward pass reads it as it
// lies, the input gradients transposed.
void Mlp::refresh_bf16() {
    for (Layer &L : layer) {
        const uint64_t nw = (uint64_t)L.out * L.in;
        k_f32_to_bf16<<<grid_for(nw), 256, 0, S()>>>(L.w.as<float>(),
                                                     L.wt_bf.as<__nv_bfloat16>(), nw);
        g_kernel_launches += 1;
    }
    XG_CUDA(cudaGetLastError());
}

void Mlp::ensure(uint32_t batch) {
    XG_REQUIRE(batch > 0 && batch % 128 == 0, XAMG_ERR_INVALID_ARG,
               "mlp: the batch must be a positive multiple of 128");
    if (batch <= cap) return;
    cap = 0;  // until every buffer is there: an allocation may throw
    const uint64_t B = batch;
    X.alloc(B * n_in * 2);
    H1.alloc(B * h * 2);
    H2.alloc(B * h * 2);
    dY.alloc(B * n_out * 2);
    dH2.alloc(B * h * 2);
    dH1.alloc(B * h * 2);
    const size_t parts = ops::mm::gemm_mse_parts(B, n_out);
    sse.alloc(parts * sizeof(double));
    if (sse_host) XG_CUDA(cudaFreeHost(sse_host));
    sse_host = nullptr;
    XG_CUDA(cudaMallocHost((void **)&sse_host, parts * sizeof(double)));
    cap = batch;
}

Mlp::~Mlp() {
    if (bounce) cudaFreeHost(bounce);
    for (cudaStream_t c : copy_streams)
        if (c) cudaStreamDestroy(c);
    if (sse_host) cudaFreeHost(sse_host);
}

// The first two layers, activations kept in BF16.
void Mlp::hidden(uint32_t batch, const float *Xf, bool split) {
    ensure(batch);
    const uint64_t B = batch;
    k_f32_to_bf16<<<grid_for(B * n_in), 256, 0, S()>>>(Xf, X.as<__nv_bfloat16>(), B * n_in);
    ++g_kernel_launches;
    using ops::mm::gemm_bf16;
    gemm_bf16(B, h, n_in, X.p, layer[0].wt_bf.p, H1.p, h, 2, layer[0].b.as<float>(), nullptr, 0,
              S(), false, false, split);
    gemm_bf16(B, h, h, H1.p, layer[1].wt_bf.p, H2.p, h, 2, layer[1].b.as<float>(), nullptr, 0,
              S(), false, false, split);
}

void Mlp::forward(uint32_t batch, const float *Xf, float *Yout) {
    hidden(batch, Xf, true);
    ops::mm::gemm_bf16(batch, n_out, h, H2.p, layer[2].wt_bf.p, Yout, n_out, 0,
                       layer[2].b.as<float>(), nullptr, 0, S());
}

// Forward and backward pass; the partial sums of the loss are on their way to
// the host when it returns (loss()). Its products never split their sums over
// K: a step's weights depend on every rounding before it (Adam divides small
// gradients by their own size), so training keeps one summation order whatever
// the shapes.
void Mlp::backward(uint32_t batch, const float *Xf, const float *T) {
    hidden(batch, Xf, false);
    const uint64_t B = batch;
    using ops::mm::gemm_bf16;
    const float scale = 2.0f / (float)(B * n_out);
    // layer 3: dY and the loss from the forward product's epilogue; dW3^T = dY^T H2,
    // dH2 = dY W3 masked by H2 > 0
    sse_n = ops::mm::gemm_mse_grad(B, n_out, h, H2.p, layer[2].wt_bf.p, dY.p,
                                   layer[2].b.as<float>(), T, scale, sse.as<double>(), S());
    loss_n = B * n_out;
    XG_CUDA(cudaMemcpyAsync(sse_host, sse.p, sse_n * sizeof(double), cudaMemcpyDeviceToHost, S()));
    gemm_bf16(n_out, h, B, dY.p, H2.p, layer[2].gw.p, h, 0, nullptr, nullptr, 0, S(), true, true,
              false);
    gemm_bf16(B, h, n_out, dY.p, layer[2].wt_bf.p, dH2.p, h, 3, nullptr, H2.p, h, S(), false, true,
              false);
    // layer 2
    gemm_bf16(h, h, B, dH2.p, H1.p, layer[1].gw.p, h, 0, nullptr, nullptr, 0, S(), true, true,
              false);
    gemm_bf16(B, h, h, dH2.p, layer[1].wt_bf.p, dH1.p, h, 3, nullptr, H1.p, h, S(), false, true,
              false);
    // layer 1
    gemm_bf16(h, n_in, B, dH1.p, X.p, layer[0].gw.p, n_in, 0, nullptr, nullptr, 0, S(), true, true,
              false);
    // bias gradients
    ColSums cs;
    cs.l[0] = ColSum{dY.as<__nv_bfloat16>(), layer[2].gb.as<float>(), n_out, 0};
    cs.l[1] = ColSum{dH2.as<__nv_bfloat16>(), layer[1].gb.as<float>(), h, n_out / 64};
    cs.l[2] = ColSum{dH1.as<__nv_bfloat16>(), layer[0].gb.as<float>(), h, (n_out + h) / 64};
    k_colsum_bf16<<<(n_out + 2 * h) / 64, CS_THREADS, 0, S()>>>(cs, batch);
    ++g_kernel_launches;
    XG_CUDA(cudaGetLastError());
}

double Mlp::loss() const {
    double s = 0;
    for (uint64_t i = 0; i < sse_n; ++i) s += sse_host[i];
    return s / (double)loss_n;
}

void Mlp::train_step(uint32_t batch, const float *Xf, const float *T, float lr) {
    backward(batch, Xf, T);
    ++step;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float c1 = 1.f - std::pow(b1, (float)step), c2 = 1.f - std::pow(b2, (float)step);
    AdamSegs a;
    uint64_t most = 0;
    for (int l = 0; l < 3; ++l) {
        Layer &L = layer[l];
        const uint64_t nw = (uint64_t)L.out * L.in;
        a.s[2 * l] = AdamSeg{L.w.as<float>(),  L.gw.as<float>(), L.mw.as<float>(),
                             L.vw.as<float>(), L.wt_bf.as<__nv_bfloat16>(), nw / 4};
        a.s[2 * l + 1] = AdamSeg{L.b.as<float>(),  L.gb.as<float>(), L.mb.as<float>(),
                                 L.vb.as<float>(), nullptr, L.out / 4};
        most = std::max(most, nw / 4);
    }
    k_adam<<<grid_for(most), 256, 0, S()>>>(a, lr, b1, b2, eps, c1, c2);
    ++g_kernel_launches;
    XG_CUDA(cudaGetLastError());
}

// Device values to the caller's pageable memory. One cudaMemcpy moves 5 GB/s
// there (the driver's single staging copy, and the first touch of the caller's
// pages): 9.3 ms for the 47 MB of a 5,248-1,024 network. COPIERS threads each
// take every COPIERS-th megabyte through a pinned buffer and a stream of their
// own, so the transfers overlap the copies out.
void Mlp::download(float *host, const float *dev, uint64_t count) {
    constexpr uint64_t CHUNK = 1u << 20;
    const uint64_t bytes = count * sizeof(float);
    if (bytes < 4 * CHUNK) {
        XG_CUDA(cudaMemcpy(host, dev, bytes, cudaMemcpyDeviceToHost));
        return;
    }
    if (!bounce) XG_CUDA(cudaMallocHost((void **)&bounce, COPIERS * CHUNK));
    for (cudaStream_t &c : copy_streams)
        if (!c) XG_CUDA(cudaStreamCreateWithFlags(&c, cudaStreamNonBlocking));
    const int device = ctx().device;
    cudaError_t err[COPIERS];
    auto copier = [&](int t) {
        cudaError_t e = cudaSetDevice(device);
        char *buf = bounce + (uint64_t)t * CHUNK;
        for (uint64_t o = (uint64_t)t * CHUNK; o < bytes && e == cudaSuccess; o += COPIERS * CHUNK) {
            const uint64_t len = std::min(CHUNK, bytes - o);
            e = cudaMemcpyAsync(buf, (const char *)dev + o, len, cudaMemcpyDeviceToHost,
                                copy_streams[t]);
            if (e == cudaSuccess) e = cudaStreamSynchronize(copy_streams[t]);
            if (e == cudaSuccess) std::memcpy((char *)host + o, buf, len);
        }
        err[t] = e;
    };
    std::thread th[COPIERS - 1];
    int started = 0;
    try {
        for (; started < COPIERS - 1; ++started) th[started] = std::thread(copier, started + 1);
    } catch (...) {  // no more threads: this one takes their share
    }
    copier(0);
    for (int t = 0; t < started; ++t) th[t].join();
    for (int t = started + 1; t < COPIERS; ++t) copier(t);
    for (cudaError_t e : err) XG_CUDA(e);
}

// Parameters in the order W1^T [h][in], b1, W2^T [h][h], b2, W3^T [out][h], b3.
uint64_t Mlp::param_count() const {
    uint64_t n = 0;
    for (const Layer &L : layer) n += (uint64_t)L.out * L.in + L.out;
    return n;
}

void Mlp::copy_params(float *host, bool set, bool grads) {
    XG_CUDA(cudaStreamSynchronize(S()));
    uint64_t off = 0;
    for (Layer &L : layer) {
        const uint64_t nw = (uint64_t)L.out * L.in;
        DevBuf &w = grads ? L.gw : L.w, &b = grads ? L.gb : L.b;
        if (set) {
            XG_CUDA(cudaMemcpy(w.p, host + off, nw * 4, cudaMemcpyHostToDevice));
            XG_CUDA(cudaMemcpy(b.p, host + off + nw, L.out * 4, cudaMemcpyHostToDevice));
        } else {
            download(host + off, w.as<float>(), nw);
            XG_CUDA(cudaMemcpy(host + off + nw, b.p, L.out * 4, cudaMemcpyDeviceToHost));
        }
        off += nw + L.out;
    }
    if (set && !grads) refresh_bf16();
}

}  // namespace xg
