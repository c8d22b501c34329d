// The MLP of the learned coarse initial guess (mlp.cu): n_in -> h -> h ->
// n_out with ReLU, BF16 weights/activations, FP32 master weights and Adam.
#pragma once

#include "device.h"

namespace xg {

struct Mlp {
    struct Layer {
        uint32_t in = 0, out = 0;
        DevBuf w, b;          // FP32 master W^T [out][in], bias [out]
        DevBuf gw, gb;        // gradients (FP32)
        DevBuf mw, vw, mb, vb;  // Adam moments
        DevBuf wt_bf;         // BF16 W^T [out][in]
    };
    uint32_t n_in = 0, h = 0, n_out = 0;
    Layer layer[3];
    uint64_t step = 0;
    uint32_t cap = 0;  // batch the activation buffers are sized for
    DevBuf X, H1, H2, dY, dH2, dH1;
    DevBuf sse;                  // the loss's partial sums (one per CTA of the last layer)
    double *sse_host = nullptr;  // their pinned copy
    uint64_t sse_n = 0;
    uint64_t loss_n = 0;  // outputs the loss is a mean over
    // parameter read-back: pinned buffers and streams of its copying threads
    static constexpr int COPIERS = 4;
    char *bounce = nullptr;
    cudaStream_t copy_streams[COPIERS] = {};

    Mlp() = default;
    Mlp(const Mlp &) = delete;
    Mlp &operator=(const Mlp &) = delete;
    ~Mlp();

    void init(uint32_t n_in, uint32_t n_hidden, uint32_t n_out, uint64_t seed);
    // Y = MLP(X) for `batch` rows of FP32 X [batch][n_in] into FP32 Y
    void forward(uint32_t batch, const float *X, float *Y);
    // gradients of the mean squared error against T at the current weights
    void backward(uint32_t batch, const float *X, const float *T);
    // one Adam step
    void train_step(uint32_t batch, const float *X, const float *T, float lr);
    // the loss of the last backward pass, before its step; once the stream has
    // been waited for
    double loss() const;
    uint64_t param_count() const;
    void copy_params(float *host, bool set, bool grads);

  private:
    void download(float *host, const float *dev, uint64_t count);
    void ensure(uint32_t batch);
    void refresh_bf16();
    void hidden(uint32_t batch, const float *X, bool split);
    static cudaStream_t S() { return ctx().stream; }
};

}  // namespace xg
