// SpMV kernels of the Jacobi smoother and the mixed-precision prolongation.
#include "spmv_launch.cuh"

namespace xg {
namespace ops {

template <typename F>
void jacobi_sweep(const DCsr &A, const F *xin, F *xout, const F *b, const F *d, F relax, int nv,
                  cudaStream_t s) {
    XG_DISPATCH(A, nv, {
        launch<F, F, I, NV, 0>(A, xin, k::EJacobi<F, NV>(xout, xin, b, d, relax), s);
    });
}
template void jacobi_sweep<double>(const DCsr &, const double *, double *, const double *,
                                   const double *, double, int, cudaStream_t);
template void jacobi_sweep<float>(const DCsr &, const float *, float *, const float *,
                                  const float *, float, int, cudaStream_t);


void prolong_mixed(const DCsr &P, const float *xH, double *x, bool x_zero, int nv,
                   cudaStream_t s) {
    XG_DISPATCH(P, nv, {
        launch<float, float, I, NV, 0>(P, xH, k::EProlongMixed<NV>(x, (int)x_zero), s);
    });
}

}  // namespace ops
}  // namespace xg
