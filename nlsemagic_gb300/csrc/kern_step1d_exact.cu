// 1D RK4 steps in registers, FP64 / FP32 (kern_step1d.cuh).  Compiled with
// -fmad=false like the other exact-class kernels: the reference's bits.
#include "kern_step1d.cuh"

namespace nlse {

template <>
cudaError_t launch_step1d_exact<double>(const Geom& g, int method, int BC, const Consts<double>& c,
                                        const C2<double>* in, const double* V, C2<double>* out,
                                        const Step1dShape& sh, int m, cudaStream_t st) {
  return step1d::launch_exact<double, 0>(g, method, BC, c, in, V, out, sh, m, st);
}
template <>
cudaError_t launch_step1d_exact<float>(const Geom& g, int method, int BC, const Consts<float>& c,
                                       const C2<float>* in, const float* V, C2<float>* out,
                                       const Step1dShape& sh, int m, cudaStream_t st) {
  return step1d::launch_exact<float, 0>(g, method, BC, c, in, V, out, sh, m, st);
}

}  // namespace nlse
