// 1D RK4 steps in registers, the FP64 class's contracted form
// (NLSE_FLAG_FMA): kern_step1d.cuh compiled with multiply-add contraction.
#include "kern_step1d.cuh"

namespace nlse {

cudaError_t launch_step1d_fma(const Geom& g, int method, int BC, const Consts<double>& c,
                              const C2<double>* in, const double* V, C2<double>* out,
                              const Step1dShape& sh, int m, cudaStream_t st) {
  return step1d::launch_exact<double, 1>(g, method, BC, c, in, V, out, sh, m, st);
}

}  // namespace nlse
