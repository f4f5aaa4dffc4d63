// 2D RK4 steps of the FP32 class with CD, one launch per step
// (kern_step2d_exact.cuh).  Compiled with -fmad=false: the reference's bits.
#include "kern_step2d_exact.cuh"

namespace nlse {

template <int BC>
static cudaError_t by_shape(const Geom& g, const Consts<float>& c, const C2<float>* in,
                            const float* V, C2<float>* out, int shape, cudaStream_t st) {
  const bool pdl = wide::g_pdl != 0;
  switch (shape) {
    case step2d::SMALL: return step2d::launch_exact_cd<BC, 32, 8, 4, 5>(g, c, in, V, out, st, pdl);
    case step2d::LARGE: return step2d::launch_exact_cd<BC, 64, 4, 8, 4>(g, c, in, V, out, st, pdl);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_step2d_exact(const Geom& g, int BC, const Consts<float>& c, const C2<float>* in,
                                const float* V, C2<float>* out, int shape, cudaStream_t st) {
  switch (BC) {
    case 1: return by_shape<1>(g, c, in, V, out, shape, st);
    case 2: return by_shape<2>(g, c, in, V, out, shape, st);
    case 3: return by_shape<3>(g, c, in, V, out, shape, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace nlse
