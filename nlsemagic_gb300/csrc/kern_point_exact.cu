// The exact classes' thread-per-point stages (kern_point.cuh).  Compiled with
// -fmad=false: the reference's bits.
#include "kern_point.cuh"

namespace nlse {

template <typename R>
cudaError_t launch_point_exact(const Geom& g, int method, int BC, const Consts<R>& c,
                               const ExactStageArgs<R>& a, int stage, cudaStream_t st) {
  if constexpr (sizeof(R) == 8)
    if (g.ndim == 2) return point::launch_ordered<R, 2, 0>(g, method, BC, c, a, stage, st);
  return point::launch_ordered<R, 3, 0>(g, method, BC, c, a, stage, st);
}

template cudaError_t launch_point_exact<double>(const Geom&, int, int, const Consts<double>&,
                                                const ExactStageArgs<double>&, int, cudaStream_t);
template cudaError_t launch_point_exact<float>(const Geom&, int, int, const Consts<float>&,
                                               const ExactStageArgs<float>&, int, cudaStream_t);

}  // namespace nlse
