// The contracted FP64 class (NLSE_FLAG_FMA) in 2D and 3D (kern_point.cuh).
#include "kern_point.cuh"

namespace nlse {

cudaError_t launch_point_fma(const Geom& g, int method, int BC, const Consts<double>& c,
                             const ExactStageArgs<double>& a, int stage, cudaStream_t st) {
  using namespace point;
  if (method == 2)
    return g.ndim == 3 ? launch<double, 3, WIDE, 1>(g, BC, c, a, stage, st)
                       : launch<double, 2, WIDE, 1>(g, BC, c, a, stage, st);
  return g.ndim == 3 ? launch<double, 3, CD, 1>(g, BC, c, a, stage, st)
                     : launch<double, 2, CD, 1>(g, BC, c, a, stage, st);
}

}  // namespace nlse
