// 2D RK4 steps of the mixed class, one launch per step (kern_step2d.cuh), and
// the form a 2D solve of any class takes.
#include "kern_step2d.cuh"

namespace nlse {
namespace step2d {

// Threads by rows, blocks per SM: see step2d_shape.
template <int METHOD, int BC>
static cudaError_t by_shape(const Geom& g, const Consts<float>& c, const float2* hi,
                            const float2* lo, const float* V, float2* K, float2* ho, float2* l2,
                            int shape, cudaStream_t st, bool pdl) {
  if constexpr (METHOD == 1) {
    switch (shape) {
      case SMALL: return launch_shape<1, BC, 32, 8, 4, 3>(g, c, hi, lo, V, K, ho, l2, st, pdl);
      case MIDDLE: return launch_shape<1, BC, 32, 8, 4, 4>(g, c, hi, lo, V, K, ho, l2, st, pdl);
      case LARGE: return launch_shape<1, BC, 64, 4, 8, 3>(g, c, hi, lo, V, K, ho, l2, st, pdl);
    }
  } else {
    switch (shape) {
      case SMALL: return launch_shape<2, BC, 64, 8, 4, 1>(g, c, hi, lo, V, K, ho, l2, st, pdl);
      case MIDDLE: return launch_shape<2, BC, 32, 8, 4, 3>(g, c, hi, lo, V, K, ho, l2, st, pdl);
      case LARGE: return launch_shape<2, BC, 64, 8, 4, 2>(g, c, hi, lo, V, K, ho, l2, st, pdl);
    }
  }
  return cudaErrorInvalidValue;
}
}  // namespace step2d

// Which tile, by the number of points.  Larger blocks lose less to the halo
// (2SHOC: 64 x 32 cells give a tile of 52 x 20, 32 x 32 one of 20 x 20), smaller
// ones spread a small grid over more SMs; more rows per thread need fewer
// shared-memory reads and more registers.  Microseconds a step of one solve
// alone / of three in flight, BC 1, against the stage launches
// (kern_wide2d.cuh, kern_tile2d.cuh):
//            stage launches   SMALL         MIDDLE        LARGE
//   mixed CD
//   256^2     9.5 /  3.6      5.2 /  2.5    5.2 /  2.6    8.3 /  3.7
//   500^2    12.3 /  6.3      7.3 /  4.1    8.5 /  3.9   11.7 /  5.0
//   900^2    25.7 / 18.9     15.6 / 12.5   14.7 / 10.9   16.1 /  9.9
//   2048^2    114 /  101     68.4 / 63.7   60.0 / 55.0   57.2 / 48.4
//   mixed 2SHOC
//   64^2      7.1 /  2.7      6.9 /  2.4    5.2 /  1.9    7.5 /  2.6
//   256^2    11.9 /  4.3      7.0 /  2.9    7.7 /  3.3    7.7 /  4.0
//   500^2    15.2 /  8.6     11.3 /  8.1   11.9 /  7.1   11.1 /  6.1
//   2048^2    130 /  116      136 /  131    119 /  115   95.7 / 89.2
//   FP32 CD (SMALL, LARGE)
//   64^2      7.2 /  2.6      3.6 /  1.3                  5.7 /  2.0
//   500^2    13.1 /  5.8      7.2 /  3.1                  8.1 /  3.8
//   1300^2   38.8 / 47.5     20.0 / 17.3                 18.3 / 13.6
// MSD adds two quotients one after the other to every stage of an edge tile,
// which small grids wait for (CD 64^2: 7.2 / 2.6 -> 7.5 / 2.6, 250^2 10.3 / 3.8
// -> 7.7 / 3.2); 2SHOC takes 32 x 32 up to 2^18 (420^2: 15.2 / 7.0, SMALL 15.4 /
// 7.6, MIDDLE 13.4 / 6.4, LARGE 19 / 7.6).  The next launch (PDL) is triggered
// before the last stage: triggered at the start, its blocks are placed while this
// launch's come and go and load the SMs unevenly (300^2 CD three in flight 2.6,
// 2.3 so).
// A grid of fewer than 16 points a side fills too little of a tile (8000 x 8:
// 3.8 against 5.4 with three in flight), and where most tiles are at a face and
// more than can all start at once, the stage launches, whose faces cost less, are
// the faster form: by step_cells.  Stage launches, this: 2SHOC MSD 16 x 62500 89 /
// 81, 161 / 158; 64 x 15625 49 / 42, 95 / 91; 15625 x 64 39 / 32, 39 / 35; 128 x 7812
// 46 / 36, 62 / 52; 64 x 1406 16 / 5.8, 12 / 10; CD MSD 32 x 31250 39 / 32, 60 / 56,
// 15625 x 64 31 / 25, 25 / 20; FP32 CD MSD 64 x 15625 32 / 27, 44 / 41.  Of 432
// narrow grids of 2e4 to 1e6 points the rule takes the slower form by more than
// 5% (mean of both figures) on 3.
// Mixed CD MSD up to 2^11 points: 24^2 6.9 / 2.6 stage launches, 7.7 / 2.8 so.
int step2d_shape(const Geom& g, int method, int BC, int precision, int kernel_kind) {
  using namespace step2d;
  if (g.ndim != 2 || kernel_kind == KERNEL_GATHER || !wide::g_wide2d || wide2d::g_ty) return 0;
  if (precision == 2 || (precision == 1 && method == 2) || BC > 3) return 0;
  if (g.M < 16 || g.N < 16 || g.N > 65535 * 20) return 0;  // tile rows: gridDim.y
  const bool cd = method == 1, single = precision == 1;
  if (cd && !single && BC == 2 && g.n <= (1LL << 11)) return 0;
  int shape = LARGE;
  if (single)
    shape = g.n <= (1LL << 19) ? SMALL : LARGE;
  else if (cd)
    shape = g.n <= (1LL << 18) ? SMALL : (g.n <= (1LL << 20) ? MIDDLE : LARGE);
  else if (g.n <= (1LL << 15) || (BC == 2 && g.n > (1LL << 17) && g.n <= (1LL << 18)))
    shape = MIDDLE;
  else if (g.n <= (1LL << 17))
    shape = SMALL;
  // the tiles of by_shape; so few all start at once
  const bool wide = cd ? shape == LARGE : shape != MIDDLE;
  const int tx = cd ? (wide ? 58 : 26) : (wide ? 52 : 20), ty = cd ? 26 : 20;
  const int nbx = (g.M + tx - 1) / tx;
  const long long tiles = (long long)nbx * ((g.N + ty - 1) / ty);
  int at_once = !cd && shape == SMALL ? 152 : 280;
  if (BC == 2 && nbx <= 2) at_once /= 2;  // none away from an x face
  if (tiles > at_once && step_cells(g, BC, tx, ty, wide ? 2048 : 1024) > stage_cells(g, method, single))
    return 0;
  return shape;
}

cudaError_t launch_step2d_mixed(const Geom& g, int method, int BC, const Consts<float>& c,
                                const float2* hi, const float2* lo, const float* V, float2* K,
                                float2* ho, float2* l2, int shape, cudaStream_t st) {
  const bool pdl = wide::g_pdl != 0;
#define NLSE_STEP2D(bc)                                                                       \
  case bc:                                                                                    \
    return method == 2 ? step2d::by_shape<2, bc>(g, c, hi, lo, V, K, ho, l2, shape, st, pdl)  \
                       : step2d::by_shape<1, bc>(g, c, hi, lo, V, K, ho, l2, shape, st, pdl)
  switch (BC) {
    NLSE_STEP2D(1);
    NLSE_STEP2D(2);
    NLSE_STEP2D(3);
  }
#undef NLSE_STEP2D
  return cudaErrorInvalidValue;
}

}  // namespace nlse
