// 1D RK4 steps in registers, mixed class (kern_step1d.cuh), and the form a
// solve of any class takes.
#include "kern_step1d.cuh"

namespace nlse {

namespace step1d {
template <int METHOD, int R>
static cudaError_t mixed_by_bc(const Geom& g, int BC, const Consts<float>& c, const float2* hi,
                               const float2* lo, const float* V, float2* ho, float2* l2, int m,
                               int warps, cudaStream_t st, bool pdl) {
  const Plan p = make_plan(g.n, METHOD, R, m, warps);
  const dim3 gr(p.blocks), bl(32 * p.warps);
  const int n = (int)g.n;
  switch (BC) {
    case 1: return launch_k(mixed_steps<METHOD, 1, R>, gr, bl, 0, st, pdl, n, c, hi, lo, V, ho, l2, p);
    case 2: return launch_k(mixed_steps<METHOD, 2, R>, gr, bl, 0, st, pdl, n, c, hi, lo, V, ho, l2, p);
    case 3: return launch_k(mixed_steps<METHOD, 3, R>, gr, bl, 0, st, pdl, n, c, hi, lo, V, ho, l2, p);
    case 4: return launch_k(mixed_steps<METHOD, 4, R>, gr, bl, 0, st, pdl, n, c, hi, lo, V, ho, l2, p);
  }
  return cudaErrorInvalidValue;
}
}  // namespace step1d

// Windows of 32 R points that store U of them; m steps a launch.  Both sides
// of each line measured on MSD solves, microseconds a step of one solve alone
// / of three in flight, against the stage launches (kern_seg1d.cuh).
//
// FP32 and mixed, R = 4 (R = 2: more shuffles per point; R = 8: 150 registers):
// more steps a launch save launches and lose more of the window, which costs
// nothing while there are fewer windows than schedulers (4 x 152).  Mixed CD,
// stage launches 3.8 / 1.3 at 1024 points, 8.0 / 3.3 at 48611, 26.9 / 26.9 at
// 10^6:  m = 10: 1.7 / 0.62, 2.2 / 1.1, -;  m = 6: 1.8 / 0.68, 1.9 / 0.98, -;
// m = 4: 2.0 / 0.76, 2.8 / 1.0, 7.5 / 5.7;  m = 3: -, -, 7.1 / 5.4.  Mixed
// 2SHOC (loses twice as much), 6.2 / 2.1, 9.6 / 3.9, 32.9 / 30.8:  m = 6:
// 3.2 / 1.1, -, -;  m = 4: 3.3 / 1.2, 4.1 / 1.7, -;  m = 2: -, 5.0 / 1.8,
// 11.2 / 8.1.  FP32 alike: 2SHOC at 10^6 points 28.6 / 27.2 -> 8.4 / 5.8.
//
// FP64 is bound by its issue rate (a warp instruction takes 16 clocks of an
// SM), so small windows spread over the SMs, one warp per block: R = 1 up to
// 2^13 points, R = 2 (fewer points lost per window) up to 2^16; above, the
// lost points cost more than the launches, and the stage launches stay.  CD,
// stage launches 16.4 / 5.7 at 1024 points, 18.4 / 10.5 at 16384, 32 / 13.8
// at 48611, 61 / 35.7 at 200003: R = 1, m = 3: 6.5 / 2.4; R = 2, m = 1: -,
// 12.4 / 5.1, 16.5 / 11.1, -; R = 4, m = 1: -, -, -, 47 / 38.  2SHOC, 25.8 /
// 8.8, 27 / 13.7, 45 / 18.3: R = 1, m = 1: 13.1 / 4.7, -, -; R = 2, m = 1:
// -, 20 / 8.8, 28 / 17.4.
Step1dShape step1d_shape(const Geom& g, int method, int precision, int kernel_kind) {
  Step1dShape sh = {0, 4, step1d::MAX_WARPS};
  const long long n = g.n;
  if (g.ndim != 1 || kernel_kind == KERNEL_GATHER || !wide::g_seg1d || n > (1LL << 30)) return sh;
  if (precision == 2) {
    if (n > (1LL << 16)) return sh;
    sh.warps = 1;
    sh.per_lane = n <= (1LL << 13) ? 1 : 2;
    sh.steps = method == 1 && sh.per_lane == 1 ? (n <= 152 * 8 ? 3 : 2) : 1;
  } else if (method == 1) {
    sh.steps = n <= (1LL << 15) ? 10 : (n <= 3LL << 15 ? 6 : (n <= (1LL << 19) ? 4 : 3));
  } else {
    sh.steps = n <= (1LL << 13) ? 6 : (n <= (1LL << 16) ? 4 : 2);
  }
  if (n <= 32 * sh.per_lane) sh.steps = 1 << 16;  // one window, nothing lost
  return sh;
}

cudaError_t launch_step1d_mixed(const Geom& g, int method, int BC, const Consts<float>& c,
                                const float2* hi, const float2* lo, const float* V, float2* ho,
                                float2* l2, const Step1dShape& sh, int m, cudaStream_t st) {
#define NLSE_STEP1D(R)                                                                            \
  return method == 2                                                                              \
             ? step1d::mixed_by_bc<2, R>(g, BC, c, hi, lo, V, ho, l2, m, sh.warps, st, wide::g_pdl != 0) \
             : step1d::mixed_by_bc<1, R>(g, BC, c, hi, lo, V, ho, l2, m, sh.warps, st, wide::g_pdl != 0)
  switch (sh.per_lane) {
    case 1: NLSE_STEP1D(1);
    case 2: NLSE_STEP1D(2);
    case 4: NLSE_STEP1D(4);
    }
#undef NLSE_STEP1D
  return cudaErrorInvalidValue;
}

}  // namespace nlse
