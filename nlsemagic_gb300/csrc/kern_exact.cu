// Exact-precision (FP64 / FP32) stage launchers.  This translation unit is
// compiled with -fmad=false: no multiply-add is contracted, so every
// operation rounds exactly as in the reference C integrators.
#include "kern_exact_impl.cuh"

namespace nlse {

static bool tile2d_path(const Geom& g, int method, int BC, int kernel_kind, bool single) {
  (void)method;
  return g.ndim == 2 && single && kernel_kind != KERNEL_GATHER && BC != 4 && wide::g_wide2d;
}

// Thread-per-point stages (kern_point.cuh).  FP64 takes them in 2D and 3D: its
// issue rate is the bound, and they waste least of it.  Microseconds a step of
// one solve alone / of three in flight, against the gather kernels (2D) and the
// tiled ones (3D), MSD:
//   CD     200^2 40.3 / 24.9 -> 25.6 / 13.2    1500^2 514 / 485 -> 480 / 469
//          61 x 72 x 67 185 / 137 -> 101 / 70  200^3 2743 / 2419 -> 1912 / 1896
//   2SHOC  200^2 108 / 43.5 -> 48.5 / 25.4     1500^2 1001 / 952 -> 930 / 912
//          61 x 72 x 67 546 / 386 -> 257 / 171 200^3 8221 / 7653 -> 4692 / 4660
// FP32 is bound by L1 there.  2SHOC in 3D gains all the same, D no longer formed
// on a tile's halo (61 x 72 x 67 124 / 62 -> 42 / 26, 220^3 1294 / 1143 -> 768 /
// 757, Dirichlet 919 / 762 -> 771 / 758); CD, which the tiled kernel streams
// through once, up to 2^20 points (96^3 52 / 32 -> 35 / 32), where the state's
// rows do not start on 16 bytes and TMA cannot stage them (161 x 150 x 155 274 /
// 248 -> 127 / 123), and with MSD (160^3 186 / 145 -> 147 / 140; Dirichlet 168 /
// 131 against 146 / 140 stays tiled).
static bool point_path(const Geom& g, int method, int BC, int kernel_kind, bool single) {
  if (kernel_kind == KERNEL_GATHER || BC > 3) return false;
  if (!single && (g.ndim == 2 || method == 1)) return g.ndim >= 2;
  if (g.ndim != 3 || kernel_kind == KERNEL_STREAM) return false;
  return !single || (method == 2 || BC == 2 || g.M % 2 || g.n <= (1LL << 20));
}

// Where one point's chain of dependent instructions is all the time there is: by
// point, a thread next to a face does that face's points after its own, up to
// seven of them at a corner; by gather each has its thread.  Microseconds a step
// of one solve alone / of three in flight, by point -> by gather:
//   FP64 2D CD    Dirichlet 8^2 13.6 / 6.0 -> 9.1 / 3.4    48^2 15.4 / 5.8 -> 14.8 / 5.6
//                 64^2 13.9 / 5.5 against 15.1 / 6.2
//                 MSD  8^2 17.8 / 7.2 -> 15.7 / 6.2  12^2 18.5 / 7.2 against 19.2 / 7.1
//           2SHOC Dirichlet 8^2 27.5 / 11.1 -> 20.2 / 7.5  18^2 30.0 / 11.2 -> 29.8 / 10.4
//                 24^2 29.0 / 10.9 against 30.8 / 10.7; LAP0 15^2 28.0 / 10.0 against
//                 28.7 / 10.1
//                 MSD 10^2 35.4 / 12.7 -> 33.0 / 11.5  12^2 34.6 / 12.8 against 40.4 / 14.2
//   3D (the streaming kernels, which 3D had before, in the middle), MSD 2SHOC
//                 FP64 3^3 80.0 / 52.2 / 40.4   FP32 3^3 25.6 / 24.2 / 14.0
bool gather_small(const Geom& g, int method, int BC, int kernel_kind, bool single) {
  if (kernel_kind != KERNEL_TILED || BC > 3) return false;
  if (g.ndim == 3) return g.n <= 64;
  if (g.ndim != 2 || single) return false;
  return g.n <= (BC == 2 ? 128 : (method == 1 ? 3 << 10 : (BC == 1 ? 320 : 240)));
}

// D scratch: 2SHOC in gather form and by point.  FP32 2D grids on the tile
// kernel take none; should the knob turn it off later, the gather kernel
// recomputes D.  The contracted class takes the wide form by point, without D
// (kern_exact_fma.cu).
long long exact_dsc_entries(const Geom& g, int method, int BC, int kernel_kind, bool single,
                            bool contracted) {
  if (method != 2) return 0;
  if (contracted && g.ndim >= 2 && kernel_kind != KERNEL_GATHER)
    return gather_small(g, method, BC, kernel_kind, false) ? g.n : 0;
  if (g.ndim == 3 && kernel_kind == KERNEL_STREAM) return 0;
  return tile2d_path(g, method, BC, kernel_kind, single) ? 0 : g.n;
}

// 3D: the tiled kernels (kern_tiled.cuh) form D on the way.
bool exact_dsc_spare(const Geom& g, int method, int BC, int kernel_kind) {
  return method == 2 && g.ndim == 3 && BC <= 3 && kernel_kind != KERNEL_GATHER;
}

int exact_stage_launches(const Geom& g, int method, int BC, int kernel_kind, bool single,
                         bool has_dsc) {
  if (tile2d_path(g, method, BC, kernel_kind, single)) return 1;
  if (!single && seg1d_exact_path(g, BC, kernel_kind)) return 1;
  if (kernel_kind != KERNEL_GATHER && tiled_supported(g, g.ndim) && BC != 4 &&
      !point_path(g, method, BC, kernel_kind, single))
    return 1;
  return method == 2 && has_dsc ? 2 : 1;  // (D,) F
}

template <typename R>
cudaError_t launch_exact_stage(const Geom& g, int method, int BC, const Consts<R>& c,
                               const ExactStageArgs<R>& a, int stage, cudaStream_t st,
                               int kernel_kind) {
  if (gather_small(g, method, BC, kernel_kind, sizeof(R) == 4)) kernel_kind = KERNEL_GATHER;
  // (2SHOC whose D scratch did not fit forms D on the way)
  if (point_path(g, method, BC, kernel_kind, sizeof(R) == 4) && (method == 1 || a.dsc))
    return launch_point_exact<R>(g, method, BC, c, a, stage, st);
  return launch_exact_stage_var<R, 0>(g, method, BC, c, a, stage, st, kernel_kind);
}

template cudaError_t launch_exact_stage<double>(const Geom&, int, int, const Consts<double>&,
                                                const ExactStageArgs<double>&, int, cudaStream_t,
                                                int);
template cudaError_t launch_exact_stage<float>(const Geom&, int, int, const Consts<float>&,
                                               const ExactStageArgs<float>&, int, cudaStream_t,
                                               int);

}  // namespace nlse
