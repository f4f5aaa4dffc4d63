// Host-side launch interface between the C ABI (nlse_abi.cu) and the
// stage-kernel translation units.
#pragma once

#include <cuda_runtime.h>

#include "nlse_common.cuh"

struct nlse_ic;  // include/nlse_gb300.h

namespace nlse {

// STREAM: as TILED, but 3D stages by the streaming kernels where the class has
// them, never by point (NLSE_FLAG_STREAM).
enum KernelKind { KERNEL_GATHER = 0, KERNEL_TILED = 1, KERNEL_STREAM = 2 };

template <typename R>
struct ExactStageArgs {
  const C2<R>* Yin;  // stage input (stage 1: Psi itself)
  C2<R>* Psi;        // RK4 base state (written in stage 4)
  const R* V;
  C2<R>* K;
  C2<R>* Yout;       // next stage input (stages 1-3)
  C2<R>* dsc;        // 2SHOC by gather or by point: D scratch (n points), or null
};

struct MixedStageArgs {
  const float2* hi_in;
  const float2* lo_in;
  const float2* e_in;  // stage input E = lo + d (unused in stage 1)
  const float* V;
  float2* K;
  float2* e_out;      // next stage input E
  float2* hi_out;      // stage 4 output (a different buffer from hi_in)
  float2* lo_out;
  // 3D 2SHOC on the tiled path (null otherwise):
  float4* gh;          // ghost values (hi, E) one cell outside each face, mixed_ghost_entries()
  float2* fq;          // F at the points next to a face (n entries, MSD only)
  float2* dsc;         // 2SHOC on the gather path: D scratch (n points), or null
  // 3D 2SHOC on the tiled path: x-face strips (null: not kept).  The x
  // faces' own lo, K and V in face-indexed order, [side][z][y], which the
  // face kernel reads and writes there instead of the full arrays' strided
  // x faces (K at the x faces is kept in the strip only), and V at the
  // points next to them (s_Vq, for the ghost kernel).
  const float2* s_lo_in;
  float2 *s_lo_out, *s_K;
  const float *s_V, *s_Vq;
};

// Entries of one x-face strip array: 2 sides x N x L.
inline long long xstrip_entries(const Geom& g) { return 2LL * g.N * g.L; }
// Whether a grid keeps x-face strips (the knob wide.strips), and their
// refill from the state's lo and V.
bool mixed_strip_path(const Geom& g, int method, int BC, int kernel_kind);
cudaError_t mixed_strip_fill(const Geom& g, const float2* lo, const float* V, float2* slo,
                             float* sV, float* sVq, cudaStream_t st);


template <typename R>
cudaError_t launch_exact_stage(const Geom& g, int method, int BC, const Consts<R>& c,
                               const ExactStageArgs<R>& a, int stage, cudaStream_t st,
                               int kernel_kind);

// The FP64 class's contracted form (NLSE_FLAG_FMA; kern_exact_fma.cu): the
// same kernels and dispatch as launch_exact_stage<double>, compiled with
// multiply-add contraction.
cudaError_t launch_exact_stage_fma(const Geom& g, int method, int BC, const Consts<double>& c,
                                   const ExactStageArgs<double>& a, int stage, cudaStream_t st,
                                   int kernel_kind);

// Whether a grid is so small that its FP64 (2D, 3D) or FP32 (3D) stages run by
// gather, not by point (kern_exact.cu).
bool gather_small(const Geom& g, int method, int BC, int kernel_kind, bool single);

// Thread-per-point stages in 2D and 3D (kern_point.cuh): exact, contracted.
template <typename R>
cudaError_t launch_point_exact(const Geom& g, int method, int BC, const Consts<R>& c,
                               const ExactStageArgs<R>& a, int stage, cudaStream_t st);
cudaError_t launch_point_fma(const Geom& g, int method, int BC, const Consts<double>& c,
                             const ExactStageArgs<double>& a, int stage, cudaStream_t st);
// 3D, mixed (kern_point_mixed.cu), and which grids take it.
bool mixed_point_path(const Geom& g, int method, int BC, int kernel_kind);
cudaError_t launch_point_mixed(const Geom& g, int method, int BC, const Consts<float>& c,
                               const MixedStageArgs& a, int stage, cudaStream_t st);

cudaError_t launch_mixed_stage(const Geom& g, int method, int BC, const Consts<float>& c,
                               const MixedStageArgs& a, int stage, cudaStream_t st,
                               int kernel_kind);

// Kernel launches one mixed stage issues (launch_mixed_stage), and the
// scratch the tiled 3D 2SHOC path needs: ghost entries (float4) and F
// entries (float2) for MixedStageArgs::gh / ::fq (0 when not needed).
// Small 1D solves: every pass of nsteps RK4 steps in one single-block launch
// (kern_small.cuh); same buffers and results as the stage launches.
template <typename R>
cudaError_t launch_small1d_exact(const Geom& g, int method, int BC, const Consts<R>& c, C2<R>* psi,
                                 C2<R>* K, C2<R>* ya, C2<R>* yb, const R* V, C2<R>* D,
                                 long long nsteps, cudaStream_t st);
cudaError_t launch_small1d_mixed(const Geom& g, int method, int BC, const Consts<float>& c,
                                 float2* const hi[2], float2* const lo[2], float2* K, float2* da,
                                 float2* db, float2* dc, const float* V, float2* D, int cur,
                                 long long nsteps, cudaStream_t st);

int mixed_stage_launches(const Geom& g, int method, int BC, int kernel_kind, bool has_dsc);
int exact_stage_launches(const Geom& g, int method, int BC, int kernel_kind, bool single,
                         bool has_dsc);
long long mixed_ghost_entries(const Geom& g, int method, int BC, int kernel_kind);
long long mixed_fq_entries(const Geom& g, int method, int BC, int kernel_kind);
// Points of D scratch (ExactStageArgs / MixedStageArgs ::dsc) a 2SHOC stage
// uses that takes two launches, else 0.  contracted: NLSE_FLAG_FMA.
long long exact_dsc_entries(const Geom& g, int method, int BC, int kernel_kind, bool single,
                            bool contracted);
// Whether a solve that uses that scratch has another form than the gather
// kernels' without it (should it not fit).
bool exact_dsc_spare(const Geom& g, int method, int BC, int kernel_kind);
long long mixed_dsc_entries(const Geom& g, int method, int BC, int kernel_kind);

// Layout conversions and reductions (kern_util.cu).  stride 2: re and im are the
// two parts of an interleaved complex array (im = re + 1).
cudaError_t planar_to_c2d(const double* re, const double* im, C2<double>* out, long long n,
                          cudaStream_t st, int stride = 1);
cudaError_t planar_to_c2f(const double* re, const double* im, C2<float>* out, long long n,
                          cudaStream_t st, int stride = 1);
cudaError_t planar_to_hilo(const double* re, const double* im, float2* hi, float2* lo,
                           long long n, cudaStream_t st, int stride = 1);
cudaError_t c2d_to_planar(const C2<double>* in, double* re, double* im, long long n,
                          cudaStream_t st, int stride = 1);
cudaError_t c2f_to_planar(const C2<float>* in, double* re, double* im, long long n,
                          cudaStream_t st, int stride = 1);
cudaError_t hilo_to_planar(const float2* hi, const float2* lo, double* re, double* im,
                           long long n, cudaStream_t st, int stride = 1);
cudaError_t real_to_float(const double* in, float* out, long long n, cudaStream_t st);
cudaError_t fill_zero_bytes(void* p, size_t bytes, cudaStream_t st);

// sum |psi|^2 into *out (device double, pre-zeroed by the callee) and set
// *bad to 1 if any component is not finite.
cudaError_t mass_c2d(const C2<double>* psi, long long n, double* out, int* bad, cudaStream_t st);
cudaError_t mass_c2f(const C2<float>* psi, long long n, double* out, int* bad, cudaStream_t st);
cudaError_t mass_hilo(const float2* hi, const float2* lo, long long n, double* out, int* bad,
                      cudaStream_t st);

// The form a 1D solve's run takes: RK4 steps per launch (0: the stage
// launches), points per lane, warps per block.
struct Step1dShape {
  int steps, per_lane, warps;
};
Step1dShape step1d_shape(const Geom& g, int method, int precision, int kernel_kind);
// Whole RK4 steps of a 1D solve in registers (kern_step1d.cuh): m <= sh.steps
// steps, from one state buffer into another.
template <typename R>
cudaError_t launch_step1d_exact(const Geom& g, int method, int BC, const Consts<R>& c,
                                const C2<R>* in, const R* V, C2<R>* out, const Step1dShape& sh, int m,
                                cudaStream_t st);
cudaError_t launch_step1d_fma(const Geom& g, int method, int BC, const Consts<double>& c,
                              const C2<double>* in, const double* V, C2<double>* out,
                              const Step1dShape& sh, int m, cudaStream_t st);
cudaError_t launch_step1d_mixed(const Geom& g, int method, int BC, const Consts<float>& c,
                                const float2* hi, const float2* lo, const float* V, float2* ho,
                                float2* l2, const Step1dShape& sh, int m, cudaStream_t st);

// Whole RK4 steps of a 2D solve, one launch each (kern_step2d.cuh): the tile
// shape (0: the stage launches), and one step from one state buffer pair into
// the other.
int step2d_shape(const Geom& g, int method, int BC, int precision, int kernel_kind);
cudaError_t launch_step2d_mixed(const Geom& g, int method, int BC, const Consts<float>& c,
                                const float2* hi, const float2* lo, const float* V, float2* K,
                                float2* ho, float2* l2, int shape, cudaStream_t st);
cudaError_t launch_step2d_exact(const Geom& g, int BC, const Consts<float>& c, const C2<float>* in,
                                const float* V, C2<float>* out, int shape, cudaStream_t st);

bool tiled_supported(const Geom& g, int dim);

// Initial conditions and diagnostics (kern_init.cu); ::nlse_ic is declared
// in include/nlse_gb300.h.
cudaError_t launch_ic(int ndim, int M, int N, int L, double h, const ::nlse_ic& ic,
                      const double* d_items, double s, double a, double* re, double* im, double* V,
                      cudaStream_t st);
cudaError_t launch_diag(int cls, int ndim, int M, int N, int L, double h, const void* a,
                        const void* b, const ::nlse_ic* ic, double s, double aa, double t,
                        void* scratch, double out[7], cudaStream_t st);

// 2D cubic-quintic 2SHOC stage (kern_cq.cu): D into Dscratch, then F and the
// RK4 update, FP64.
struct CqParams {
  int M, N, BC, guard;
  double s1, s2, a, lh2, l_a, a1_6h2, a1_12;
};
cudaError_t launch_cq_stage(const CqParams& c, const Consts<double>& k, const C2<double>* Yin,
                            C2<double>* Psi, const double* V, C2<double>* K, C2<double>* Yout,
                            C2<double>* Dscratch, int stage, cudaStream_t st);

// 3D vorticity (kern_vort.cu): planar FP64 U of M x N x L points -> wx, wy,
// wz, W; vscratch holds 3 n doubles.
cudaError_t launch_vorticity(int M, int N, int L, const double* Ur, const double* Ui, double lh2,
                             double veps, double* vscratch, double* wx, double* wy, double* wz,
                             double* W, cudaStream_t st);

// Device error word of the tiled kernels (bounded-wait timeouts, self-check
// failures): take_device_error() returns and clears it.
namespace tiled {
int* error_word();
}
int take_device_error();

}  // namespace nlse
