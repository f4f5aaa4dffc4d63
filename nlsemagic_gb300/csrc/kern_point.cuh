// 2D and 3D stages of the exact classes, a thread per point.
//
// FP64 is bound by its issue rate (a warp instruction takes 16 clocks of an
// SM), so the kernels are laid out for full warps of FP64 work and nothing
// else: the points with two cells to every face ("deep") are numbered
// consecutively and read their neighbours through L1 (3D wide form: 70 of the
// 700 clocks a warp's stage takes); every point next to a face has a thread of
// its own, in blocks of such threads only, that also does the face points whose
// MSD neighbour it is.  Nothing waits within a launch.  The tiled kernels
// (kern_tiled.cuh) form 2SHOC's D on their halo as well and idle at a barrier
// per plane; the gather kernels (kern_gather.cuh) mix face points, whose code
// is long, into warps of others.
//
// Forms:
//   CD, D, F   the gather kernels' per-point functions in their order: CD in one
//              launch; 2SHOC as D at the interior and the face-interior points
//              into scratch, then F.  In a unit compiled with -fmad=false the
//              reference's bits.
//   WIDE       2SHOC of the contracted class (NLSE_FLAG_FMA) in one launch.
//              Where every face neighbour is interior the compact scheme equals
//              the wide fourth-order Laplacian a/(12 h^2) (16 sum_f (Y_f - Y_0) -
//              sum_2 (Y_2 - Y_0)), f the face neighbours, 2 the points two cells
//              off; next to a face point b it still does once the cell beyond b
//              holds the ghost
//                G = Y_b + h^2 D_bc(b) - (Y_q - Y_b) - sum_t (Y_t - Y_b)
//              (kern_wide.cuh).  So D is never formed: 41 FP64 operations a
//              point and stage in 3D and 31 in 2D against 80 and 47 of the
//              compact form.  The second differences are taken per axis as (Y_+ - 2
//              Y_0) + Y_-: on a resolved field both operations are exact (the first
//              is a multiple of Y_0's last place and about as large as Y_0, the
//              second cancels), where Y_+ + Y_- rounds at twice |Y|, and the sums are
//              weighted by 16.  Error against extended precision after 20 steps,
//              relative L2, 2D / 3D: compact form 1.76e-16 / 2.28e-16, this one
//              1.71e-16 / 1.96e-16 (1.87e-16 / 2.08e-16 with the sums first).
//
// Measured, one solve of 128^3 points in 2SHOC: contracted class 1305 -> 651 us a
// step (Dirichlet), FP64 1630 -> 1208; the FP64 pipe's 529 G additions and 628 G
// multiply-adds a second set 600 and 1190.  Where each form is taken, with both
// sides: kern_exact.cu (point_path), kern_mixed.cu (mixed_point_path).
#pragma once

#include "kern_gather.cuh"
#include "nlse_launch.h"
#include "nlse_pdl.cuh"

namespace nlse {
namespace point {

enum Form { CD, D, F, WIDE };

// Threads per block.  FP64: small blocks spread a small grid's warps, above all
// those next to faces, over the SMs (WIDE 64^2: 26 us a step with blocks of 64,
// 36 with 256).  FP32 reads through L1 at its rate and wants blocks that share
// lines: 128 (61 x 72 x 67 CD, three solves in flight: 10.7 us a step, 17.9 with
// 64), 256 from 2^20 points (160^3 2SHOC: 319 us, 371 with 128).
// The blocks of shell threads (points next to a face), then the deep points.
struct Map {
  unsigned shell_blocks, shell, deep;  // blocks, threads, points
  unsigned pz, py;                     // shell threads of the z and the y layers
  FastDiv z_row, y_row, x_row;         // points per row of a z, y, x layer
  FastDiv z_lay, y_lay, x_lay;         // points per layer
  FastDiv d_row, d_plane;              // deep points per row and plane
};

inline Map make_map(const Geom& g, int nt) {
  auto in = [](int n) { return (unsigned)(n - 2); };
  auto dp = [](int n) { return (unsigned)(n > 4 ? n - 4 : 0); };
  auto layers = [&](int n) { return in(n) > 1 ? 2u : 1u; };  // n = 3: one
  const bool d3 = g.ndim == 3;
  const unsigned Ld = d3 ? dp(g.L) : 1;
  const unsigned zl = in(g.M) * in(g.N), yl = in(g.M) * Ld, xl = dp(g.N) * Ld;
  Map m;
  m.pz = d3 ? layers(g.L) * zl : 0;
  m.py = layers(g.N) * yl;
  m.shell = m.pz + m.py + layers(g.M) * xl;
  m.z_row = FastDiv(in(g.M));
  m.z_lay = FastDiv(zl);
  m.y_row = FastDiv(in(g.M));
  m.y_lay = FastDiv(yl);
  m.x_row = FastDiv(dp(g.N));
  m.x_lay = FastDiv(xl);
  m.d_row = FastDiv(dp(g.M));
  m.d_plane = FastDiv(dp(g.M) * dp(g.N));
  m.deep = dp(g.M) * dp(g.N) * Ld;
  m.shell_blocks = (m.shell + nt - 1) / nt;
  return m;
}

// Deep point d's index in the grid.
template <int DIM>
__device__ __forceinline__ unsigned deep_index(const Geom& g, const Map& m, unsigned d) {
  const unsigned z = DIM == 3 ? m.d_plane.div(d) : 0, e = d - z * m.d_plane.d;
  const unsigned y = m.d_row.div(e), x = e - y * m.d_row.d;
  return (DIM == 3 ? (z + 2) * (unsigned)g.P : 0u) + (y + 2) * (unsigned)g.M + x + 2;
}

// Coordinates (x, y, z) of shell thread t's point.
template <int DIM>
__device__ __forceinline__ void shell_point(const Geom& g, const Map& m, unsigned t, int* q) {
  if (DIM == 3 && t < m.pz) {
    const unsigned l = m.z_lay.div(t), e = t - l * m.z_lay.d, y = m.z_row.div(e);
    q[0] = 1 + (int)(e - y * m.z_row.d);
    q[1] = 1 + (int)y;
    q[2] = l ? g.L - 2 : 1;
    return;
  }
  t -= m.pz;
  if (t < m.py) {
    const unsigned l = m.y_lay.div(t), e = t - l * m.y_lay.d, z = m.y_row.div(e);
    q[0] = 1 + (int)(e - z * m.y_row.d);
    q[1] = l ? g.N - 2 : 1;
    q[2] = DIM == 3 ? 2 + (int)z : 0;
    return;
  }
  t -= m.py;
  const unsigned l = m.x_lay.div(t), e = t - l * m.x_lay.d, z = m.x_row.div(e);
  q[0] = l ? g.M - 2 : 1;
  q[1] = 2 + (int)(e - z * m.x_row.d);
  q[2] = DIM == 3 ? 2 + (int)z : 0;
}

template <typename R>
__device__ __forceinline__ C2<R> add(C2<R> a, C2<R> b) {
  return {a.r + b.r, a.i + b.i};
}
// a + w b
template <typename R>
__device__ __forceinline__ C2<R> axpy(C2<R> a, R w, C2<R> b) {
  return {fma(w, b.r, a.r), fma(w, b.i, a.i)};
}

// (p - 2 y) + m: the second difference along an axis, exact on a resolved field
template <typename R>
__device__ __forceinline__ C2<R> second(C2<R> p, C2<R> y, C2<R> m) {
  return add(axpy(p, (R)-2, y), m);
}

// F = i (c12 (16 t1 - s2 + 2 DIM y) + (s|y|^2 - V) y), t1 the sum of the second
// differences, s2 the sum over the points two cells off
template <typename R, int DIM>
__device__ __forceinline__ C2<R> rhs_wide(const Consts<R>& c, C2<R> y, R v, C2<R> t1, C2<R> s2) {
  const R nl = fma(c.s, fma(y.r, y.r, y.i * y.i), -v);
  const R wr = fma((R)(2 * DIM), y.r, -s2.r), wi = fma((R)(2 * DIM), y.i, -s2.i);
  const R lr = fma((R)16, t1.r, wr), li = fma((R)16, t1.i, wi);
  return {-fma(c.a12lh2, li, nl * y.i), fma(c.a12lh2, lr, nl * y.r)};
}

// D or F at an interior point from U (and D): exact::d_int_at, f_int, f_int_d
template <typename R, int DIM, Form FORM>
__device__ __forceinline__ C2<R> interior(const Geom& g, const Consts<R>& c, const C2<R>* u, R v,
                                          const C2<R>* d) {
  const int M = g.M, P = g.P;
  if (FORM == CD) {
    if (DIM == 2) return exact::f_cd_2d<R>(c, u[0], v, u[M], u[-M], u[1], u[-1]);
    return exact::f_cd_3d<R>(c, u[0], v, u[P], u[-P], u[M], u[-M], u[1], u[-1]);
  }
  if (FORM == D) {
    if (DIM == 2) return exact::d_int_2d<R>(c, u[M], u[-M], u[0], u[1], u[-1]);
    return exact::d_int_3d<R>(c, u[P], u[-P], u[M], u[-M], u[1], u[-1], u[0]);
  }
  if (DIM == 2) {
    const C2<R> dn[4] = {d[M], d[-M], d[1], d[-1]};
    const C2<R> dg[4] = {u[M + 1], u[M - 1], u[-M + 1], u[-M - 1]};
    return exact::f_2shoc_2d<R>(c, u[0], v, d[0], dn, dg);
  }
  const C2<R> dn[6] = {d[P], d[-P], d[M], d[-M], d[1], d[-1]};
  const C2<R> e[12] = {u[P + M], u[M + 1], u[P + 1], u[-P - M], u[-M - 1], u[-P - 1],
                       u[P - M], u[M - 1], u[P - 1], u[-P + M], u[-M + 1], u[-P + 1]};
  return exact::f_2shoc_3d<R>(c, u[0], v, d[0], dn, e);
}

// One launch of a stage.  The deep points trigger the next launch once F is
// formed, not at the start: its blocks are then placed as this launch ends, which
// hides its latency.  Placed at the start, while this launch's blocks still come
// and go, they load the SMs unevenly (FP64 2SHOC on 200 x 333, one solve: 110 us a
// step; 49 without overlap, 47 so; with three in flight 37, 31 and 30).
// FORM D writes Ds and reads Yin and V only.  VAR: as
// exact::gather_stage (1: the contracted class).
template <typename R, int DIM, Form FORM, int BC, int VAR, int NT>
__global__ void __launch_bounds__(NT)
    pass(Geom g, Consts<R> c, const C2<R>* Yin, C2<R>* Psi, const R* V, C2<R>* K, C2<R>* Yout,
         C2<R>* Ds, int stage, Map m) {
  typedef C2<R> T2;
  const int M = g.M, P = g.P;
  if (blockIdx.x >= m.shell_blocks) {
    const unsigned d = (blockIdx.x - m.shell_blocks) * NT + threadIdx.x;
    if (d >= m.deep) return;
    const unsigned p = deep_index<DIM>(g, m, d);
    pdl_wait();  // the previous kernel's output
    const T2* u = Yin + p;
    if (FORM == WIDE) {
      const T2 y0 = u[0];
      T2 t1 = second(u[1], y0, u[-1]), s2 = add(u[2], u[-2]);
      t1 = add(t1, second(u[M], y0, u[-M]));
      s2 = add(s2, add(u[2 * M], u[-2 * M]));
      if (DIM == 3) {
        t1 = add(t1, second(u[P], y0, u[-P]));
        s2 = add(s2, add(u[2 * P], u[-2 * P]));
      }
      const T2 f0 = rhs_wide<R, DIM>(c, y0, V[p], t1, s2);
      pdl_trigger();
      exact::update<R>(c, stage, p, f0, Psi, K, Yout);
    } else if (FORM == D) {
      const T2 d0 = interior<R, DIM, D>(g, c, u, (R)0, nullptr);
      pdl_trigger();
      Ds[p] = d0;
    } else {
      const T2 f0 = interior<R, DIM, FORM>(g, c, u, V[p], Ds + p);
      pdl_trigger();
      exact::update<R>(c, stage, p, f0, Psi, K, Yout);
    }
    return;
  }
  // a point next to a face
  const unsigned t = blockIdx.x * NT + threadIdx.x;
  if (t >= m.shell) return;
  const int n[3] = {M, g.N, DIM == 3 ? g.L : 3}, s[3] = {1, M, P};
  int q[3];
  shell_point<DIM>(g, m, t, q);
  const int p = (DIM == 3 ? q[2] * P : 0) + q[1] * M + q[0];
  pdl_wait();  // the previous kernel's output
  const T2 yq = Yin[p];
  const R vq = V[p];
  if (FORM == D) {  // and D at the face-interior points beside it
    const T2 dq = interior<R, DIM, D>(g, c, Yin + p, (R)0, nullptr);
    Ds[p] = dq;
#pragma unroll
    for (int a = 0; a < DIM; ++a)
#pragma unroll
      for (int d = -1; d <= 1; d += 2) {
        if (q[a] != (d < 0 ? 1 : n[a] - 2)) continue;
        const int b = p + d * s[a];
        Ds[b] = exact::d_bnd<R, BC>(c, Yin[b], V[b], yq, vq, dq);
      }
    return;
  }
  T2 Fq;
  if (FORM == WIDE) {
    T2 t1 = second(Yin[p + 1], yq, Yin[p - 1]), s2;
#pragma unroll
    for (int a = 1; a < DIM; ++a)
      t1 = add(t1, second(Yin[p + s[a]], yq, Yin[p - s[a]]));
    const T2 dq = {c.lh2 * t1.r, c.lh2 * t1.i};
#pragma unroll
    for (int a = 0; a < DIM; ++a)
#pragma unroll
      for (int d = -1; d <= 1; d += 2) {
        T2 far;
        if (q[a] != (d < 0 ? 1 : n[a] - 2)) {
          far = Yin[p + 2 * d * s[a]];
        } else {  // the ghost beyond the face point b
          const int b = p + d * s[a];
          const T2 yb = Yin[b];
          const T2 db = exact::d_bnd<R, BC>(c, yb, BC == 3 ? (R)0 : V[b], yq, vq, dq);
          T2 st = axpy(yq, (R)-1, yb);
#pragma unroll
          for (int e = 0; e < DIM; ++e)
            if (e != a) st = add(st, second(Yin[b + s[e]], yb, Yin[b - s[e]]));
          far = axpy(axpy(yb, (R)-1, st), c.h2, db);
        }
        s2 = a == 0 && d < 0 ? far : add(s2, far);
      }
    Fq = rhs_wide<R, DIM>(c, yq, vq, t1, s2);
  } else {
    Fq = interior<R, DIM, FORM>(g, c, Yin + p, vq, Ds + p);
  }
  exact::update<R>(c, stage, p, Fq, Psi, K, Yout);
  // the face points whose inward neighbour this is: every nonzero choice of a
  // step to a face per axis
  const int lo[3] = {q[0] == 1 ? -1 : 0, q[1] == 1 ? -1 : 0, DIM == 3 && q[2] == 1 ? -1 : 0};
  const int hi[3] = {q[0] == n[0] - 2, q[1] == n[1] - 2, DIM == 3 && q[2] == n[2] - 2};
#pragma unroll 1
  for (int dz = lo[2]; dz <= hi[2]; ++dz)
#pragma unroll 1
    for (int dy = lo[1]; dy <= hi[1]; ++dy)
#pragma unroll 1
      for (int dx = lo[0]; dx <= hi[0]; ++dx) {
        if (!(dx | dy | dz)) continue;
        const int b = p + dz * P + dy * M + dx;
        const T2 Fb = exact::f_bnd<R, BC>(c, Yin[b], BC == 3 ? V[b] : (R)0, yq, Fq);
        exact::update<R>(c, stage, b, Fb, Psi, K, Yout);
      }
}

template <typename R, int DIM, Form FORM, int VAR, int NT>
cudaError_t by_bc(const Geom& g, int BC, const Consts<R>& c, const ExactStageArgs<R>& a, int stage,
                  cudaStream_t st) {
  const Map m = make_map(g, NT);
  const unsigned blocks = m.shell_blocks + (m.deep + NT - 1) / NT;
  const dim3 gr(blocks), bl(NT);
  const bool pdl = wide::g_pdl != 0;
#define NLSE_POINT(bc)                                                                          \
  case bc:                                                                                      \
    return launch_k(pass<R, DIM, FORM, bc, VAR, NT>, gr, bl, 0, st, pdl, g, c, a.Yin, a.Psi,  \
                    a.V, a.K, a.Yout, a.dsc, stage, m)
  switch (BC) {
    NLSE_POINT(1);
    NLSE_POINT(2);
    NLSE_POINT(3);
  }
#undef NLSE_POINT
  return cudaErrorInvalidValue;
}

template <typename R, int DIM, Form FORM, int VAR>
cudaError_t launch(const Geom& g, int BC, const Consts<R>& c, const ExactStageArgs<R>& a, int stage,
                   cudaStream_t st) {
  if constexpr (sizeof(R) == 8) return by_bc<R, DIM, FORM, VAR, 64>(g, BC, c, a, stage, st);
  else if (g.n < (1LL << 20)) return by_bc<R, DIM, FORM, VAR, 128>(g, BC, c, a, stage, st);
  else return by_bc<R, DIM, FORM, VAR, 256>(g, BC, c, a, stage, st);
}

// A stage in the reference's order: CD, or D and F.
template <typename R, int DIM, int VAR>
cudaError_t launch_ordered(const Geom& g, int method, int BC, const Consts<R>& c,
                           const ExactStageArgs<R>& a, int stage, cudaStream_t st) {
  if (method == 1) return launch<R, DIM, CD, VAR>(g, BC, c, a, stage, st);
  cudaError_t e = launch<R, DIM, D, VAR>(g, BC, c, a, stage, st);
  return e != cudaSuccess ? e : launch<R, DIM, F, VAR>(g, BC, c, a, stage, st);
}

}  // namespace point
}  // namespace nlse
