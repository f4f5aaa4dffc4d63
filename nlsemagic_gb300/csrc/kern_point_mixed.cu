// 3D stages of the mixed class, a thread per point, one launch per stage
// (small grids; the layout of kern_point.cuh).
//
// The streaming kernels (kern_wide.cuh) take three launches a 2SHOC stage
// (ghosts, interior, faces) and one CTA per 32 x 8 column and z chunk, few on a
// small grid; without 16-byte rows they stage planes by plain loads.  Here the
// neighbours are read through L1 and a point next to a face forms its ghosts,
// its F and then its face points, with the same per-point functions of the same
// operands: the same bits.  The next launch (PDL) is not triggered before a block
// ends (32^3 2SHOC, one solve: 29 us a step when triggered at the start, 21 so).
#include "kern_point.cuh"
#include "kern_wide.cuh"

namespace nlse {
namespace point {

constexpr int MIXED_NT = 128;

template <int METHOD, int BC>
__global__ void __launch_bounds__(MIXED_NT)
    mixed3d(Geom g, Consts<float> c, MixedStageArgs a, int stage, Map m) {
  using namespace mixed;
  const int M = g.M, P = g.P;
  const YIn Y{a.hi_in, stage == 1 ? a.lo_in : a.e_in};
  // stage update of point p from F; u its own (hi, E)
  auto upd = [&](unsigned p, float2 T, const HE& u) {
    const float2 lo = stage == 1 ? u.e : a.lo_in[p];
    const float2 kv = stage == 4 ? a.K[p] : lo;
    float2 eo, ko, ho, l2;
    stage_update(c, stage, T, u.h, lo, u.e, kv, eo, ko, ho, l2);
    if (stage == 2) a.K[p] = ko;
    if (stage < 4) {
      a.e_out[p] = eo;
    } else {
      a.hi_out[p] = ho;
      a.lo_out[p] = l2;
    }
  };
  if (blockIdx.x >= m.shell_blocks) {
    const unsigned d = (blockIdx.x - m.shell_blocks) * MIXED_NT + threadIdx.x;
    if (d >= m.deep) return;
    const unsigned p = deep_index<3>(g, m, d);
    pdl_wait();  // the previous kernel's output
    const HE u0 = Y.at(p);
    const HE fn[6] = {Y.at(p + P), Y.at(p - P), Y.at(p + M),
                      Y.at(p - M), Y.at(p + 1), Y.at(p - 1)};
    float2 T;
    if (METHOD == 1) {
      T = f_interior_cd<3>(c, u0, a.V[p], fn);
    } else {
      const HE f2n[6] = {Y.at(p + 2 * P), Y.at(p - 2 * P), Y.at(p + 2 * M),
                         Y.at(p - 2 * M), Y.at(p + 2),     Y.at(p - 2)};
      T = f_wide_2shoc<3>(c, u0, a.V[p], fn, f2n);
    }
    upd(p, T, u0);
    return;
  }
  // a point next to a face
  const unsigned t = blockIdx.x * MIXED_NT + threadIdx.x;
  if (t >= m.shell) return;
  const int n[3] = {M, g.N, g.L}, s[3] = {1, M, P};
  int q[3];
  shell_point<3>(g, m, t, q);
  const int p = q[2] * P + q[1] * M + q[0];
  pdl_wait();  // the previous kernel's output
  const HE uq = Y.at(p);
  const float vq = a.V[p];
  const HE nq[6] = {Y.at(p + P), Y.at(p - P), Y.at(p + M), Y.at(p - M), Y.at(p + 1), Y.at(p - 1)};
  float2 T;
  if (METHOD == 1) {
    T = f_interior_cd<3>(c, uq, vq, nq);
  } else {
    HE far[6];  // z+, z-, y+, y-, x+, x-
    unsigned ghosts = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const int ax = 2 - i / 2, d = i % 2 ? -1 : 1;
      if (q[ax] != (d < 0 ? 1 : n[ax] - 2))
        far[i] = Y.at(p + 2 * d * s[ax]);
      else
        ghosts |= 1u << i;
    }
    // the ghost beyond face point b (wide::ghost_value), one copy of the code;
    // in-face neighbours in its order: y, z for an x face, else x and the
    // other axis
#pragma unroll 1
    for (; ghosts; ghosts &= ghosts - 1) {
      const int i = __ffs(ghosts) - 1, ax = 2 - i / 2;
      const int sa = ax == 2 ? P : (ax == 1 ? M : 1);
      const int b = p + (i % 2 ? -sa : sa), t1 = ax == 0 ? M : 1, t2 = ax == 2 ? M : P;
      const HE ub = Y.at(b);
      const HE tn[4] = {Y.at(b + t1), Y.at(b - t1), Y.at(b + t2), Y.at(b - t2)};
      const float4 gv = wide::ghost_value<BC>(c, ub, a.V[b], uq, vq, nq, tn);
#pragma unroll
      for (int k = 0; k < 6; ++k)
        if (ghosts & -ghosts & (1u << k)) {
          far[k].h = make_float2(gv.x, gv.y);
          far[k].e = make_float2(gv.z, gv.w);
        }
    }
    T = f_wide_2shoc<3>(c, uq, vq, nq, far);
  }
  upd((unsigned)p, T, uq);
  // the face points whose inward neighbour this is
  const int lo[3] = {q[0] == 1 ? -1 : 0, q[1] == 1 ? -1 : 0, q[2] == 1 ? -1 : 0};
  const int hi[3] = {q[0] == n[0] - 2, q[1] == n[1] - 2, q[2] == n[2] - 2};
#pragma unroll 1
  for (int dz = lo[2]; dz <= hi[2]; ++dz)
#pragma unroll 1
    for (int dy = lo[1]; dy <= hi[1]; ++dy)
#pragma unroll 1
      for (int dx = lo[0]; dx <= hi[0]; ++dx) {
        if (!(dx | dy | dz)) continue;
        const int b = p + dz * P + dy * M + dx;
        const HE ub = Y.at(b);
        upd((unsigned)b, f_boundary<METHOD, BC>(c, ub, a.V[b], uq, T, nullptr), ub);
      }
}

}  // namespace point

cudaError_t launch_point_mixed(const Geom& g, int method, int BC, const Consts<float>& c,
                               const MixedStageArgs& a, int stage, cudaStream_t st) {
  using namespace point;
  const Map m = make_map(g, MIXED_NT);
  const dim3 grid(m.shell_blocks + (m.deep + MIXED_NT - 1) / MIXED_NT), block(MIXED_NT);
  const bool pdl = wide::g_pdl != 0;
#define NLSE_POINT(bc)                                                                         \
  case bc:                                                                                     \
    return method == 2 ? launch_k(mixed3d<2, bc>, grid, block, 0, st, pdl, g, c, a, stage, m)  \
                       : launch_k(mixed3d<1, bc>, grid, block, 0, st, pdl, g, c, a, stage, m)
  switch (BC) {
    NLSE_POINT(1);
    NLSE_POINT(2);
    NLSE_POINT(3);
  }
#undef NLSE_POINT
  return cudaErrorInvalidValue;
}

}  // namespace nlse
