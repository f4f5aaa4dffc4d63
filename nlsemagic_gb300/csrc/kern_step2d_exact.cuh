// FP32, 2D, CD: a whole RK4 step per launch (the tiling of kern_step2d.cuh).
//
// Stage s is evaluated on the tile and a halo of 4 - s cells.  The state, the
// accumulator and the potential of a thread's R cells stay in registers; two
// shared-memory planes hold the stage input and output in turn.  Every value
// is the same per-point function of the same operands as in the gather
// kernels, in a unit compiled with -fmad=false: the reference's bits.  The
// stage launches pass 36 B per point and stage through L2 or HBM; this passes
// 20 B per step and is bound by instruction issue (1537 x 1203, three solves in
// flight: 14.9 us a step against 52.5).
#pragma once

#include "kern_step2d.cuh"
#include "nlse_exact.cuh"

namespace nlse {
namespace step2d {

template <int XT, int G, int R>
struct ExactShape {
  static constexpr int YT = G * R, NT = XT * G;
  static constexpr int TX = XT - 6, TY = YT - 6;  // largest tile
  static constexpr int SX = XT + 2, SY = YT + 2;  // staged cells
  static constexpr int FACES = 2 * YT + 2 * XT;
  static constexpr int SMEM = (2 * SX * SY + FACES) * (int)sizeof(C2<float>);
};

template <int BC, int XT, int G, int R, bool EDGE>
__device__ __forceinline__ void exact_cd_tile(const Geom& g, const Consts<float>& c,
                                              const C2<float>* in, const float* V,
                                              C2<float>* out, const Tile& t, C2<float>* ya) {
  using namespace exact;
  typedef C2<float> T2;
  typedef ExactShape<XT, G, R> S;
  constexpr int SX = S::SX, SY = S::SY, YT = S::YT, NT = S::NT;
  T2* const yb = ya + SX * SY;
  T2* const fqx = yb + SX * SY;  // F next to the x faces, [side][row]
  T2* const fqy = fqx + 2 * YT;  // and the y faces, [side][column]
  const int M = g.M, N = g.N, x0 = t.x0, y0 = t.y0;
  const int tid = (int)threadIdx.x, lx = tid % XT, l0 = tid / XT * R;
  const int x = x0 + lx;

  // stage the state (a warp per row); cells clamped into the grid are not read
  for (int cy = tid / 32; cy < SY; cy += NT / 32) {
    const unsigned row = (unsigned)min(max(y0 - 1 + cy, 0), N - 1) * M;
#pragma unroll
    for (int cx = tid % 32; cx < SX; cx += 32)
      cp_async<8>(&ya[cy * SX + cx], in + row + min(max(x0 - 1 + cx, 0), M - 1), true);
  }
  float v[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
    v[r] = V[(unsigned)min(max(y0 + l0 + r, 0), N - 1) * M + min(max(x, 0), M - 1)];
  cp_async_wait_all();
  __syncthreads();

  const int w0 = (l0 + 1) * SX + lx + 1;  // own column, first row
  T2 ps[R], K[R];
#pragma unroll
  for (int r = 0; r < R; ++r) ps[r] = ya[w0 + r * SX];

#pragma unroll
  for (int stage = 1; stage <= 4; ++stage) {
    if (stage == 4) pdl_trigger();  // the next kernel may launch; it waits for this one
    const int m = stage - 1;  // margin of this stage's cells
    T2* const yin = stage & 1 ? ya : yb;
    T2* const yout = stage & 1 ? yb : ya;
    const int cx0 = m, cx1 = t.tx1 - x0 + 3 - m, cy0 = m, cy1 = t.ty1 - y0 + 3 - m;
    // exact::update of the thread's row r from F
    auto upd = [&](int r, T2 T) {
      if (stage == 1)
        K[r] = T;
      else if (stage < 4)
        K[r] = T2{K[r].r + 2.0f * T.r, K[r].i + 2.0f * T.i};
      else
        K[r] = T2{K[r].r + 1.0f * T.r, K[r].i + 1.0f * T.i};
      if (stage < 4) {
        const float cf = stage == 3 ? c.k : c.k2;
        yout[w0 + r * SX] = T2{ps[r].r + cf * T.r, ps[r].i + cf * T.i};
      } else {
        const int y = y0 + l0 + r;
        if (x >= t.tx0 && x < t.tx1 && y >= t.ty0 && y < t.ty1)
          out[(unsigned)y * M + x] = T2{ps[r].r + c.k6 * K[r].r, ps[r].i + c.k6 * K[r].i};
      }
    };
    // 1. interior points
    const bool some =
        EDGE ? lx >= cx0 && lx < cx1 && x >= 1 && x <= M - 2 : l0 + R > cy0 && l0 < cy1;
    if (some) {
      T2 dn = yin[w0 - SX], u0 = yin[w0];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int l = l0 + r, y = y0 + l, i = w0 + r * SX;
        const T2 up = yin[i + SX];
        if (!EDGE || (l >= cy0 && l < cy1 && y >= 1 && y <= N - 2)) {
          const T2 T = f_cd_2d<float>(c, u0, v[r], up, dn, yin[i + 1], yin[i - 1]);
          if (BC == 2 && EDGE) {
            if (x == 1) fqx[l] = T;
            if (x == M - 2) fqx[YT + l] = T;
            if (y == 1) fqy[lx] = T;
            if (y == N - 2) fqy[XT + lx] = T;
          }
          upd(r, T);
        }
        dn = u0;
        u0 = up;
      }
    }
    // 2. face points, from their MSD neighbour
    if (EDGE) {
      if (BC == 2) __syncthreads();  // F next to the faces
      if (lx >= cx0 && lx < cx1 && x >= 0 && x < M) {
        const int qx = min(max(x, 1), M - 2);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int l = l0 + r, y = y0 + l;
          if (l < cy0 || l >= cy1 || y < 0 || y >= N) continue;
          const int qy = min(max(y, 1), N - 2);
          if (qx == x && qy == y) continue;
          const T2 ub = yin[w0 + r * SX], uq = yin[(qy - y0 + 1) * SX + qx - x0 + 1];
          T2 fq = {0, 0};
          if (BC == 2) fq = qx != x ? fqx[(x ? YT : 0) + qy - y0] : fqy[(y ? XT : 0) + lx];
          upd(r, f_bnd<float, BC>(c, ub, v[r], uq, fq));
        }
      }
    }
    if (stage < 4) __syncthreads();
  }
}

template <int BC, int XT, int G, int R, int MINB>
__global__ void __launch_bounds__(XT* G, MINB)
    exact_cd_step(Geom g, Consts<float> c, const C2<float>* in, const float* V, C2<float>* out,
                  int nbx, int nby) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2<float>* const sm = reinterpret_cast<C2<float>*>(smem_raw);
  const Tile t = tile_of<1>(g, (int)blockIdx.x, (int)blockIdx.y, nbx, nby);
  pdl_wait();  // the previous kernel's output
  if (at_edge<1>(g, t))
    exact_cd_tile<BC, XT, G, R, true>(g, c, in, V, out, t, sm);
  else
    exact_cd_tile<BC, XT, G, R, false>(g, c, in, V, out, t, sm);
}

template <int BC, int XT, int G, int R, int MINB>
cudaError_t launch_exact_cd(const Geom& g, const Consts<float>& c, const C2<float>* in,
                            const float* V, C2<float>* out, cudaStream_t st, bool pdl) {
  typedef ExactShape<XT, G, R> S;
  const int nbx = (g.M + S::TX - 1) / S::TX, nby = (g.N + S::TY - 1) / S::TY;
  auto k = exact_cd_step<BC, XT, G, R, MINB>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
  if (e != cudaSuccess) return e;
  return launch_k(k, dim3((unsigned)nbx, (unsigned)nby), dim3(S::NT), S::SMEM, st, pdl, g, c, in, V,
                  out, nbx, nby);
}

}  // namespace step2d
}  // namespace nlse
