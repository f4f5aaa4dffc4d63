// Mixed-precision 2D: a whole RK4 step per launch.
//
// A CTA owns a tile and computes all four stages of it from shared memory.
// Stage s is evaluated on the tile and a halo of (4 - s) H cells (H = 2 for
// 2SHOC, 1 for CD), so the halo's points are computed by several CTAs (every
// one to the same bits: the per-point functions and operands are those of the
// stage kernel, kern_wide2d.cuh) and the state crosses HBM once per step
// instead of four times, with one launch instead of four.
//
// Within a step the hi parts do not change, so their share of the Laplacian
// sums (the differences h_n - h_0 of mixed::lapsum, face neighbours and, for
// 2SHOC, the neighbours two cells off) is formed once per step and kept in
// registers; a stage reads only the E plane of its neighbours.  Each thread
// owns R consecutive cells of a column, so that a cell's neighbours along the
// column come from a register window.
//
// Shared memory: hi and two E planes (the first is staged as lo, the E of
// stage 1; a thread's own lo stays in registers).  The ghost
// beyond a face point is its hi (constant) and an E that each stage writes
// into the E plane's cell beyond the face before it is read.
//
// What bounds it: shared-memory reads and FP32 latency (2048^2 2SHOC: 33 B of HBM
// traffic per point and step against 160 B of the stage launches; shared memory at
// 73% of its rate); what both took is beside step2d_shape.
//
// Tiles start at floor(i M / nbx), floor(j N / nby): sizes that differ by one
// cell at most and are at least 2, so a face point and its MSD neighbour are
// in the same tile.
#pragma once

#include "kern_wide2d.cuh"

namespace nlse {
namespace step2d {

enum { SMALL = 1, MIDDLE = 2, LARGE = 3 };  // step2d_shape

// What a step of a grid costs in tiles of tx x ty cells, `cells` evaluated in
// stage 1, in cells of an inner tile: a tile at a face runs the tests of every
// cell and, with MSD, waits for a quotient twice a stage; where the face is one
// lane of each warp (x) more than where it is whole rows (y).  Weights from
// launches of such tiles only (sides of 16 to 128 points by up to 62500).
inline double step_cells(const Geom& g, int BC, int tx, int ty, int cells) {
  const double nbx = (g.M + tx - 1) / tx, nby = (g.N + ty - 1) / ty;
  const double ix = nbx > 2 ? nbx - 2 : 0, iy = nby > 2 ? nby - 2 : 0;
  const double wx = BC == 2 ? 2.6 : 1.65, wy = BC == 2 ? 1.8 : 1.5;
  return cells * ((nbx - ix) * nby * wx + ix * (nby - iy) * wy + ix * iy);
}
// The stage launches' share: a stage of a step in the cells of their tiles, over
// the cost of an inner tile's cell.
inline double stage_cells(const Geom& g, int method, bool single) {
  const double ratio = method == 2 ? 0.30 : (single ? 0.22 : 0.27);
  const int ty = wide2d::pick_ty(g);
  return (double)wide2d::tiles(g, ty) * 32 * ty / ratio;
}

// XT x G threads of R rows: the cells stage 1 is evaluated on.
template <int METHOD, int XT, int G, int R>
struct Shape {
  static constexpr int H = METHOD == 2 ? 2 : 1;
  static constexpr int YT = G * R, NT = XT * G;
  static constexpr int TX = XT - 6 * H, TY = YT - 6 * H;  // largest tile
  static constexpr int SX = XT + 2 * H, SY = YT + 2 * H;  // staged cells
  static constexpr int FACES = 2 * YT + 2 * XT;
  static constexpr int SMEM = (3 * SX * SY + FACES) * (int)sizeof(float2);
};

// Tile of one CTA: its cells, and stage 1's cell (0, 0).
struct Tile {
  int tx0, tx1, ty0, ty1, x0, y0;
};

template <int H>
__device__ __forceinline__ Tile tile_of(const Geom& g, int bx, int by, int nbx, int nby) {
  Tile t;
  t.tx0 = (int)((long long)bx * g.M / nbx);
  t.tx1 = (int)((long long)(bx + 1) * g.M / nbx);
  t.ty0 = (int)((long long)by * g.N / nby);
  t.ty1 = (int)((long long)(by + 1) * g.N / nby);
  t.x0 = t.tx0 - 3 * H;
  t.y0 = t.ty0 - 3 * H;
  return t;
}
// Whether the cells a tile reads (4 H around it) hold face points.
template <int H>
__device__ __forceinline__ bool at_edge(const Geom& g, const Tile& t) {
  return t.tx0 <= 4 * H || t.tx1 + 4 * H >= g.M || t.ty0 <= 4 * H || t.ty1 + 4 * H >= g.N;
}

// EDGE: the staged cells hold face points.  A tile without any evaluates
// every cell of its threads' rows in every stage (rows beyond the stage's
// halo give values nobody reads), which costs fewer instructions than the
// tests that would skip them; only rows that are all beyond it are skipped.
template <int METHOD, int BC, int XT, int G, int R, bool EDGE>
__device__ __forceinline__ void mixed_tile(const Geom& g, const Consts<float>& c,
                                           const float2* hi_in, const float2* lo_in,
                                           const float* V, float2* Kg, float2* hi_out,
                                           float2* lo_out, const Tile& t, float2* sh) {
  using namespace mixed;
  typedef Shape<METHOD, XT, G, R> S;
  constexpr int H = S::H, SX = S::SX, SY = S::SY, YT = S::YT, NT = S::NT;
  float2* const ea = sh + SX * SY;  // lo as staged: the E of stage 1
  float2* const eb = ea + SX * SY;
  float2* const fqx = eb + SX * SY;  // F next to the x faces, [side][row]
  float2* const fqy = fqx + 2 * YT;  // and the y faces, [side][column]
  const int M = g.M, N = g.N, x0 = t.x0, y0 = t.y0;
  const int tid = (int)threadIdx.x, lx = tid % XT, l0 = tid / XT * R;
  const int x = x0 + lx;

  // stage the state (a warp per row); the hi of a ghost is the face point's
  for (int cy = tid / 32; cy < SY; cy += NT / 32) {
    const int gy = y0 - H + cy;
#pragma unroll
    for (int cx = tid % 32; cx < SX; cx += 32) {
      const int gx = x0 - H + cx;
      if (EDGE) {
        const bool in = gx >= 0 && gx < M && gy >= 0 && gy < N;
        const unsigned p = (unsigned)min(max(gy, 0), N - 1) * M + min(max(gx, 0), M - 1);
        cp_async<8>(&sh[cy * SX + cx], hi_in + p, true);
        cp_async<8>(&ea[cy * SX + cx], lo_in + p, in);
      } else {  // a tile narrower than XT - 6 H stages cells it does not read
        const unsigned p = (unsigned)min(gy, N - 1) * M + min(gx, M - 1);
        cp_async<8>(&sh[cy * SX + cx], hi_in + p, true);
        cp_async<8>(&ea[cy * SX + cx], lo_in + p, true);
      }
    }
  }
  float v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int y = y0 + l0 + r;
    if (EDGE)
      v[r] = x >= 0 && x < M && y >= 0 && y < N ? V[(unsigned)y * M + x] : 0.f;
    else
      v[r] = V[(unsigned)min(y, N - 1) * M + min(x, M - 1)];
  }
  // ghost task of this thread (2SHOC, edge tiles): face point b, inward step
  bool gt = false;
  int bx = 0, by = 0, dx = 0, dy = 0;
  float vb = 0.f, vq = 0.f;
  if (METHOD == 2 && EDGE && tid < S::FACES) {
    if (tid < 2 * YT) {
      const int side = tid / YT;
      bx = side == 0 ? 0 : M - 1;
      by = y0 + (tid - side * YT);
      dx = side == 0 ? 1 : -1;
      gt = by >= 1 && by <= N - 2;
    } else {
      const int side = (tid - 2 * YT) / XT;
      by = side == 0 ? 0 : N - 1;
      bx = x0 + (tid - 2 * YT - side * XT);
      dy = side == 0 ? 1 : -1;
      gt = bx >= 1 && bx <= M - 2;
    }
    // its inward neighbour among stage 1's cells (else no stage needs it)
    gt = gt && bx + dx >= x0 && bx + dx < x0 + XT && by + dy >= y0 && by + dy < y0 + YT;
    if (gt && BC != 3) vb = V[(unsigned)by * M + bx];
    if (gt && BC == 2) vq = V[(unsigned)(by + dy) * M + bx + dx];
  }
  cp_async_wait_all();
  __syncthreads();

  const int w0 = (l0 + H) * SX + lx + H;  // own column, first row
  float2 lo[R];
#pragma unroll
  for (int r = 0; r < R; ++r) lo[r] = ea[w0 + r * SX];
  // hi parts of the Laplacian sums
  float2 sf[R], s2[METHOD == 2 ? R : 1];
  {
    float2 w[R + 2 * H];
#pragma unroll
    for (int r = 0; r < R + 2 * H; ++r) w[r] = sh[w0 + (r - H) * SX];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float2* q = sh + w0 + r * SX;
      const float2 c0 = w[r + H];
      float2 d = psub(w[r + H + 1], c0);
      d = padd(d, psub(w[r + H - 1], c0));
      d = padd(d, psub(q[1], c0));
      sf[r] = padd(d, psub(q[-1], c0));
      if (METHOD == 2) {
        d = psub(w[r + H + H], c0);
        d = padd(d, psub(w[r], c0));
        d = padd(d, psub(q[2], c0));
        s2[r] = padd(d, psub(q[-2], c0));
      }
    }
  }

#pragma unroll
  for (int stage = 1; stage <= 4; ++stage) {
    if (stage == 4) pdl_trigger();  // the next kernel may launch; it waits for this one
    const int m = (stage - 1) * H;  // margin of this stage's cells
    float2* const ein = stage & 1 ? ea : eb;
    float2* const eout = stage & 1 ? eb : ea;
    // columns and rows of this stage: the tile and its remaining halo
    const int cx0 = m, cx1 = t.tx1 - x0 + 3 * H - m, cy0 = m, cy1 = t.ty1 - y0 + 3 * H - m;
    // the accumulators that stage 4 ends with, all in flight before its work
    float2 kv[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int y = y0 + l0 + r;
      kv[r] = make_float2(0.f, 0.f);
      if (stage == 4 && x >= t.tx0 && x < t.tx1 && y >= t.ty0 && y < t.ty1)
        kv[r] = Kg[(unsigned)y * M + x];
    }
    auto at = [&](int gx, int gy) -> HE {
      const int i = (gy - y0 + H) * SX + gx - x0 + H;
      HE q;
      q.h = sh[i];
      q.e = ein[i];
      return q;
    };
    // 1. ghosts beyond the face points
    if (METHOD == 2 && EDGE) {
      const int qx = bx + dx, qy = by + dy;
      if (gt && qx - x0 >= cx0 && qx - x0 < cx1 && qy - y0 >= cy0 && qy - y0 < cy1) {
        const HE ub = at(bx, by), uq = at(qx, qy);
        float2 dq = make_float2(0.f, 0.f);
        if (BC == 2) {
          const HE nq[4] = {at(qx, qy + 1), at(qx, qy - 1), at(qx + 1, qy), at(qx - 1, qy)};
          dq = d_interior<2>(c, uq, nq);
        }
        const float2 dbc = d_boundary<BC>(c, ub, vb, uq, vq, dq, nullptr);
        const HE tn[2] = {at(bx + dy, by + dx), at(bx - dy, by - dx)};  // along the face
        const float2 st = lapsum<2>(ub, tn);
        const float2 sq = lapsum<1>(ub, &uq);
        const float2 delta = psub(pmul(P2(c.h2), dbc), padd(sq, st));
        ein[(by - dy - y0 + H) * SX + bx - dx - x0 + H] = padd(ub.e, delta);
      }
      __syncthreads();
    }
    // stage update of the cell in row l from F; h, e, kv its own values
    auto upd = [&](int l, int i, float2 T, float2 h, float2 lo, float2 e, float2 kv) {
      const unsigned p = (unsigned)(y0 + l) * M + x;
      const bool own = x >= t.tx0 && x < t.tx1 && y0 + l >= t.ty0 && y0 + l < t.ty1;
      float2 eo, ko, ho, l2;
      stage_update(c, stage, T, h, lo, e, kv, eo, ko, ho, l2);
      if (stage == 2 && own) Kg[p] = ko;
      if (stage < 4) {
        eout[i] = eo;
      } else if (own) {
        hi_out[p] = ho;
        lo_out[p] = l2;
      }
    };
    // 2. interior points
    const bool some =
        EDGE ? lx >= cx0 && lx < cx1 && x >= 1 && x <= M - 2 : l0 + R > cy0 && l0 < cy1;
    if (some) {
      float2 w[2 * H + 1];  // E of the column, rows l - H .. l + H
#pragma unroll
      for (int k = 0; k < 2 * H; ++k) w[k + 1] = ein[w0 + (k - H) * SX];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int l = l0 + r, y = y0 + l, i = w0 + r * SX;
#pragma unroll
        for (int k = 0; k < 2 * H; ++k) w[k] = w[k + 1];
        w[2 * H] = ein[i + H * SX];
        if (EDGE && (l < cy0 || l >= cy1 || y < 1 || y > N - 2)) continue;
        const float2 e0 = w[H], h0 = sh[i];
        float2 se = padd(padd(padd(w[H + 1], w[H - 1]), ein[i + 1]), ein[i - 1]);
        const float2 s = padd(sf[r], pfma(e0, P2(-4.f), se));
        float2 lin;
        if (METHOD == 1) {
          lin = pmul(P2(c.ah2), s);
        } else {
          se = padd(padd(padd(w[2 * H], w[0]), ein[i + 2]), ein[i - 2]);
          const float2 d = padd(s2[r], pfma(e0, P2(-4.f), se));
          lin = pmul(P2(c.a12lh2), pfma(P2(16.f), s, f2(-d.x, -d.y)));
        }
        const float2 u = padd(h0, e0);
        const float2 T = rhs(lin, nl_term(c, u, v[r]), u);
        if (BC == 2 && EDGE) {
          if (x == 1) fqx[l] = T;
          if (x == M - 2) fqx[YT + l] = T;
          if (y == 1) fqy[lx] = T;
          if (y == N - 2) fqy[XT + lx] = T;
        }
        upd(l, i, T, h0, lo[r], e0, kv[r]);
      }
    }
    // 3. face points, from their MSD neighbour
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
          const HE ub = at(x, y), uq = at(qx, qy);
          float2 fq = make_float2(0.f, 0.f);
          if (BC == 2) fq = qx != x ? fqx[(x ? YT : 0) + qy - y0] : fqy[(y ? XT : 0) + lx];
          const float2 T = f_boundary<METHOD, BC>(c, ub, v[r], uq, fq, nullptr);
          upd(l, w0 + r * SX, T, ub.h, lo[r], ub.e, kv[r]);
        }
      }
    }
    if (stage < 4) __syncthreads();
  }
}

template <int METHOD, int BC, int XT, int G, int R, int MINB>
__global__ void __launch_bounds__(XT* G, MINB)
    mixed_step(Geom g, Consts<float> c, const float2* hi_in, const float2* lo_in, const float* V,
               float2* Kg, float2* hi_out, float2* lo_out, int nbx, int nby) {
  constexpr int H = Shape<METHOD, XT, G, R>::H;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* const sm = reinterpret_cast<float2*>(smem_raw);
  const Tile t = tile_of<H>(g, (int)blockIdx.x, (int)blockIdx.y, nbx, nby);
  pdl_wait();  // the previous kernel's output
  if (at_edge<H>(g, t))
    mixed_tile<METHOD, BC, XT, G, R, true>(g, c, hi_in, lo_in, V, Kg, hi_out, lo_out, t, sm);
  else
    mixed_tile<METHOD, BC, XT, G, R, false>(g, c, hi_in, lo_in, V, Kg, hi_out, lo_out, t, sm);
}

template <int METHOD, int BC, int XT, int G, int R, int MINB>
cudaError_t launch_shape(const Geom& g, const Consts<float>& c, const float2* hi, const float2* lo,
                         const float* V, float2* K, float2* ho, float2* l2, cudaStream_t st,
                         bool pdl) {
  typedef Shape<METHOD, XT, G, R> S;
  const int nbx = (g.M + S::TX - 1) / S::TX, nby = (g.N + S::TY - 1) / S::TY;
  auto k = mixed_step<METHOD, BC, XT, G, R, MINB>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
  if (e != cudaSuccess) return e;
  return launch_k(k, dim3((unsigned)nbx, (unsigned)nby), dim3(S::NT), S::SMEM, st, pdl, g, c, hi, lo,
                  V, K, ho, l2, nbx, nby);
}

}  // namespace step2d
}  // namespace nlse
