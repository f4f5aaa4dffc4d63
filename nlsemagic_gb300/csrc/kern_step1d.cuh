// 1D RK4 steps in registers: several whole steps of a run per launch.
//
// A warp owns a window of W = 32 R consecutive points, R per lane, and keeps
// everything a point needs (state, stage input, accumulator, potential) in
// registers.  Neighbours across lanes come by shuffles, so a stage has no
// barrier, no shared memory and no memory traffic.  The window's ends have no
// neighbours: each stage loses H points per side (H = 1 for CD, 2 for 2SHOC),
// so m steps lose 4 H m and the warp stores only the middle U = W - 8 H m
// points; windows overlap by what is lost.  A grid of at most W points is one
// window that loses nothing.  Every point's value is the same per-point
// function of the same operands as in the gather kernels (kern_gather.cuh) in
// the same order, so the results are the same bits however often a point is
// computed.
//
// What bounds it: FP32 (FP64) issue; on small grids one window's chain of
// dependent instructions, the MSD quotient of its end above all.  The stage
// launches this replaces (kern_seg1d.cuh, kern_gather.cuh) pass the state
// through L2 or HBM 4 times a step and pay a launch for each pass.  10^6
// points, mixed CD MSD: 5.4 us a step (184 Gpt-steps/s) against 26.9; what
// both sides took on other sizes is beside step1d_shape.
//
// The ends of the grid: a window that holds one evaluates its boundary
// formula in every lane on broadcast operands (the end point and its inward
// neighbours lie at warp-uniform positions) and the owner keeps the value, so
// there is one copy of that code per pass and no divergence in it.  One copy
// per slot did not fit the instruction cache (2SHOC MSD on 1024 points, R = 8:
// 13 us a step).
//
// The next launch (PDL) is triggered when a window is done, not at the start: its
// blocks are then placed as this one's end, which hides its latency.  Placed at
// the start they load the SMs unevenly (FP64 CD on 48611 points, one solve: 49 us a
// step; 16.5 without overlap, 15.1 so).
//
// Slots outside the grid hold zeros; nothing inside reads them.  The state is
// read from one buffer and written to another (neighbouring windows still
// read the old one).
#pragma once

#include "kern_gather.cuh"
#include "nlse_launch.h"
#include "nlse_pdl.cuh"

namespace nlse {
namespace step1d {

constexpr int MAX_WARPS = 4;  // per block; warps are independent of each other

struct Plan {
  int m, lost, U;  // steps, window points left of the stored ones, stored points
  unsigned blocks, warps;  // warps per block
};

// Windows of m steps over n points, R per lane.
__host__ __device__ inline Plan make_plan(long long n, int method, int R, int m, int warps) {
  Plan p;
  p.m = m;
  p.lost = n <= 32 * R ? 0 : 4 * (method == 2 ? 2 : 1) * m;
  p.U = 32 * R - 2 * p.lost;
  // The formula of end point n-1 reads up to two points further in than an
  // interior point's does (F at its MSD neighbour; the one-sided difference):
  // where the last window would store one or two points, all windows keep two
  // more on the left.
  if (p.lost && (n % p.U == 1 || n % p.U == 2)) {
    p.lost += 2;
    p.U -= 2;
  }
  const long long windows = (n + p.U - 1) / p.U;
  p.warps = (unsigned)warps;
  p.blocks = (unsigned)((windows + warps - 1) / warps);
  return p;
}

__device__ __forceinline__ float2 shfl(float2 v, int lane) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}
template <typename F>
__device__ __forceinline__ C2<F> shfl(C2<F> v, int lane) {
  return {__shfl_sync(0xffffffffu, v.r, lane), __shfl_sync(0xffffffffu, v.i, lane)};
}
template <typename F>
__device__ __forceinline__ F shfl(F v, int lane) {
  return __shfl_sync(0xffffffffu, v, lane);
}
__device__ __forceinline__ float2 up(float2 v) {  // the lane below's value
  return make_float2(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1));
}
__device__ __forceinline__ float2 dn(float2 v) {  // the lane above's value
  return make_float2(__shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1));
}
template <typename F>
__device__ __forceinline__ C2<F> up(C2<F> v) {
  return {__shfl_up_sync(0xffffffffu, v.r, 1), __shfl_up_sync(0xffffffffu, v.i, 1)};
}
template <typename F>
__device__ __forceinline__ C2<F> dn(C2<F> v) {
  return {__shfl_down_sync(0xffffffffu, v.r, 1), __shfl_down_sync(0xffffffffu, v.i, 1)};
}

// The slot of window position pos as a one-bit mask.  Opaque to the compiler,
// which otherwise recognises the selections below as indexing and puts the
// arrays in local memory (4x slower on every window).
template <int R>
__device__ __forceinline__ unsigned slot_bit(int pos) {
  unsigned b = 1u << (pos % R);
  asm("" : "+r"(b));
  return b;
}
// The value at window position pos (warp-uniform), in every lane; and its
// replacement.
template <int R, typename T>
__device__ __forceinline__ T get(const T (&a)[R], int pos) {
  const unsigned bit = slot_bit<R>(pos);
  T q = a[0];
#pragma unroll
  for (int r = 1; r < R; ++r)
    if (bit & (1u << r)) q = a[r];
  return shfl(q, pos / R);
}
template <int R, typename T>
__device__ __forceinline__ void put(T (&a)[R], int pos, int lane, T v) {
  const unsigned bit = lane == pos / R ? slot_bit<R>(pos) : 0u;
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (bit & (1u << r)) a[r] = v;
}

// ---- mixed class --------------------------------------------------------------
// The hi parts do not change within a step: their share of the Laplacian,
// (h+ - h0) + (h- - h0), is formed once per step (mixed::lapsum, split).
// One window, by the calling warp; first: the first point it stores.
template <int METHOD, int BC, int R>
__device__ __forceinline__ void mixed_window(int n, const Consts<float>& c, const float2* hi_in,
                                             const float2* lo_in, const float* V, float2* hi_out,
                                             float2* lo_out, const Plan& pl, int first) {
  using namespace mixed;
  constexpr int W = 32 * R;
  const int lane = (int)(threadIdx.x & 31);
  const int x0 = first - pl.lost, x = x0 + lane * R;
  const bool ends = x0 <= 0 || x0 + W >= n;  // an end of the grid in the window
  float2 hi[R], lo[R], e[R], sh[R], K[R], T[R];
  float v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const bool in = x + r >= 0 && x + r < n;
    hi[r] = in ? hi_in[x + r] : make_float2(0.f, 0.f);
    lo[r] = in ? lo_in[x + r] : make_float2(0.f, 0.f);
    v[r] = in ? V[x + r] : 0.f;
    K[r] = make_float2(0.f, 0.f);
  }
  auto he = [&](int pos) -> HE {
    HE q;
    q.h = get<R>(hi, pos);
    q.e = get<R>(e, pos);
    return q;
  };
  // f(position of an end point, inward step) for each end in the window
  auto at_ends = [&](auto f) {
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      const int b = side ? n - 1 - x0 : -x0;
      if (b >= 0 && b < W) f(b, side ? -1 : 1);
    }
  };
  for (int s = 0; s < pl.m; ++s) {
    {
      const float2 hm = up(hi[R - 1]), hp = dn(hi[0]);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        sh[r] = padd(psub(r + 1 < R ? hi[r + 1] : hp, hi[r]), psub(r ? hi[r - 1] : hm, hi[r]));
        e[r] = lo[r];
      }
    }
#pragma unroll
    for (int stage = 1; stage <= 4; ++stage) {
      const float2 em = up(e[R - 1]), ep = dn(e[0]);
#pragma unroll
      for (int r = 0; r < R; ++r) {  // a/h2 times the Laplacian sum, or D
        const float2 se = padd(r + 1 < R ? e[r + 1] : ep, r ? e[r - 1] : em);
        T[r] = pmul(P2(METHOD == 1 ? c.ah2 : c.lh2), padd(sh[r], pfma(e[r], P2(-2.f), se)));
      }
      if (METHOD == 2) {
        if (ends)
          at_ends([&](int b, int d) {
            HE os[4] = {he(b), he(b + d)};
            if (BC == 4) os[2] = he(b + 2 * d), os[3] = he(b + 3 * d);
            put<R>(T, b, lane, d_boundary<BC>(c, os[0], get<R>(v, b), os[1], get<R>(v, b + d),
                                              get<R>(T, b + d), os));
          });
        const float2 dm = up(T[R - 1]), dp = dn(T[0]);
        float2 prev = dm;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float2 d0 = T[r];
          T[r] = pfma(P2(c.a76), d0, pmul(P2(-c.a112), padd(r + 1 < R ? T[r + 1] : dp, prev)));
          prev = d0;
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float2 y = padd(hi[r], e[r]);
        T[r] = rhs(T[r], nl_term(c, y, v[r]), y);
      }
      if (ends)
        at_ends([&](int b, int d) {
          HE os[4] = {he(b), he(b + d)};
          if (BC == 4) os[2] = he(b + 2 * d), os[3] = he(b + 3 * d);
          put<R>(T, b, lane, f_boundary<METHOD, BC>(c, os[0], get<R>(v, b), os[1],
                                                    get<R>(T, b + d), os));
        });
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float2 eo, Ko, ho, l2;
        if (stage == 1) {
          stage_update(c, 1, T[r], hi[r], lo[r], e[r], K[r], e[r], Ko, ho, l2);
        } else if (stage == 2) {
          stage_update(c, 2, T[r], hi[r], lo[r], e[r], K[r], eo, Ko, ho, l2);
          e[r] = eo;
          K[r] = Ko;
        } else if (stage == 3) {
          stage_update(c, 3, T[r], hi[r], lo[r], e[r], K[r], e[r], Ko, ho, l2);
        } else {
          stage_update(c, 4, T[r], hi[r], lo[r], e[r], K[r], eo, Ko, ho, l2);
          hi[r] = ho;
          lo[r] = l2;
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = lane * R + r;
    if (i >= pl.lost && i < pl.lost + pl.U && x + r < n) {
      hi_out[x + r] = hi[r];
      lo_out[x + r] = lo[r];
    }
  }
}

template <int METHOD, int BC, int R>
__global__ void __launch_bounds__(32 * MAX_WARPS)
    mixed_steps(int n, Consts<float> c, const float2* hi_in, const float2* lo_in, const float* V,
                float2* hi_out, float2* lo_out, Plan pl) {
  const int first = (int)(blockIdx.x * pl.warps + (threadIdx.x >> 5)) * pl.U;
  if (first >= n) return;
  pdl_wait();  // the previous kernel's output
  mixed_window<METHOD, BC, R>(n, c, hi_in, lo_in, V, hi_out, lo_out, pl, first);
}

// ---- exact classes (FP64 / FP32) ---------------------------------------------
// VAR: as exact::gather_stage (contracted copy of the FP64 class)
template <typename F, int METHOD, int BC, int R, int VAR>
__global__ void __launch_bounds__(32 * MAX_WARPS)
    exact_steps(int n, Consts<F> c, const C2<F>* psi_in, const F* V, C2<F>* psi_out, Plan pl) {
  using namespace exact;
  typedef C2<F> T2;
  constexpr int W = 32 * R;
  const int lane = (int)(threadIdx.x & 31);
  const int first = (int)(blockIdx.x * pl.warps + (threadIdx.x >> 5)) * pl.U;
  if (first >= n) return;
  const int x0 = first - pl.lost, x = x0 + lane * R;
  const bool ends = x0 <= 0 || x0 + W >= n;  // an end of the grid in the window
  pdl_wait();  // the previous kernel's output
  T2 ps[R], y[R], K[R], T[R];
  F v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const bool in = x + r >= 0 && x + r < n;
    ps[r] = in ? psi_in[x + r] : T2{0, 0};
    v[r] = in ? V[x + r] : (F)0;
    K[r] = T2{0, 0};
  }
  // f(position of an end point, inward step) for each end in the window
  auto at_ends = [&](auto f) {
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      const int b = side ? n - 1 - x0 : -x0;
      if (b >= 0 && b < W) f(b, side ? -1 : 1);
    }
  };
  for (int s = 0; s < pl.m; ++s) {
#pragma unroll
    for (int r = 0; r < R; ++r) y[r] = ps[r];
#pragma unroll
    for (int stage = 1; stage <= 4; ++stage) {
      const T2 ym = up(y[R - 1]), yp = dn(y[0]);
      if (METHOD == 1) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          T[r] = f_cd_1d<F>(c, y[r], v[r], r + 1 < R ? y[r + 1] : yp, r ? y[r - 1] : ym);
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r)
          T[r] = d_int_1d<F>(c, r + 1 < R ? y[r + 1] : yp, y[r], r ? y[r - 1] : ym);
        if (ends)
          at_ends([&](int b, int d) {
            if constexpr (BC == 4)
              put<R>(T, b, lane,
                     d_onesided<F>(c, get<R>(y, b + 3 * d), get<R>(y, b + 2 * d),
                                   get<R>(y, b + d), get<R>(y, b)));
            else
              put<R>(T, b, lane, d_bnd<F, BC>(c, get<R>(y, b), get<R>(v, b), get<R>(y, b + d),
                                              get<R>(v, b + d), get<R>(T, b + d)));
          });
        const T2 dm = up(T[R - 1]), dp = dn(T[0]);
        T2 prev = dm;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const T2 d0 = T[r];
          T[r] = f_2shoc_1d<F>(c, y[r], v[r], d0, r + 1 < R ? T[r + 1] : dp, prev);
          prev = d0;
        }
      }
      if (ends)
        at_ends([&](int b, int d) {
          if constexpr (BC == 4)
            put<R>(T, b, lane,
                   f_onesided<F, METHOD>(c, get<R>(y, b), get<R>(v, b), get<R>(y, b + 3 * d),
                                         get<R>(y, b + 2 * d), get<R>(y, b + d), get<R>(y, b)));
          else
            put<R>(T, b, lane, f_bnd<F, BC>(c, get<R>(y, b), get<R>(v, b), get<R>(y, b + d),
                                            get<R>(T, b + d)));
        });
      // exact::update, in registers
      if (stage == 1) {
#pragma unroll
        for (int r = 0; r < R; ++r) K[r] = T[r];
      } else {
        const F w = stage == 4 ? (F)1.0 : (F)2.0;
#pragma unroll
        for (int r = 0; r < R; ++r) K[r] = T2{K[r].r + w * T[r].r, K[r].i + w * T[r].i};
      }
      if (stage < 4) {
        const F cf = stage == 3 ? c.k : c.k2;
#pragma unroll
        for (int r = 0; r < R; ++r) y[r] = T2{ps[r].r + cf * T[r].r, ps[r].i + cf * T[r].i};
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r)
          ps[r] = T2{ps[r].r + c.k6 * K[r].r, ps[r].i + c.k6 * K[r].i};
      }
    }
  }
  pdl_trigger();  // the next kernel may launch; it waits for this one
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = lane * R + r;
    if (i >= pl.lost && i < pl.lost + pl.U && x + r < n) psi_out[x + r] = ps[r];
  }
}

template <typename F, int METHOD, int R, int VAR>
cudaError_t exact_by_bc(const Geom& g, int BC, const Consts<F>& c, const C2<F>* in, const F* V,
                        C2<F>* out, int m, int warps, cudaStream_t st, bool pdl) {
  const Plan p = make_plan(g.n, METHOD, R, m, warps);
  const dim3 gr(p.blocks), bl(32 * p.warps);
  const int n = (int)g.n;
  switch (BC) {
    case 1: return launch_k(exact_steps<F, METHOD, 1, R, VAR>, gr, bl, 0, st, pdl, n, c, in, V, out, p);
    case 2: return launch_k(exact_steps<F, METHOD, 2, R, VAR>, gr, bl, 0, st, pdl, n, c, in, V, out, p);
    case 3: return launch_k(exact_steps<F, METHOD, 3, R, VAR>, gr, bl, 0, st, pdl, n, c, in, V, out, p);
    case 4: return launch_k(exact_steps<F, METHOD, 4, R, VAR>, gr, bl, 0, st, pdl, n, c, in, V, out, p);
  }
  return cudaErrorInvalidValue;
}

template <typename F, int VAR>
cudaError_t launch_exact(const Geom& g, int method, int BC, const Consts<F>& c, const C2<F>* in,
                         const F* V, C2<F>* out, const Step1dShape& sh, int m, cudaStream_t st) {
#define NLSE_STEP1D(R)                                                                     \
  return method == 2 ? exact_by_bc<F, 2, R, VAR>(g, BC, c, in, V, out, m, sh.warps, st, wide::g_pdl != 0) \
                     : exact_by_bc<F, 1, R, VAR>(g, BC, c, in, V, out, m, sh.warps, st, wide::g_pdl != 0)
  switch (sh.per_lane) {
    case 1: NLSE_STEP1D(1);
    case 2: NLSE_STEP1D(2);
    case 4: NLSE_STEP1D(4);
  }
#undef NLSE_STEP1D
  return cudaErrorInvalidValue;
}

}  // namespace step1d
}  // namespace nlse
