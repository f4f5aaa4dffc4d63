// The batched launch of mixed 1D and 2D solves: whole RK4 steps per task.
//
// A task is one tile of one round of one solve: a 2D tile's RK4 step
// (kern_step2d.cuh) or 16 windows of a 1D solve's next steps in registers
// (kern_step1d.cuh), so a step of a solve is one pass over its tiles where the
// stage passes of the general kernel (batch_kern.cuh) are four.  Tasks are
// numbered round by round; CTAs claim them in that order from one counter.
// Before a task of a later round a CTA waits until its solve's tiles of the round
// before are all done (a counter per solve): no barrier over the grid, and the
// solves' rounds overlap.  Every task waited for has a smaller number, so the
// CTA that holds it is running and waits, if at all, for smaller ones still: the
// wait ends whatever CTAs are resident.  It is bounded all the same
// (NLSE_ERR_TIMEOUT in the error word, every CTA returns).
//
// The same per-point functions as the single-solve kernels: the same bits.
//
// Gpt-steps/s of the uneven batch's first 512 / 128 / 24 / 6 solves, the general
// kernel's stage passes (25.1 / 20.8 / 12.2 / 8.6) and this one with CTAs of
//   64 x 8 threads, two per SM (64 registers)    27.1 / 29.1 / 28.2 / 17.9
//   64 x 8, one per SM (128 registers)           19.2 / 20.4 / 23.0 / 19.6
//   32 x 8, three or four per SM                 21.7 / 23.5 / 27.4 / 20.4
// What bounds it: the edge tiles, most of a small solve's, whose MSD quotients
// follow one another in every stage.
#include "batch_kern.cuh"
#include "kern_step1d.cuh"
#include "kern_step2d.cuh"

namespace {

constexpr int ST = 512;                 // threads per CTA, two CTAs per SM
constexpr int XT = 64, GT = 8, RT = 4;  // 2D: threads by rows (ST = XT GT)
constexpr int R1 = 4, WARPS1 = ST / 32;      // 1D: points per lane, windows per tile
typedef step2d::Shape<1, XT, GT, RT> Shape1;
typedef step2d::Shape<2, XT, GT, RT> Shape2;
constexpr int SMEM = Shape1::SMEM > Shape2::SMEM ? Shape1::SMEM : Shape2::SMEM;

__host__ __device__ inline int tiles_x(int M, int method) {
  const int w = method == 1 ? Shape1::TX : Shape2::TX;
  return (M + w - 1) / w;
}
__host__ __device__ inline int tiles_y(int N, int method) {
  const int h = method == 1 ? Shape1::TY : Shape2::TY;
  return (N + h - 1) / h;
}
// Steps of a 1D solve per round, whatever its size: what single solves of 2^15 to 3
// 2^15 (CD) and 2^13 to 2^16 points (2SHOC) take, between fewer waits and less halo.
__host__ __device__ inline int round_steps(const BSolve& d) {
  return d.g.ndim == 2 ? 1 : (d.method == 1 ? 6 : 4);
}

template <int METHOD, int BC>
__device__ __noinline__ void step_2d(const BSolve& s, int par, int t, float2* sm) {
  constexpr int H = Shape1::H * METHOD;
  const int nbx = tiles_x(s.g.M, METHOD), nby = tiles_y(s.g.N, METHOD);
  const step2d::Tile tl = step2d::tile_of<H>(s.g, t % nbx, t / nbx, nbx, nby);
  const float2 *hi = (const float2*)s.buf[par], *lo = (const float2*)s.buf[2 + par];
  float2 *ho = (float2*)s.buf[1 - par], *l2 = (float2*)s.buf[3 - par], *K = (float2*)s.buf[4];
  const float* V = (const float*)s.buf[7];
  if (step2d::at_edge<H>(s.g, tl))
    step2d::mixed_tile<METHOD, BC, XT, GT, RT, true>(s.g, s.cf, hi, lo, V, K, ho, l2, tl, sm);
  else
    step2d::mixed_tile<METHOD, BC, XT, GT, RT, false>(s.g, s.cf, hi, lo, V, K, ho, l2, tl, sm);
}

template <int METHOD, int BC>
__device__ __noinline__ void steps_1d(const BSolve& s, int par, int t, int m) {
  const step1d::Plan pl = step1d::make_plan(s.g.n, METHOD, R1, m, WARPS1);
  // windows of a shorter last round store more: the tiles cover them with room
  const long long first = ((long long)t * WARPS1 + (threadIdx.x >> 5)) * pl.U;
  if (first >= s.g.n) return;
  step1d::mixed_window<METHOD, BC, R1>(
      (int)s.g.n, s.cf, (const float2*)s.buf[par], (const float2*)s.buf[2 + par],
      (const float*)s.buf[7], (float2*)s.buf[1 - par], (float2*)s.buf[3 - par], pl, (int)first);
}

template <int METHOD>
__device__ void run_tile(const BSolve& s, int par, int t, int m, float2* sm) {
  if (s.g.ndim == 1) {
    switch (s.bc) {
      case 1: steps_1d<METHOD, 1>(s, par, t, m); break;
      case 2: steps_1d<METHOD, 2>(s, par, t, m); break;
      case 3: steps_1d<METHOD, 3>(s, par, t, m); break;
      default: steps_1d<METHOD, 4>(s, par, t, m); break;
    }
  } else {
    switch (s.bc) {
      case 1: step_2d<METHOD, 1>(s, par, t, sm); break;
      case 2: step_2d<METHOD, 2>(s, par, t, sm); break;
      default: step_2d<METHOD, 3>(s, par, t, sm); break;
    }
  }
}

// done[solve]: tiles of that solve finished so far; tile_n[solve]: tiles a round.
__global__ void __launch_bounds__(ST, 2)
    batch_steps(const BSolve* __restrict__ solves, const BTile* __restrict__ tiles, int ntiles,
                const int* __restrict__ tile_n, int max_steps, long long tasks,
                unsigned long long* queue, unsigned long long* done, int* err,
                long long budget) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ BSolve s;
  __shared__ int s_solve, s_ok;  // the solve whose descriptor s holds
  __shared__ long long s_task[2];  // this task and the next one claimed
  if (threadIdx.x == 0) {
    s_solve = -1;
    s_ok = 1;
    s_task[0] = (long long)atomicAdd(queue, 1ull);
  }
  __syncthreads();
  for (int it = 0;; ++it) {
    const long long task = s_task[it & 1];
    if (task >= tasks) return;
    // claim the next task now; it is stored when this one is done
    unsigned long long nx = 0;
    if (threadIdx.x == 0) nx = atomicAdd(queue, 1ull);
    const long long round = task / ntiles;
    const BTile tl = tiles[task - round * ntiles];
    if (tl.solve != s_solve) {
      __syncthreads();  // every thread has compared s_solve
      const int* src = reinterpret_cast<const int*>(&solves[tl.solve]);
      int* dst = reinterpret_cast<int*>(&s);
      for (int w = threadIdx.x; w < (int)(sizeof(BSolve) / sizeof(int)); w += blockDim.x)
        dst[w] = src[w];
      if (threadIdx.x == 0) s_solve = tl.solve;
      __syncthreads();
    }
    const int per = round_steps(s);
    const long long most = s.steps_left < max_steps ? s.steps_left : max_steps;
    const long long left = most - round * per;
    if (left > 0) {
      if (threadIdx.x == 0 && round > 0) {
        const unsigned long long want = (unsigned long long)round * tile_n[tl.solve];
        volatile unsigned long long* d = done + tl.solve;
        const long long t0 = clock64();
        while (*d < want) {
          if (*(volatile int*)err) {
            s_ok = 0;
            break;
          }
          if (clock64() - t0 > budget) {
            atomicExch(err, NLSE_ERR_TIMEOUT);
            s_ok = 0;
            break;
          }
          __nanosleep(32);
        }
        __threadfence();
      }
      __syncthreads();
      if (!s_ok) return;
      const int par = s.cur ^ (int)(round & 1), m = left < per ? (int)left : per;
      if (s.method == 1)
        run_tile<1>(s, par, (int)tl.start, m, reinterpret_cast<float2*>(smem));
      else
        run_tile<2>(s, par, (int)tl.start, m, reinterpret_cast<float2*>(smem));
      __syncthreads();  // the tile is written
      if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(done + tl.solve, 1ull);
      }
    }
    if (threadIdx.x == 0) s_task[(it + 1) & 1] = (long long)nx;
    __syncthreads();
  }
}

}  // namespace

namespace nlse {

// Solves this launch takes, and their tiles a round and rounds for adv steps.
bool batch_steps_takes(const nlse_problem& p) {
  return p.precision == NLSE_PREC_MIXED && (p.ndim == 1 || (p.ndim == 2 && p.bc <= 3));
}
long long batch_steps_tiles(const void* solve) {
  const BSolve& d = *(const BSolve*)solve;
  if (d.g.ndim == 2)
    return (long long)tiles_x(d.g.M, d.method) * tiles_y(d.g.N, d.method);
  const step1d::Plan pl = step1d::make_plan(d.g.n, d.method, R1, round_steps(d), WARPS1);
  return pl.blocks;
}
// Estimated time of a step of a solve, nanoseconds of the whole chip, in this launch
// and by stage passes on segments and rectangles (batch_kern.cuh), whose four grid
// barriers cost batch_barriers_time whatever the solves.  Measured and (estimated),
// microseconds a step of 24 solves, by stage passes / here:
//   8 x 8000 MSD    CD 262 (274) / 353 (394)   2SHOC 314 (328) / 580 (665)
//   3 x 9000        CD 211 (230) / 286 (281)   2SHOC 248 (277) / 475 (474)
//   64 x 1500 MSD   CD 121 (128) / 152 (148)   2SHOC 153 (148) / 240 (249)
//   128 x 700 MSD   CD 112 (122) /  91 (88)    2SHOC 139 (141) / 143 (140)
//   300 x 300 MSD   CD 114 (134) /  69 (57)    2SHOC 133 (155) / 103 (92)
double batch_steps_time(const void* solve) {
  const BSolve& d = *(const BSolve*)solve;
  const bool cd = d.method == 1;
  if (d.g.ndim == 1) return d.g.n * (cd ? 6e-3 : 9e-3);
  return step2d::step_cells(d.g, d.bc, cd ? Shape1::TX : Shape2::TX, cd ? Shape1::TY : Shape2::TY,
                            XT * GT * RT) *
         (cd ? 10e-3 : 13e-3);
}
double batch_stages_time(const void* solve) {
  const BSolve& d = *(const BSolve*)solve;
  const bool cd = d.method == 1;
  if (d.g.ndim == 1) return d.g.n * 28e-3;
  return wide2d::tiles(d.g, W2_TY) * (d.bc == 2 ? (cd ? 39.0 : 48.0) : (cd ? 28.0 : 35.0));
}
double batch_barriers_time() { return 40000.0; }

long long batch_steps_rounds(const void* solve, long long adv) {
  const int per = round_steps(*(const BSolve*)solve);
  return (adv + per - 1) / per;
}

// queue: one counter, then one per solve, all zero; tables on the device.
cudaError_t batch_steps_launch(const void* solves, const void* tiles, int ntiles,
                               const int* tile_n, int max_steps, long long rounds,
                               unsigned long long* queue, int* err, long long budget, int sms,
                               cudaStream_t st) {
  cudaError_t e =
      cudaFuncSetAttribute(batch_steps, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (e != cudaSuccess) return e;
  const long long tasks = rounds * ntiles;
  const int most = 2 * sms;
  batch_steps<<<ntiles < most ? ntiles : most, ST, SMEM, st>>>(
      (const BSolve*)solves, (const BTile*)tiles, ntiles, tile_n, max_steps, tasks, queue,
      queue + 1, err, budget);
  return cudaGetLastError();
}

}  // namespace nlse
