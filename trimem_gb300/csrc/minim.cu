// Energy minimisation on device-resident positions: limited-memory BFGS
// (Nocedal, "Updating quasi-Newton matrices with limited storage", Math.
// Comp. 35, 1980; two-loop recursion) with a backtracking line search on
// the Armijo condition.  The reference's minimisation path
// (src/trimem/mc/util.py:240-306) runs scipy's L-BFGS-B over the energy and
// gradient with the neighbour list refreshed at every evaluation; here the
// iterate, the gradient and the correction pairs stay in device memory, each
// evaluation refreshes the cell list and evaluates on the device.  The search
// direction with its trial point is one cooperative kernel (k_direction), the
// correction pair of the trial, its dot products and the energy another
// (k_finish), and the host waits once per evaluation for a few scalars to
// decide on the step.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "tm_energy.cuh"
#include "tm_grid.h"
#include "tm_internal.h"

using namespace tmg;

#define TM_API_BEGIN try {
#define TM_API_END                  \
  }                                 \
  catch (const tmg::Error& e) {     \
    tmg::set_last_error(e.what());  \
    return e.code;                  \
  }                                 \
  catch (const std::exception& e) { \
    tmg::set_last_error(e.what());  \
    return TM_ERR_ARG;              \
  }                                 \
  return TM_OK;

namespace {

constexpr int DB = 256, DG = 296;  // dot-product blocks: 2 per SM
constexpr int MAXHIST = 64;

// Sums in a fixed order: grid-stride partials per thread, the block's 256 by
// halving (256 -> 128 -> .. -> 1), then the blocks' partials the same way.
// block_tree: the block's sum, in thread 0
__device__ __forceinline__ double halve32(double r) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  return r;
}
__device__ __forceinline__ double block_tree(double acc, double* s) {
  const int t = threadIdx.x;
  __syncthreads();  // s may still be read
  s[t] = acc;
  __syncthreads();
  double r = 0.0;
  if (t < 32)
    r = halve32(((s[t] + s[t + 128]) + (s[t + 64] + s[t + 192])) + ((s[t + 32] + s[t + 160]) + (s[t + 96] + s[t + 224])));
  return r;
}
// the sum of nb <= DG block partials, in every lane; a warp of its own
__device__ __forceinline__ double total_of(const double* part, int nb) {
  static_assert(DG <= 9 * 32 + 8, "two partials for the first 40 of 256 sums");
  const int l = threadIdx.x & 31;
  double v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int b = l + 32 * q;
    v[q] = b < nb ? __ldcg(part + b) : 0.0;
    if (q < 2 && b + DB < nb) v[q] += __ldcg(part + b + DB);
  }
  return __shfl_sync(0xffffffffu, halve32(((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]))), 0);
}

// scalars the host reads (page-locked)
enum { R_E, R_SY, R_YY, R_AMAX, R_GD, R_STEP, R_RESTART, R_N };

// y = x + a d
__global__ void k_step(int n, double a, const double* __restrict__ x, const double* __restrict__ d,
                       double* __restrict__ y) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = x[i] + a * d[i];
}

struct Direction {
  int n, stored, head, rows, accept;
  size_t pitch;          // doubles from one row of S or Y to the next
  double gamma, amax;
  double *x, *g;         // iterate and its gradient
  double *xn;            // trial point: in, the accepted one (accept); out, the next
  const double* gn;      // gradient at the accepted trial point
  const double *S, *Y;   // correction pairs, [rows][pitch]
  double *d, *part, *out;
  double rho[MAXHIST + 1];
};

// Two-loop recursion d = -H g, the slope g . d, the restart from steepest
// descent when d is not a descent direction, and the trial point x + a d.
// The recursion is a chain of 2 stored + 1 dot products over the whole
// vector: one kernel with one barrier per dot product.  The update of d
// stays within the thread (E elements in registers; E = 0: in memory), and the
// vectors of the next update and dot product are loaded before the barrier.
// FP64 instructions of one SM queue on a pipe of two lanes, so one warp sums the
// block partials and forms the update's coefficient for its block (every warp
// for itself: 1.53 ms for ten iterations at 10,242 vertices, so 1.28; one
// cluster of 16 blocks with its faster barrier, but the vectors' FP64 work on
// 16 SMs: 1.38, all in one program; the whole call takes 1.31 to 1.40 ms).  As
// separate kernels with the dot product read by the host, 10,242 vertices and
// ten iterations took 330 launches and 140 waits of the 600 launches and 5.7
// ms of the whole minimisation.
template <int E>
__global__ void __launch_bounds__(DB, 2) k_direction(const __grid_constant__ Direction q) {
  __shared__ double s[DB];
  __shared__ double alpha[MAXHIST], coef;
  constexpr int M = E > 0 ? E : 1;
  const cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  const int n = q.n, first = blockIdx.x * DB + threadIdx.x, step = gridDim.x * DB;
  double d[M], dv[M], av[M], nv[M];
  // f(e, i) for every element i of this thread (e: its register)
  auto each = [&](auto&& f) {
    if (E > 0) {
#pragma unroll
      for (int e = 0; e < M; ++e) {
        const int i = first + e * step;
        if (i < n) f(e, i);
      }
    } else {
      for (int i = first; i < n; i += step) f(0, i);
    }
  };
  const double* g = q.accept ? q.gn : q.g;
  each([&](int e, int i) {
    if (q.accept) {
      q.x[i] = q.xn[i];
      q.g[i] = g[i];
    }
    d[e] = -1.0 * g[i];
    if (E == 0) q.d[i] = d[e];
  });
  auto pair = [&](int k) { return (q.head - 1 - k + q.rows) % q.rows; };
  auto row = [&](int k) { return pair(k) * q.pitch; };
  const int nd = 2 * q.stored;
  auto dot_vec = [&](int k) { return k < q.stored ? q.S + row(k) : (k < nd ? q.Y + row(nd - 1 - k) : g); };
  auto add_vec = [&](int k) { return k < q.stored ? q.Y + row(k) : q.S + row(nd - 1 - k); };
  const double* v = dot_vec(0);
  if (E > 0) each([&](int e, int i) { dv[e] = v[i]; });
  double r = 0.0;
  bool restart = false;
  for (int k = 0;; ++k) {
    double acc = 0.0;
    each([&](int e, int i) { acc += (E > 0 ? dv[e] : v[i]) * (E > 0 ? d[e] : q.d[i]); });
    double* part = q.part + (k & 1) * DG;
    acc = block_tree(acc, s);
    if (threadIdx.x == 0) part[blockIdx.x] = acc;
    const double* a = k < nd ? add_vec(k) : g;
    const double* w = k < nd ? dot_vec(k + 1) : g;
    if (E > 0)
      each([&](int e, int i) {
        av[e] = a[i];
        nv[e] = w[i];
      });
    grid.sync();
    if (threadIdx.x < 32) {  // the slope, or the coefficient of the update
      double c = total_of(part, gridDim.x);
      if (threadIdx.x == 0) {
        if (k < q.stored) {
          alpha[k] = __dmul_rn(q.rho[pair(k)], c);
          c = -alpha[k];
        } else if (k < nd) {
          c = __dsub_rn(alpha[nd - 1 - k], __dmul_rn(q.rho[pair(nd - 1 - k)], c));
        }
        coef = c;
      }
    }
    __syncthreads();
    r = coef;
    if (k >= nd) {
      if (restart || r < 0.0) break;
      restart = true;
      each([&](int e, int i) {
        d[e] = -1.0 * g[i];
        if (E == 0) q.d[i] = d[e];
      });
    } else {
      const bool scale = k == q.stored - 1;
      each([&](int e, int i) {
        if (E > 0) {
          d[e] += r * av[e];
          if (scale) d[e] = q.gamma * d[e];
        } else {
          double y = q.d[i] + r * a[i];
          if (scale) y = q.gamma * y;
          q.d[i] = y;
        }
      });
    }
    v = w;
#pragma unroll
    for (int e = 0; e < M; ++e) dv[e] = nv[e];
  }
  // the first step along -g is limited to a move of 1e-3 of the largest
  // gradient component
  const double a = restart || q.stored == 0 ? fmin(1.0, 1e-3 / fmax(q.amax, 1e-300)) : 1.0;
  each([&](int e, int i) {
    const double di = E > 0 ? d[e] : q.d[i];
    if (E > 0) q.d[i] = di;
    q.xn[i] = q.x[i] + a * di;
  });
  if (first == 0) {
    q.out[R_GD] = r;
    q.out[R_STEP] = a;
    q.out[R_RESTART] = restart ? 1.0 : 0.0;
  }
}

// After an evaluation: max |gn| and the energy for the host; with PAIR the
// correction pair s = xn - x, y = gn - g of the trial point into the rows
// sk, yk with s . y and y . y.  The last block sums the partials.
template <bool PAIR>
__global__ void __launch_bounds__(DB) k_finish(int n, const double* __restrict__ x, const double* __restrict__ g,
                                               const double* __restrict__ xn, const double* __restrict__ gn,
                                               double* __restrict__ sk, double* __restrict__ yk, double* part,
                                               unsigned int* ticket, const double* energy, double* out) {
  __shared__ double s[DB];
  __shared__ bool last;
  double sy = 0.0, yy = 0.0, m = 0.0;
  for (int i = blockIdx.x * DB + threadIdx.x; i < n; i += gridDim.x * DB) {
    const double b = gn[i];
    m = fmax(m, fabs(b));
    if (PAIR) {
      const double a = xn[i] - x[i], y = b - g[i];
      sk[i] = a;
      yk[i] = y;
      sy += a * y;
      yy += y * y;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (PAIR) {
    sy = block_tree(sy, s);
    yy = block_tree(yy, s);
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < DB / 32; ++w) m = fmax(m, s[w]);
    part[blockIdx.x] = sy;
    part[DG + blockIdx.x] = yy;
    part[2 * DG + blockIdx.x] = m;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last || threadIdx.x >= 32) return;
  __threadfence();
  if (PAIR) {
    sy = total_of(part, gridDim.x);
    yy = total_of(part + DG, gridDim.x);
  }
  m = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) m = fmax(m, __ldcg(part + 2 * DG + b));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (threadIdx.x == 0) {
    out[R_E] = *energy;
    out[R_SY] = sy;
    out[R_YY] = yy;
    out[R_AMAX] = m;
    *ticket = 0;
  }
}

inline int nblk(long n, int b) { return (int)((n + b - 1) / b); }

using DirectionKernel = void (*)(const Direction);
DirectionKernel direction_kernel(int n, int blocks) {
  switch (elements_held(n, (long long)blocks * DB)) {
    case 1: return k_direction<1>;
    case 2: return k_direction<2>;
    case 4: return k_direction<4>;
    case 8: return k_direction<8>;
    default: return k_direction<0>;
  }
}

}  // namespace

extern "C" int tm_minimize_device(tm_energy* e, tm_mesh* m, double* d_x, int maxiter, int history, double gtol,
                                  double ftol, int32_t* iterations, double* energy, void* stream) {
  TM_API_BEGIN
  if (!e || !m || !d_x) fail(TM_ERR_ARG, "NULL argument");
  if (maxiter < 0 || history < 1 || history > 64) fail(TM_ERR_ARG, "invalid L-BFGS settings");
  cudaStream_t s = stream ? (cudaStream_t)stream : e->stream;
  const int n = 3 * m->nv;
  // work space of the handle, kept between calls: d, g, trial point and its
  // gradient, the pairs, block partials and a ticket.  One pair more than the
  // history: every trial's pair is written before its s . y is known, and a
  // refused one must not have replaced the oldest that is still in use.
  const int rows = history + 1;
  const size_t row = ((size_t)n + 1) & ~(size_t)1;  // 16-byte boundaries
  const size_t need = (4 + 2 * (size_t)rows) * row + 3 * DG + 2;
  e->mwork.ensure(need);
  double* d = e->mwork.get();
  double *g = d + row, *xn = g + row, *gn = xn + row, *S = gn + row, *Y = S + rows * row;
  double* part = Y + rows * row;
  unsigned int* ticket = reinterpret_cast<unsigned int*>(part + 3 * DG);
  TM_CUDA(cudaMemsetAsync(ticket, 0, sizeof(unsigned int), s));
  double* out = e->host_scalars();
  const int grid = std::max(1, std::min(DG, nblk(n, DB)));
  int dgrid = grid;  // of the direction: fewer where they cannot all be resident
  // energy and gradient at x, neighbour list refreshed first
  auto eval = [&](const double* x, double* gx) {
    nlist_make(&e->nl, m, e->prm, x, s);
    energy_eval(e, m, x, true, false, gx, s);
  };
  eval(d_x, g);
  const double* energy_at = &e->glob.get()->comps[6];
  k_finish<false><<<grid, DB, 0, s>>>(n, nullptr, nullptr, nullptr, g, nullptr, nullptr, part, ticket, energy_at, out);
  TM_LAUNCH();
  TM_CUDA(cudaStreamSynchronize(s));
  double f = out[R_E];
  Direction q{};
  q.n = n;
  q.rows = rows;
  q.pitch = row;
  q.gamma = 1.0;
  q.amax = out[R_AMAX];
  q.x = d_x;
  q.g = g;
  q.xn = xn;
  q.gn = gn;
  q.S = S;
  q.Y = Y;
  q.d = d;
  q.part = part;
  q.out = out;
  int k = 0;
  for (; k < maxiter; ++k) {
    if (q.amax <= gtol) break;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(DB);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    TM_CUDA(launch_as_fits(dgrid, cudaErrorCooperativeLaunchTooLarge, [&](int blocks) {
      cfg.gridDim = dim3(blocks);
      const cudaError_t r = cudaLaunchKernelEx(&cfg, direction_kernel(n, blocks), q);
      if (r == cudaErrorCooperativeLaunchTooLarge) cudaGetLastError();
      return r;
    }));
    q.accept = 0;  // x and g are the accepted ones again
    double a = 0.0, gd = 0.0, fn = 0.0;
    bool ok = false;
    for (int ls = 0; ls < 40; ++ls) {
      if (ls > 0) {
        k_step<<<nblk(n, DB), DB, 0, s>>>(n, a, d_x, d, xn);
        TM_LAUNCH();
      }
      eval(xn, gn);
      k_finish<true><<<grid, DB, 0, s>>>(n, d_x, g, xn, gn, S + q.head * row, Y + q.head * row, part,
                                          ticket, energy_at, out);
      TM_LAUNCH();
      TM_CUDA(cudaStreamSynchronize(s));
      fn = out[R_E];
      if (ls == 0) {
        gd = out[R_GD];
        a = out[R_STEP];
        if (out[R_RESTART] != 0.0) {
          q.stored = 0;
          q.gamma = 1.0;
        }
      }
      if (std::isfinite(fn) && fn <= f + 1e-4 * a * gd) {
        ok = true;
        break;
      }
      a *= 0.5;
    }
    if (!ok) break;  // no decrease along d
    q.accept = 1;    // the next direction takes the trial point over
    q.amax = out[R_AMAX];
    const double sy = out[R_SY], fprev = f;
    f = fn;
    if (sy > 1e-300) {
      q.rho[q.head] = 1.0 / sy;
      q.gamma = sy / out[R_YY];
      q.head = (q.head + 1) % rows;
      q.stored = std::min(q.stored + 1, history);
    }
    if ((fprev - f) <= ftol * std::max({std::fabs(fprev), std::fabs(f), 1.0})) {
      ++k;
      break;
    }
  }
  if (q.accept) TM_CUDA(cudaMemcpyAsync(d_x, xn, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
  TM_CUDA(cudaStreamSynchronize(s));
  if (iterations) *iterations = k;
  if (energy) *energy = f;
  TM_API_END
}
