// Double-float stencil variant of the energy / gradient evaluation
// (tm_energy_set_stencil_precision(e, 2)).
//
// GB300's FP64 pipe retires a small fraction of the FP32 rate, and the FP64
// kernels of energy.cu keep it ~85% busy.  These kernels compute the same
// quantities with double-word numbers (df64.cuh: pairs of floats, ~48-bit
// significands) on the FP32 pipe:
//   * positions are split once per evaluation into float hi / lo parts (one
//     32-byte sector per vertex); edge vectors are double-word differences,
//     so |x| >> |x_b - x_a| costs no accuracy;
//   * products are exact TwoProds, sums collect their rounding errors in one
//     float (Dot2 / Sum2 style) and are renormalised once, normalisations
//     and reciprocals are a float estimate plus one Newton step;
//   * the dihedral angle is refined from a float atan2 estimate on the grid
//     t0 = k/128 (double-word sine and cosine table), theta = t0 + asin(x)
//     with x = sin(theta - t0) from the sine and cosine of the face normals;
//   * FP64 stays for the flat-bottom potentials below lc1 with non-positive
//     exponents, the repulsion pairs (exact pair decisions), the global sums
//     and the penalty assembly.
// The results agree with the FP64 oracle to ~1e-13 relative (the parity
// tests hold them to 1e-10); they are not bitwise equal to the FP64 kernels.
//
// An evaluation is a chain of five kernels (positions, faces + repulsion,
// edges + queued repulsion, vertices, gradient).  What bounds it: on large
// meshes issue slots (each double-word operation is 7-20 FP32 instructions)
// and gathers over the 1-ring, on small ones the kernels' latencies.  Against
// the former chain of eight kernels on two streams (a graph replay, 64- and
// 32-byte records gathered in 16-byte pieces, cross products per ring slot):
// 113 to 87 us at 163,842 vertices (the gradient 41 to 25), 53 to 37 at
// 40,962, 43 to 23 at 642, 84 to 32 for an open tube of 7,566 vertices with
// Verlet rows; the errors against 64 bits are the same (gradient 6.7e-13 at
// 163,842 vertices, energy 1.9e-14).  A variant with all stages in one
// cooperative kernel (grid barriers instead of launches) was slower at every
// size: 32 us at 642 vertices, 40 at 10,242, 150 at 163,842.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "df64.cuh"
#include "tm_dw.cuh"
#include "tm_chain.cuh"
#include "tm_energy.cuh"
#include "tm_internal.h"
#include "tm_math.cuh"

namespace tmg {

namespace {

// Face record, four float4 (two sectors) per face:
//   [0] (nx, ny)  [1] (nz, A)  [2] (cot a, cot b)  [3] (cot c, -)
// with n the unit normal, A the area and the cotangents of the corners in
// the face's stored vertex order; (A, V), V the signed volume about the
// origin, again in a compact record for the ring sums.
// Edge records, one float4 each: (l theta, bond value) for the ring sums and
// (theta / l, kt dB/dl / l) for the gradient.
// Every entry is a double-word (hi, lo).

// What the stages of one evaluation work on.
struct DwEval {
  Topo t;
  const double* P;  // positions
  float4* X;        // PosDW records
  float* P32;       // float copy of the positions (repulsion prefilter)
  float4 *fd, *fav, *eg, *elt;
  const float4* sct;
  EP ep;
  EPD epd;
  // repulsion: rep 0 none, 1 with near rows or Verlet rows, 2 without
  int rep, use_near, excl_fresh;
  NLView nl;
  const double* xb;  // positions the near rows were built at
  double thr2;
  float thr;
  int* moved;  // per block of the split stage: some vertex left its skin
  int nmoved;
  double *pot, *repg;
  int *slow, *nslow;
  double* partial;
  Globals* g;
  double* energy;  // energy of the evaluation, may be NULL
  double* grad;    // NULL: energy only
};

// The velocity-Verlet update that precedes an evaluation inside an HMC move
// (kick with the last two forces, drift): per vertex, so the split stage
// does it on the fly instead of a pass of its own over x, p and g.
struct DwMove {
  double *x, *p;
  const double *g0, *g1;  // g1 NULL: drift only, with g0
  double dt, hdt, hdt2, im;  // step, dt / 2, dt^2 / 2, 1 / mass
};

__device__ __forceinline__ df3 pos_of(const float4* X, int v) { return PosDW{X}.at(v); }
__device__ __forceinline__ df3 pos_of(const float4* X, int v, df* kr) { return PosDW{X}.at(v, kr); }

// ---- stage 1: positions ------------------------------------------------------
// Returns whether the vertex has left the skin of the near rows (the test of
// k_moved, decided in float when the float distance is clearly inside: the
// margin is four times the rounding of the two positions).
template <bool MOVE>
__device__ __forceinline__ bool split_vertex(const DwEval& a, const DwMove& mv, int v) {
  double x[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const size_t i = 3 * (size_t)v + k;
    if (MOVE) {
      double pn = mv.p[i], f = -mv.g0[i];
      if (mv.g1) {
        const double f1 = -mv.g1[i];
        pn = pn + (f + f1) * mv.hdt;
        mv.p[i] = pn;
        f = f1;
      }
      x[k] = mv.x[i] + (pn * mv.dt + f * mv.hdt2) * mv.im;
      mv.x[i] = x[k];
    } else {
      x[k] = a.P[i];
    }
  }
  float h[3], l[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) split_bits(x[k], &h[k], &l[k]);
  st32(a.X + 2 * (size_t)v, make_float4(h[0], h[1], h[2], 0.0f), make_float4(l[0], l[1], l[2], 0.0f));
  if (!a.rep) return false;
#pragma unroll
  for (int k = 0; k < 3; ++k) a.P32[3 * (size_t)v + k] = h[k];
  if (!a.use_near) return false;
  double b[3];
  float s = 0.0f, m = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    b[k] = __ldg(a.xb + 3 * (size_t)v + k);
    float bh, bl;
    split_bits(b[k], &bh, &bl);
    const float d = h[k] - bh;
    s = fmaf(d, d, s);
    m = fmaxf(m, fmaxf(fabsf(h[k]), fabsf(bh)));
  }
  const float in = a.thr - 1e-6f * m;
  if (in > 0.0f && s < 0.999f * in * in) return false;
  const double dx = x[0] - b[0], dy = x[1] - b[1], dz = x[2] - b[2];
  return !(dx * dx + dy * dy + dz * dz < a.thr2);  // NaN counts as moved
}

// ---- stage 2: faces, and the repulsion of the vertices -----------------------
__device__ __forceinline__ void face_dw(const DwEval& q, int a, int b, int c, int f) {
  const df3 pa = pos_of(q.X, a), pb = pos_of(q.X, b), pc = pos_of(q.X, c);
  const df3 eab = sub3(pb, pa), eac = sub3(pc, pa), ebc = sub3(pc, pb);
  const df3 N = cross3(eab, eac);
  const df n2 = dot3(N, N);
  const df r = rsqrt_dw(n2);  // 1 / |N|
  const df A = half(mul_s(n2, r));
  // (p_a x p_b) . p_c = p_a . ((p_b - p_a) x (p_c - p_a)) = p_a . N
  const df V = mul_s(dot3(pa, N), sixth());
  const df nx = mul_s(N.x, r), ny = mul_s(N.y, r), nz = mul_s(N.z, r);
  const df c0 = mul_s(dot3(eab, eac), r);
  const df c1 = neg(mul_s(dot3(eab, ebc), r));
  const df c2 = mul_s(dot3(eac, ebc), r);
  float4* o = q.fd + 4 * (size_t)f;
  st32(o, make_float4(nx.hi, nx.lo, ny.hi, ny.lo), make_float4(nz.hi, nz.lo, A.hi, A.lo));
  st32(o + 2, make_float4(c0.hi, c0.lo, c1.hi, c1.lo), make_float4(c2.hi, c2.lo, 0.0f, 0.0f));
  q.fav[f] = make_float4(A.hi, A.lo, V.hi, V.lo);
}

// Whether the near rows serve this evaluation: 0 no, 1 rows and exclusion
// flags, 2 rows with the exclusion tested (the topology has changed since).
// Called by whole blocks.
__device__ __forceinline__ int near_mode_of(const DwEval& q) {
  if (!q.use_near) return 0;
  bool mv = false;
  for (int b = threadIdx.x; b < q.nmoved; b += blockDim.x) mv = mv || ((volatile int*)q.moved)[b] != 0;
  if (__syncthreads_or(mv)) return 0;
  if (q.nl.nflag[1] != 0) return 0;
  return q.nl.nflag[2] == *q.nl.dtopo ? 1 : 2;
}

// Pair term of the repulsion and (grad) its derivative over l times the
// distance vector
struct RepTerm {
  double pot, gx, gy, gz;
};
template <bool GRAD>
__device__ __forceinline__ RepTerm rep_term(const EP& ep, double l, d3 dv) {
  const double lmc = l - ep.rlc1;
  const double ilmc = 1.0 / lmc, il = 1.0 / l;
  const double ex = exp(l * ilmc) * ipow(il, ep.rr);
  RepTerm r{ex, 0.0, 0.0, 0.0};
  if (GRAD) {
    const double fac = -(ep.rlc1 * (ilmc * ilmc) + ep.rr * il) * (ex * il);
    r.gx = fac * dv.x;
    r.gy = fac * dv.y;
    r.gz = fac * dv.z;
  }
  return r;
}

constexpr int SB = 256;  // threads per block of the split, face and edge kernels

// The repulsion runs a block at a time in two steps: the threads test their
// rows and set the accepted pairs aside in shared memory, then the block
// evaluates those densely, and each vertex adds its terms in a fixed order.  A
// term is about 200 FP64 instructions of 16 cycles an SM each, whatever part of a
// warp takes them: with every thread evaluating its own pairs where it found
// them, a sphere of 642 vertices with near rows and 1.5 accepted pairs a vertex
// took 159 us an evaluation (so 35), one of 161,292 715 (260), a tube of
// 7,566 vertices with Verlet rows and 1,220 active pairs 35.3 (32.9).
constexpr int VL = 8;  // lanes per vertex, where several share one
struct RepPair {
  double a, x, y, z;  // squared distance and vector, then potential and gradient
};
template <bool LANES>
struct RepBlock {
  RepPair pair[LANES ? SB : 1];   // one per thread (one lane per vertex: in pot and repg)
  long long key[LANES ? SB : 1];  // near rows by VL lanes: NEAR_HITS per vertex
  unsigned short list[SB];
  int n[2];  // list lengths of a round and the next, zero at the start
};
static_assert(VL == NEAR_HITS, "one lane per accepted pair of a near row");
// the n pairs named by list, dense
template <bool GRAD>
__device__ __forceinline__ void rep_dense(const EP& ep, RepBlock<true>& sh, int n) {
  for (int i = threadIdx.x; i < n; i += SB) {
    RepPair& c = sh.pair[sh.list[i]];
    const RepTerm r = rep_term<GRAD>(ep, __dsqrt_rn(c.a), mk(c.x, c.y, c.z));
    c = {r.pot, r.gx, r.gy, r.gz};
  }
  __syncthreads();
}
__device__ __forceinline__ void add_term(RepTerm& sum, const RepTerm& r) {
  sum.pot += r.pot;
  sum.gx += r.gx;
  sum.gy += r.gy;
  sum.gz += r.gz;
}
template <bool GRAD>
__device__ __forceinline__ void store_rep(const DwEval& q, int v, const RepTerm& sum) {
  q.pot[v] = sum.pot;
  if (GRAD) st3(q.repg, v, 2.0 * mk(sum.gx, sum.gy, sum.gz));
}

// appends v to the queue of the cell walk (one atomic for the threads that do
// so together; the order does not matter, each vertex is written by one warp)
__device__ __forceinline__ void queue_vertex(const DwEval& q, int v) {
  const cooperative_groups::coalesced_group g = cooperative_groups::coalesced_threads();
  int at = 0;
  if (g.thread_rank() == 0) at = atomicAdd(q.nslow, (int)g.size());
  q.slow[g.shfl(at, 0) + g.thread_rank()] = v;
}

// Vertex v by one thread without near rows: its candidate row (the others are
// queued for the cell walk) or its Verlet row
template <bool GRAD>
__device__ __forceinline__ void rep_vertex(const DwEval& q, int v) {
  const NLView& nl = q.nl;
  const EP& ep = q.ep;
  const d3 p = ld3p(q.P, v);
  const PairTest pt = make_pair_test(nl, v, ep.rlc1, ep.rT);
  TableExclSlim x{q.t, nl.excl};
  RepTerm sum{0.0, 0.0, 0.0, 0.0};
  auto add = [&](int, double l, d3 dv) { add_term(sum, rep_term<GRAD>(ep, l, dv)); };
  if (nl.kind == 0) {
    int co[3];
    if (!in_build_cell(nl, v, p, co)) {
      queue_vertex(q, v);
      return;
    }
    visit_candidates(pt, nl, q.P, v, p, x, add);
  } else {
    const int lo = nl.vrow[v], hi = nl.vrow[v + 1];
    for (int e = lo; e < hi; ++e) {
      const int j = nl.vcol[e];
      d3 pj;
      double s;
      if (!pair_within(pt, nl, q.P, p, j, &pj, &s)) continue;
      // the rows leave out the pairs excluded when they were built
      if (!q.excl_fresh && nl.excl > 0 && x(v, j)) continue;
      add(j, __dsqrt_rn(s), exact_diff(p, pj));
    }
  }
  store_rep<GRAD>(q, v, sum);
}

// the cell-list pair of v (in cell co) and j, as visit_near takes it: its key
// in the reference's visiting order, or -1
__device__ __forceinline__ long long near_key(const NLView& nl, const int* co, int j) {
  const int ox = nl.bcoord[3 * j] - co[0], oy = nl.bcoord[3 * j + 1] - co[1], oz = nl.bcoord[3 * j + 2] - co[2];
  if (ox < -1 || ox > 1 || oy < -1 || oy > 1 || oz < -1 || oz > 1) return -1;
  return ((long long)((ox + 1) * 9 + (oy + 1) * 3 + (oz + 1)) << 32) | (long long)j;
}

// Near rows by one thread per vertex (mode: see visit_near), the first accepted
// pairs of all vertices in one round, then the second ones, and so on.  A pair is
// set aside in its vertex's own result entries, not in shared memory, which would
// take L1 from the faces' gathers.
template <bool GRAD>
__device__ __forceinline__ void rep_near_block(const DwEval& q, int mode, RepBlock<false>& sh) {
  const NLView& nl = q.nl;
  const EP& ep = q.ep;
  const int v = blockIdx.x * SB + threadIdx.x;
  long long key[NEAR_HITS];
  double dist2[NEAR_HITS];
  int hits = 0;
  bool walk = false;
  d3 p = mk(0, 0, 0);
  if (v < q.t.nv) {
    p = ld3p(q.P, v);
    const PairTest pt = make_pair_test(nl, v, ep.rlc1, ep.rT);
    TableExclSlim x{q.t, nl.excl};
    int co[3];
    in_build_cell(nl, v, p, co);
    // four entries per load (a row starts on a 192-byte boundary)
    const int4* row4 = reinterpret_cast<const int4*>(nl.nent + (size_t)v * TM_NEAR_CAP);
    const int n = nl.ncnt[v];
    int4 r4 = make_int4(0, 0, 0, 0);
    for (int e = 0; e < n; ++e) {
      if ((e & 3) == 0) r4 = row4[e >> 2];
      const int c = r4.x, j = c & 0x7fffffff;
      r4 = make_int4(r4.y, r4.z, r4.w, 0);
      if (mode == 1 && c < 0) continue;
      d3 pj;
      double s;
      if (!pair_within(pt, nl, q.P, p, j, &pj, &s)) continue;
      const long long k = near_key(nl, co, j);
      if (k < 0 || (mode == 2 && nl.excl > 0 && x(v, j))) continue;
      if (hits == NEAR_HITS) {
        walk = true;
        break;
      }
      int h = hits++;
      while (h > 0 && key[h - 1] > k) {
        key[h] = key[h - 1];
        dist2[h] = dist2[h - 1];
        --h;
      }
      key[h] = k;
      dist2[h] = s;
    }
    if (walk) {
      hits = 0;
      queue_vertex(q, v);
    }
  }
  RepTerm sum{0.0, 0.0, 0.0, 0.0};
  for (int r = 0; __syncthreads_or(r < hits); ++r) {
    int& n = sh.n[r & 1];
    if (r < hits) {
      q.pot[v] = dist2[r];
      st3(q.repg, v, exact_diff(p, ld3p(q.P, (int)(key[r] & 0xffffffff))));
      sh.list[atomicAdd(&n, 1)] = (unsigned short)threadIdx.x;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += SB) {
      const int u = blockIdx.x * SB + sh.list[i];
      const RepTerm t = rep_term<GRAD>(ep, __dsqrt_rn(q.pot[u]), ld3p(q.repg, u));
      q.pot[u] = t.pot;
      if (GRAD) st3(q.repg, u, mk(t.gx, t.gy, t.gz));
    }
    __syncthreads();
    if (r < hits) {
      sum.pot += q.pot[v];
      if (GRAD) {
        const d3 g = ld3p(q.repg, v);
        sum.gx += g.x;
        sum.gy += g.y;
        sum.gz += g.z;
      }
    }
    if (threadIdx.x == 0) n = 0;  // for the round after the next
  }
  if (v < q.t.nv && !walk) store_rep<GRAD>(q, v, sum);
}

// Near rows by VL lanes per vertex
template <bool GRAD>
__device__ __forceinline__ void rep_near_lanes(const DwEval& q, int mode, RepBlock<true>& sh) {
  const NLView& nl = q.nl;
  const EP& ep = q.ep;
  const int v = (blockIdx.x * SB + threadIdx.x) / VL, sub = threadIdx.x % VL, base = threadIdx.x & ~(VL - 1);
  const bool act = v < q.t.nv;
  const unsigned gmask = ((1u << VL) - 1u) << (threadIdx.x & 31 & ~(VL - 1));
  int total = 0;
  if (act) {
    const d3 p = ld3p(q.P, v);
    const PairTest pt = make_pair_test(nl, v, ep.rlc1, ep.rT);
    TableExclSlim x{q.t, nl.excl};
    const int* row = nl.nent + (size_t)v * TM_NEAR_CAP;
    const int n = nl.ncnt[v];
    int co[3];
    in_build_cell(nl, v, p, co);
    for (int e0 = 0; e0 < n; e0 += VL) {
      const int e = e0 + sub;
      long long key = -1;
      double s = 0.0;
      d3 pj = p;
      if (e < n) {
        const int c = row[e], j = c & 0x7fffffff;
        if (!(mode == 1 && c < 0) && pair_within(pt, nl, q.P, p, j, &pj, &s)) {
          key = near_key(nl, co, j);
          if (mode == 2 && key >= 0 && nl.excl > 0 && x(v, j)) key = -1;
        }
      }
      const unsigned b = __ballot_sync(gmask, key >= 0);
      const int pos = total + __popc(b & ((1u << (threadIdx.x & 31)) - 1u));
      if (key >= 0 && pos < NEAR_HITS) {
        const d3 dv = exact_diff(p, pj);
        sh.key[base + pos] = key;
        sh.pair[base + pos] = {s, dv.x, dv.y, dv.z};
      }
      total += __popc(b);
    }
    if (total > NEAR_HITS) {
      if (sub == 0) queue_vertex(q, v);
    } else if (sub < total) {
      sh.list[atomicAdd(&sh.n[0], 1)] = (unsigned short)(base + sub);
    }
  }
  if (__syncthreads_or(total > 0)) rep_dense<GRAD>(ep, sh, sh.n[0]);
  if (!act || total > NEAR_HITS) return;
  // in the order of the keys
  int rank = -1;
  if (sub < total) {
    rank = 0;
    for (int o = 0; o < total; ++o) rank += sh.key[base + o] < sh.key[base + sub] ? 1 : 0;
  }
  RepTerm sum{0.0, 0.0, 0.0, 0.0};
  for (int h = 0; h < total; ++h) {
    const int src = __ffs(__ballot_sync(gmask, rank == h)) - 1 - (threadIdx.x & 31 & ~(VL - 1));
    const RepPair c = sh.pair[base + src];
    add_term(sum, {c.a, c.x, c.y, c.z});
  }
  if (sub == 0) store_rep<GRAD>(q, v, sum);
}

// Verlet rows by VL lanes per vertex: a lane's first accepted pair is set aside,
// further ones are evaluated where they are found; each lane adds its own in row
// order, then a fixed shuffle tree
template <bool GRAD>
__device__ __forceinline__ void rep_verlet_lanes(const DwEval& q, RepBlock<true>& sh) {
  const NLView& nl = q.nl;
  const EP& ep = q.ep;
  const int v = (blockIdx.x * SB + threadIdx.x) / VL, sub = threadIdx.x % VL;
  const bool act = v < q.t.nv;
  const unsigned gmask = ((1u << VL) - 1u) << (threadIdx.x & 31 & ~(VL - 1));
  RepTerm more{0.0, 0.0, 0.0, 0.0};  // past the first
  bool mine = false;
  if (act) {
    const d3 p = ld3p(q.P, v);
    const PairTest pt = make_pair_test(nl, v, ep.rlc1, ep.rT);
    TableExclSlim x{q.t, nl.excl};
    const int lo = nl.vrow[v], hi = nl.vrow[v + 1];
    for (int e = lo + sub; e < hi; e += VL) {
      const int j = nl.vcol[e];
      d3 pj;
      double s;
      if (!pair_within(pt, nl, q.P, p, j, &pj, &s)) continue;
      // the rows leave out the pairs excluded when they were built
      if (!q.excl_fresh && nl.excl > 0 && x(v, j)) continue;
      const d3 dv = exact_diff(p, pj);
      if (!mine) {
        mine = true;
        sh.pair[threadIdx.x] = {s, dv.x, dv.y, dv.z};
        sh.list[atomicAdd(&sh.n[0], 1)] = (unsigned short)threadIdx.x;
      } else {
        add_term(more, rep_term<GRAD>(ep, __dsqrt_rn(s), dv));
      }
    }
  }
  if (__syncthreads_or(mine)) rep_dense<GRAD>(ep, sh, sh.n[0]);
  if (!act) return;
  RepTerm sum{0.0, 0.0, 0.0, 0.0};
  if (mine) {
    const RepPair c = sh.pair[threadIdx.x];
    sum = {c.a, c.x, c.y, c.z};
  }
  if (__ballot_sync(gmask, mine)) {  // (no FP64 shuffle tree where no lane has a pair)
    add_term(sum, more);
#pragma unroll
    for (int o = VL / 2; o > 0; o >>= 1) {
      sum.pot += __shfl_down_sync(gmask, sum.pot, o);
      if (GRAD) {
        sum.gx += __shfl_down_sync(gmask, sum.gx, o);
        sum.gy += __shfl_down_sync(gmask, sum.gy, o);
        sum.gz += __shfl_down_sync(gmask, sum.gz, o);
      }
    }
  }
  if (sub == 0) store_rep<GRAD>(q, v, sum);
}

// ---- stage 3: edges, and the queued repulsion --------------------------------
// Flat-bottom bond of an edge shorter than lc1 (src/mesh_tether.h:29-85)
// in double-word arithmetic: value e^(l/(l-lc1)) / l^r, derivative
// -(lc1/(l-lc1)^2 + r/l) e^(l/(l-lc1)) / l^r (plus the l > lc0 branch when
// lc1 > lc0).
__device__ __forceinline__ void edge_bond_short_dw(const EP& ep, const EPD& epd, df l, df* val, df* fac) {
  const int r = ep.r;
  df v = df_make(0.0f), f = df_make(0.0f);
  const bool above = df_less(epd.lc0, l);
  if (above) {
    const df d = sub_s(l, epd.lc0);
    v = mul_s(epd.br1, ipow_dw(d, r));
    f = mul_s(epd.br2, ipow_dw(d, r - 1));
  }
  const df ilmc = rcp_dw(sub_s(l, epd.lc1)), il = rcp_dw(l);
  const df ex = df_exp_nonpos(mul_s(l, ilmc));
  const df ilr = ipow_dw(il, r);
  if (!above) v = mul_s(ex, ilr);
  f = sub_s(f, add_s(mul_s(epd.lc1, mul_s(ilmc, ilmc)), mul_s(il, df_make((float)r))));
  *val = v;
  *fac = mul_s(mul_s(f, ilr), ex);
}


__device__ __forceinline__ void edge_dw(const DwEval& q, int4 E, int e) {
  const EP& ep = q.ep;
  const EPD& epd = q.epd;
  const df3 ev = sub3(pos_of(q.X, E.y), pos_of(q.X, E.x));
  const df l2 = dot3(ev, ev);
  const df il = rsqrt_dw(l2);
  const df l = mul_s(l2, il);
  df th = df_make(0.0f);
  const bool interior = E.z >= 0 && E.w >= 0;
  if (interior) {
    float4 a0, a1, b0, b1;
    ld32(q.fd + 4 * (size_t)E.z, a0, a1);
    ld32(q.fd + 4 * (size_t)E.w, b0, b1);
    const df3 n0 = {{a0.x, a0.y}, {a0.z, a0.w}, {a1.x, a1.y}};
    const df3 n1 = {{b0.x, b0.y}, {b0.z, b0.w}, {b1.x, b1.y}};
    // n0 x n1 lies along the shared edge: its projection on the unit edge
    // is the signed sine, with the sign of the reference's test
    // (n0 x n1) . e >= 0
    const df sd = mul_s(dot3(cross3(n0, n1), ev), il);
    th = angle_dw(sd, dot3(n0, n1), q.sct);
  }
  // flat-bottom edge penalty: above the flat bottom products only, below it
  // the exponential (a warp with any short edge takes that branch; on the
  // jittered benchmark membrane nearly every warp has one, which costs less
  // than a list of short edges and a kernel of their own)
  df val = df_make(0.0f), db = df_make(0.0f);
  const bool shortb = ep.btype == 0 && df_less(l, epd.lc1);
  if (ep.btype == 0 && !shortb && df_less(epd.lc0, l) && ep.r >= 1) {
    const df d = sub_s(l, epd.lc0);
    const df dr1 = ipow_dw(d, ep.r - 1);
    val = mul_s(epd.br1, mul_s(dr1, d));
    db = mul_s(epd.br2, dr1);
  }
  if (shortb) {
    if (ep.r >= 1) {
      edge_bond_short_dw(ep, epd, l, &val, &db);
    } else {  // non-positive exponents: FP64
      double v, f;
      const double ld = df_to(l);
      edge_bond(ep, ld, 1.0 / ld, &v, &f);
      val = df_from(v);
      db = df_from(f);
    }
  }
  const df lt = mul_s(l, th), tl = mul_s(th, il), kd = mul_s(mul_s(epd.kt, db), il);
  q.eg[e] = make_float4(tl.hi, tl.lo, kd.hi, kd.lo);
  q.elt[e] = make_float4(lt.hi, lt.lo, val.hi, val.lo);
}

// One warp per queued vertex: lane l < 27 looks up neighbour cell l (the
// reference's x-outer / z-inner order), then all lanes take the cells' members
// in that order, every 32nd each, so that the pair terms (about 200 FP64
// instructions) are evaluated by as many lanes as there are pairs; the lanes'
// sums are combined by a fixed shuffle tree, so the result does not depend on
// timing.
template <bool GRAD>
__device__ __forceinline__ void rep_queue(const DwEval& q, int n, int warp, int nwarps) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const NLView& nl = q.nl;
  const NLGeom& G = *nl.geom;
  TableExclSlim x{q.t, nl.excl};
  for (int i = warp; i < n; i += nwarps) {
    const int v = ((volatile int*)q.slow)[i];
    const d3 p = ld3p(q.P, v);
    const PairTest pt = make_pair_test(nl, v, q.ep.rlc1, q.ep.rT);
    RepTerm sum{0.0, 0.0, 0.0, 0.0};
    auto add = [&](int, double l, d3 dv) { add_term(sum, rep_term<GRAD>(q.ep, l, dv)); };
    int co[3];
    in_build_cell(nl, v, p, co);
    int st = 0, cnt = 0;
    if (lane < 27) {
      const int ii = co[0] + lane / 9 - 1, jj = co[1] + (lane / 3) % 3 - 1, kk = co[2] + lane % 3 - 1;
      if (ii >= 0 && ii < G.shape[0] && jj >= 0 && jj < G.shape[1] && kk >= 0 && kk < G.shape[2])
        cnt = cell_find(nl, cell_key(ii * G.stride[0] + jj * G.stride[1] + kk * G.stride[2], 0), &st);
    }
    int end = cnt;  // members of the cells up to this lane's
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL, end, o);
      if (lane >= o) end += y;
    }
    const int total = __shfl_sync(FULL, end, 31), first = st + cnt - end;
    for (int m = lane; m - lane < total; m += 32) {
      int c = 0;  // the cell of member m: as many cells end at or before it
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(FULL, end, c + o - 1) <= m) c += o;
      const int at = __shfl_sync(FULL, first, c);
      if (m < total) {
        const int j = nl.cell_verts[at + m];
        if (j != v) visit_pair(pt, nl, q.P, v, p, j, x, add);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum.pot += __shfl_down_sync(FULL, sum.pot, o);
      if (GRAD) {
        sum.gx += __shfl_down_sync(FULL, sum.gx, o);
        sum.gy += __shfl_down_sync(FULL, sum.gy, o);
        sum.gz += __shfl_down_sync(FULL, sum.gz, o);
      }
    }
    if (lane == 0) store_rep<GRAD>(q, v, sum);
  }
}

// ---- stage 4: vertices and global sums ---------------------------------------
// Sum of x over the L lanes of a vertex (adjacent lanes, L a power of two);
// every lane ends with the same sum.  Called by whole warps.
template <int L>
__device__ __forceinline__ df lane_sum(df x) {
#pragma unroll
  for (int q = L / 2; q > 0; q >>= 1)
    x = add_s(x, df{__shfl_xor_sync(0xffffffffu, x.hi, q), __shfl_xor_sync(0xffffffffu, x.lo, q)});
  return x;
}

// The six properties of vertex v from its ring into pr (lane 0 of the
// vertex's L lanes, each with a run of ceil(d / L) ring slots), and the
// curvature weight kb c/a for the gradient into the free entries of the
// position record.
template <int L>
__device__ __forceinline__ void vertex_dw(const DwEval& q, int v, int sub, df* pr) {
  const Topo& t = q.t;
  dacc A = {0.0f, 0.0f}, Vo = A, LT = A, T = A;
#pragma unroll
  for (int k = 0; k < 6; ++k) pr[k] = df_make(0.0f);
  if (v < t.nv) {
    const int d = t.val[v];
    const int run = (d + L - 1) / L, m1 = min(d, (sub + 1) * run);
    // slots in groups (one group at the usual valence): all loads of a group
    // are issued before the sums, which keep the slot order
    constexpr int G = (6 + L - 1) / L;
    for (int m0 = sub * run; m0 < m1; m0 += G) {
      int4 s[G];
#pragma unroll
      for (int k = 0; k < G; ++k) s[k] = m0 + k < m1 ? t.slot[(size_t)(m0 + k) * t.nv + v] : make_int4(0, -1, 0, 0);
      float4 av[G], lb[G];
#pragma unroll
      for (int k = 0; k < G; ++k) {
        const int f = slot_face(s[k].y);
        av[k] = lb[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (f >= 0) {
          av[k] = q.fav[f];
          lb[k] = q.elt[s[k].z];
        }
      }
#pragma unroll
      for (int k = 0; k < G; ++k) {
        if (slot_face(s[k].y) < 0) continue;
        acc_add(A, lo_hi(av[k].x, av[k].y));
        acc_add(Vo, lo_hi(av[k].z, av[k].w));
        acc_add(LT, lo_hi(lb[k].x, lb[k].y));
        if (q.ep.btype == 0) {
          acc_add(T, lo_hi(lb[k].z, lb[k].w));
        } else {
          const df z = sub_s(mul_s(lo_hi(av[k].x, av[k].y), q.epd.inv_a0), df_make(1.0f));
          acc_add(T, mul_s(z, z));
        }
      }
    }
  }
  const df sA = lane_sum<L>(acc_val(A)), sV = lane_sum<L>(acc_val(Vo)), sLT = lane_sum<L>(acc_val(LT)),
           sT = lane_sum<L>(acc_val(T));
  if (v < t.nv && sub == 0) {
    const df a = mul_s(sA, third());
    const df c = ldexp2(sLT, 0.25f);
    const df rho = mul_s(c, rcp_dw(a));
    pr[0] = a;
    pr[1] = mul_s(sV, third());
    pr[2] = c;
    pr[3] = ldexp2(mul_s(c, rho), 2.0f);  // 2 c^2 / a
    pr[4] = mul_s(sT, q.epd.inv_tdiv);
    if (q.rep) split_bits(q.pot[v], &pr[5].hi, &pr[5].lo);
    const df kr = mul_s(q.epd.kb, rho);
    q.X[2 * (size_t)v].w = kr.hi;
    q.X[2 * (size_t)v + 1].w = kr.lo;
  }
}

// Sums of the six properties over a block into partial[0..5] (FP64).  Warp
// sums by halving (each step a lane keeps half of its values and adds the
// partner's): 8 additions per lane instead of the 30 of six shuffle trees,
// which were half of the vertex stage's instructions.  The lanes' bits 4..2
// select the property they end with.  Then property k is summed over the
// warps in warp order by thread k, with one FP64 conversion per block
// (GB300's FP64 pipe is the scarce one).
template <int NW>
__device__ __forceinline__ void block_props(const df* pr, float2 (*wsum)[NW], double* partial) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  auto swap_add = [](bool up, const df& a, const df& b, int o) {  // keep a (up: b), add the partner's same one
    const df keep = up ? b : a, send = up ? a : b;
    return add_s(keep, df{__shfl_xor_sync(0xffffffffu, send.hi, o), __shfl_xor_sync(0xffffffffu, send.lo, o)});
  };
  const df zero = df_make(0.0f);
  const df q0 = swap_add(lane & 16, pr[0], pr[3], 16), q1 = swap_add(lane & 16, pr[1], pr[4], 16),
           q2 = swap_add(lane & 16, pr[2], pr[5], 16);
  const df r0 = swap_add(lane & 8, q0, q2, 8), r1 = swap_add(lane & 8, q1, zero, 8);
  df r = swap_add(lane & 4, r0, r1, 4);
#pragma unroll
  for (int o = 2; o > 0; o >>= 1)
    r = add_s(r, df{__shfl_xor_sync(0xffffffffu, r.hi, o), __shfl_xor_sync(0xffffffffu, r.lo, o)});
  const int prop = (lane & 16 ? 3 : 0) + (lane & 8 ? 2 : (lane & 4 ? 1 : 0));
  if ((lane & 3) == 0 && (lane & 12) != 12) wsum[prop][w] = make_float2(r.hi, r.lo);
  __syncthreads();
  if (threadIdx.x < 6) {
    df s = df_make(0.0f);
    for (int k = 0; k < NW; ++k) s = add_s(s, lo_hi(wsum[threadIdx.x][k].x, wsum[threadIdx.x][k].y));
    partial[threadIdx.x] = df_to(s);
  }
}
// ---- stage 5: gradient ---------------------------------------------------------
// Gradient gather per vertex i over its ring (slot m: face (i, j = r_m,
// k = r_{m-1})), the reference's gather (src/mesh_properties.cpp:51-148 with
// src/kernel.h:124-137) with every term written along the edge vectors
// d_j = x_j - x_i and the face normals n, so that each slot needs two scaled
// vectors and no cross product (the area gradient in its cotangent form and
// the volume gradient through the normal, Meyer, Desbrun, Schroeder & Barr,
// "Discrete differential-geometry operators for triangulated 2-manifolds",
// 2003).  With h = alpha / 2, alpha = gA - 2/3 kb (rho_i^2 + rho_j^2 +
// rho_k^2), and w = gC/2 + kb (rho_i + rho_j):
//   area       -h (cot_k d_j + cot_j d_k)       [= h n x (x_k - x_j)]
//   volume     gV/3 A n                         [= gV/6 d_j x d_k; the
//              x_i x (d_k - d_j) / 6 parts cancel around a closed fan]
//   length     -(w theta + kt dB/dl) / l d_j    for edge (i, j)
//   dihedral   (w_ij cot_j + w_ik cot_k - w_jk (cot_j + cot_k)) n
// Positions enter relative to x_i, so the sums stay near the size of the
// result.  Per slot a lane gathers four sectors: the neighbour's position
// and weight, the face's two, the edge's 16 bytes.
// L lanes share a vertex, each with a run of ceil(d / L) slots; the part of
// a run's first face on d_k (the previous run's last vector) is added
// directly, later ones complete the coefficient of the vector before.
__device__ __forceinline__ df cot_of(const float4& F2, const float4& F3, int c) {
  return c == 0 ? lo_hi(F2.x, F2.y) : (c == 1 ? lo_hi(F2.z, F2.w) : lo_hi(F3.x, F3.y));
}
// 2/3 kb rho^2 from kb rho (epd.kq = 2 s / (3 kb), epd.iks = 1 / s with s the
// power of two at kb: no under- or overflow of the square)
__device__ __forceinline__ df kq_of(const EPD& epd, df kr) {
  return mul_s(mul_s(ldexp2(kr, epd.iks), kr), epd.kq);
}

template <bool CLOSED, int L>
__device__ __forceinline__ void grad_dw(const DwEval& q, int i, int sub, df gA, df gV, df gC) {
  const Topo& t = q.t;
  const EPD& epd = q.epd;
  dacc3 acc = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
  dacc3 vtel = acc;
  df3 xi = {df_make(0.0f), df_make(0.0f), df_make(0.0f)};
  if (i < t.nv) {
    const df gV3 = mul_s(gV, third());
    const df hgC = half(gC);
    df kri;
    xi = pos_of(q.X, i, &kri);
    const df ai = sub_s(gA, kq_of(epd, kri));
    const df wi = add_s(hgC, kri);
    const int d = t.val[i];
    const int run = (d + L - 1) / L, mb = sub * run, m1 = min(d, mb + run);
    const size_t nv = t.nv;
    if (mb < m1) {
      const int4 sp = t.slot[(size_t)(mb == 0 ? d - 1 : mb - 1) * nv + i];
      df krk;
      df3 dk = sub3(pos_of(q.X, sp.x, &krk), xi);
      df qk = kq_of(epd, krk);
      df uk = add_s(hgC, krk);
      df wk = add_s(wi, krk);  // weight of edge (i, k)
      bool fprev = slot_face(sp.y) >= 0;
      int4 sc = t.slot[(size_t)mb * nv + i];
      dacc s = {0.0f, 0.0f};  // coefficient of d_k still open
      for (int m = mb; m < m1; ++m) {
        // the next slot's row is fetched one slot ahead; on an open fan it
        // also tells whether edge (i, j) has a face on either side
        int4 sn = sc;
        if (!CLOSED || m + 1 < m1) sn = t.slot[(size_t)(m + 1 == d ? 0 : m + 1) * nv + i];
        df krj;
        const df3 dj = sub3(pos_of(q.X, sc.x, &krj), xi);
        const df qj = kq_of(epd, krj);
        const df wj = add_s(wi, krj);
        const int f = slot_face(sc.y);
        const float4 E = q.eg[sc.z];
        dacc sj = {0.0f, 0.0f};
        if (CLOSED || f >= 0) {
          float4 F0, F1, F2, F3;
          ld32(q.fd + 4 * (size_t)f, F0, F1);
          ld32(q.fd + 4 * (size_t)f + 2, F2, F3);
          const int ci = slot_corner(sc.y);
          const df cj = cot_of(F2, F3, ci == 2 ? 0 : ci + 1), ck = cot_of(F2, F3, ci == 0 ? 2 : ci - 1);
          df alpha = sub_s(sub_s(ai, qj), qk);
          if (q.ep.btype == 1) {
            const df z = sub_s(mul_s(lo_hi(F1.z, F1.w), epd.inv_a0), df_make(1.0f));
            alpha = add_s(alpha, ldexp2(mul_s(mul_s(epd.kt, z), epd.inv_a0), 2.0f));
          }
          const df h = half(neg(alpha));
          // edge (i, k): this face completes its coefficient
          acc_fma(s, h, cj);
          acc_fma3(acc, acc_val(s), dk);
          // edge (i, j): length and area terms
          acc_fma(sj, neg(wj), lo_hi(E.x, E.y));
          if (q.ep.btype == 0) acc_add(sj, neg(lo_hi(E.z, E.w)));
          acc_fma(sj, h, ck);
          // along n
          dacc c = {0.0f, 0.0f};
          acc_fma(c, gV3, lo_hi(F1.z, F1.w));
          bool in_ij = true, in_ik = true, in_jk = true;
          if (!CLOSED) {
            in_ij = slot_face(sn.y) >= 0;
            in_ik = fprev;
            const int4 ejk = t.edge[sc.w];
            in_jk = ejk.z >= 0 && ejk.w >= 0;
          }
          if (in_ij) acc_fma(c, wj, cj);
          if (in_ik) acc_fma(c, wk, ck);
          if (in_jk) acc_fma(c, neg(add_s(uk, krj)), add_s(cj, ck));
          acc_fma3(acc, acc_val(c), {{F0.x, F0.y}, {F0.z, F0.w}, {F1.x, F1.y}});
          if (!CLOSED) acc_add3(vtel, sub3(dk, dj));
        } else {
          // no face: the edge before it has no more terms
          acc_fma3(acc, acc_val(s), dk);
        }
        fprev = f >= 0;
        s = sj;
        dk = dj;
        qk = qj;
        uk = add_s(hgC, krj);
        wk = wj;
        sc = sn;
      }
      acc_fma3(acc, acc_val(s), dk);  // the run's last edge
    }
  }
  df3 r = acc_val3(acc);
  if (L > 1) r = {lane_sum<L>(r.x), lane_sum<L>(r.y), lane_sum<L>(r.z)};
  if (!CLOSED) {
    df3 tel = acc_val3(vtel);
    if (L > 1) tel = {lane_sum<L>(tel.x), lane_sum<L>(tel.y), lane_sum<L>(tel.z)};
    const df3 tx = scale3(mul_s(gV, sixth()), cross3(xi, tel));
    r = {add_s(r.x, tx.x), add_s(r.y, tx.y), add_s(r.z, tx.z)};
  }
  if (i >= t.nv || sub != 0) return;
  double o[3] = {df_to(r.x), df_to(r.y), df_to(r.z)};
  if (q.rep) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      o[k] = o[k] + q.ep.kr * q.repg[3 * (size_t)i + k];
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) q.grad[3 * (size_t)i + k] = o[k];
}

// ---- the five kernels ----------------------------------------------------------
// Each stage is a kernel; the repulsion runs as extra blocks of the face and
// edge kernels (its queue between the two), so the kernels form one chain.
// Every kernel but the first is launched with programmatic stream
// serialisation: it may start while the one before drains, fetches its
// topology rows (which no evaluation writes) and only then waits.

template <bool MOVE>
__global__ void __launch_bounds__(SB) k_split_dw(const __grid_constant__ DwEval q, const __grid_constant__ DwMove mv) {
  let_next_start();
  const int v = blockIdx.x * SB + threadIdx.x;
  const bool m = v < q.t.nv && split_vertex<MOVE>(q, mv, v);
  if (q.use_near) {
    const int any = __syncthreads_or(m);
    if (threadIdx.x == 0) q.moved[blockIdx.x] = any;
  }
  if (v == 0) *q.nslow = 0;
}

// blocks [0, nrep): repulsion, with LANES by VL lanes per vertex (near or Verlet
// rows) or else by one; the others: faces
template <bool GRAD, bool LANES>
__global__ void __launch_bounds__(SB) k_face_dw(const __grid_constant__ DwEval q, int nrep) {
  __shared__ RepBlock<LANES> sh;
  let_next_start();
  if ((int)blockIdx.x < nrep) {
    if (threadIdx.x < 2) sh.n[threadIdx.x] = 0;
    __syncthreads();
    wait_previous();
    const int mode = near_mode_of(q);  // the same in every thread
    const int v = (blockIdx.x * SB + threadIdx.x) / (LANES ? VL : 1);
    if constexpr (LANES) {
      if (mode != 0)
        rep_near_lanes<GRAD>(q, mode, sh);
      else if (q.nl.kind == 1)
        rep_verlet_lanes<GRAD>(q, sh);
      else if (v < q.t.nv && threadIdx.x % VL == 0)
        rep_vertex<GRAD>(q, v);
    } else {
      if (mode != 0)
        rep_near_block<GRAD>(q, mode, sh);
      else if (v < q.t.nv)
        rep_vertex<GRAD>(q, v);
    }
    return;
  }
  const int f = (blockIdx.x - nrep) * SB + threadIdx.x;
  int a = 0, b = 0, c = 0;
  if (f < q.t.nf) {
    a = __ldg(q.t.fv + 3 * (size_t)f);
    b = __ldg(q.t.fv + 3 * (size_t)f + 1);
    c = __ldg(q.t.fv + 3 * (size_t)f + 2);
  }
  wait_previous();
  if (f < q.t.nf) face_dw(q, a, b, c, f);
}

// blocks [0, nqueue): the queued repulsion, one warp per vertex; the others:
// edges.  Blocks [0, nwalk) share the queue, the edges' after their edges: once
// a vertex has left its skin, or a near row has overflowed, it holds every
// vertex of the mesh.  nwalk is the number of resident blocks (four per SM at
// 62 registers), since blocks of a second wave would begin their walks when
// those of the first have ended.
template <bool GRAD>
__global__ void __launch_bounds__(SB) k_edge_dw(const __grid_constant__ DwEval q, int nqueue, int nwalk) {
  let_next_start();
  const int e = (blockIdx.x - nqueue) * SB + threadIdx.x;
  int4 E = make_int4(0, 0, -1, -1);
  if (e >= 0 && e < q.t.ne) E = __ldg(q.t.edge + e);
  wait_previous();
  const int n = nqueue ? *(volatile int*)q.nslow : 0;
  if (e >= 0 && e < q.t.ne) edge_dw(q, E, e);
  if ((int)blockIdx.x < nwalk) rep_queue<GRAD>(q, n, (blockIdx.x * SB + threadIdx.x) >> 5, nwalk * (SB / 32));
}

// The last block (atomic ticket) reduces the block partials in block order
// and assembles energy and penalty factors.  Fixed order throughout: results
// are bit-reproducible.
template <int L>
__global__ void __launch_bounds__(VB) k_vertex_dw(const __grid_constant__ DwEval q) {
  __shared__ float2 wsum[6][VB / 32];
  __shared__ double redd[6];
  __shared__ bool last;
  let_next_start();
  wait_previous();
  df pr[6];
  vertex_dw<L>(q, (blockIdx.x * VB + threadIdx.x) / L, threadIdx.x % L, pr);
  block_props<VB / 32>(pr, wsum, q.partial + 8 * (size_t)blockIdx.x);
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned int tk = atomicAdd(&q.g->ticket, 1u);
    last = (tk == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  total_props(q.partial, gridDim.x, redd);
  __syncthreads();
  if (threadIdx.x < 32) assemble_warp(q.ep, redd, q.g, q.energy);
}

template <bool CLOSED, int L>
__global__ void __launch_bounds__(128, 5) k_grad_dw(const __grid_constant__ DwEval q) {
  wait_previous();
  const Globals* g = q.g;
  grad_dw<CLOSED, L>(q, (blockIdx.x * 128 + threadIdx.x) / L, threadIdx.x % L, {g->gdf[0], g->gdf[1]}, {g->gdf[2], g->gdf[3]},
                            {g->gdf[4], g->gdf[5]});
}

__global__ void k_split_only(int nv, const double* __restrict__ P, float4* __restrict__ X, float* __restrict__ P32) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  float hx, hy, hz, lx, ly, lz;
  split_bits(P[3 * v], &hx, &lx);
  split_bits(P[3 * v + 1], &hy, &ly);
  split_bits(P[3 * v + 2], &hz, &lz);
  st32(X + 2 * (size_t)v, make_float4(hx, hy, hz, 0.0f), make_float4(lx, ly, lz, 0.0f));
  P32[3 * v] = hx;
  P32[3 * v + 1] = hy;
  P32[3 * v + 2] = hz;
}

inline int nblk(long n, int b) { return (int)((n + b - 1) / b); }

df host_df(double x) {
  float h = (float)x;
  return {h, (float)(x - (double)h)};
}

}  // namespace

EPD make_epd(const EP& ep) {
  EPD epd;
  epd.kb = host_df(ep.kb);
  epd.kt = host_df(ep.kt);
  epd.kr = host_df(ep.kr);
  int ex = 0;
  std::frexp(ep.kb, &ex);
  ex = std::min(std::max(ex, -100), 100);
  epd.iks = (float)std::ldexp(1.0, -ex);
  // (none where kb is zero as a float: kb rho, which it multiplies, is zero then)
  epd.kq = host_df((float)ep.kb != 0.0f ? std::ldexp(2.0 / 3.0, ex) / ep.kb : 0.0);
  epd.a0 = host_df(ep.a0);
  epd.inv_a0 = host_df(1.0 / ep.a0);
  epd.inv_tdiv = host_df(1.0 / ep.tdiv);
  epd.lc0 = host_df(ep.lc0);
  epd.lc1 = host_df(ep.lc1);
  epd.br1 = host_df(ep.br1);
  epd.br2 = host_df(ep.br2);
  return epd;
}

const float4* split_positions_dw(tm_energy* e, int nv, const double* P, cudaStream_t s) {
  const size_t n = std::max(nv, 1);
  e->pos32.ensure(3 * n);
  e->posdw.ensure(2 * n);
  if (nv) k_split_only<<<nblk(nv, 256), 256, 0, s>>>(nv, P, e->posdw.get(), e->pos32.get());
  TM_LAUNCH();
  return e->posdw.get();
}

void energy_eval_df(tm_energy* e, tm_mesh* m, const double* P, bool want_grad, double* d_grad, double* d_energy,
                    const Leap* leap, cudaStream_t s, cudaEvent_t* ev) {
  e->ensure(m->nv, m->ne, m->nf);
  const size_t nv = std::max(m->nv, 1);
  DwEval q{};
  q.t = m->topo();
  q.P = P;
  q.X = e->posdw.get();
  q.P32 = e->pos32.get();
  q.fd = reinterpret_cast<float4*>(e->face.get());    // 64 bytes per face
  q.eg = reinterpret_cast<float4*>(e->edge.get());    // (theta / l, kt dB/dl / l) per edge, 16 bytes
  q.elt = reinterpret_cast<float4*>(e->ebond.get());  // (l theta, bond) per edge, 16 bytes
  q.fav = reinterpret_cast<float4*>(e->fav.get());    // (area, volume) per face, 16 bytes
  q.sct = e->sctf.get();
  q.ep = make_ep(e);
  q.epd = make_epd(q.ep);
  q.nl = e->nl.view;
  q.nl.pos32 = q.P32;
  q.rep = q.ep.rlc1 > 0 ? 1 : 0;  // no pair can be closer than a non-positive cut-off
  q.use_near = q.rep && q.nl.kind == 0 && q.nl.nent && e->nl.near_nv == m->nv && e->nl.near_lc1 == q.ep.rlc1;
  q.excl_fresh = e->nl.built_topo == m->topo_version;
  q.xb = e->nl.xb.get();
  q.thr2 = e->nl.near_move2;
  q.thr = (float)std::sqrt(std::max(q.thr2, 0.0));
  q.moved = e->moved.get();
  q.pot = e->reppot.get();
  q.repg = e->repg.get();
  q.slow = e->slow.get();
  q.nslow = q.slow + nv;
  q.partial = e->partials.get();
  q.g = e->glob.get();
  q.energy = d_energy;
  q.grad = want_grad ? d_grad : nullptr;
  DwMove mv{};
  if (leap)
    mv = DwMove{leap->x, leap->p, leap->g0, leap->g1, leap->dt, 0.5 * leap->dt, 0.5 * (leap->dt * leap->dt), leap->im};
  const Topo& t = q.t;
  const int nsb = std::max(1, nblk(t.nv, SB));
  q.nmoved = nsb;
  if (ev) TM_CUDA(cudaEventRecord(ev[0], s));
  if (leap)
    k_split_dw<true><<<nsb, SB, 0, s>>>(q, mv);
  else
    k_split_dw<false><<<nsb, SB, 0, s>>>(q, mv);
  TM_LAUNCH();
  // Eight lanes share a vertex over Verlet rows that hold a few entries each
  // (the tube of 7,566 vertices with 1,220 active pairs: 38.6 us per evaluation
  // against 57.5 with one, before the pairs were set aside) and over near rows
  // up to 8,000 vertices, where one lane per vertex leaves SMs idle (at 10,242
  // vertices 54 us against 90 where pairs are accepted, but 30.2 against 28.6
  // where none is, the usual case; at 5,762 the latter are equal, 26.4); above,
  // and over sparse Verlet rows, almost every entry is skipped without a test
  // and one lane walks them (163,842 vertices: 85 us against 105).
  const bool lanes8 = q.nl.kind == 1 ? e->nl.vtotal >= 2LL * t.nv : q.use_near && t.nv <= 8000;
  const int nrep = q.rep ? nblk((long)t.nv * (lanes8 ? VL : 1), SB) : 0;
  auto* kf = lanes8 ? (want_grad ? k_face_dw<true, true> : k_face_dw<false, true>)
                    : (want_grad ? k_face_dw<true, false> : k_face_dw<false, false>);
  launch_after(kf, std::max(1, nrep + nblk(t.nf, SB)), SB, s, q, nrep);
  if (ev) TM_CUDA(cudaEventRecord(ev[1], s));
  // One block per SM for the queue alone: more cost evaluations without a queue
  // (two per SM 0.6 us of 28.4 at 10,242 vertices).  Whole evaluations with
  // every vertex queued, in us, of the separate kernel of 1,216 blocks that it
  // once was / of 152 blocks with one lane per cell / now, at 642, 10,242,
  // 46,242 and 163,842 vertices: one vertex past its skin (cut-off 0.8 l,
  // exclusion 2) 43/27/27, 64/66/57, 125/134/107, 381/801/324; rows overflowing
  // (2.2 l, exclusion 0) 96/61/37, 489/611/192, 1,930/-/466, 6,560/13,020/1,580.
  const int nqueue = q.rep && q.nl.kind == 0 ? e->sm_count() : 0;
  const int edge_grid = std::max(1, nqueue + nblk(t.ne, SB));
  launch_after(want_grad ? k_edge_dw<true> : k_edge_dw<false>, edge_grid, SB, s, q, nqueue,
               std::min(edge_grid, 4 * nqueue));
  if (ev) TM_CUDA(cudaEventRecord(ev[2], s));
  // Several lanes per vertex shorten the chain of one thread's walk over its
  // ring and fill more SMs, one lane per vertex issues fewer instructions.
  // Whole evaluations of spheres on a GB300 in us, lanes of the vertex stage /
  // of the gradient:
  //   vertices    1 / 1   1 / 2   2 / 2   2 / 4   2 / 8   8 / 8
  //        642    26.7    24.8    24.3    23.4    22.9    23.2
  //      4,002    27.0    26.3    25.3    25.1    25.1    26.5
  //     10,242    29.6    28.5    28.4    28.3    28.6    30.7
  //     23,042    32.6    31.0    30.7    30.6    34.5    39.1
  //     40,962    39.0    37.7    37.8    41.0    46.0    51.0
  //     81,002    44.0    47.1    49.7    56.2    65.2    79.7
  const bool two = t.nv <= 50000;
  launch_after(two ? k_vertex_dw<2> : k_vertex_dw<1>, std::max(1, nblk((long)t.nv * (two ? 2 : 1), VB)), VB, s, q);
  if (ev) TM_CUDA(cudaEventRecord(ev[3], s));
  if (want_grad && t.nv) {
    const int lanes = t.nv <= 4500 ? 8 : (two ? 2 : 1);
    auto* kg = lanes == 8   ? (m->closed ? k_grad_dw<true, 8> : k_grad_dw<false, 8>)
               : lanes == 2 ? (m->closed ? k_grad_dw<true, 2> : k_grad_dw<false, 2>)
                            : (m->closed ? k_grad_dw<true, 1> : k_grad_dw<false, 1>);
    launch_after(kg, nblk((long)t.nv * lanes, 128), 128, s, q);
  }
  if (ev) TM_CUDA(cudaEventRecord(ev[4], s));
}

}  // namespace tmg
