// Neighbour lists: cell list and Verlet list (src/nlists/cell_list.h,
// verlet_list.h, nlist.cpp).
//
// Cell list build (every rebuild, all on the device; five kernels in one
// chain of programmatic dependent launches, each a pass over the vertices):
//   k_box     bounding-box partials with the reference's initial values
//             {DBL_MAX,0,0} / {-1,0,0} (cell_list.h:46-47); on the side the
//             hash table is cleared and the near rows' skin is tested
//   k_insert  every block finishes the box and derives r_list/shape/strides
//             exactly like cell_list.h:56-65; cell id per vertex with C
//             truncation (cell_list.h:71-78), inserted into an open-addressing
//             hash table of the non-empty cells (2x the vertex count, power of
//             two), which counts the members
//   k_alloc   a cell's first arrival takes the cell's run of the member array
//             (the order of the runs is not observable)
//   k_scatter members into their cell's run in order of arrival
//   k_rank    rank of each member by vertex id, so a cell lists its vertices
//             in ascending order like the reference's
//             std::map<int, std::vector<int>>
// What bounds it is the chain's length: at 10,242 vertices a rebuild was 13
// launches and 75 us, with passes over all table slots, a three-kernel scan
// of them and one thread sorting a cell, and is 28 now (with new near rows 340
// then, 104 now); at 163,842 vertices 97 and 57 (554 and 511).
// Queries bin the query point with its CURRENT position but look up the
// cells' build-time members, as the reference does (cell_list.h:131-219).
// Distances are rounded operation by operation (no FMA), so pair sets match
// the sequential CPU code bit for bit.
// The Verlet list is a CSR built from the cell list with cut-off rlist
// (verlet_list.h:18-35); its queries apply `< dmax`.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <memory>

#include "tm_chain.cuh"
#include "tm_energy.cuh"
#include "tm_internal.h"
#include "tm_math.cuh"

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

namespace tmg {

__device__ __forceinline__ unsigned long long cell_hash2(long long key) {
  unsigned long long z = (unsigned long long)key + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ int cell_lookup(const NLView& nl, long long key, int* start) {
  unsigned long long h = cell_hash2(key) & nl.tmask;
  for (unsigned long long p = 0; p <= nl.tmask; ++p) {
    CellEntry c = nl.table[h];
    if (c.key == key) {
      *start = c.start;
      return c.count;
    }
    if (c.key == -1) return 0;
    h = (h + 1) & nl.tmask;
  }
  return 0;
}

namespace {

constexpr int BB = 256;
constexpr int NBOX = 296;  // most box partials of one mesh: two blocks per SM

// smaller / larger by the reference's comparisons (a NaN never replaces)
__device__ __forceinline__ double box_min(double a, double b) { return b < a ? b : a; }
__device__ __forceinline__ double box_max(double a, double b) { return b > a ? b : a; }

// skin test of the near rows: they go stale once some vertex has moved lc1/2
// or more from where they were built (thr2 rounded down; NaN moves)
struct NearCheck {
  const double* xb;  // NULL: no rows to test
  double thr2;
  int* flag;
  const EP* eps;  // batch: the replica's skin
};

// Box partials, one per block: a block takes every gridDim-th 256 vertices
// (batch: exactly its 256, which belong to one replica)
__global__ void __launch_bounds__(BB) k_box(int nv, const double* __restrict__ P, const int* __restrict__ vrep,
                                            double* __restrict__ part, CellEntry* __restrict__ T, size_t tsize,
                                            int* cursor, NearCheck nc) {
  __shared__ double s[6][BB / 32];
  let_next_start();
  const int first = blockIdx.x * BB + threadIdx.x, step = gridDim.x * BB;
  if (first == 0) *cursor = 0;
  for (size_t i = first; i < tsize; i += step) T[i] = CellEntry{-1, 0, 0};
  const bool check = nc.xb && !nc.flag[1];
  double m[6] = {DBL_MAX, 0.0, 0.0, -1.0, 0.0, 0.0};
  for (int i = first; i < nv; i += step) {
    const int rep = vrep ? vrep[i] : 0;
    if (rep < 0) continue;  // padding vertex of a batch: in no box, never moves
    const double x[3] = {P[3 * (size_t)i], P[3 * (size_t)i + 1], P[3 * (size_t)i + 2]};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      m[k] = box_min(m[k], x[k]);
      m[3 + k] = box_max(m[3 + k], x[k]);
    }
    if (check) {
      double thr2 = nc.thr2;
      if (vrep) thr2 = 0.25 * nc.eps[rep].rlc1 * nc.eps[rep].rlc1 * (1.0 - 1e-12);
      const double dx = x[0] - nc.xb[3 * (size_t)i], dy = x[1] - nc.xb[3 * (size_t)i + 1],
                   dz = x[2] - nc.xb[3 * (size_t)i + 2];
      if (!(dx * dx + dy * dy + dz * dz < thr2)) nc.flag[1] = 1;
    }
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double y = __shfl_xor_sync(0xffffffffu, m[k], o);
      m[k] = k < 3 ? box_min(m[k], y) : box_max(m[k], y);
    }
    if ((threadIdx.x & 31) == 0) s[k][threadIdx.x >> 5] = m[k];
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double r = s[threadIdx.x][0];
    for (int w = 1; w < BB / 32; ++w)
      r = threadIdx.x < 3 ? box_min(r, s[threadIdx.x][w]) : box_max(r, s[threadIdx.x][w]);
    part[6 * (size_t)blockIdx.x + threadIdx.x] = r;
  }
}

// Bounding box from nb partials, then r_list, shape and strides exactly like
// src/nlists/cell_list.h:56-65 (min/max are exact, so the order does not
// matter).  Called by a whole block.
__device__ void box_geometry(int nb, const double* part, double rlist, NLGeom& G) {
  __shared__ double s[6];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (w < 6) {
    double r = w == 0 ? DBL_MAX : (w == 3 ? -1.0 : 0.0);
    for (int b = lane; b < nb; b += 32) {
      const double y = part[6 * (size_t)b + w];
      r = w < 3 ? box_min(r, y) : box_max(r, y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double y = __shfl_xor_sync(0xffffffffu, r, o);
      r = w < 3 ? box_min(r, y) : box_max(r, y);
    }
    if (lane == 0) s[w] = r;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    const int k = threadIdx.x;
    const double box_eps = 1.0e-6;
    const double dim = __dadd_rn(__dsub_rn(s[3 + k], s[k]), box_eps);
    const int nk = (int)__ddiv_rn(dim, rlist);
    G.rl[k] = nk > 0 ? __ddiv_rn(dim, (double)nk) : dim;
    G.inv_rl[k] = 1.0 / G.rl[k];
    G.inv_rlf[k] = (float)G.inv_rl[k];
    G.bminf[k] = (float)s[k];
    G.shape[k] = nk > 0 ? nk : 1;
    G.bmin[k] = s[k];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    G.stride[0] = 1;
    G.stride[1] = G.shape[0];
    G.stride[2] = (long long)G.shape[0] * G.shape[1];
  }
  __syncthreads();
}

// cell of every vertex and its hash slot; vrank takes the order of arrival
// in the cell.  rblocks: the box partials of each replica of a batch.
__global__ void __launch_bounds__(BB) k_insert(int nv, const double* __restrict__ P, NLView nl, CellEntry* T,
                                               const double* part, int nb,
                                               const int2* __restrict__ rblocks, double rlist,
                                               const double* __restrict__ rlists, NLGeom* geoms, long long* vcid,
                                               int* vcoord, int* vslot, int* vrank, int* status) {
  __shared__ NLGeom G;
  let_next_start();
  const int v = blockIdx.x * BB + threadIdx.x;
  const int brep = nl.vrep ? nl.vrep[blockIdx.x * BB] : 0;  // the block's replica (its first vertex is real)
  int b0 = 0;
  if (nl.vrep) {
    const int2 rb = rblocks[brep];
    b0 = rb.x;
    nb = rb.y - rb.x;
    rlist = rlists[brep];
  }
  wait_previous();
  box_geometry(nb, part + 6 * (size_t)b0, rlist, G);
  if (threadIdx.x == 0 && (int)blockIdx.x == b0) geoms[brep] = G;
  if (v >= nv) return;
  const int rep = rep_of(nl, v);
  if (rep < 0) {  // padding vertex of a batch: in no cell
    vslot[v] = -1;
    vcid[v] = -1;
    vcoord[3 * v] = vcoord[3 * v + 1] = vcoord[3 * v + 2] = -1000000;
    return;
  }
  long long id = 0;
  for (int k = 0; k < 3; ++k) {
    const int c = cell_coord(P[3 * (size_t)v + k], G, k);
    vcoord[3 * v + k] = c;
    id += (long long)c * G.stride[k];
  }
  vcid[v] = id;
  id = cell_key(id, rep);
  unsigned long long h = cell_hash2(id) & nl.tmask;
  int slot = -1;
  for (unsigned long long p = 0; p <= nl.tmask; ++p) {
    unsigned long long prev =
        atomicCAS(reinterpret_cast<unsigned long long*>(&T[h].key), (unsigned long long)(-1LL), (unsigned long long)id);
    if (prev == (unsigned long long)(-1LL) || prev == (unsigned long long)id) {
      slot = (int)h;
      break;
    }
    h = (h + 1) & nl.tmask;
  }
  if (slot < 0) {
    atomicExch(status, 1);
    vslot[v] = -1;
    return;
  }
  vslot[v] = slot;
  vrank[v] = atomicAdd(&T[slot].count, 1);
}

// a cell's first arrival takes the cell's run of members (one atomic a warp)
__global__ void __launch_bounds__(BB) k_alloc(int nv, const int* vslot, const int* vrank,
                                              CellEntry* T, int* cursor) {
  let_next_start();
  wait_previous();
  const int v = blockIdx.x * BB + threadIdx.x, lane = threadIdx.x & 31;
  const int slot = v < nv ? vslot[v] : -1;
  const bool first = slot >= 0 && vrank[v] == 0;
  const int n = first ? T[slot].count : 0;
  int incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  int base = 0;
  if (lane == 31 && incl > 0) base = atomicAdd(cursor, incl);
  base = __shfl_sync(0xffffffffu, base, 31);
  if (first) T[slot].start = base + incl - n;
}
__global__ void __launch_bounds__(BB) k_scatter(int nv, const int* vslot, const int* vrank,
                                                const CellEntry* T, int* members) {
  let_next_start();
  wait_previous();
  const int v = blockIdx.x * BB + threadIdx.x;
  if (v >= nv) return;
  const int s = vslot[v];
  if (s >= 0) members[T[s].start + vrank[v]] = v;
}
// rank of each vertex among its cell's members (ascending vertex id).  early:
// the next kernel may start at once, and otherwise when these blocks have ended.
// Near rows that are rebuilt fill the GPU for long, and blocks that were placed
// while others held most of the SMs stay stacked on the few that were free
// (10,242 vertices, a rebuild with new rows: 130 us against 104; 163,842, one
// lane a vertex: 1,370 against 998).
__global__ void __launch_bounds__(BB) k_rank(int nv, const int* vslot, const CellEntry* T,
                                             const int* members, int* cell_verts,
                                             int* vrank, bool early) {
  if (early) let_next_start();
  wait_previous();
  const int v = blockIdx.x * BB + threadIdx.x;
  if (v >= nv) return;
  const int s = vslot[v];
  if (s < 0) return;
  const CellEntry c = T[s];
  int r = 0;
  for (int q = 0; q < c.count; ++q) r += members[c.start + q] < v ? 1 : 0;
  cell_verts[c.start + r] = v;
  vrank[v] = r;
}

// Position of the pair {v, u} in the reference's distance_matrix traversal
// (cell pairs in ascending first-cell id, neighbour offsets x-outer/z-inner,
// then the rank of the first-cell vertex, then of the second).
struct PairKey {
  long long icell;
  int off, ra, rb;
};
__device__ __forceinline__ PairKey pair_key(int v, int u, const long long* vcid, const int* vcoord,
                                            const int* vrank) {
  long long cv = vcid[v], cu = vcid[u];
  int a = v, b = u;
  if (cu < cv || (cu == cv && u < v)) {
    a = u;
    b = v;
  }
  PairKey k;
  k.icell = vcid[a];
  int dx = vcoord[3 * b] - vcoord[3 * a], dy = vcoord[3 * b + 1] - vcoord[3 * a + 1];
  int dz = vcoord[3 * b + 2] - vcoord[3 * a + 2];
  k.off = (dx + 1) * 9 + (dy + 1) * 3 + (dz + 1);
  k.ra = vrank[a];
  k.rb = vrank[b];
  return k;
}
__device__ __forceinline__ bool key_less(const PairKey& x, const PairKey& y) {
  if (x.icell != y.icell) return x.icell < y.icell;
  if (x.off != y.off) return x.off < y.off;
  if (x.ra != y.ra) return x.ra < y.ra;
  return x.rb < y.rb;
}

// order each Verlet row like the reference's push_back sequence
// (src/nlists/verlet_list.h:26-34)
__global__ void k_verlet_sort(int nv, const int* vrow, int* vcol, double* vd, const long long* vcid,
                              const int* vcoord, const int* vrank) {
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  int lo = vrow[v], hi = vrow[v + 1];
  for (int x = lo + 1; x < hi; ++x) {
    int u = vcol[x];
    double du = vd[x];
    PairKey ku = pair_key(v, u, vcid, vcoord, vrank);
    int y = x - 1;
    while (y >= lo && key_less(ku, pair_key(v, vcol[y], vcid, vcoord, vrank))) {
      vcol[y + 1] = vcol[y];
      vd[y + 1] = vd[y];
      --y;
    }
    vcol[y + 1] = u;
    vd[y + 1] = du;
  }
}

// Exclusion of the pairs of a build: with both rings in registers up to 60,000
// vertices (2,562 with exclusion 2 and 1.6 l: 419 us a Verlet build, 567 one
// vertex at a time), one vertex at a time above, where the GPU is full and the
// registers cost more (163,842: 1,262 and 1,264; exclusion 0 1,332 and 1,214;
// the distance matrix 701 and 665)
constexpr int SLIM_FROM = 60000;
template <bool SLIM>
__device__ __forceinline__ bool excluded_pair(const Topo& t, int excl, int a, int b) {
  return SLIM ? TableExclSlim{t, excl}(a, b) : excluded(t, excl, a, b);
}

// Pairs of the build-time cell neighbourhood of vertex a:
//   mode 0: Verlet build, all b != a, d <= rd        (both orders)
//   mode 1: distance_matrix of the cell list, each pair once with
//           (cid_b > cid_a) or (same cell and b > a), d <= rd
// pass 0 counts, pass 1 writes (d, i, j) at row offsets.
template <bool SLIM>
__global__ void k_cell_pairs(int nv, const double* P, NLView nl, Topo t, const int* vcoord, const long long* vcid,
                             double rd, int mode, int pass, int* cnt, const int* off, double* od, int* oi, int* oj) {
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= nv) return;
  d3 pa = ld3(P, a);
  long long ca = vcid[a];
  const NLGeom& G = *nl.geom;
  int n = 0;
  int base = pass ? off[a] : 0;
  for (int x = -1; x < 2; ++x) {
    int ii = vcoord[3 * a] + x;
    if (ii < 0 || ii >= G.shape[0]) continue;
    for (int y = -1; y < 2; ++y) {
      int jj = vcoord[3 * a + 1] + y;
      if (jj < 0 || jj >= G.shape[1]) continue;
      for (int z = -1; z < 2; ++z) {
        int kk = vcoord[3 * a + 2] + z;
        if (kk < 0 || kk >= G.shape[2]) continue;
        long long cid = ii * G.stride[0] + jj * G.stride[1] + kk * G.stride[2];
        if (mode == 1 && cid < ca) continue;
        int st = 0;
        int cnt_c = cell_lookup(nl, cid, &st);
        for (int q = 0; q < cnt_c; ++q) {
          int b = nl.cell_verts[st + q];
          if (b == a) continue;
          if (mode == 1 && cid == ca && b < a) continue;
          double dd = exact_dist(pa, ld3(P, b));
          if (!(dd <= rd)) continue;
          if (excluded_pair<SLIM>(t, nl.excl, a, b)) continue;
          if (pass) {
            od[base + n] = dd;
            if (mode == 0) {
              oj[base + n] = b;
            } else {
              oi[base + n] = a < b ? a : b;
              oj[base + n] = a < b ? b : a;
            }
          }
          ++n;
        }
      }
    }
  }
  if (!pass) cnt[a] = n;
}

// Verlet rows of a batch of replicas (src/nlists/verlet_list.h:18-35): the
// members of the 27 build-time neighbour cells of vertex a in its own
// replica's grid (replica-tagged cell keys) closer than that replica's
// cut-off rlist[rep], not excluded at that replica's level; padding
// vertices have empty rows.  pass 0 counts, pass 1 writes (then ordered by
// k_verlet_sort like the single-mesh rows).
template <bool SLIM>
__global__ void k_verlet_batch(int nv, const double* P, NLView nl, Topo t, const int* vcoord,
                               const double* __restrict__ rlist, int pass, int* cnt, const int* off, double* od,
                               int* oj) {
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= nv) return;
  const int rep = rep_of(nl, a);
  if (rep < 0) {
    if (!pass) cnt[a] = 0;
    return;
  }
  const NLGeom& G = nl.geom[rep];
  const double rd = rlist[rep];
  const int excl = excl_of(nl, a);
  const d3 pa = ld3(P, a);
  int n = 0;
  int base = pass ? off[a] : 0;
  for (int x = -1; x < 2; ++x) {
    int ii = vcoord[3 * a] + x;
    if (ii < 0 || ii >= G.shape[0]) continue;
    for (int y = -1; y < 2; ++y) {
      int jj = vcoord[3 * a + 1] + y;
      if (jj < 0 || jj >= G.shape[1]) continue;
      for (int z = -1; z < 2; ++z) {
        int kk = vcoord[3 * a + 2] + z;
        if (kk < 0 || kk >= G.shape[2]) continue;
        long long cid = ii * G.stride[0] + jj * G.stride[1] + kk * G.stride[2];
        int st = 0;
        int c = cell_lookup(nl, cell_key(cid, rep), &st);
        for (int q = 0; q < c; ++q) {
          int b = nl.cell_verts[st + q];
          if (b == a) continue;
          double dd = exact_dist(pa, ld3(P, b));
          if (!(dd <= rd)) continue;
          if (excluded_pair<SLIM>(t, excl, a, b)) continue;
          if (pass) {
            od[base + n] = dd;
            oj[base + n] = b;
          }
          ++n;
        }
      }
    }
  }
  if (!pass) cnt[a] = n;
}

// candidate rows: members of the 27 build-time neighbour cells of vertex a in
// the reference's scan order (x outer, z inner; members ascending), self
// excluded.  pass 0 counts, pass 1 writes.  Eight lanes look up consecutive
// cells of the scan and place their members by a prefix of the counts (one
// thread through 27 dependent hash probes took 81 us at 218,000 vertices).
__global__ void __launch_bounds__(256) k_cand(int nv, NLView nl, const int* vcoord, int pass, int* cnt,
                                              const int* off, int* out) {
  constexpr int L = 8;
  const int a = (blockIdx.x * 256 + threadIdx.x) / L, sub = threadIdx.x % L;
  const unsigned gmask = ((1u << L) - 1u) << (threadIdx.x & 31 & ~(L - 1));
  if (a >= nv) return;
  const int rep = rep_of(nl, a);
  if (rep < 0) {
    if (!pass && sub == 0) cnt[a] = 0;
    return;
  }
  const NLGeom& G = nl.geom[rep];
  const int ci = vcoord[3 * a], cj = vcoord[3 * a + 1], ck = vcoord[3 * a + 2];
  // The vertex itself is in the cell with its own id: the middle one, or, for a
  // vertex on the upper face of a box so wide that the margin of its sides is
  // lost in rounding, the one that the id past the side wraps to
  const bool inside = ci >= 0 && ci < G.shape[0] && cj >= 0 && cj < G.shape[1] && ck >= 0 && ck < G.shape[2];
  const long long home = inside ? 0 : ci * G.stride[0] + cj * G.stride[1] + ck * G.stride[2];
  int n = pass ? off[a] : 0;
  for (int c0 = 0; c0 < 27; c0 += L) {
    const int c = c0 + sub;
    const int ii = ci + c / 9 - 1, jj = cj + (c / 3) % 3 - 1, kk = ck + c % 3 - 1;
    int st = 0, m = 0;
    bool self = false;
    if (c < 27 && ii >= 0 && ii < G.shape[0] && jj >= 0 && jj < G.shape[1] && kk >= 0 && kk < G.shape[2]) {
      const long long id = ii * G.stride[0] + jj * G.stride[1] + kk * G.stride[2];
      m = cell_lookup(nl, cell_key(id, rep), &st);
      self = inside ? c == 13 : id == home;
    }
    const int own = m - (self && m > 0 ? 1 : 0);
    int incl = own;
#pragma unroll
    for (int o = 1; o < L; o <<= 1) {
      const int y = __shfl_up_sync(gmask, incl, o, L);
      if (sub >= o) incl += y;
    }
    if (pass) {
      int w = n + incl - own;
      for (int q = 0; q < m; ++q) {
        const int b = nl.cell_verts[st + q];
        if (b != a) out[w++] = b;
      }
    }
    n += __shfl_sync(gmask, incl, L - 1, L);
  }
  if (!pass && sub == 0) cnt[a] = n;
}

// Near rows (rebuilt only when flagged stale): the vertices closer than rn
// to each vertex (squared threshold rn2, rounded up), found through the cell
// table (the cells that meet the ball of radius rn), with a flag for pairs
// excluded on the current topology.  A row longer than TM_NEAR_CAP marks the
// rows unusable (flag[3]).
// With eight lanes a vertex (NLN) each looks up every eighth of the up to 343
// cells around the ball (most are empty, so the time is the chain of hash
// probes) and walks the rings of every eighth ring vertex for the exclusion
// flags; one lane a vertex runs the chain but works out whole planes and lines
// of cells to be too far at once.  A row's order does not matter to its
// readers, which visit accepted pairs by their cell and id; it is the same from
// run to run.
constexpr int NB = 128;   // threads per block of k_near
constexpr int NEAR_BLOCKS = 8 * 152;  // resident blocks of eight lanes a vertex, looping over the vertices
template <int NLN>
__global__ void __launch_bounds__(NB) k_near(int nv, const double* __restrict__ P, NLView nl, Topo t, int excl,
                                             double rn, double rn2, int* flag, const int* dtopo, int* ncnt,
                                             int* nent, double* xb, const EP* eps) {
  __shared__ int srow[NB / NLN][TM_NEAR_CAP + 1];  // (an odd pitch: no bank conflicts)
  let_next_start();
  wait_previous();
  if (flag[1] == 0) return;  // rows still valid
  const int sub = threadIdx.x % NLN, lane = threadIdx.x & 31;
  const unsigned gmask = ((1u << NLN) - 1u) << (lane & ~(NLN - 1)), below = (1u << lane) - 1u;
  int* row = srow[threadIdx.x / NLN];
  for (int a = (blockIdx.x * NB + threadIdx.x) / NLN; a < nv; a += gridDim.x * (NB / NLN)) {
    const int rep = rep_of(nl, a);
    if (rep < 0) {  // padding vertex of a batch
      if (sub == 0) ncnt[a] = 0;
      continue;
    }
    if (eps) {  // batch: the replica's cut-off
      rn = 2.0 * eps[rep].rlc1;
      rn2 = rn * rn * (1.0 + 1e-12);
    }
    const NLGeom& G = nl.geom[rep];
    const d3 pa = ld3(P, a);
    const double* pp = &pa.x;
    int lo[3], hi[3];
    // position in cell units (float) for the box-distance pruning; a cell is
    // skipped only when it is farther than rn after every axis distance is
    // shortened by 1e-3 cell widths plus 8 float ulps of the coordinate, far
    // above the float rounding of the cell coordinate
    float u[3], rlf[3], mg[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      lo[k] = max(0, (int)floor((pp[k] - rn - G.bmin[k]) * G.inv_rl[k]) - 1);
      hi[k] = min(G.shape[k] - 1, (int)floor((pp[k] + rn - G.bmin[k]) * G.inv_rl[k]) + 1);
      u[k] = (float)((pp[k] - G.bmin[k]) * G.inv_rl[k]);
      rlf[k] = (float)G.rl[k];
      mg[k] = 1e-3f + 9.6e-7f * fabsf(u[k]);
    }
    const float rnf2 = (float)rn2 * 1.0001f;
    // distance of the ball's centre from a plane of cells, cell c along axis k
    auto away = [&](int k, int c) {
      return fmaxf(fmaxf((float)c - u[k], u[k] - (float)(c + 1)) - mg[k], 0.0f) * rlf[k];
    };
    auto lookup = [&](int ii, int jj, int kk, int* st) {
      return cell_lookup(nl, cell_key(ii * G.stride[0] + jj * G.stride[1] + kk * G.stride[2], rep), st);
    };
    auto near = [&](int b) {
      const d3 pb = ld3(P, b);
      const double ex = pa.x - pb.x, ey = pa.y - pb.y, ez = pa.z - pb.z;
      return b != a && !(ex * ex + ey * ey + ez * ez >= rn2);
    };
    int n = 0;
    if constexpr (NLN == 1) {
      for (int ii = lo[0]; ii <= hi[0]; ++ii) {
        const float dx = away(0, ii);
        for (int jj = lo[1]; jj <= hi[1]; ++jj) {
          const float dy = away(1, jj), gxy = dx * dx + dy * dy;
          if (gxy > rnf2) continue;
          for (int kk = lo[2]; kk <= hi[2]; ++kk) {
            const float dz = away(2, kk);
            if (gxy + dz * dz > rnf2) continue;
            int st = 0;
            const int cnt = lookup(ii, jj, kk, &st);
            for (int q = 0; q < cnt; ++q) {
              const int b = nl.cell_verts[st + q];
              if (!near(b)) continue;
              if (n < TM_NEAR_CAP) row[n] = b;
              ++n;
            }
          }
        }
      }
    } else {
      const int ny = hi[1] - lo[1] + 1, nz = hi[2] - lo[2] + 1;
      const int ncell = hi[0] >= lo[0] && ny > 0 && nz > 0 ? (hi[0] - lo[0] + 1) * ny * nz : 0;
      for (int c0 = 0; c0 < ncell; c0 += NLN) {
        const int c = c0 + sub;
        int cnt = 0, st = 0;
        if (c < ncell) {
          const int kk = lo[2] + c % nz, ij = c / nz;
          const int jj = lo[1] + ij % ny, ii = lo[0] + ij / ny;
          const float dx = away(0, ii), dy = away(1, jj), dz = away(2, kk);
          if (!(dx * dx + dy * dy + dz * dz > rnf2)) cnt = lookup(ii, jj, kk, &st);
        }
        for (int q = 0; __any_sync(gmask, q < cnt); ++q) {
          const int b = q < cnt ? nl.cell_verts[st + q] : a;
          const bool acc = q < cnt && near(b);
          const unsigned bal = __ballot_sync(gmask, acc);
          const int pos = n + __popc(bal & below);
          if (acc && pos < TM_NEAR_CAP) row[pos] = b;
          n += __popc(bal);
        }
      }
    }
    if (sub == 0 && n > TM_NEAR_CAP) atomicOr(&flag[3], 1);
    n = min(n, TM_NEAR_CAP);
    __syncwarp(gmask);
    // exclusion flags: an entry is excluded when it is in the
    // ring of a or, at level 2, in the ring of a ring vertex of a; the rings
    // are walked once and their vertices looked up in the row
    const int level = nl.rexcl ? nl.rexcl[rep] : excl;  // batch: the replica's level
    if (level > 0 && n > 0) {
      const int d = t.val[a];
      auto mark = [&](int w) {
        for (int e = 0; e < n; ++e)
          if ((row[e] & 0x7fffffff) == w) {
            if constexpr (NLN == 1)
              row[e] |= (int)0x80000000u;
            else
              atomicOr(&row[e], (int)0x80000000u);
          }
      };
      for (int m = sub; m < d; m += NLN) {
        const int w = t.nbr[(size_t)m * t.nv + a];
        mark(w);
        if (level > 1) {
          const int dw = t.val[w];
          for (int q = 0; q < dw; ++q) mark(t.nbr[(size_t)q * t.nv + w]);
        }
      }
      __syncwarp(gmask);
    }
    int* out = nent + (size_t)a * TM_NEAR_CAP;
    for (int e = sub; e < n; e += NLN) out[e] = row[e];
    if (sub == 0) ncnt[a] = n;
    if constexpr (NLN == 1)
      st3(xb, a, pa);
    else if (sub < 3)
      xb[3 * (size_t)a + sub] = pp[sub];
    __syncwarp(gmask);  // the row is reused
  }
  // the last block (it follows every block's reads of the flag): usable
  // unless a row overflowed; record the topology version
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&flag[4], 1) == (int)gridDim.x - 1) {
      flag[1] = atomicExch(&flag[3], 0);
      flag[2] = *dtopo;
      flag[4] = 0;
    }
  }
}

// distance_matrix of the Verlet list: rows in vertex order, d < rd
__global__ void k_verlet_dm(int nv, const double* P, const int* vrow, const int* vcol, double rd, int pass, int* cnt,
                            const int* off, double* od, int* oi, int* oj) {
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= nv) return;
  d3 pa = ld3(P, a);
  int n = 0;
  int base = pass ? off[a] : 0;
  for (int q = vrow[a]; q < vrow[a + 1]; ++q) {
    int b = vcol[q];
    double dd = exact_dist(pa, ld3(P, b));
    if (dd < rd) {
      if (pass) {
        od[base + n] = dd;
        oi[base + n] = a;
        oj[base + n] = b;
      }
      ++n;
    }
  }
  if (!pass) cnt[a] = n;
}

// point_distances for one vertex (single thread; API use only)
__global__ void k_point(int pid, const double* P, NLView nl, Topo t, double rd, int pass, int* count, double* od,
                        int* oj) {
  if (threadIdx.x || blockIdx.x) return;
  d3 p = ld3(P, pid);
  int n = 0;
  if (nl.kind == 0) {
    const NLGeom& G = *nl.geom;
    int co[3];
    const double* pp = &p.x;
    for (int k = 0; k < 3; ++k) co[k] = (int)__ddiv_rn(__dsub_rn(pp[k], G.bmin[k]), G.rl[k]);
    for (int a = -1; a < 2; ++a) {
      int ii = co[0] + a;
      if (ii < 0 || ii >= G.shape[0]) continue;
      for (int b = -1; b < 2; ++b) {
        int jj = co[1] + b;
        if (jj < 0 || jj >= G.shape[1]) continue;
        for (int c = -1; c < 2; ++c) {
          int kk = co[2] + c;
          if (kk < 0 || kk >= G.shape[2]) continue;
          long long cid = ii * G.stride[0] + jj * G.stride[1] + kk * G.stride[2];
          int st = 0;
          int cc = cell_lookup(nl, cid, &st);
          for (int q = 0; q < cc; ++q) {
            int j = nl.cell_verts[st + q];
            if (j == pid) continue;
            if (excluded(t, nl.excl, pid, j)) continue;
            d3 pj = ld3(P, j);
            if (exact_dist(p, pj) < rd) {
              if (pass) {
                st3(od, n, exact_diff(p, pj));
                oj[n] = j;
              }
              ++n;
            }
          }
        }
      }
    }
  } else {
    for (int q = nl.vrow[pid]; q < nl.vrow[pid + 1]; ++q) {
      int j = nl.vcol[q];
      d3 pj = ld3(P, j);
      if (exact_dist(p, pj) < rd) {
        if (pass) {
          st3(od, n, exact_diff(p, pj));
          oj[n] = j;
        }
        ++n;
      }
    }
  }
  if (!pass) *count = n;
}

inline int nblk(long n, int b) { return (int)((n + b - 1) / b); }

}  // namespace

// What a build needs beside the mesh: one box (rlist) or one per replica of
// a batch (vrep in the view, rblocks, rlists)
struct BoxInput {
  double rlist;
  const int2* rblocks;
  const double* rlists;
  int boxes;
};

// The cell list (header comment) and the candidate rows, shared by single
// meshes and batches; V.vrep is set by the caller.  near: test the near
// rows' skin on the side.
static void build_cells(tm_nlist* nl, NLView& V, int nv, const double* P, const BoxInput& in, const NearCheck& near,
                        cudaStream_t s, bool candidates) {
  // hash table of the non-empty cells: 2x the vertex count, power of two
  size_t tsize = 64;
  while (tsize < 2 * (size_t)std::max(nv, 1)) tsize <<= 1;
  nl->table.ensure(tsize);
  V.tmask = tsize - 1;
  nl->vcid.ensure(std::max(nv, 1));
  nl->vcoord.ensure(3 * (size_t)std::max(nv, 1));
  nl->vslot.ensure(std::max(nv, 1));
  nl->vrank.ensure(std::max(nv, 1));
  nl->fill.ensure((size_t)std::max(nv, 1));
  nl->cell_verts.ensure(std::max(nv, 1));
  nl->d_count.ensure(4);
  const int vb = std::max(1, nblk(nv, BB));
  const int nb = V.vrep ? vb : std::min(NBOX, vb);
  nl->bbox.ensure(6 * (size_t)nb);
  nl->geom.ensure(in.boxes);
  V.geom = nl->geom.get();
  V.table = nl->table.get();
  V.cell_verts = nl->cell_verts.get();
  V.bcoord = nl->vcoord.get();  // build-time cell of every vertex
  int* status = nl->d_count.get();
  int* cursor = status + 1;
  k_box<<<nb, BB, 0, s>>>(nv, P, V.vrep, nl->bbox.get(), nl->table.get(), tsize, cursor, near);
  TM_LAUNCH();
  launch_after(k_insert, vb, BB, s, nv, P, V, nl->table.get(), nl->bbox.get(), nb, in.rblocks, in.rlist, in.rlists,
               nl->geom.get(), nl->vcid.get(), nl->vcoord.get(), nl->vslot.get(), nl->vrank.get(), status);
  launch_after(k_alloc, vb, BB, s, nv, nl->vslot.get(), nl->vrank.get(), nl->table.get(), cursor);
  launch_after(k_scatter, vb, BB, s, nv, nl->vslot.get(), nl->vrank.get(), nl->table.get(), nl->fill.get());
  launch_after(k_rank, vb, BB, s, nv, nl->vslot.get(), nl->table.get(), nl->fill.get(), nl->cell_verts.get(),
               nl->vrank.get(), nblk(8L * nv, NB) <= NEAR_BLOCKS / 8);
  if (candidates && nv > 0) {
    // candidate rows for the queries of points that stay in their build cell
    nl->crow.ensure((size_t)nv + 1);
    nl->cnt.ensure((size_t)nv + 1);
    k_cand<<<nblk(8L * nv, 256), 256, 0, s>>>(nv, V, nl->vcoord.get(), 0, nl->cnt.get(), nullptr, nullptr);
    TM_LAUNCH();
    TM_CUDA(cudaMemsetAsync(nl->cnt.get() + nv, 0, sizeof(int), s));
    int total = 0;
    exclusive_scan_int(nl->cnt.get(), nl->crow.get(), nv + 1, &total, nl->tmp, s);
    // rows are only kept while they stay small (coarse grids fall back to the
    // cell table)
    if ((long long)total <= 64LL * nv) {
      nl->ccol.ensure(std::max(total, 1));
      k_cand<<<nblk(8L * nv, 256), 256, 0, s>>>(nv, V, nl->vcoord.get(), 1, nullptr, nl->crow.get(), nl->ccol.get());
      TM_LAUNCH();
      V.crow = nl->crow.get();
      V.ccol = nl->ccol.get();
    }
  }
}

// Near rows for repulsion queries at cut-off lc1 (skin lc1/2).  A pair
// closer than lc1 at query time whose vertices both moved less than lc1/2
// since the rows were built was closer than 2 lc1 then, so the row holds
// every neighbour the query can accept; the query keeps the ones whose
// build-time cell of the current cell list is among the 27 around its own
// current cell and visits them in the reference's order.  The rows do not
// depend on the cell list, so a cell-list rebuild rebuilds them only when a
// vertex has moved lc1/2 since they were built (decided on the device).
static NearCheck prepare_near(tm_nlist* nl, int nv, double lc1, cudaStream_t s, const EP* eps = nullptr) {
  if (nl->near_nv != nv || nl->near_lc1 != lc1) {
    nl->nent.ensure((size_t)nv * TM_NEAR_CAP);
    nl->ncnt.ensure(nv);
    nl->xb.ensure(3 * (size_t)nv);
    nl->nflag.ensure(5);
    int init[5] = {0, 1, 0, 0, 0};  // stale until built
    TM_CUDA(cudaMemcpyAsync(nl->nflag.get(), init, sizeof(init), cudaMemcpyHostToDevice, s));
    TM_CUDA(cudaStreamSynchronize(s));
    nl->near_nv = nv;
    nl->near_lc1 = lc1;
    nl->near_move2 = 0.25 * lc1 * lc1 * (1.0 - 1e-12);
  }
  return NearCheck{nl->xb.get(), nl->near_move2, nl->nflag.get(), eps};
}
// after build_cells with the check of prepare_near
static void refresh_near(tm_nlist* nl, tm_mesh* m, NLView& V, const double* P, double lc1, cudaStream_t s,
                         const EP* eps = nullptr) {
  const int nv = nl->nv;
  const double rn = 2.0 * lc1;
  int* flag = nl->nflag.get();
  // A rebuild with new rows, us, of one / eight lanes a vertex at 10,242, 40,962,
  // 51,842, 81,002 and 163,842 vertices: 0.8 l, exclusion 2: 292/105, 319/241,
  // 325/277, 302/367, 510/677; 2.2 l, exclusion 0: 745/252, 843/672, 677/821,
  // 893/1,242, 1,416/2,325
  const bool eight = nv <= 45000;
  launch_after(eight ? k_near<8> : k_near<1>, eight ? std::min(NEAR_BLOCKS, nblk(8L * nv, NB)) : nblk(nv, NB), NB, s, nv,
               P, V, m->topo(), V.excl, rn, rn * rn * (1.0 + 1e-12), flag, m->d_topo_ver.get(), nl->ncnt.get(),
               nl->nent.get(), nl->xb.get(), eps);
  V.nent = nl->nent.get();
  V.ncnt = nl->ncnt.get();
  V.nflag = flag;
  V.dtopo = m->d_topo_ver.get();
}

void nlist_make(tm_nlist* nl, tm_mesh* m, const tm_params& p, const double* P, cudaStream_t s) {
  if (p.n_search != 0 && p.n_search != 1) fail(TM_ERR_ARG, "Unknown neighbour search algorithm.");
  if (p.exclusion_level < 0 || p.exclusion_level > 2) fail(TM_ERR_ARG, "Unsupported exclusion level");
  nl->prm = p;
  nl->built_topo = m->topo_version;
  nl->vtotal = 0;
  int nv = m->nv;
  nl->nv = nv;
  NLView& V = nl->view;
  V = NLView{};
  V.kind = 0;
  V.excl = p.exclusion_level;
  // with near rows the candidate rows are not needed: the rare fallback
  // (a vertex moved lc1/2 since the rows were built) takes the cell walk
  const bool near = p.n_search == 0 && p.rep_lc1 > 0 && p.rlist >= p.rep_lc1 && nv > 0;
  NearCheck nc{};
  if (near) nc = prepare_near(nl, nv, p.rep_lc1, s);
  build_cells(nl, V, nv, P, BoxInput{p.rlist, nullptr, nullptr, 1}, nc, s, p.n_search == 0 && !near);
  if (near) refresh_near(nl, m, V, P, p.rep_lc1, s);
  if (p.n_search == 1) {
    // Verlet CSR from the cell list at cut-off rlist, rows in the reference's
    // insertion order
    nl->vrow.ensure((size_t)nv + 1);
    Topo t = m->topo();
    int total = 0;
    if (nv > 0) {
      nl->cnt.ensure((size_t)nv + 1);
      auto* pairs = nv > SLIM_FROM ? k_cell_pairs<true> : k_cell_pairs<false>;
      pairs<<<nblk(nv, 256), 256, 0, s>>>(nv, P, V, t, nl->vcoord.get(), nl->vcid.get(), p.rlist, 0, 0, nl->cnt.get(),
                                          nullptr, nullptr, nullptr, nullptr);
      TM_LAUNCH();
      TM_CUDA(cudaMemsetAsync(nl->cnt.get() + nv, 0, sizeof(int), s));
      exclusive_scan_int(nl->cnt.get(), nl->vrow.get(), nv + 1, &total, nl->tmp, s);
      nl->vcol.ensure(std::max(total, 1));
      nl->vtotal = total;
      nl->d_res.ensure(std::max(total, 1));
      pairs<<<nblk(nv, 256), 256, 0, s>>>(nv, P, V, t, nl->vcoord.get(), nl->vcid.get(), p.rlist, 0, 1, nullptr,
                                          nl->vrow.get(), nl->d_res.get(), nullptr, nl->vcol.get());
      TM_LAUNCH();
      k_verlet_sort<<<nblk(nv, 128), 128, 0, s>>>(nv, nl->vrow.get(), nl->vcol.get(), nl->d_res.get(),
                                                  nl->vcid.get(), nl->vcoord.get(), nl->vrank.get());
      TM_LAUNCH();
    } else {
      TM_CUDA(cudaMemsetAsync(nl->vrow.get(), 0, sizeof(int), s));
      nl->vcol.ensure(1);
    }
    V.kind = 1;
    V.vrow = nl->vrow.get();
    V.vcol = nl->vcol.get();
  }
}

void nlist_make_batch(tm_nlist* nl, tm_mesh* m, int R, const int* d_vrep, const int2* d_rblocks,
                      const double* d_rlist, int excl, const int* d_rexcl, const double* P, cudaStream_t s,
                      const EP* d_eps, bool near, bool verlet) {
  if (excl < 0 || excl > 2) fail(TM_ERR_ARG, "Unsupported exclusion level");
  int nv = m->nv;
  nl->nv = nv;
  nl->built_topo = m->topo_version;
  nl->vtotal = 0;
  nl->prm.n_search = verlet ? 1 : 0;
  nl->prm.exclusion_level = excl;
  NLView& V = nl->view;
  V = NLView{};
  V.kind = 0;
  V.excl = excl;
  V.rexcl = d_rexcl;
  V.vrep = d_vrep;
  const BoxInput in{0.0, d_rblocks, d_rlist, R};
  if (verlet) {
    // Verlet rows at each replica's cut-off, ordered like the single-mesh
    // rows (the reference's insertion order)
    build_cells(nl, V, nv, P, in, NearCheck{}, s, false);
    nl->vrow.ensure((size_t)nv + 1);
    Topo t = m->topo();
    int total = 0;
    if (nv > 0) {
      nl->cnt.ensure((size_t)nv + 1);
      auto* rows = nv > SLIM_FROM ? k_verlet_batch<true> : k_verlet_batch<false>;
      rows<<<nblk(nv, 256), 256, 0, s>>>(nv, P, V, t, nl->vcoord.get(), d_rlist, 0, nl->cnt.get(), nullptr, nullptr,
                                         nullptr);
      TM_LAUNCH();
      TM_CUDA(cudaMemsetAsync(nl->cnt.get() + nv, 0, sizeof(int), s));
      exclusive_scan_int(nl->cnt.get(), nl->vrow.get(), nv + 1, &total, nl->tmp, s);
      nl->vcol.ensure(std::max(total, 1));
      nl->vtotal = total;
      nl->d_res.ensure(std::max(total, 1));
      rows<<<nblk(nv, 256), 256, 0, s>>>(nv, P, V, t, nl->vcoord.get(), d_rlist, 1, nullptr, nl->vrow.get(),
                                         nl->d_res.get(), nl->vcol.get());
      TM_LAUNCH();
      k_verlet_sort<<<nblk(nv, 128), 128, 0, s>>>(nv, nl->vrow.get(), nl->vcol.get(), nl->d_res.get(),
                                                  nl->vcid.get(), nl->vcoord.get(), nl->vrank.get());
      TM_LAUNCH();
    } else {
      TM_CUDA(cudaMemsetAsync(nl->vrow.get(), 0, sizeof(int), s));
      nl->vcol.ensure(1);
    }
    V.kind = 1;
    V.vrow = nl->vrow.get();
    V.vcol = nl->vcol.get();
    return;
  }
  // candidate rows as well: unrelaxed replicas can move a skin's width
  // within a few steps, and then the candidate rows keep most vertices off
  // the cell walk
  // near rows with each replica's cut-off (the lc1 argument only tags the
  // rows: any positive value)
  NearCheck nc{};
  if (near && nv > 0) nc = prepare_near(nl, nv, 1.0, s, d_eps);
  build_cells(nl, V, nv, P, in, nc, s, true);
  if (near && nv > 0) refresh_near(nl, m, V, P, 1.0, s, d_eps);
}

int64_t nlist_distance_matrix(tm_nlist* nl, tm_mesh* m, const double* P, double rd, cudaStream_t s) {
  int nv = m->nv;
  nl->res_d.clear();
  nl->res_i.clear();
  nl->res_j.clear();
  if (nv == 0) return 0;
  if (nv != nl->nv) fail(TM_ERR_ARG, "mesh does not match the neighbour list");
  nl->cnt.ensure((size_t)nv + 1);
  nl->fill.ensure((size_t)nv + 1);
  Topo t = m->topo();
  int total = 0;
  auto* pairs = nv > SLIM_FROM ? k_cell_pairs<true> : k_cell_pairs<false>;
  if (nl->view.kind == 0)
    pairs<<<nblk(nv, 256), 256, 0, s>>>(nv, P, nl->view, t, nl->vcoord.get(), nl->vcid.get(), rd, 1, 0, nl->cnt.get(),
                                        nullptr, nullptr, nullptr, nullptr);
  else
    k_verlet_dm<<<nblk(nv, 256), 256, 0, s>>>(nv, P, nl->vrow.get(), nl->vcol.get(), rd, 0, nl->cnt.get(), nullptr,
                                              nullptr, nullptr, nullptr);
  TM_LAUNCH();
  TM_CUDA(cudaMemsetAsync(nl->cnt.get() + nv, 0, sizeof(int), s));
  exclusive_scan_int(nl->cnt.get(), nl->fill.get(), nv + 1, &total, nl->tmp, s);
  nl->d_res.ensure(std::max(total, 1));
  nl->d_resi.ensure(std::max(total, 1));
  nl->d_resj.ensure(std::max(total, 1));
  if (nl->view.kind == 0)
    pairs<<<nblk(nv, 256), 256, 0, s>>>(nv, P, nl->view, t, nl->vcoord.get(), nl->vcid.get(), rd, 1, 1, nullptr,
                                        nl->fill.get(), nl->d_res.get(), nl->d_resi.get(), nl->d_resj.get());
  else
    k_verlet_dm<<<nblk(nv, 256), 256, 0, s>>>(nv, P, nl->vrow.get(), nl->vcol.get(), rd, 1, nullptr, nl->fill.get(),
                                              nl->d_res.get(), nl->d_resi.get(), nl->d_resj.get());
  TM_LAUNCH();
  nl->res_d.resize(total);
  nl->res_i.resize(total);
  nl->res_j.resize(total);
  if (total) {
    TM_CUDA(cudaMemcpyAsync(nl->res_d.data(), nl->d_res.get(), sizeof(double) * total, cudaMemcpyDeviceToHost, s));
    TM_CUDA(cudaMemcpyAsync(nl->res_i.data(), nl->d_resi.get(), sizeof(int) * total, cudaMemcpyDeviceToHost, s));
    TM_CUDA(cudaMemcpyAsync(nl->res_j.data(), nl->d_resj.get(), sizeof(int) * total, cudaMemcpyDeviceToHost, s));
  }
  TM_CUDA(cudaStreamSynchronize(s));
  return total;
}

int64_t nlist_point_distances(tm_nlist* nl, tm_mesh* m, const double* P, int pid, double rd, cudaStream_t s) {
  nl->res_d.clear();
  nl->res_i.clear();
  nl->res_j.clear();
  if (pid < 0 || pid >= m->nv) fail(TM_ERR_ARG, "pid out of range");
  if (m->nv != nl->nv) fail(TM_ERR_ARG, "mesh does not match the neighbour list");
  Topo t = m->topo();
  nl->d_count.ensure(4);
  k_point<<<1, 1, 0, s>>>(pid, P, nl->view, t, rd, 0, nl->d_count.get(), nullptr, nullptr);
  TM_LAUNCH();
  int n = 0;
  TM_CUDA(cudaMemcpyAsync(&n, nl->d_count.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
  TM_CUDA(cudaStreamSynchronize(s));
  nl->d_res.ensure(3 * (size_t)std::max(n, 1));
  nl->d_resj.ensure(std::max(n, 1));
  k_point<<<1, 1, 0, s>>>(pid, P, nl->view, t, rd, 1, nullptr, nl->d_res.get(), nl->d_resj.get());
  TM_LAUNCH();
  nl->res_d.resize(3 * (size_t)n);
  nl->res_j.resize(n);
  if (n) {
    TM_CUDA(cudaMemcpyAsync(nl->res_d.data(), nl->d_res.get(), sizeof(double) * 3 * n, cudaMemcpyDeviceToHost, s));
    TM_CUDA(cudaMemcpyAsync(nl->res_j.data(), nl->d_resj.get(), sizeof(int) * n, cudaMemcpyDeviceToHost, s));
  }
  TM_CUDA(cudaStreamSynchronize(s));
  return n;
}

}  // namespace tmg

// --------------------------------------------------------------------------
// C ABI
// --------------------------------------------------------------------------


extern "C" {

int tm_nlist_create(tm_mesh* m, const tm_params* p, tm_nlist** out) {
  TM_API_BEGIN
  if (!m || !p || !out) fail(TM_ERR_ARG, "NULL argument");
  *out = nullptr;
  std::unique_ptr<tm_nlist> nl(new tm_nlist());
  m->upload_points(m->stream);
  tmg::nlist_make(nl.get(), m, *p, m->d_pts.get(), m->stream);
  TM_CUDA(cudaStreamSynchronize(m->stream));
  *out = nl.release();
  TM_API_END
}

int tm_nlist_destroy(tm_nlist* nl) {
  delete nl;
  return TM_OK;
}

int tm_nlist_distance_matrix(tm_nlist* nl, tm_mesh* m, double rdist, int64_t* count) {
  TM_API_BEGIN
  if (!nl || !m || !count) fail(TM_ERR_ARG, "NULL argument");
  m->upload_points(m->stream);
  *count = tmg::nlist_distance_matrix(nl, m, m->d_pts.get(), rdist, m->stream);
  TM_API_END
}

int tm_nlist_point_distances(tm_nlist* nl, tm_mesh* m, int64_t pid, double rdist, int64_t* count) {
  TM_API_BEGIN
  if (!nl || !m || !count) fail(TM_ERR_ARG, "NULL argument");
  m->upload_points(m->stream);
  *count = tmg::nlist_point_distances(nl, m, m->d_pts.get(), (int)pid, rdist, m->stream);
  TM_API_END
}

int tm_nlist_fetch(tm_nlist* nl, double* d, int32_t* i, int32_t* j) {
  if (!nl) return TM_ERR_ARG;
  if (d && !nl->res_d.empty()) std::memcpy(d, nl->res_d.data(), sizeof(double) * nl->res_d.size());
  if (i && !nl->res_i.empty()) std::memcpy(i, nl->res_i.data(), sizeof(int) * nl->res_i.size());
  if (j && !nl->res_j.empty()) std::memcpy(j, nl->res_j.data(), sizeof(int) * nl->res_j.size());
  return TM_OK;
}

}  // extern "C"
