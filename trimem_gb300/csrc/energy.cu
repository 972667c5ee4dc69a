// Energy manager: vertex properties, penalty assembly and gradient.
//
// The reference evaluates, per vertex, every incident face and edge again
// (src/mesh_properties.cpp:12-148), i.e. each face three times and each edge
// two to four times per pass, with acos/tan per call.  On GB300 (FP64 issue
// rate ~1/58 of FP32) the kernels instead compute each face and each edge once
// per evaluation and gather them per vertex:
//
//   k_face   (one thread per face)  unit normal, area, signed volume and the
//            cotangents of the three corners (u.v / |u x v|, no acos/tan)
//   k_edge   (one thread per edge)  length, signed dihedral angle, tether
//            bond value and derivative
//   k_vertex (one thread per vertex) area/volume/curvature/tether sums of
//            the ring, bending 2c^2/a, repulsion (and its gradient), a
//            fixed-order block reduction of the six global sums; the last
//            block reduces the block partials in fixed order and assembles
//            energy and the penalty gradient factors on the device
//   k_grad   (one thread per vertex) gather of dE/dx_i over the ring
//
// No atomics touch floating-point data, so every result is bit-reproducible.
// With w_e = gC/2 + kb (rho_i + rho_j) (rho = curvature/area per vertex) the
// gradient is
//   sum_f [gA - 2/3 kb (rho_a^2+rho_b^2+rho_c^2) (+ kt dpen)] dA_f
//   + gV dV_f + sum_e (w_e theta_e + kt dbond_e) dl_e + w_e l_e dtheta_e
//   + kr drep,
// which is the reference's gather (src/mesh_properties.cpp:51-148 with
// src/kernel.h:124-137) regrouped per face and edge.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "tm_internal.h"
#include "tm_math.cuh"
#include "tm_energy.cuh"

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

// ---- per-face and per-edge quantities ------------------------------------
// Sign tests and absolute values as integer operations on the bits (no
// FP64 compare or absolute value: FP64 is GB300's scarce pipe).  For
// non-negative doubles the bit patterns order like the values, so a length
// l >= 0 is compared with a threshold by its bits (NaN lengths compare as
// above every threshold).
__device__ __forceinline__ double abs_bits(double x) {
  return __longlong_as_double(__double_as_longlong(x) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ bool len_below(double l, double c) {
  return __double_as_longlong(l) < __double_as_longlong(c);
}
__device__ __forceinline__ bool len_above(double l, double c) {
  return __double_as_longlong(l) > __double_as_longlong(c);
}
// fav: (area, volume) of each face again, compact, for k_vertex's gathers
__global__ void k_face(Topo t, const double* __restrict__ P, FaceD* __restrict__ fd, float* __restrict__ P32,
                       double2* __restrict__ fav) {
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  // the float copy of the positions used by the neighbour prefilter
  for (int v = f; v < t.nv; v += gridDim.x * blockDim.x) {
    P32[3 * v] = (float)P[3 * v];
    P32[3 * v + 1] = (float)P[3 * v + 1];
    P32[3 * v + 2] = (float)P[3 * v + 2];
  }
  if (f >= t.nf) return;
  int a = t.fv[3 * f], b = t.fv[3 * f + 1], c = t.fv[3 * f + 2];
  d3 pa = ld3(P, a), pb = ld3(P, b), pc = ld3(P, c);
  d3 eab = pb - pa, eac = pc - pa, ebc = pc - pb;
  d3 N = cross(eab, eac);
  double n2 = dot(N, N);
  double inv = rsqrt(n2);
  double nn = n2 * inv;
  FaceD F;
  F.nx = N.x * inv;
  F.ny = N.y * inv;
  F.nz = N.z * inv;
  F.A = 0.5 * nn;
  // (p_a x p_b) . p_c = p_a . ((p_b - p_a) x (p_c - p_a)) = p_a . N
  F.V = dot(pa, N) * (1.0 / 6.0);
  F.c0 = dot(eab, eac) * inv;
  F.c1 = -dot(eab, ebc) * inv;
  F.c2 = dot(eac, ebc) * inv;
  fd[f] = F;
  fav[f] = make_double2(F.A, F.V);
}

// Per edge eg: (theta / l, kt dB/dl / l) for the gradient (theta 0 on
// boundary edges) and elt: (l theta, bond value) for k_vertex, 16 bytes per
// gather each.  Edges below the flat bottom (exp and a division in FP64) are
// collected per block and handled by its first threads, so that whole warps
// do not wait on a few lanes.
constexpr int EB = 256;
__global__ void __launch_bounds__(EB) k_edge(Topo t, const double* __restrict__ P, const FaceD* __restrict__ fd,
                                             double2* __restrict__ eg, double2* __restrict__ elt, EP ep,
                                             const double2* __restrict__ sct) {
  __shared__ double sl[EB], sil[EB];
  __shared__ int se[EB], nshort;
  if (threadIdx.x == 0) nshort = 0;
  __syncthreads();
  const int e = blockIdx.x * EB + threadIdx.x;
  if (e < t.ne) {
    int4 E = t.edge[e];
    d3 pi = ld3(P, E.x), pj = ld3(P, E.y);
    d3 ev = pj - pi;
    double l2 = dot(ev, ev);
    double il = rsqrt(l2);
    double l = l2 * il;
    double th = 0.0;
    if (E.z >= 0 && E.w >= 0) {
      const FaceD F0 = fd[E.z], F1 = fd[E.w];
      d3 n0 = mk(F0.nx, F0.ny, F0.nz), n1 = mk(F1.nx, F1.ny, F1.nz);
      // both normals are perpendicular to the shared edge, so n0 x n1 lies
      // along it: its projection on the unit edge is the signed sine, whose
      // sign is the reference's sign test (n0 x n1) . e >= 0
      double sd = dot(cross(n0, n1), ev) * il;
      double a = angle_sc(abs_bits(sd), dot(n0, n1), sct);
      th = sd >= 0.0 ? a : -a;
    }
    // flat-bottom edge penalty: above the flat bottom inline (products only,
    // edge_bond's l > lc0 branch)
    double val = 0.0, fac = 0.0;
    if (ep.btype == 0) {
      if (len_below(l, ep.lc1)) {
        const int k = atomicAdd(&nshort, 1);
        se[k] = e;
        sl[k] = l;
        sil[k] = il;
      } else if (len_above(l, ep.lc0)) {
        const double d = l - ep.lc0;
        val = ep.br1 * ipow(d, ep.r);
        fac = ep.kt * (ep.br2 * ipow(d, ep.r - 1)) * il;
      }
    }
    eg[e] = make_double2(th * il, fac);
    elt[e] = make_double2(l * th, val);
  }
  __syncthreads();
  if ((int)threadIdx.x < nshort) {
    const int k = threadIdx.x;
    double val, fac;
    edge_bond(ep, sl[k], sil[k], &val, &fac);
    eg[se[k]].y = ep.kt * fac * sil[k];
    elt[se[k]].y = val;
  }
}

constexpr int VG = 6;  // ring slots loaded together by k_vertex
template <bool VPROPS>
__global__ void __launch_bounds__(VB) k_vertex(Topo t, const double2* __restrict__ fav,
                                              const double2* __restrict__ elt, const double* __restrict__ reppot,
                                              EP ep, double2* __restrict__ rk, double* __restrict__ vprops,
                                              double* partial, Globals* g) {
  int v = blockIdx.x * VB + threadIdx.x;
  double pr[6] = {0, 0, 0, 0, 0, 0};
  if (v < t.nv) {
    int d = t.val[v];
    double A = 0, V = 0, LT = 0, T = 0;
    // slots in groups of six (one group at the usual valence): all loads of
    // a group are issued before the sums, which keep the slot order
    for (int m0 = 0; m0 < d; m0 += VG) {
      int4 s[VG];
#pragma unroll
      for (int k = 0; k < VG; ++k) s[k] = m0 + k < d ? t.slot[(size_t)(m0 + k) * t.nv + v] : make_int4(0, -1, 0, 0);
      double fa[VG], fv[VG], lt[VG], tb[VG];
#pragma unroll
      for (int k = 0; k < VG; ++k) {
        int f = slot_face(s[k].y);
        fa[k] = fv[k] = lt[k] = tb[k] = 0.0;
        if (f >= 0) {
          const double2 av = fav[f], lb = elt[s[k].z];
          fa[k] = av.x;
          fv[k] = av.y;
          lt[k] = lb.x;
          if (ep.btype == 0) tb[k] = lb.y;
        }
      }
#pragma unroll
      for (int k = 0; k < VG; ++k) {
        if (slot_face(s[k].y) < 0) continue;
        A += fa[k];
        V += fv[k];
        LT += lt[k];
        if (ep.btype == 0) {
          T += tb[k];
        } else {
          double q = fa[k] / ep.a0 - 1.0;
          T += q * q;
        }
      }
    }
    double a = A * (1.0 / 3.0), c = 0.25 * LT;
    double ia = 1.0 / a;
    pr[0] = a;
    pr[1] = V * (1.0 / 3.0);
    pr[2] = c;
    pr[3] = 2 * c * c * ia;
    pr[4] = T * ep.itdiv;
    pr[5] = reppot[v];
    const double rho = c * ia;
    rk[v] = make_double2(ep.kb * rho, (ep.kb * (2.0 / 3.0)) * (rho * rho));
    if (VPROPS)
      for (int k = 0; k < 6; ++k) vprops[6 * (size_t)v + k] = pr[k];
  }
  finish_props(pr, partial, gridDim.x, blockIdx.x, ep, g);
}

__global__ void k_assemble_props(EP ep, const double* props6, Globals* g) {
  if (threadIdx.x || blockIdx.x) return;
  for (int k = 0; k < 6; ++k) g->props[k] = props6[k];
  assemble(ep, g);
}

// ---- gradient gather ------------------------------------------------------
// Per vertex i over its ring (slot m: face (i, j = r_m, k = r_{m-1})), every
// term along an edge vector d_j = x_j - x_i or a face normal n (area gradient
// in its cotangent form, volume through the normal; Meyer, Desbrun, Schroeder
// & Barr 2003), as in the double-word evaluation: with h = alpha / 2, alpha =
// gA - 2/3 kb (rho_i^2 + rho_j^2 + rho_k^2), and w = gC/2 + kb (rho_i + rho_j)
//   area -h (cot_k d_j + cot_j d_k), volume gV/3 A n, length -(w theta + kt
//   dB/dl) / l d_j, dihedral (w_ij cot_j + w_ik cot_k - w_jk (cot_j + cot_k)) n
// 25 FP64 operations per slot on GB300's narrow FP64 pipe (35 with cross
// products of absolute positions).  Two lanes share a vertex, each with half
// of its slots: twice the warps to cover the latency of gathers and FP64
// chains for an eighth more operations.  rk[v] = (kb rho_v, 2/3 kb rho_v^2),
// written by k_vertex.
constexpr int GL = 2, GB = 128;
template <bool CLOSED>
__global__ void __launch_bounds__(GB) k_grad(Topo t, const double* __restrict__ P, const FaceD* __restrict__ fd,
                                             const double2* __restrict__ eg, const double2* __restrict__ rk,
                                             const double* __restrict__ repg, const Globals* __restrict__ g, EP ep,
                                             double* __restrict__ grad) {
  const int i = (blockIdx.x * GB + threadIdx.x) / GL, sub = threadIdx.x % GL;
  d3 acc = mk(0, 0, 0), tel = mk(0, 0, 0), xi = mk(0, 0, 0);
  const double gV = g->gV;
  if (i < t.nv) {
    const double gA = g->gA, hgC = 0.5 * g->gC, gV3 = gV * (1.0 / 3.0);
    xi = ld3(P, i);
    const double2 qi = rk[i];
    const double ai = gA - qi.y, wi = hgC + qi.x;
    const int d = t.val[i];
    const int run = (d + GL - 1) / GL, mb = sub * run, m1 = min(d, mb + run);
    const size_t nv = t.nv;
    if (mb < m1) {
      const int4 sp = t.slot[(size_t)(mb == 0 ? d - 1 : mb - 1) * nv + i];
      d3 dk = ld3(P, sp.x) - xi;
      double2 qk = rk[sp.x];
      double uk = hgC + qk.x, wk = wi + qk.x;
      bool fprev = slot_face(sp.y) >= 0;
      int4 sc = t.slot[(size_t)mb * nv + i];
      double s = 0.0;  // coefficient of d_k still open
      for (int m = mb; m < m1; ++m) {
        int4 sn = sc;
        if (!CLOSED || m + 1 < m1) sn = t.slot[(size_t)(m + 1 == d ? 0 : m + 1) * nv + i];
        const d3 dj = ld3(P, sc.x) - xi;
        const double2 qj = rk[sc.x];
        const double wj = wi + qj.x;
        const int f = slot_face(sc.y);
        double sj = 0.0;
        if (CLOSED || f >= 0) {
          const FaceD F = fd[f];
          const double2 E = eg[sc.z];
          const int ci = slot_corner(sc.y);
          const double cj = cot_at(F, ci == 2 ? 0 : ci + 1), ck = cot_at(F, ci == 0 ? 2 : ci - 1);
          double alpha = (ai - qj.y) - qk.y;
          if (ep.btype == 1) alpha += ep.kt * 2.0 * (F.A / ep.a0 - 1.0) / ep.a0;
          const double h = -0.5 * alpha;
          // edge (i, k): this face completes its coefficient
          s = fma(h, cj, s);
          acc.x = fma(s, dk.x, acc.x);
          acc.y = fma(s, dk.y, acc.y);
          acc.z = fma(s, dk.z, acc.z);
          // edge (i, j): length and area terms
          sj = fma(h, ck, -fma(wj, E.x, E.y));
          // along n
          double c = gV3 * F.A;
          bool in_ij = true, in_ik = true, in_jk = true;
          if (!CLOSED) {
            in_ij = slot_face(sn.y) >= 0;
            in_ik = fprev;
            const int4 ejk = t.edge[sc.w];
            in_jk = ejk.z >= 0 && ejk.w >= 0;
          }
          if (in_ij) c = fma(wj, cj, c);
          if (in_ik) c = fma(wk, ck, c);
          if (in_jk) c = fma(-(uk + qj.x), cj + ck, c);
          acc.x = fma(c, F.nx, acc.x);
          acc.y = fma(c, F.ny, acc.y);
          acc.z = fma(c, F.nz, acc.z);
          if (!CLOSED) tel += dk - dj;
        } else {
          // no face: the edge before it has no more terms
          acc += s * dk;
        }
        fprev = f >= 0;
        s = sj;
        dk = dj;
        qk = qj;
        uk = hgC + qj.x;
        wk = wj;
        sc = sn;
      }
      acc += s * dk;  // the run's last edge
    }
  }
  auto lanes = [](double x) { return x + __shfl_xor_sync(0xffffffffu, x, 1); };
  acc = mk(lanes(acc.x), lanes(acc.y), lanes(acc.z));
  if (!CLOSED) {  // x_i x (d_k - d_j) / 6 cancels around a closed fan only
    tel = mk(lanes(tel.x), lanes(tel.y), lanes(tel.z));
    acc += (gV * (1.0 / 6.0)) * cross(xi, tel);
  }
  if (i >= t.nv || sub) return;
  acc += ep.kr * ld3(repg, i);
  st3(grad, i, acc);
}

inline int nblk(long n, int b) { return (int)((n + b - 1) / b); }
// the FP64 path's per-vertex curvature weights (kb rho, 2/3 kb rho^2)
inline double2* rk2(tm_energy* e) { return reinterpret_cast<double2*>(e->rho.get()); }
// the FP64 path's compact (area, volume) per face and (l theta, bond) per edge
inline double2* fav2(tm_energy* e) { return reinterpret_cast<double2*>(e->fav.get()); }
inline double2* elt2(tm_energy* e) { return reinterpret_cast<double2*>(e->ebond.get()); }

EP make_ep(const tm_energy* e) {
  const tm_params& p = e->prm;
  EP ep;
  std::memset(&ep, 0, sizeof ep);  // padding too: evaluation graphs compare EP bytes
  ep.kb = p.kappa_b;
  ep.ka = p.kappa_a;
  ep.kv = p.kappa_v;
  ep.kc = p.kappa_c;
  ep.kt = p.kappa_t;
  ep.kr = p.kappa_r;
  double lam = p.cont_lambda;
  ep.refA = (1.0 - lam * (1.0 - p.area_frac)) * e->initial[0];
  ep.refV = (1.0 - lam * (1.0 - p.volume_frac)) * e->initial[1];
  ep.refC = (1.0 - lam * (1.0 - p.curvature_frac)) * e->initial[2];
  ep.lc0 = p.bond_lc0;
  ep.lc1 = p.bond_lc1;
  ep.a0 = p.bond_a0;
  ep.r = p.bond_r;
  ep.btype = p.bond_type;
  ep.rlc1 = p.rep_lc1;
  ep.rT = sq_threshold(p.rep_lc1);
  ep.rr = p.rep_r;
  ep.tdiv = p.bond_type == 0 ? 2.0 : 3.0;
  ep.itdiv = 1.0 / ep.tdiv;
  auto ipow_h = [](double x, int n) {  // the device's ipow, on the host
    double r = 1.0;
    for (int k = 0; k < std::abs(n); ++k) r *= x;
    return n < 0 ? 1.0 / r : r;
  };
  ep.br1 = ipow_h((double)p.bond_r, p.bond_r + 1);
  ep.br2 = ipow_h((double)p.bond_r, p.bond_r + 2);
  return ep;
}

void energy_eval(tm_energy* e, tm_mesh* m, const double* P, bool want_grad, bool want_vprops, double* d_grad,
                 cudaStream_t s, double* d_energy) {
  if (e->stencil == 2 && !want_vprops) {
    energy_eval_df(e, m, P, want_grad, d_grad, d_energy, nullptr, s, nullptr);
    return;
  }
  energy_eval_marked(e, m, P, want_grad, want_vprops, d_grad, s, nullptr);
  if (d_energy)
    TM_CUDA(cudaMemcpyAsync(d_energy, &e->glob.get()->comps[6], sizeof(double), cudaMemcpyDeviceToDevice, s));
}

bool energy_eval_moved(tm_energy* e, tm_mesh* m, const Leap& leap, double* d_grad, cudaStream_t s) {
  if (e->stencil != 2) return false;
  energy_eval_df(e, m, leap.x, true, d_grad, nullptr, &leap, s, nullptr);
  return true;
}

static void eval_fp64_launches(tm_energy* e, tm_mesh* m, const double* P, bool want_grad, bool want_vprops,
                               double* d_grad, cudaStream_t s, cudaEvent_t* ev);

// the launches of one FP32 or FP64 evaluation (the double-word path is short
// enough to need no graph)
static void eval_launches(tm_energy* e, tm_mesh* m, const double* P, bool want_grad, double* d_grad,
                          cudaStream_t s) {
  if (e->stencil == 1)
    energy_eval32(e, m, P, want_grad, false, d_grad, s, nullptr);
  else
    eval_fp64_launches(e, m, P, want_grad, false, d_grad, s, nullptr);
}

// What the launches of an evaluation depend on besides device memory:
// arguments, stencil precision, buffers, parameters and the neighbour-list
// view.  Equal keys mean a captured graph replays the same launches.
static std::vector<unsigned char> eval_key(tm_energy* e, tm_mesh* m, const double* P, bool want_grad,
                                           double* d_grad) {
  std::vector<unsigned char> k;
  auto add = [&k](const void* p, size_t n) {
    const unsigned char* b = static_cast<const unsigned char*>(p);
    k.insert(k.end(), b, b + n);
  };
  // (the launch stream is not part of the key: a graph replays on any stream)
  const void* ptrs[] = {P, d_grad, e->face.get(), e->edge.get(), e->ebond.get(), e->fav.get(), e->rho.get(),
                        e->repg.get(), e->reppot.get(), e->slow.get(), e->pos32.get(), e->partials.get(),
                        e->glob.get(), e->sct.get(), e->aux, e->ev_fork, e->ev_join, e->nl.xb.get(),
                        e->posdw.get(), e->sctf.get()};
  add(ptrs, sizeof ptrs);
  const Topo t = m->topo();
  const int sizes[] = {t.nv, t.ne, t.nf, want_grad ? 1 : 0, e->stencil, e->nl.near_nv};
  add(sizes, sizeof sizes);
  const void* tp[] = {t.to, t.next, t.face, t.vout, t.fhe, t.slot, t.nbr, t.val, t.fv, t.edge};
  add(tp, sizeof tp);
  const double nd[] = {e->nl.near_lc1, e->nl.near_move2};
  add(nd, sizeof nd);
  const EP ep = make_ep(e);
  add(&ep, sizeof ep);
  add(&e->nl.view, sizeof(NLView));
  return k;
}

// Evaluation replayed from a CUDA graph: the launch sequence (about a dozen
// kernels, memsets and the fork/join of the repulsion stream) is captured
// per key and then issued as one graph launch, which removes the gaps
// between the short kernels.  On a miss the launches run directly first
// (any allocation they make happens outside a capture), then they are
// captured for the next call.  A few graphs are kept (with and without the
// gradient, several buffers), the least recently used is replaced.
static void eval_graph(tm_energy* e, tm_mesh* m, const double* P, bool want_grad, double* d_grad, cudaStream_t s) {
  constexpr size_t MAX_GRAPHS = 4;
  std::vector<unsigned char> key = eval_key(e, m, P, want_grad, d_grad);
  for (auto& g : e->eval_graphs)
    if (g.exec && g.key == key) {
      g.used = ++e->eval_tick;
      TM_CUDA(cudaGraphLaunch(g.exec, s));
      return;
    }
  eval_launches(e, m, P, want_grad, d_grad, s);
  key = eval_key(e, m, P, want_grad, d_grad);
  cudaGraph_t g = nullptr;
  TM_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  try {
    eval_launches(e, m, P, want_grad, d_grad, s);
  } catch (...) {
    cudaStreamEndCapture(s, &g);  // leave capture mode before reporting
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    throw;
  }
  TM_CUDA(cudaStreamEndCapture(s, &g));
  cudaGraphExec_t exec = nullptr;
  cudaError_t rc = cudaGraphInstantiate(&exec, g, 0);
  cudaGraphDestroy(g);
  TM_CUDA(rc);
  tm_energy::EvalGraph* slot = nullptr;
  if (e->eval_graphs.size() < MAX_GRAPHS) {
    e->eval_graphs.emplace_back();
    slot = &e->eval_graphs.back();
  } else {
    slot = &e->eval_graphs[0];
    for (auto& c : e->eval_graphs)
      if (c.used < slot->used) slot = &c;
    cudaGraphExecDestroy(slot->exec);
  }
  slot->exec = exec;
  slot->key.swap(key);
  slot->used = ++e->eval_tick;
}

void energy_eval_marked(tm_energy* e, tm_mesh* m, const double* P, bool want_grad, bool want_vprops, double* d_grad,
                        cudaStream_t s, cudaEvent_t* ev) {
  // graphs need a capturable stream (not the legacy default stream)
  if (!ev && !want_vprops && s != nullptr && e->use_graphs) {
    eval_graph(e, m, P, want_grad, d_grad, s);
    return;
  }
  if (e->stencil == 1 && !want_vprops) {
    energy_eval32(e, m, P, want_grad, want_vprops, d_grad, s, ev);
    return;
  }
  eval_fp64_launches(e, m, P, want_grad, want_vprops, d_grad, s, ev);
}

static void eval_fp64_launches(tm_energy* e, tm_mesh* m, const double* P, bool want_grad, bool want_vprops,
                               double* d_grad, cudaStream_t s, cudaEvent_t* ev) {
  if (ev) TM_CUDA(cudaEventRecord(ev[0], s));
  e->ensure(m->nv, m->ne, m->nf);
  Topo t = m->topo();
  EP ep = make_ep(e);
  FaceD* fd = reinterpret_cast<FaceD*>(e->face.get());
  double2* eg = reinterpret_cast<double2*>(e->edge.get());
  int nfb = std::max(nblk(std::max(t.nf, t.nv), 256), 1);
  k_face<<<nfb, 256, 0, s>>>(t, P, fd, e->pos32.get(), fav2(e));
  TM_LAUNCH();
  if (ev) TM_CUDA(cudaEventRecord(ev[1], s));
  // the repulsion pass needs only the positions: it overlaps the edge kernels
  // (in sequence when the stages are timed)
  const bool conc = ev == nullptr;
  if (conc) fork_repulsion(e, m, P, want_grad, s, true);
  if (t.ne) k_edge<<<nblk(t.ne, EB), EB, 0, s>>>(t, P, fd, eg, elt2(e), ep, e->sct.get());
  TM_LAUNCH();
  if (ev) TM_CUDA(cudaEventRecord(ev[2], s));
  if (conc)
    join_repulsion(e, s, true);
  else
    fork_repulsion(e, m, P, want_grad, s, false);
  int nb = std::max(1, nblk(t.nv, VB));
  if (want_vprops)
    k_vertex<true><<<nb, VB, 0, s>>>(t, fav2(e), elt2(e), e->reppot.get(), ep, rk2(e),
                                     e->vprops.get(), e->partials.get(), e->glob.get());
  else
    k_vertex<false><<<nb, VB, 0, s>>>(t, fav2(e), elt2(e), e->reppot.get(), ep, rk2(e), nullptr,
                                      e->partials.get(), e->glob.get());
  TM_LAUNCH();
  if (ev) TM_CUDA(cudaEventRecord(ev[3], s));
  if (want_grad && t.nv)
    (m->closed ? k_grad<true> : k_grad<false>)<<<nblk((long)GL * t.nv, GB), GB, 0, s>>>(
        t, P, fd, eg, rk2(e), e->repg.get(), e->glob.get(), ep, d_grad);
  TM_LAUNCH();
  if (ev) TM_CUDA(cudaEventRecord(ev[4], s));
}

void energy_from_props_device(tm_energy* e, const double* d_props6, double* /*unused*/, cudaStream_t s) {
  EP ep = make_ep(e);
  k_assemble_props<<<1, 1, 0, s>>>(ep, d_props6, e->glob.get());
  TM_LAUNCH();
}

}  // namespace tmg

void tm_energy::ensure(int nv_, int ne_, int nf_) {
  if (nv_ == nv && ne_ == ne && nf_ == nf && glob.get()) return;
  nv = nv_;
  ne = ne_;
  nf = nf_;
  face.ensure(8 * (size_t)std::max(nf, 1));
  edge.ensure(2 * (size_t)std::max(ne, 1));  // 16 bytes per edge in every stencil precision
  ebond.ensure(2 * (size_t)std::max(ne, 1));  // FP64 path: (l theta, bond value) per edge
  fav.ensure(2 * (size_t)std::max(nf, 1));    // FP64 path: (area, volume) per face
  rho.ensure(2 * (size_t)std::max(nv, 1));  // FP64 path: (kb rho, 2/3 kb rho^2) per vertex
  repg.ensure(3 * (size_t)std::max(nv, 1));
  reppot.ensure(std::max(nv, 1));
  slow.ensure((size_t)std::max(nv, 1) + 1);  // repulsion slow list
  vprops.ensure(6 * (size_t)std::max(nv, 1));
  pos32.ensure(3 * (size_t)std::max(nv, 1));
  posdw.ensure(2 * (size_t)std::max(nv, 1));
  int nb = std::max(1, (nv + tmg::VB - 1) / tmg::VB);
  partials.ensure(8 * (size_t)nb * 2);  // up to two lanes per vertex
  moved.ensure(nb);
  grad.ensure(3 * (size_t)std::max(nv, 1));
  // workspace of an HMC move: position, momentum, two forces, partials and scalars
  work.ensure(12 * (size_t)std::max(nv, 1) + 1024 + 64);
  glob.ensure(1);
  TM_CUDA(cudaMemsetAsync(glob.get(), 0, sizeof(tmg::Globals), stream));
}

int tm_energy::sm_count() {
  if (!sms) {
    int dev = 0;
    TM_CUDA(cudaGetDevice(&dev));
    TM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  }
  return sms;
}

void tm_energy::to_host(double* dst, const double* src, size_t n) {
  // direct copy: for pageable destinations the driver's own staged copy beat
  // a page-locked staging buffer plus memcpy (the destination is a fresh
  // array whose pages are touched for the first time either way)
  if (n) TM_CUDA(cudaMemcpyAsync(dst, src, sizeof(double) * n, cudaMemcpyDeviceToHost, stream));
  TM_CUDA(cudaStreamSynchronize(stream));
}

double* tm_energy::host_scalars(bool required) {
  if (!pinned && cudaMallocHost(&pinned, sizeof(tmg::Globals) + 16 * sizeof(double)) != cudaSuccess) {
    cudaGetLastError();
    pinned = nullptr;
    if (required) fail(TM_ERR_NOMEM, "page-locked allocation failed");
  }
  return pinned;
}

tm_energy::~tm_energy() {
  if (pinned) cudaFreeHost(pinned);
  for (auto& g : eval_graphs)
    if (g.exec) cudaGraphExecDestroy(g.exec);
  if (flip_graph.exec) cudaGraphExecDestroy(flip_graph.exec);
  if (ev_fork) cudaEventDestroy(ev_fork);
  if (ev_join) cudaEventDestroy(ev_join);
  if (aux) cudaStreamDestroy(aux);
  if (stream) cudaStreamDestroy(stream);
}

// --------------------------------------------------------------------------
// C ABI
// --------------------------------------------------------------------------
static void check_params(const tm_params& p) {
  if (p.bond_type != 0 && p.bond_type != 1) fail(TM_ERR_ARG, "Unknown bond potential");
  if (p.n_search != 0 && p.n_search != 1) fail(TM_ERR_ARG, "Unknown neighbour search algorithm.");
  if (p.exclusion_level < 0 || p.exclusion_level > 2) fail(TM_ERR_ARG, "Unsupported exclusion level");
}

// staged: through the handle's page-locked memory (where there is none, the
// driver does so for a pageable destination: energy() of 642 vertices takes 35
// us instead of 33); not at creation, where allocating it would cost more
static void fetch_globals(tm_energy* e, tmg::Globals* g, bool staged = true) {
  void* pinned = staged ? e->host_scalars(false) : nullptr;
  void* h = pinned ? pinned : (void*)g;
  TM_CUDA(cudaMemcpyAsync(h, e->glob.get(), sizeof(tmg::Globals), cudaMemcpyDeviceToHost, e->stream));
  TM_CUDA(cudaStreamSynchronize(e->stream));
  if (pinned) std::memcpy(g, pinned, sizeof(tmg::Globals));
}

static void eval_host(tm_energy* e, tm_mesh* m, bool grad, bool vprops) {
  if (!e || !m) fail(TM_ERR_ARG, "NULL handle");
  m->upload_points(e->stream);
  tmg::energy_eval(e, m, m->d_pts.get(), grad, vprops, e->grad.get(), e->stream);
}

extern "C" {

int tm_energy_create(tm_mesh* m, const tm_params* p, tm_energy** out) {
  TM_API_BEGIN
  if (!m || !p || !out) fail(TM_ERR_ARG, "NULL argument");
  *out = nullptr;
  check_params(*p);
  std::unique_ptr<tm_energy> e(new tm_energy());
  e->prm = *p;
  TM_CUDA(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking));
  TM_CUDA(cudaStreamCreateWithFlags(&e->aux, cudaStreamNonBlocking));
  TM_CUDA(cudaEventCreateWithFlags(&e->ev_fork, cudaEventDisableTiming));
  TM_CUDA(cudaEventCreateWithFlags(&e->ev_join, cudaEventDisableTiming));
  {
    std::vector<double2> sc(tmg::TM_SCT_N);
    std::vector<float4> scf(tmg::TM_SCT_N);
    auto split = [](double x, float* h, float* l) {
      *h = (float)x;
      *l = (float)(x - (double)*h);
    };
    for (int k = 0; k < tmg::TM_SCT_N; ++k) {
      sc[k] = make_double2(std::sin(k / 128.0), std::cos(k / 128.0));
      split(sc[k].x, &scf[k].x, &scf[k].y);
      split(sc[k].y, &scf[k].z, &scf[k].w);
    }
    e->sct.ensure(tmg::TM_SCT_N);
    e->sctf.ensure(tmg::TM_SCT_N);
    TM_CUDA(cudaMemcpyAsync(e->sct.get(), sc.data(), sizeof(double2) * tmg::TM_SCT_N, cudaMemcpyHostToDevice,
                            e->stream));
    TM_CUDA(cudaMemcpyAsync(e->sctf.get(), scf.data(), sizeof(float4) * tmg::TM_SCT_N, cudaMemcpyHostToDevice,
                            e->stream));
    TM_CUDA(cudaStreamSynchronize(e->stream));
  }
  m->upload_points(e->stream);
  tmg::nlist_make(&e->nl, m, e->prm, m->d_pts.get(), e->stream);
  // initial properties: the reference properties are still unset (zero) and
  // only the sums matter here; taken with the FP64 stencil whatever the
  // handle's stencil precision
  const int stencil = e->stencil;
  e->stencil = 0;
  tmg::energy_eval(e.get(), m, m->d_pts.get(), false, false, nullptr, e->stream);
  e->stencil = stencil;
  tmg::Globals g;
  fetch_globals(e.get(), &g, false);
  for (int k = 0; k < 6; ++k) e->initial[k] = g.props[k];
  *out = e.release();
  TM_API_END
}

int tm_energy_destroy(tm_energy* e) {
  delete e;
  return TM_OK;
}

int tm_energy_get_params(tm_energy* e, tm_params* out) {
  if (!e || !out) return TM_ERR_ARG;
  *out = e->prm;
  return TM_OK;
}

int tm_energy_initial_props(tm_energy* e, double* out6) {
  if (!e || !out6) return TM_ERR_ARG;
  std::memcpy(out6, e->initial, sizeof(double) * 6);
  return TM_OK;
}

int tm_energy_set_initial_props(tm_energy* e, const double* in6) {
  TM_API_BEGIN
  if (!e || !in6) fail(TM_ERR_ARG, "NULL argument");
  std::memcpy(e->initial, in6, sizeof(double) * 6);
  TM_API_END
}

int tm_energy_properties(tm_energy* e, tm_mesh* m, double* out6) {
  TM_API_BEGIN
  if (!out6) fail(TM_ERR_ARG, "NULL output");
  eval_host(e, m, false, false);
  tmg::Globals g;
  fetch_globals(e, &g);
  std::memcpy(out6, g.props, sizeof(double) * 6);
  TM_API_END
}

int tm_energy_vertex_properties(tm_energy* e, tm_mesh* m, double* out6v) {
  TM_API_BEGIN
  if (!out6v) fail(TM_ERR_ARG, "NULL output");
  eval_host(e, m, false, true);
  TM_CUDA(cudaMemcpyAsync(out6v, e->vprops.get(), sizeof(double) * 6 * m->nv, cudaMemcpyDeviceToHost, e->stream));
  TM_CUDA(cudaStreamSynchronize(e->stream));
  TM_API_END
}

int tm_energy_energy(tm_energy* e, tm_mesh* m, double* energy) {
  TM_API_BEGIN
  if (!energy) fail(TM_ERR_ARG, "NULL output");
  eval_host(e, m, false, false);
  tmg::Globals g;
  fetch_globals(e, &g);
  *energy = g.comps[6];
  TM_API_END
}

int tm_energy_energy_props(tm_energy* e, const double* props6, double* energy) {
  TM_API_BEGIN
  if (!e || !props6 || !energy) fail(TM_ERR_ARG, "NULL argument");
  e->ensure(std::max(e->nv, 1), std::max(e->ne, 1), std::max(e->nf, 1));
  TM_CUDA(cudaMemcpyAsync(e->work.get(), props6, sizeof(double) * 6, cudaMemcpyHostToDevice, e->stream));
  tmg::energy_from_props_device(e, e->work.get(), nullptr, e->stream);
  tmg::Globals g;
  fetch_globals(e, &g);
  *energy = g.comps[6];
  TM_API_END
}

int tm_energy_components(tm_energy* e, tm_mesh* m, double* out7) {
  TM_API_BEGIN
  if (!out7) fail(TM_ERR_ARG, "NULL output");
  eval_host(e, m, false, false);
  tmg::Globals g;
  fetch_globals(e, &g);
  std::memcpy(out7, g.comps, sizeof(double) * 7);
  TM_API_END
}

int tm_energy_gradient(tm_energy* e, tm_mesh* m, double* grad, double* energy) {
  TM_API_BEGIN
  if (!grad) fail(TM_ERR_ARG, "NULL output");
  eval_host(e, m, true, false);
  if (energy)
    TM_CUDA(cudaMemcpyAsync(energy, &e->glob.get()->comps[6], sizeof(double), cudaMemcpyDeviceToHost, e->stream));
  e->to_host(grad, e->grad.get(), 3 * (size_t)m->nv);
  TM_API_END
}

int tm_energy_update_reference_properties(tm_energy* e) {
  if (!e) return TM_ERR_ARG;
  if (e->prm.cont_lambda < 1.0) e->prm.cont_lambda += e->prm.cont_delta;
  return TM_OK;
}

int tm_energy_update_repulsion(tm_energy* e, tm_mesh* m) {
  TM_API_BEGIN
  if (!e || !m) fail(TM_ERR_ARG, "NULL handle");
  m->upload_points(e->stream);
  tmg::nlist_make(&e->nl, m, e->prm, m->d_pts.get(), e->stream);
  TM_CUDA(cudaStreamSynchronize(e->stream));
  TM_API_END
}

int tm_energy_set_stencil_precision(tm_energy* e, int mode) {
  TM_API_BEGIN
  if (!e) fail(TM_ERR_ARG, "NULL handle");
  if (mode < 0 || mode > 2) fail(TM_ERR_ARG, "mode must be 0 (FP64), 1 (FP32) or 2 (double-float)");
  e->stencil = mode;
  TM_API_END
}

int tm_energy_eval_device(tm_energy* e, tm_mesh* m, const double* d_points, double* d_grad, double* d_energy,
                          void* stream) {
  TM_API_BEGIN
  if (!e || !m || !d_points) fail(TM_ERR_ARG, "NULL argument");
  cudaStream_t s = stream ? (cudaStream_t)stream : e->stream;
  tmg::energy_eval(e, m, d_points, d_grad != nullptr, false, d_grad, s, d_energy);
  TM_API_END
}

int tm_energy_eval_timed(tm_energy* e, tm_mesh* m, const double* d_points, double* d_grad, float* ms5,
                         void* stream) {
  TM_API_BEGIN
  if (!e || !m || !d_points || !ms5) fail(TM_ERR_ARG, "NULL argument");
  cudaStream_t s = stream ? (cudaStream_t)stream : e->stream;
  cudaEvent_t ev[5];
  for (int k = 0; k < 5; ++k) TM_CUDA(cudaEventCreate(&ev[k]));
  if (e->stencil == 2)
    tmg::energy_eval_df(e, m, d_points, d_grad != nullptr, d_grad, nullptr, nullptr, s, ev);
  else
    tmg::energy_eval_marked(e, m, d_points, d_grad != nullptr, false, d_grad, s, ev);
  TM_CUDA(cudaEventSynchronize(ev[4]));
  for (int k = 0; k < 4; ++k) TM_CUDA(cudaEventElapsedTime(&ms5[k], ev[k], ev[k + 1]));
  TM_CUDA(cudaEventElapsedTime(&ms5[4], ev[0], ev[4]));
  for (int k = 0; k < 5; ++k) cudaEventDestroy(ev[k]);
  TM_API_END
}

int tm_energy_update_repulsion_device(tm_energy* e, tm_mesh* m, const double* d_points, void* stream) {
  TM_API_BEGIN
  if (!e || !m || !d_points) fail(TM_ERR_ARG, "NULL argument");
  cudaStream_t s = stream ? (cudaStream_t)stream : e->stream;
  tmg::nlist_make(&e->nl, m, e->prm, d_points, s);
  TM_API_END
}

int tm_fd_gradient(tm_mesh* m, tm_energy* e, double eps, double* grad) {
  TM_API_BEGIN
  if (!m || !e || !grad) fail(TM_ERR_ARG, "NULL argument");
  double e0 = 0;
  int rc = tm_energy_energy(e, m, &e0);
  if (rc) return rc;
  for (int i = 0; i < m->nv; ++i)
    for (int k = 0; k < 3; ++k) {
      double* x = m->h_pts + 3 * (size_t)i + k;
      *x += eps;
      double en = 0;
      rc = tm_energy_energy(e, m, &en);
      *x -= eps;
      if (rc) return rc;
      grad[3 * (size_t)i + k] = (en - e0) / eps;
    }
  TM_API_END
}

}  // extern "C"

// --------------------------------------------------------------------------
// Evaluation without allocation.
//
// Some callers cannot call cudaMalloc while they evaluate the energy: a host
// that runs under a strict device-memory budget owned by someone else (an
// embedding application or a pool allocator that forbids side allocations),
// or code that must not enter the CUDA allocator while other streams of the
// process are busy.  tm_energy_eval_device_noalloc evaluates the FP64 energy
// and gradient of a mesh whose scratch (face and edge records, per-vertex
// intermediates, block partials and the reduction state) fits into one
// file-scope device array of TM_NOALLOC_SCRATCH_BYTES, instead of the energy
// manager's own buffers.  It allocates nothing and frees nothing.
//
// The array's host-side name is only a stand-in for the device symbol, so its
// device address is looked up with cudaGetSymbolAddress once per device, on
// the first call made with that device current; make that first call before
// any stream capture.  All calls share the array and it keeps the last call's
// contents: each call clears the reduction state it needs at zero, and calls
// whose executions overlap on the GPU (other streams, other threads) race on
// the shared scratch and must be serialised by the caller.
// --------------------------------------------------------------------------
#include <mutex>

namespace {
static __device__ __align__(256) unsigned char g_noalloc_scratch[TM_NOALLOC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
unsigned char* g_noalloc_ptr[kMaxDevices] = {nullptr};

unsigned char* noalloc_scratch_for_current_device() {
  int dev = 0;
  TM_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) fail(TM_ERR_ARG, "device index out of range for the no-alloc scratch");
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    TM_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    g_noalloc_ptr[dev] = static_cast<unsigned char*>(p);
  }
  return g_noalloc_ptr[dev];
}

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
}  // namespace

extern "C" int tm_energy_eval_device_noalloc(tm_energy* e, tm_mesh* m, const double* d_points, double* d_grad,
                                             double* d_energy, void* stream) {
  TM_API_BEGIN
  if (!e || !m || !d_points || !d_grad) fail(TM_ERR_ARG, "NULL argument");
  const size_t nv = std::max(m->nv, 1), ne = std::max(m->ne, 1), nf = std::max(m->nf, 1);
  const int nb = std::max(1, (m->nv + VB - 1) / VB);
  // scratch layout, 256-byte aligned pieces (the mesh sizes that fit are part of
  // the interface: each edge keeps the 32 bytes and the list entry it had)
  size_t off_face = 0;
  size_t off_edge = off_face + align256(sizeof(FaceD) * nf);
  size_t off_ebond = off_edge + align256(4 * sizeof(double) * ne);
  size_t off_fav = off_ebond + align256(sizeof(double2) * ne);
  size_t off_rho = off_fav + align256(sizeof(double2) * nf);
  size_t off_repg = off_rho + align256(sizeof(double2) * nv);
  size_t off_pos32 = off_repg + align256(3 * sizeof(double) * nv);
  size_t off_pot = off_pos32 + align256(3 * sizeof(float) * nv);
  size_t off_slow = off_pot + align256(sizeof(double) * nv);
  size_t off_part = off_slow + align256(sizeof(int) * (nv + 1)) + align256(sizeof(int) * (ne + 1));
  size_t off_glob = off_part + align256(8 * sizeof(double) * nb);
  size_t need = off_glob + align256(sizeof(Globals));
  if (need > (size_t)TM_NOALLOC_SCRATCH_BYTES)
    fail(TM_ERR_ARG, "mesh needs " + std::to_string(need) + " bytes of scratch, more than the " +
                         std::to_string((size_t)TM_NOALLOC_SCRATCH_BYTES) +
                         " bytes of tm_energy_eval_device_noalloc (about 44,000 vertices)");
  unsigned char* base = noalloc_scratch_for_current_device();
  cudaStream_t s = stream ? (cudaStream_t)stream : e->stream;
  FaceD* fd = reinterpret_cast<FaceD*>(base + off_face);
  double2* eg = reinterpret_cast<double2*>(base + off_edge);
  double2* ebond = reinterpret_cast<double2*>(base + off_ebond);
  double2* fav = reinterpret_cast<double2*>(base + off_fav);
  double2* rho = reinterpret_cast<double2*>(base + off_rho);
  double* repg = reinterpret_cast<double*>(base + off_repg);
  float* pos32 = reinterpret_cast<float*>(base + off_pos32);
  double* reppot = reinterpret_cast<double*>(base + off_pot);
  int* slow = reinterpret_cast<int*>(base + off_slow);
  double* part = reinterpret_cast<double*>(base + off_part);
  Globals* g = reinterpret_cast<Globals*>(base + off_glob);
  // the block ticket of the reduction must start at zero
  TM_CUDA(cudaMemsetAsync(g, 0, sizeof(Globals), s));
  Topo t = m->topo();
  EP ep = make_ep(e);
  int nfb = std::max(nblk(std::max(t.nf, t.nv), 256), 1);
  k_face<<<nfb, 256, 0, s>>>(t, d_points, fd, pos32, fav);
  TM_LAUNCH();
  if (t.ne) k_edge<<<nblk(t.ne, EB), EB, 0, s>>>(t, d_points, fd, eg, ebond, ep, e->sct.get());
  TM_LAUNCH();
  repulsion_eval(e, m, d_points, pos32, true, reppot, repg, slow, slow + nv, s);
  k_vertex<false><<<nb, VB, 0, s>>>(t, fav, ebond, reppot, ep, rho, nullptr, part, g);
  TM_LAUNCH();
  if (t.nv)
    (m->closed ? k_grad<true> : k_grad<false>)<<<nblk((long)GL * t.nv, GB), GB, 0, s>>>(t, d_points, fd, eg, rho,
                                                                                       repg, g, ep, d_grad);
  TM_LAUNCH();
  if (d_energy) TM_CUDA(cudaMemcpyAsync(d_energy, &g->comps[6], sizeof(double), cudaMemcpyDeviceToDevice, s));
  TM_API_END
}
