// FP32-stencil variant of the energy / gradient evaluation
// (tm_energy_set_stencil_precision(e, 1)).
//
// Positions stay FP64 in memory.  Each evaluation splits them into float
// hi + lo parts, so an edge vector (x_b - x_a) = (hi_b - hi_a) + (lo_b - lo_a)
// keeps FP32 relative accuracy even though |x| >> |x_b - x_a|; everything
// local (normals, areas, cotangents, dihedral angles, potentials, the
// gradient gather) is then FP32.  Face volumes use x_a . N_f / 6 (N_f from the
// accurate edge vectors), not the triple product of absolute positions.  The
// dihedral angle is atan2(|n0 x n1|, n0 . n1), accurate for the small angles
// of fine meshes where acosf is not.  The global sums, the penalty assembly
// and the neighbour-pair decisions (exact FP64 threshold) stay FP64, so the
// pair set is the same as in FP64.
#include <algorithm>
#include <cmath>

#include "tm_energy.cuh"
#include "tm_internal.h"
#include "tm_math.cuh"
#include "tm_dw.cuh"
#include "tm_fp32.cuh"

namespace tmg {

namespace {

using namespace fp32;

// Positions as float hi + lo (and the float copy of the repulsion
// prefilter).  MOVE 1: drifts the positions first (with g0), 2: kicks with g0
// and g1, then drifts (with g1): the velocity-Verlet update in the pass that
// reads the positions anyway.  With the products of constants from the host
// it is five FP64 operations per coordinate on GB300's narrow FP64 pipe
// (218,000 vertices: 11 us, where a kick-drift pass of eight operations and a
// split with conversions took 13 + 4).
struct SplitMove {
  double *x, *p;
  const double *g0, *g1;
  double dt, hdt, hdt2, im;
};
template <int MOVE>
__global__ void __launch_bounds__(256) k_split(int nv, const double* __restrict__ P, SplitMove mv, float4* X,
                                               float* __restrict__ P32) {
  const int v = blockIdx.x * 256 + threadIdx.x;
  if (v >= nv) return;
  float h[3], l[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const size_t i = 3 * (size_t)v + k;
    double x;
    if (MOVE) {
      double p = mv.p[i], f = -mv.g0[i];
      if (MOVE == 2) {
        const double f1 = -mv.g1[i];
        p = p + (f + f1) * mv.hdt;
        mv.p[i] = p;
        f = f1;
      }
      x = mv.x[i] + (p * mv.dt + f * mv.hdt2) * mv.im;
      mv.x[i] = x;
    } else {
      x = P[i];
    }
    split_bits(x, &h[k], &l[k]);
    P32[i] = h[k];
  }
  st32(X + 2 * (size_t)v, make_float4(h[0], h[1], h[2], 0.0f), make_float4(l[0], l[1], l[2], 0.0f));
}

// faces [f0, f1)
__global__ void k_face32(int f0, int f1, Topo t, Split S, FaceF* __restrict__ fd) {
  int f = f0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= f1) return;
  const Pos32 a = S.at(t.fv[3 * f]), b = S.at(t.fv[3 * f + 1]), c = S.at(t.fv[3 * f + 2]);
  f3 eab = diff(b, a), eac = diff(c, a), ebc = diff(c, b);
  f3 N = fcross(eab, eac);
  float nn = fnorm(N);
  float inv = 1.0f / nn;
  FaceF F;
  F.nx = N.x * inv;
  F.ny = N.y * inv;
  F.nz = N.z * inv;
  F.A = 0.5f * nn;
  F.V = fdot(a.hi, N) * (1.0f / 6.0f);
  F.c0 = fdot(eab, eac) * inv;
  F.c1 = -fdot(eab, ebc) * inv;
  F.c2 = fdot(eac, ebc) * inv;
  fd[f] = F;
}

__device__ __forceinline__ EdgeF edge32(const int4& E, const Split& S, const FaceF* __restrict__ fd, const EP& ep) {
  f3 ev = diff(S.at(E.y), S.at(E.x));
  float l = fnorm(ev);
  EdgeF o;
  o.l = -l;
  o.th = 0.0f;
  if (E.z >= 0 && E.w >= 0) {
    const float4 F0 = *reinterpret_cast<const float4*>(fd + E.z), F1 = *reinterpret_cast<const float4*>(fd + E.w);
    f3 n0 = {F0.x, F0.y, F0.z}, n1 = {F1.x, F1.y, F1.z};
    f3 cr = fcross(n0, n1);
    float a = atan2f(fnorm(cr), fdot(n0, n1));
    o.th = fdot(cr, ev) >= 0.0f ? a : -a;
    o.l = l;
  }
  float val = 0.0f, fac = 0.0f;
  if (ep.btype == 0) {
    int r = ep.r;
    float lc0 = (float)ep.lc0, lc1 = (float)ep.lc1;
    if (l > lc0) {
      val = fipow((float)r, r + 1) * fipow(l - lc0, r);
      fac = fipow((float)r, r + 2) * fipow(l - lc0, r - 1);
    } else if (l < lc1) {
      val = expf(l / (l - lc1)) / fipow(l, r);
    }
    if (l < lc1) {
      float lmc = l - lc1;
      fac -= lc1 / (lmc * lmc) + r / l;
      fac /= fipow(l, r);
      fac *= expf(l / lmc);
    }
  }
  o.db = fac;
  o.bond = val;
  return o;
}
__global__ void k_edge32(Topo t, Split S, const FaceF* __restrict__ fd, EdgeF* __restrict__ ed, EP ep) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < t.ne) ed[e] = edge32(t.edge[e], S, fd, ep);
}

// The six properties of vertex v from its ring, in slot order; the records
// of six slots (one group at the usual valence) are loaded before the sums,
// 32 bytes per slot.
constexpr int VG32 = 6;
__device__ __forceinline__ void vertex32(const Topo& t, const FaceF* __restrict__ fd, const EdgeF* __restrict__ ed,
                                         const double* __restrict__ reppot, const EP& ep, int v,
                                         float4* X, float* __restrict__ rho, double* pr) {
  const int d = t.val[v];
  float A = 0, V = 0, LT = 0, T = 0;
  for (int m0 = 0; m0 < d; m0 += VG32) {
    int4 s[VG32];
#pragma unroll
    for (int k = 0; k < VG32; ++k) s[k] = m0 + k < d ? t.slot[(size_t)(m0 + k) * t.nv + v] : make_int4(0, -1, 0, 0);
    float fa[VG32], fv[VG32];
    EdgeF E[VG32];
#pragma unroll
    for (int k = 0; k < VG32; ++k) {
      const int f = slot_face(s[k].y);
      if (f < 0) continue;
      const float2 av = *reinterpret_cast<const float2*>(&fd[f].A);
      fa[k] = av.x;
      fv[k] = av.y;
      E[k] = ed[s[k].z];
    }
#pragma unroll
    for (int k = 0; k < VG32; ++k) {
      if (slot_face(s[k].y) < 0) continue;
      A += fa[k];
      V += fv[k];
      LT += E[k].length() * E[k].th;
      if (ep.btype == 0) {
        T += E[k].bond;
      } else {
        float q = fa[k] / (float)ep.a0 - 1.0f;
        T += q * q;
      }
    }
  }
  float a = A / 3, c = 0.25f * LT;
  pr[0] = a;
  pr[1] = V / 3;
  pr[2] = c;
  pr[3] = 2 * c * c / a;
  pr[4] = T / (float)ep.tdiv;
  pr[5] = reppot[v];
  const float rv = c / a;
  X[2 * (size_t)v].w = rv;
  rho[v] = rv;
}

__global__ void __launch_bounds__(VB) k_vertex32(Topo t, const FaceF* __restrict__ fd, const EdgeF* __restrict__ ed,
                                                const double* __restrict__ reppot, EP ep, float4* X,
                                                float* __restrict__ rho, double* partial, Globals* g) {
  int v = blockIdx.x * VB + threadIdx.x;
  double pr[6] = {0, 0, 0, 0, 0, 0};
  if (v < t.nv) vertex32(t, fd, ed, reppot, ep, v, X, rho, pr);
  finish_props(pr, partial, gridDim.x, blockIdx.x, ep, g);
}

__device__ __forceinline__ float cotf_at(const FaceF& F, int c) { return c == 0 ? F.c0 : (c == 1 ? F.c1 : F.c2); }

// Gradient of vertex i over its ring.  Per slot three gathers (neighbour with
// its rho, face and edge record; on an open mesh also the opposite edge's
// flag), where separate position and rho arrays took eleven.
template <bool CLOSED>
__device__ __forceinline__ f3 grad32(const Topo& t, const Split& S, const FaceF* __restrict__ fd,
                                     const EdgeF* __restrict__ ed, const double* __restrict__ repg, const Globals* g,
                                     const EP& ep, int i) {
  const float gA = (float)g->gA, gV = (float)g->gV, gC = (float)g->gC;
  const float kb = (float)ep.kb, kt = (float)ep.kt, a0 = (float)ep.a0;
  const float hgC = 0.5f * gC;
  const float kb23 = kb * (2.0f / 3.0f);
  f3 acc = (float)ep.kr * f3{(float)repg[3 * i], (float)repg[3 * i + 1], (float)repg[3 * i + 2]};
  const int d = t.val[i];
  if (d <= 0) return acc;
  const size_t nv = t.nv;
  auto face = [&](int f) {
    float4 a, b;
    ld32(reinterpret_cast<const float4*>(fd + f), a, b);
    return FaceF{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  };
  const Pos32 xi = S.at(i);
  const float ri = xi.rho;
  // neighbour positions relative to x_i (accurate small vectors)
  int4 sc = t.slot[i];
  const Pos32 pk = S.at(t.slot[(size_t)(d - 1) * nv + i].x);
  f3 xk = diff(pk, xi);
  float rk = pk.rho;
  Pos32 pj = S.at(sc.x);
  f3 xj = diff(pj, xi);
  float rj = pj.rho;
  FaceF Fc;
  int fcur = slot_face(sc.y);
  if (CLOSED || fcur >= 0) Fc = face(fcur);
  // normal multiples summed per face; the dihedral part of edge (i, j) on
  // the next face is carried to the next slot
  float carry = 0.0f;
  f3 n0 = {0.0f, 0.0f, 0.0f};
  for (int m = 0; m < d; ++m) {
    int4 sn = t.slot[(size_t)((m + 1) == d ? 0 : m + 1) * nv + i];
    int fnx = slot_face(sn.y);
    FaceF Fn;
    if (CLOSED || fnx >= 0) Fn = face(fnx);
    pj = S.at(sn.x);
    float carry_next = 0.0f;
    if (CLOSED || fcur >= 0) {
      int ci = slot_corner(sc.y);
      float cj = cotf_at(Fc, ci == 2 ? 0 : ci + 1);
      float ck = cotf_at(Fc, ci == 0 ? 2 : ci - 1);
      f3 n = {Fc.nx, Fc.ny, Fc.nz};
      if (m == 0) n0 = n;
      float alpha = gA - kb23 * (ri * ri + rj * rj + rk * rk);
      if (ep.btype == 1) alpha += kt * 2.0f * (Fc.A / a0 - 1.0f) / a0;
      acc += (0.5f * alpha) * fcross(n, xk - xj);
      // (x_j x x_k)/6 with x = x_i + d: x_i x (d_k - d_j) + d_j x d_k
      f3 vj = fcross(xi.hi, xk - xj) + fcross(xj, xk);
      acc += (gV * (1.0f / 6.0f)) * vj;
      EdgeF E = ed[sc.z];
      float w = hgC + kb * (ri + rj);
      float cl = w * E.th + (ep.btype == 0 ? kt * E.db : 0.0f);
      acc += (-cl / E.length()) * xj;
      float cn = carry;
      if (CLOSED || E.interior()) {
        int cin = slot_corner(sn.y);
        cn += w * cj;
        carry_next = w * cotf_at(Fn, cin == 0 ? 2 : cin - 1);
      }
      if (CLOSED || ed[sc.w].interior()) cn -= (hgC + kb * (rj + rk)) * (cj + ck);
      acc += cn * n;
    }
    carry = carry_next;
    xk = xj;
    rk = rj;
    sc = sn;
    fcur = fnx;
    Fc = Fn;
    xj = diff(pj, xi);
    rj = pj.rho;
  }
  acc += carry * n0;
  return acc;
}

template <bool CLOSED>
__global__ void __launch_bounds__(256) k_grad32(Topo t, Split S, const FaceF* __restrict__ fd,
                                               const EdgeF* __restrict__ ed, const double* __restrict__ repg,
                                               const Globals* __restrict__ g, EP ep, double* __restrict__ grad) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= t.nv) return;
  const f3 r = grad32<CLOSED>(t, S, fd, ed, repg, g, ep, i);
  grad[3 * i] = r.x;
  grad[3 * i + 1] = r.y;
  grad[3 * i + 2] = r.z;
}

// ---- batch of replicas (disjoint-union mesh, replica-aligned blocks) -----
// Same arithmetic as the single-mesh FP32 kernels; the parameters and the
// global sums are per replica (vrep: vertex -> replica, -1 for padding).

// edges [e0, e1)
__global__ void k_edge32b(int e0, int e1, Topo t, Split S, const FaceF* __restrict__ fd, EdgeF* __restrict__ ed,
                          const EP* __restrict__ eps, const int* __restrict__ vrep) {
  int e = e0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= e1) return;
  const int4 E = t.edge[e];
  ed[e] = edge32(E, S, fd, eps[vrep[E.x]]);
}

__global__ void __launch_bounds__(VB) k_vertex32b(Topo t, const FaceF* __restrict__ fd, const EdgeF* __restrict__ ed,
                                                 const double* __restrict__ reppot, const EP* __restrict__ eps,
                                                 const int* __restrict__ vrep, const int2* __restrict__ rblocks,
                                                 float4* X, float* __restrict__ rho, double* partial, Globals* gs) {
  const int rep = vrep[blockIdx.x * VB];  // blocks never straddle replicas
  const EP& ep = eps[rep];
  const int2 rb = rblocks[rep];
  int v = blockIdx.x * VB + threadIdx.x;
  double pr[6] = {0, 0, 0, 0, 0, 0};
  if (v < t.nv && vrep[v] >= 0) vertex32(t, fd, ed, reppot, ep, v, X, rho, pr);
  finish_props(pr, partial + 8 * (size_t)rb.x, rb.y - rb.x, blockIdx.x - rb.x, ep, gs + rep);
}

// vertices [v0, v1)
template <bool CLOSED>
__global__ void __launch_bounds__(256) k_grad32b(int v0, int v1, Topo t, Split S, const FaceF* __restrict__ fd,
                                                const EdgeF* __restrict__ ed, const double* __restrict__ repg,
                                                const Globals* __restrict__ gs, const EP* __restrict__ eps,
                                                const int* __restrict__ vrep, double* __restrict__ grad) {
  int i = v0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= v1) return;
  const int rep = vrep[i];
  f3 r = {0.0f, 0.0f, 0.0f};
  if (rep >= 0) r = grad32<CLOSED>(t, S, fd, ed, repg, gs + rep, eps[rep], i);
  grad[3 * i] = r.x;
  grad[3 * i + 1] = r.y;
  grad[3 * i + 2] = r.z;
}

inline int nblk(long n, int b) { return (int)((n + b - 1) / b); }

}  // namespace

void energy_eval32(tm_energy* e, tm_mesh* m, const double* P, bool want_grad, bool want_vprops, double* d_grad,
                   cudaStream_t s, cudaEvent_t* ev) {
  e->ensure(m->nv, m->ne, m->nf);
  size_t nv = std::max(m->nv, 1), ne = std::max(m->ne, 1), nf = std::max(m->nf, 1);
  // FP32 records live in the FP64 buffers (they are smaller)
  Topo t = m->topo();
  EP ep = make_ep(e);
  float4* X = e->posdw.get();
  Split S{X};
  FaceF* fd = reinterpret_cast<FaceF*>(e->face.get());
  EdgeF* ed = reinterpret_cast<EdgeF*>(e->edge.get());
  float* rho = reinterpret_cast<float*>(e->rho.get());
  double* repg = e->repg.get();
  (void)nf;
  (void)ne;
  if (ev) TM_CUDA(cudaEventRecord(ev[0], s));
  if (m->nv) k_split<0><<<nblk(m->nv, 256), 256, 0, s>>>(m->nv, P, SplitMove{}, X, e->pos32.get());
  TM_LAUNCH();
  const bool conc = ev == nullptr;  // repulsion overlaps the face and edge kernels
  if (conc) fork_repulsion(e, m, P, want_grad, s, true);
  if (t.nf) k_face32<<<nblk(t.nf, 256), 256, 0, s>>>(0, t.nf, t, S, fd);
  TM_LAUNCH();
  if (ev) TM_CUDA(cudaEventRecord(ev[1], s));
  if (t.ne) k_edge32<<<nblk(t.ne, 256), 256, 0, s>>>(t, S, fd, ed, ep);
  TM_LAUNCH();
  if (ev) TM_CUDA(cudaEventRecord(ev[2], s));
  if (conc)
    join_repulsion(e, s, true);
  else
    fork_repulsion(e, m, P, want_grad, s, false);
  (void)repg;
  int nb = std::max(1, nblk(t.nv, VB));
  (void)want_vprops;
  k_vertex32<<<nb, VB, 0, s>>>(t, fd, ed, e->reppot.get(), ep, X, rho, e->partials.get(), e->glob.get());
  TM_LAUNCH();
  if (ev) TM_CUDA(cudaEventRecord(ev[3], s));
  if (want_grad && t.nv)
    (m->closed ? k_grad32<true> : k_grad32<false>)<<<nblk(t.nv, 256), 256, 0, s>>>(t, S, fd, ed, repg, e->glob.get(),
                                                                                     ep, d_grad);
  TM_LAUNCH();
  if (ev) TM_CUDA(cudaEventRecord(ev[4], s));
}

// The local terms of the energy only (bending and repulsion weights set to
// zero, no neighbour pass) with FP32 stencils: the exact part of the
// surrogate force.  Leaves the FP32 face / edge records, rho = c/a per vertex
// and the split positions (e->posdw) filled for the caller.
void energy_eval32_local(tm_energy* e, tm_mesh* m, const double* P, double* d_grad, cudaStream_t s) {
  e->ensure(m->nv, m->ne, m->nf);
  size_t nv = std::max(m->nv, 1);
  Topo t = m->topo();
  EP ep = make_ep(e);
  ep.kb = 0.0;
  ep.kr = 0.0;
  float4* X = e->posdw.get();
  Split S{X};
  FaceF* fd = reinterpret_cast<FaceF*>(e->face.get());
  EdgeF* ed = reinterpret_cast<EdgeF*>(e->edge.get());
  float* rho = reinterpret_cast<float*>(e->rho.get());
  TM_CUDA(cudaMemsetAsync(e->reppot.get(), 0, sizeof(double) * nv, s));
  TM_CUDA(cudaMemsetAsync(e->repg.get(), 0, sizeof(double) * 3 * nv, s));
  if (m->nv) k_split<0><<<nblk(m->nv, 256), 256, 0, s>>>(m->nv, P, SplitMove{}, X, e->pos32.get());
  TM_LAUNCH();
  if (t.nf) k_face32<<<nblk(t.nf, 256), 256, 0, s>>>(0, t.nf, t, S, fd);
  TM_LAUNCH();
  if (t.ne) k_edge32<<<nblk(t.ne, 256), 256, 0, s>>>(t, S, fd, ed, ep);
  TM_LAUNCH();
  int nb = std::max(1, nblk(t.nv, VB));
  k_vertex32<<<nb, VB, 0, s>>>(t, fd, ed, e->reppot.get(), ep, X, rho, e->partials.get(), e->glob.get());
  TM_LAUNCH();
  if (t.nv)
    (m->closed ? k_grad32<true> : k_grad32<false>)<<<nblk(t.nv, 256), 256, 0, s>>>(t, S, fd, ed, e->repg.get(),
                                                                                     e->glob.get(), ep, d_grad);
  TM_LAUNCH();
}

// One element kernel of one size class of a batch: which 1 face, 2 edge, 3
// gradient, with block size blk, on stream s.
void batch32_class_kernel(int which, const BatchClass& c, int blk, tm_energy* e, tm_mesh* m, double* d_grad,
                          const EP* eps, const int* vrep, const Globals* gs, cudaStream_t s) {
  Topo t = m->topo();
  Split S{e->posdw.get()};
  FaceF* fd = reinterpret_cast<FaceF*>(e->face.get());
  EdgeF* ed = reinterpret_cast<EdgeF*>(e->edge.get());
  if (which == 1 && c.f1 > c.f0) k_face32<<<nblk(c.f1 - c.f0, blk), blk, 0, s>>>(c.f0, c.f1, t, S, fd);
  if (which == 2 && c.e1 > c.e0)
    k_edge32b<<<nblk(c.e1 - c.e0, blk), blk, 0, s>>>(c.e0, c.e1, t, S, fd, ed, eps, vrep);
  if (which == 3 && c.v1 > c.v0)
    (m->closed ? k_grad32b<true> : k_grad32b<false>)<<<nblk(c.v1 - c.v0, blk), blk, 0, s>>>(
        c.v0, c.v1, t, S, fd, ed, e->repg.get(), gs, eps, vrep, d_grad);
  TM_LAUNCH();
}

// The batch's evaluation: the positions' split for all replicas (after the
// velocity-Verlet update of leap, when given), then per size class
// (consecutive replicas of similar size, each with its own tuned block sizes)
// the face and edge kernels, the repulsion beside them on a stream of its
// own, the vertex stage for all replicas, and the gradient per class.  With
// side streams the classes' kernels run side by side (fork and join events),
// so the small replicas' launches fill the SMs the large ones leave idle.
void energy_eval_batch32(tm_energy* e, tm_mesh* m, const double* P, double* d_grad, const EP* eps,
                         const int* vrep, const int2* rblocks, Globals* gs, const BatchClass* cls, int ncls,
                         const BatchStreams& bs, const Leap* leap, cudaStream_t s) {
  e->ensure(m->nv, m->ne, m->nf);
  size_t nv = std::max(m->nv, 1);
  Topo t = m->topo();
  FaceF* fd = reinterpret_cast<FaceF*>(e->face.get());
  EdgeF* ed = reinterpret_cast<EdgeF*>(e->edge.get());
  float* rho = reinterpret_cast<float*>(e->rho.get());
  SplitMove mv{};
  if (leap)
    mv = SplitMove{leap->x, leap->p, leap->g0, leap->g1, leap->dt, 0.5 * leap->dt, 0.5 * (leap->dt * leap->dt), leap->im};
  auto* ks = !leap ? k_split<0> : (leap->g1 ? k_split<2> : k_split<1>);
  ks<<<std::max(1, nblk(m->nv, 256)), 256, 0, s>>>(m->nv, P, mv, e->posdw.get(), e->pos32.get());
  TM_LAUNCH();
  const bool side = ncls > 1;
  auto stream_of = [&](int c) { return side ? bs.cs[c] : s; };
  auto fork = [&](int k) {
    TM_CUDA(cudaEventRecord(bs.fork[k], s));
    if (k == 0) TM_CUDA(cudaStreamWaitEvent(bs.rep, bs.fork[k], 0));
    for (int c = 0; side && c < ncls; ++c) TM_CUDA(cudaStreamWaitEvent(bs.cs[c], bs.fork[k], 0));
  };
  auto join = [&]() {
    for (int c = 0; side && c < ncls; ++c) {
      TM_CUDA(cudaEventRecord(bs.join[c], bs.cs[c]));
      TM_CUDA(cudaStreamWaitEvent(s, bs.join[c], 0));
    }
  };
  fork(0);
  repulsion_eval(e, m, P, e->pos32.get(), true, e->reppot.get(), e->repg.get(), e->slow.get(),
                 e->slow.get() + std::max(m->nv, 1), bs.rep, eps);
  TM_CUDA(cudaEventRecord(bs.join_rep, bs.rep));
  for (int c = 0; c < ncls; ++c)
    for (int k = 1; k < 3; ++k)
      batch32_class_kernel(k, cls[c], cls[c].blk[k], e, m, d_grad, eps, vrep, gs, stream_of(c));
  join();
  TM_CUDA(cudaStreamWaitEvent(s, bs.join_rep, 0));
  int nb = std::max(1, nblk(t.nv, VB));
  k_vertex32b<<<nb, VB, 0, s>>>(t, fd, ed, e->reppot.get(), eps, vrep, rblocks, e->posdw.get(), rho,
                                e->partials.get(), gs);
  TM_LAUNCH();
  fork(1);
  for (int c = 0; c < ncls; ++c)
    batch32_class_kernel(3, cls[c], cls[c].blk[3], e, m, d_grad, eps, vrep, gs, stream_of(c));
  join();
}

}  // namespace tmg
