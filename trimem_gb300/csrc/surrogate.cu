// Learned surrogate force for hybrid HMC: the leapfrog integrates
//   -grad E(x)  ~  -(g_local(x) - F_nn(x)),
// where g_local is the exact gradient of the local penalty terms (area,
// volume, area difference, tether; FP32 stencils, one pass without the
// neighbour list) and F_nn is a message-passing network that stands in for
// the bending and repulsion forces.  Acceptance always uses the exact FP64
// Hamiltonian, so the chain samples the exact distribution; the surrogate
// only changes how often proposals are accepted.
//
// Network (width H = 64, SiLU, three rounds), per vertex i with ring j:
//   u_i   = 8 rotation-invariant vertex features (area, curvature, valence,
//           dihedral and edge-length statistics of the ring)
//   e_ij  = 4 edge features (length, dihedral, curvature difference / mean)
//   h_i   = SiLU(W_in u_i + b_in)
//   round r:  m_i = sum_j (W_e^r e_ij + b_e^r) * h_j          (gather, CUDA cores)
//             h_i = h_i + SiLU(W^r [h_i ; m_i] + b^r)          (tcgen05 BF16 GEMM)
//   F_i   = s ( sum_j c_ij (x_j - x_i)/|x_j - x_i| + c_i N_i ),
//           c_ij = sum_c w_o,c h_i,c h_j,c + b_o,  c_i = w_n . h_i + b_n,
//           N_i the area-weighted vertex normal.
// F is equivariant by construction (invariant coefficients on the edge
// directions and the normal).  Activations h, m are stored as bf16, the
// dense weights W^r are bf16 with FP32 accumulation in tensor memory; the
// small layers are FP32.
//
// A round is one CTA per 128 vertices (k_layer): TMA loads h (a 128 x 64 bf16
// box) and W^r (two 64 x 64 boxes) into 128-byte-swizzled shared memory while
// the threads gather the messages m into the other operand tile; one thread
// issues 8 tcgen05.mma (M 128, N 64, K 16), the accumulator (128 lanes x 64
// FP32 columns) is read back by eight warps, the epilogue adds bias, SiLU and
// the residual h (in the swizzled tile), and TMA stores the tile.  k_dense is
// the dense layer alone, on given [h | m] (tm_dense_silu_bf16).
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "tm_energy.cuh"
#include "tm_fp32.cuh"
#include "tm_internal.h"
#include "tm_math.cuh"
#include "tm_tc.cuh"

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

constexpr int H = 64, FV = 8, FE = 4, NR = 3, BM = 128;
constexpr int BLOB_HEADER = 8;
constexpr int BLOB_SIZE = BLOB_HEADER + H * FV + H + NR * (H * FE + H + H * 2 * H + H) + H + 1 + H + 1;

// FP32 parameters of the small layers (device copy)
struct SurW {
  float win[H * FV], bin[H];
  float we[NR][H * FE], be[NR][H], b[NR][H];
  float wo[H], wn[H];
  float bo, bn, lbar, abar, fscale;
};

}  // namespace

struct tm_surrogate {
  int nv = 0;
  SurW hw{};
  DevBuf<SurW> w;
  DevBuf<__nv_bfloat16> wd;  // dense weights [NR][H][2H] (row n, column k)
  DevBuf<float> nrm;
  DevBuf<__nv_bfloat16> hb[2];
  DevBuf<double> gloc;
  DevBuf<int> status;
  alignas(64) CUtensorMap map_h[2];
  alignas(64) CUtensorMap map_w[NR];
};

namespace {

using namespace tmg::fp32;
using tmg::tc::smem_u32;

inline int nblk(long n, int b) { return (int)((n + b - 1) / b); }

__device__ __forceinline__ float silu(float x) { return x / (1.0f + __expf(-x)); }

__device__ __forceinline__ uint4 pack8(const float* f) {
  uint4 v;
  __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int q = 0; q < 4; ++q) b[q] = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
  return v;
}

// the input layer's weights of channels 8 sub .. 8 sub + 7, in registers
struct Embed8 {
  float w[8][FV], b[8];
  __device__ __forceinline__ Embed8(const float* win, const float* bin, int sub) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float4* r = reinterpret_cast<const float4*>(win + (8 * sub + q) * FV);
      const float4 w0 = r[0], w1 = r[1];
      w[q][0] = w0.x, w[q][1] = w0.y, w[q][2] = w0.z, w[q][3] = w0.w;
      w[q][4] = w1.x, w[q][5] = w1.y, w[q][6] = w1.z, w[q][7] = w1.w;
      b[q] = bin[8 * sub + q];
    }
  }
  __device__ __forceinline__ void operator()(const float* x, float* y) const {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      y[q] = b[q];
#pragma unroll
      for (int k = 0; k < FV; ++k) y[q] += w[q][k] * x[k];
    }
  }
};

// vertex features and normal (one thread per vertex), then the embedding of
// the block's vertices by eight threads each, with the weights in registers
// and whole rows of h per store (one thread per vertex with 32 four-byte
// stores took 53 us at 163,842 vertices, now 35)
constexpr int SFB = 128;
__global__ void __launch_bounds__(SFB) k_sfeat(Topo t, const FaceF* __restrict__ fd, const EdgeF* __restrict__ ed,
                                               const float* __restrict__ rho, const SurW* __restrict__ W,
                                               float* __restrict__ u, float* __restrict__ nrm,
                                               __nv_bfloat16* __restrict__ h) {
  __shared__ float sx[SFB][FV + 1];
  const int i = blockIdx.x * SFB + threadIdx.x;
  if (i < t.nv) {
    const float lbar = W->lbar, abar = W->abar;
    const int d = t.val[i];
    float A = 0.f, ls = 0.f, l2 = 0.f, ths = 0.f, th2 = 0.f;
    f3 N = {0.f, 0.f, 0.f};
    int4 s = d > 0 ? t.slot[i] : make_int4(0, -1, 0, 0);
    for (int m = 0; m < d; ++m) {
      const int4 sn = m + 1 < d ? t.slot[(size_t)(m + 1) * t.nv + i] : s;
      const int f = slot_face(s.y);
      if (f >= 0) {
        FaceF F = fd[f];
        A += F.A;
        N += F.A * f3{F.nx, F.ny, F.nz};
      }
      EdgeF E = ed[s.z];
      float lr = E.length() / lbar;
      ls += lr;
      l2 += lr * lr;
      ths += E.th;
      th2 += E.th * E.th;
      s = sn;
    }
    float inv_d = d > 0 ? 1.0f / d : 0.0f;
    float* x = sx[threadIdx.x];
    float rl = rho[i] * lbar;
    x[0] = (A / 3.0f) / abar - 1.0f;
    x[1] = rl;
    x[2] = rl * rl;
    x[3] = (d - 6) * (1.0f / 6.0f);
    x[4] = ths * inv_d;
    x[5] = sqrtf(th2 * inv_d);
    x[6] = ls * inv_d - 1.0f;
    x[7] = sqrtf(fmaxf(l2 * inv_d - (ls * inv_d) * (ls * inv_d), 0.0f));
    float nn = fnorm(N);
    float in = nn > 0.f ? 1.0f / nn : 0.0f;
    reinterpret_cast<float4*>(nrm)[i] = make_float4(N.x * in, N.y * in, N.z * in, 0.f);
  }
  __syncthreads();
  const int v0 = blockIdx.x * SFB, n = min(SFB, t.nv - v0);
  if (u)
    for (int q = threadIdx.x; q < n * FV; q += SFB) u[(size_t)FV * v0 + q] = sx[q / FV][q % FV];
  const int sub = threadIdx.x & 7;
  const Embed8 emb(W->win, W->bin, sub);
  for (int v = threadIdx.x >> 3; v < n; v += SFB / 8) {
    float y[8];
    emb(sx[v], y);
#pragma unroll
    for (int q = 0; q < 8; ++q) y[q] = silu(y[q]);
    reinterpret_cast<uint4*>(h)[(size_t)(v0 + v) * (H / 8) + sub] = pack8(y);
  }
}

__device__ __forceinline__ void edge_feat(const EdgeF& E, float ri, float rj, float lbar, float* ef) {
  ef[0] = E.length() / lbar - 1.0f;
  ef[1] = E.th;
  ef[2] = (rj - ri) * lbar;
  ef[3] = 0.5f * (rj + ri) * lbar;
}

__device__ __forceinline__ void unpack8(uint4 v, float* f) {
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float2 x = __bfloat1622float2(b[q]);
    f[2 * q] = x.x;
    f[2 * q + 1] = x.y;
  }
}
// h_out = h + SiLU([h | m] W^T + b) for 128 vertices per CTA on the tensor cores
constexpr int DENSE_SMEM = 1024 + 49152 + 64;

// Every wait is bounded: wait_polls polls for the tile loads and for the MMA
// completion.  When a wait gives up the CTA records it in *status (1 loads,
// 2 MMA), skips the work that depended on it, waits (with the long default
// limit) for the copies and the MMA it did issue to land, and frees its
// tensor memory before it returns.
constexpr int WAIT_POLLS = 1 << 22;
__global__ void __launch_bounds__(128) k_dense(const __grid_constant__ CUtensorMap mh,
                                               const __grid_constant__ CUtensorMap mm,
                                               const __grid_constant__ CUtensorMap mw, const float* __restrict__ bias,
                                               __nv_bfloat16* __restrict__ out, int M, int* status, int wait_polls) {
  using namespace tmg::tc;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* A0 = base;           // h tile, 128 rows x 128 B
  uint8_t* A1 = base + 16384;   // m tile
  uint8_t* B0 = base + 32768;   // W[:, 0:64], 64 rows x 128 B
  uint8_t* B1 = base + 40960;   // W[:, 64:128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + 49152);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(base + 49152 + 16);
  int* issued = reinterpret_cast<int*>(base + 49152 + 20);  // the MMA was issued
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * BM;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&mh);
    tma_prefetch_desc(&mm);
    tma_prefetch_desc(&mw);
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    mbar_fence_init();
    *issued = 0;
  }
  if (warp == 0) {
    tmem_alloc(tslot, 64);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  if (threadIdx.x == 0) {
    mbar_expect_tx(&bars[0], 49152);
    tma_load_2d(A0, &mh, &bars[0], 0, m0);
    tma_load_2d(A1, &mm, &bars[0], 0, m0);
    tma_load_2d(B0, &mw, &bars[0], 0, 0);
    tma_load_2d(B1, &mw, &bars[0], 64, 0);
    if (mbar_wait(&bars[0], 0, wait_polls)) {
      tc_fence_after();
      constexpr uint32_t idesc = idesc_bf16_f32(BM, H);
#pragma unroll
      for (int kc = 0; kc < 2; ++kc) {
        const uint32_t a = smem_u32(kc ? A1 : A0), b = smem_u32(kc ? B1 : B0);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mma_bf16(tmem, sdesc_sw128(a + 32 * k, 1024), sdesc_sw128(b + 32 * k, 1024), idesc, (kc | k) != 0);
      }
      mma_commit(&bars[1]);
      *issued = 1;
    } else {
      atomicExch(status, 1);  // tile loads did not arrive in time
      // the copies are still this CTA's: let them land before it exits
      if (!mbar_wait(&bars[0], 0, WAIT_POLLS)) atomicExch(status, 3);
    }
  }
  __syncthreads();
  bool done = __all_sync(0xffffffffu, mbar_wait(&bars[1], 0, wait_polls));
  tc_fence_after();
  if (done) {
    const int r = warp * 32 + lane;
    float acc[H];
    const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
    tmem_ld32(taddr, acc);
    tmem_ld32(taddr + 32, acc + 32);
    if (m0 + r < M) {
      const uint8_t* rowp = A0 + (r >> 3) * 1024 + (r & 7) * 128;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint4 hv = *reinterpret_cast<const uint4*>(rowp + ((c ^ (r & 7)) * 16));
        const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&hv);
        uint4 ov;
        __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int n = c * 8 + 2 * q;
          float2 hf = __bfloat1622float2(h2[q]);
          const float z0 = acc[n] + bias[n], z1 = acc[n + 1] + bias[n + 1];
          o2[q] = __floats2bfloat162_rn(hf.x + silu(z0), hf.y + silu(z1));
        }
        *reinterpret_cast<uint4*>(out + (size_t)(m0 + r) * H + c * 8) = ov;
      }
    }
  } else {
    if (lane == 0) atomicExch(status, 2);  // the MMA completion did not arrive in time
    // an MMA that was issued still writes the accumulator: wait for it
    // before the tensor memory is freed
    if (threadIdx.x == 0 && *issued && !mbar_wait(&bars[1], 0, WAIT_POLLS)) atomicExch(status, 3);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 64);
}

// One round for 128 vertices per CTA: m_i = sum_j (W_e e_ij + b_e) * h_j into
// the second operand tile, then h_out = h + SiLU([h | m] W^T + b) as in
// k_dense.  What bounds it is the gather of h_j (six rows of 128 bytes per
// vertex, from L2): eight threads share a vertex with eight channels (16
// bytes) each, lane k of the eight loads ring slot k (index and edge features
// once per slot, the next vertex's while the current one is summed) and hands
// them around, and four gathers are in flight per thread.  The message weights
// stay in registers over a thread's four vertices.  Separate kernels with 16
// threads per vertex, every one of them loading every slot's features, took
// 70 + 29 us a round at 163,842 vertices, this one 64; three CTAs per SM (80
// registers, 50 bytes spilled) beat two (112) by 13 us a round.
struct LayerIn {
  // inference: rings and edge records of the mesh
  Topo t;
  const EdgeF* ed;
  const float* rho;
  float lbar;
  // training: exported rings [D][n]
  const int* nbr;
  const float4* ef;
  int D;
  const float *we, *be, *bias;  // W_e (64 x 4), b_e, dense bias
  const uint4* h;               // activations in, 8 x 16 bytes per vertex
  float* z;                     // training: pre-activations out
  int M;
  int* status;
};
struct RingSlot {
  int j, edge, lim;  // neighbour (-1: none), its edge, ring slots of the vertex
};
constexpr int LT = 256;
constexpr int LAYER_SMEM = DENSE_SMEM;
template <bool TRAIN>
__device__ __forceinline__ RingSlot ring_slot(const LayerIn& q, int i, int m) {
  if (TRAIN) return {i < q.M && m < q.D ? q.nbr[(size_t)m * q.M + i] : -1, 0, q.D};
  if (i >= q.M || m >= TM_MAXVAL) return {-1, 0, 0};
  const int d = q.t.val[i];
  const int4 s = q.t.slot[(size_t)m * q.M + i];
  return {m < d ? s.x : -1, s.z, d};
}
// e_ij of slot m
template <bool TRAIN>
__device__ __forceinline__ float4 ring_feat(const LayerIn& q, const RingSlot& r, int i, int m) {
  if (r.j < 0) return make_float4(0.f, 0.f, 0.f, 0.f);
  if (TRAIN) return q.ef[(size_t)m * q.M + i];
  float e[FE];
  edge_feat(q.ed[r.edge], q.rho[i], q.rho[r.j], q.lbar, e);
  return make_float4(e[0], e[1], e[2], e[3]);
}

template <bool TRAIN>
__global__ void __launch_bounds__(LT, 3) k_layer(const __grid_constant__ CUtensorMap mh,
                                                 const __grid_constant__ CUtensorMap mw,
                                                 const __grid_constant__ CUtensorMap mout,
                                                 const __grid_constant__ CUtensorMap mm,
                                                 const __grid_constant__ LayerIn q) {
  using namespace tmg::tc;
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* A0 = base;           // h tile, 128 rows x 128 B; later the result
  uint8_t* A1 = base + 16384;   // m tile
  uint8_t* B0 = base + 32768;   // W[:, 0:64], 64 rows x 128 B
  uint8_t* B1 = base + 40960;   // W[:, 64:128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + 49152);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(base + 49152 + 16);
  int* issued = reinterpret_cast<int*>(base + 49152 + 20);  // the MMA was issued
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * BM;
  if (threadIdx.x == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    mbar_fence_init();
    *issued = 0;
    mbar_expect_tx(&bars[0], 32768);
    tma_load_2d(A0, &mh, &bars[0], 0, m0);
    tma_load_2d(B0, &mw, &bars[0], 0, 0);
    tma_load_2d(B1, &mw, &bars[0], 64, 0);
  }
  if (warp == 0) {
    __syncwarp();
    tmem_alloc(tslot, 64);
    tmem_relinquish();
  }
  // messages: rows 32 it + (thread >> 3), it < 4
  {
    const int sub = threadIdx.x & 7, grp = threadIdx.x >> 3;
    float4 w[8];
    float b[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      w[c] = *reinterpret_cast<const float4*>(q.we + (8 * sub + c) * FE);
      b[c] = q.be[8 * sub + c];
    }
    RingSlot r = ring_slot<TRAIN>(q, m0 + grp, sub);
    float4 e = ring_feat<TRAIN>(q, r, m0 + grp, sub);
    for (int it = 0; it < 4; ++it) {
      const int row = 32 * it + grp, i = m0 + row;
      RingSlot rn = {-1, 0, 0};
      if (it < 3) rn = ring_slot<TRAIN>(q, i + 32, sub);
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int m = 0;;) {  // eight slots at a time; the ring ends at the first absent one
        const unsigned have = (__ballot_sync(FULL, r.j >= 0) >> (lane & 24)) & 0xffu;
        const int cnt = have == 0xffu ? 8 : __ffs(~have) - 1;
        const int most = __reduce_max_sync(FULL, cnt);
#pragma unroll
        for (int k0 = 0; k0 < 8; k0 += 4) {
          if (k0 >= most) break;
          uint4 hv[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int j = __shfl_sync(FULL, r.j, k0 + k, 8);
            hv[k] = make_uint4(0u, 0u, 0u, 0u);
            if (k0 + k < cnt) hv[k] = q.h[(size_t)j * (H / 8) + sub];
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float4 f = make_float4(__shfl_sync(FULL, e.x, k0 + k, 8), __shfl_sync(FULL, e.y, k0 + k, 8),
                                         __shfl_sync(FULL, e.z, k0 + k, 8), __shfl_sync(FULL, e.w, k0 + k, 8));
            float hj[8];
            unpack8(hv[k], hj);
            if (k0 + k < cnt) {
#pragma unroll
              for (int c = 0; c < 8; ++c)
                acc[c] += (b[c] + w[c].x * f.x + w[c].y * f.y + w[c].z * f.z + w[c].w * f.w) * hj[c];
            }
          }
        }
        m += 8;
        const bool more = cnt == 8 && m < r.lim;
        if (!__any_sync(FULL, more)) break;
        r.j = -1;
        if (more) r = ring_slot<TRAIN>(q, i, m + sub);
        e = ring_feat<TRAIN>(q, r, i, m + sub);
      }
      *reinterpret_cast<uint4*>(A1 + (row >> 3) * 1024 + (row & 7) * 128 + ((sub ^ (row & 7)) * 16)) = pack8(acc);
      r = rn;
      if (it < 3) e = ring_feat<TRAIN>(q, r, i + 32, sub);
    }
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  if (threadIdx.x == 0) {
    if (mbar_wait(&bars[0], 0, WAIT_POLLS)) {
      constexpr uint32_t idesc = idesc_bf16_f32(BM, H);
#pragma unroll
      for (int kc = 0; kc < 2; ++kc) {
        const uint32_t a = smem_u32(kc ? A1 : A0), b = smem_u32(kc ? B1 : B0);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mma_bf16(tmem, sdesc_sw128(a + 32 * k, 1024), sdesc_sw128(b + 32 * k, 1024), idesc, (kc | k) != 0);
      }
      mma_commit(&bars[1]);
      *issued = 1;
    } else {
      atomicExch(q.status, 1);  // tile loads did not arrive in time
      // the copies are still this CTA's: let them land before it exits
      if (!mbar_wait(&bars[0], 0, WAIT_POLLS)) atomicExch(q.status, 3);
    }
  }
  __syncthreads();
  const bool done = __syncthreads_and(*issued && mbar_wait(&bars[1], 0, WAIT_POLLS));
  tc_fence_after();
  if (done) {
    // warp w: rows 32 (w & 3) + lane, columns 32 (w >> 2) .. + 31
    const int r = (warp & 3) * 32 + lane, n0 = (warp >> 2) * 32;
    float acc[32];
    tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + n0, acc);
    uint8_t* rowp = A0 + (r >> 3) * 1024 + (r & 7) * 128;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint4* hp = reinterpret_cast<uint4*>(rowp + (((n0 / 8 + c) ^ (r & 7)) * 16));
      float hf[8], o[8];
      unpack8(*hp, hf);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float z = acc[8 * c + k] + q.bias[n0 + 8 * c + k];
        acc[8 * c + k] = z;
        o[k] = hf[k] + silu(z);
      }
      *hp = pack8(o);
    }
    if (TRAIN && m0 + r < q.M) {
      float4* z4 = reinterpret_cast<float4*>(q.z + (size_t)(m0 + r) * H + n0);
#pragma unroll
      for (int c = 0; c < 8; ++c) z4[c] = make_float4(acc[4 * c], acc[4 * c + 1], acc[4 * c + 2], acc[4 * c + 3]);
    }
    fence_async_smem();
  } else if (threadIdx.x == 0) {
    atomicExch(q.status, 2);  // the MMA completion did not arrive in time
    // an MMA that was issued still writes the accumulator: wait for it
    // before the tensor memory is freed
    if (*issued && !mbar_wait(&bars[1], 0, WAIT_POLLS)) atomicExch(q.status, 3);
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && done) {
    tma_store_2d(&mout, A0, 0, m0);
    if (TRAIN) tma_store_2d(&mm, A1, 0, m0);
    tma_store_wait();
  }
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem, 64);
  }
}

// output head: g = g_local - s (sum_j c_ij d_ij + c_i N_i), eight threads
// per vertex with eight channels each; lane k of the eight holds ring slot
// k's neighbour and direction, the eight slots' products are gathered in
// flight together and reduced so that lane k ends with slot k's sum (7
// shuffles for eight slots, the same pairs as eight butterflies), and three
// lanes add the slots in order.  Every lane computing every direction, 24
// shuffles: 53 us at 163,842 vertices, now 38.
__global__ void __launch_bounds__(256) k_out(Topo t, Split S, const float* __restrict__ nrm,
                                             const SurW* __restrict__ W, const __nv_bfloat16* __restrict__ h,
                                             const double* __restrict__ gloc, double* __restrict__ g) {
  __shared__ float4 term[256];  // (c_ij / |e|, e) of each slot
  constexpr unsigned FULL = 0xffffffffu;
  const int gt = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = gt >> 3, sub = gt & 7;
  const bool act = i < t.nv;
  const int ii = act ? i : 0, d = act ? t.val[i] : 0;
  const uint4* h4 = reinterpret_cast<const uint4*>(h);
  float hi[8], pi[8];
  unpack8(h4[(size_t)ii * (H / 8) + sub], hi);
  float cn = 0.f;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    pi[c] = W->wo[8 * sub + c] * hi[c];
    cn += W->wn[8 * sub + c] * hi[c];
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) cn += __shfl_xor_sync(FULL, cn, o);
  cn += W->bn;
  const float bo = W->bo;
  float F = cn * nrm[4 * (size_t)ii + (sub < 3 ? sub : 3)];  // lane k < 3: component k
  const float4* mine = term + (threadIdx.x & ~7);
  const Pos32 xi = S.at(ii);
  for (int m = 0; __any_sync(FULL, m < d); m += 8) {
    const int cnt = min(8, d - m);
    int j = -1;
    f3 e = {0.f, 0.f, 0.f};
    if (sub < cnt) {
      j = t.nbr[(size_t)(m + sub) * t.nv + ii];
      e = diff(S.at(j), xi);
    }
    float c[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int jk = __shfl_sync(FULL, j, k, 8);
      c[k] = 0.f;
      if (k < cnt) {
        float hj[8];
        unpack8(h4[(size_t)jk * (H / 8) + sub], hj);
#pragma unroll
        for (int q = 0; q < 8; ++q) c[k] += pi[q] * hj[q];
      }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {  // keep the slots whose bit o is this lane's
      const bool up = (sub & o) != 0;
#pragma unroll
      for (int k = 0; k < 8 / (2 * o); ++k) {
        const float keep = up ? c[2 * k + 1] : c[2 * k], send = up ? c[2 * k] : c[2 * k + 1];
        c[k] = keep + __shfl_xor_sync(FULL, send, o);
      }
    }
    const float s = j >= 0 ? (c[0] + bo) / fnorm(e) : 0.f;
    term[threadIdx.x] = make_float4(e.x, e.y, e.z, s);
    __syncwarp();
    if (sub < 3)
      for (int k = 0; k < cnt; ++k) F += mine[k].w * (sub == 0 ? mine[k].x : (sub == 1 ? mine[k].y : mine[k].z));
    __syncwarp();
  }
  if (act && sub < 3) g[3 * (size_t)i + sub] = gloc[3 * (size_t)i + sub] - (double)(W->fscale * F);
}

// training inputs: ring neighbours, edge features and unit edge directions,
// slot-major [D][nv] (neighbour -1 and zeros past the valence)
__global__ void k_export(Topo t, Split S, const EdgeF* __restrict__ ed, const float* __restrict__ rho,
                         const SurW* __restrict__ W, int D, int* __restrict__ nbr, float* __restrict__ ef,
                         float* __restrict__ tv) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= t.nv) return;
  int d = t.val[i];
  for (int m = 0; m < D; ++m) {
    size_t o = (size_t)m * t.nv + i;
    float f[FE] = {0.f, 0.f, 0.f, 0.f};
    f3 dir = {0.f, 0.f, 0.f};
    int j = -1;
    if (m < d) {
      int4 s = t.slot[o];
      j = s.x;
      edge_feat(ed[s.z], rho[i], rho[j], W->lbar, f);
      f3 e = diff(S.at(j), S.at(i));
      dir = (1.0f / fnorm(e)) * e;
    }
    nbr[o] = j;
    for (int k = 0; k < FE; ++k) ef[FE * o + k] = f[k];
    tv[3 * o] = dir.x;
    tv[3 * o + 1] = dir.y;
    tv[3 * o + 2] = dir.z;
  }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    TM_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q));
    if (q != cudaDriverEntryPointSuccess || !p) fail(TM_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// bf16 row-major [rows][cols] matrix, boxes of 64 columns x box_rows rows,
// 128-byte swizzle
void make_map(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_rows) {
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0) fail(TM_ERR_ARG, "tensor base not 16-byte aligned");
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * sizeof(__nv_bfloat16)};
  cuuint32_t box[2] = {64, box_rows};
  cuuint32_t es[2] = {1, 1};
  CUresult r = encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, es,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) fail(TM_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
}

// a kernel's limit of dynamic shared memory belongs to the current device: set
// for every handle at its creation, and on every call without one
template <class K>
void allow_smem(K* k, int bytes) {
  TM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}

void dense_launch(const CUtensorMap& mh, const CUtensorMap& mm, const CUtensorMap& mw, const float* bias,
                  __nv_bfloat16* out, int M, int* status, cudaStream_t s, int wait_polls) {
  allow_smem(k_dense, DENSE_SMEM);
  if (M > 0) k_dense<<<nblk(M, BM), BM, DENSE_SMEM, s>>>(mh, mm, mw, bias, out, M, status, wait_polls);
  TM_LAUNCH();
}

template <bool TRAIN>
void layer_launch(const CUtensorMap& mh, const CUtensorMap& mw, const CUtensorMap& mout, const CUtensorMap& mm,
                  const LayerIn& in, cudaStream_t s) {
  k_layer<TRAIN><<<nblk(in.M, BM), LT, LAYER_SMEM, s>>>(mh, mw, mout, mm, in);
  TM_LAUNCH();
}

void parse_blob(const float* b, int64_t n, SurW& w, std::vector<__nv_bfloat16>& wd) {
  if (n != BLOB_SIZE) fail(TM_ERR_ARG, "surrogate weights: expected " + std::to_string(BLOB_SIZE) + " floats");
  if (b[0] != 1.0f || b[1] != FV || b[2] != FE || b[3] != H || b[4] != NR)
    fail(TM_ERR_ARG, "surrogate weights: unsupported layout");
  w.lbar = b[5];
  w.abar = b[6];
  w.fscale = b[7];
  if (!(w.lbar > 0) || !(w.abar > 0)) fail(TM_ERR_ARG, "surrogate weights: non-positive length or area scale");
  const float* q = b + BLOB_HEADER;
  auto take = [&](float* dst, int k) {
    std::memcpy(dst, q, sizeof(float) * k);
    q += k;
  };
  take(w.win, H * FV);
  take(w.bin, H);
  wd.resize((size_t)NR * H * 2 * H);
  for (int r = 0; r < NR; ++r) {
    take(w.we[r], H * FE);
    take(w.be[r], H);
    for (int k = 0; k < H * 2 * H; ++k) wd[(size_t)r * H * 2 * H + k] = __float2bfloat16_rn(q[k]);
    q += H * 2 * H;
    take(w.b[r], H);
  }
  take(w.wo, H);
  take(&w.bo, 1);
  take(w.wn, H);
  take(&w.bn, 1);
}

}  // namespace

namespace tmg {

// surrogate gradient at positions P into g (device arrays of 3 nv doubles)
void surrogate_grad(tm_surrogate* sg, tm_energy* e, tm_mesh* m, const double* P, double* g, cudaStream_t s) {
  if (m->nv != sg->nv) fail(TM_ERR_ARG, "surrogate built for another mesh size");
  int nv = m->nv;
  if (nv == 0) return;
  energy_eval32_local(e, m, P, sg->gloc.get(), s);
  Topo t = m->topo();
  const FaceF* fd = reinterpret_cast<const FaceF*>(e->face.get());
  const EdgeF* ed = reinterpret_cast<const EdgeF*>(e->edge.get());
  const float* rho = reinterpret_cast<const float*>(e->rho.get());
  Split S{e->posdw.get()};
  SurW* W = sg->w.get();
  k_sfeat<<<nblk(nv, SFB), SFB, 0, s>>>(t, fd, ed, rho, W, nullptr, sg->nrm.get(), sg->hb[0].get());
  TM_LAUNCH();
  int cur = 0;
  LayerIn in{};
  in.t = t;
  in.ed = ed;
  in.rho = rho;
  in.lbar = sg->hw.lbar;
  in.M = nv;
  in.status = sg->status.get();
  for (int r = 0; r < NR; ++r) {
    in.we = W->we[r];
    in.be = W->be[r];
    in.bias = W->b[r];
    in.h = reinterpret_cast<const uint4*>(sg->hb[cur].get());
    layer_launch<false>(sg->map_h[cur], sg->map_w[r], sg->map_h[cur ^ 1], sg->map_h[cur ^ 1], in, s);
    cur ^= 1;
  }
  k_out<<<nblk(8L * nv, 256), 256, 0, s>>>(t, S, sg->nrm.get(), W, sg->hb[cur].get(), sg->gloc.get(), g);
  TM_LAUNCH();
}

}  // namespace tmg

// --------------------------------------------------------------------------
// Training on the GPU: hand-written forward and backward kernels of the
// network above and Adam, on the inputs tm_surrogate_inputs_device exports.
//
// Parameters live as one FP32 vector theta in the blob's order (the
// header dropped).  The forward pass is the inference pass with its
// intermediates kept: h and m in bf16 (as the inference kernels store
// them), the dense weights rounded to bf16 with FP32 accumulation (the
// same tcgen05 layer, which also writes the pre-activations z in FP32).
// The backward pass treats the bf16 roundings as identities (straight
// through) and accumulates in FP32:
//   output   dF_i = 2 (F_i - T_i) / (3 n rms^2),  dc_ij = s dF_i . d_ij,
//            dc_i = s dF_i . N_i,  dh_i = dc_i w_n + w_o * sum_j (dc_ij + dc_ji) h_j
//   dense    dz = dh * SiLU'(z), d[h ; m] = dz W (h part added to the
//            residual), dW += dz [h ; m]^T, db += dz
//   messages dh_j += sum_i (W_e e_ij + b_e) * dm_i over the rings of j,
//            dW_e += (dm_i * h_j) e_ij^T, db_e += dm_i * h_j
//   input    dz = dh * SiLU'(z), dW_in += dz u^T, db_in += dz
// Parameter gradients are summed per block and then over the blocks in a
// fixed order (no floating-point atomics: a step is bit-reproducible).
// --------------------------------------------------------------------------
namespace {

// offsets of the parameter groups in theta
constexpr int P_WIN = 0, P_BIN = H * FV, P_R0 = P_BIN + H;
constexpr int P_RSTRIDE = H * FE + H + H * 2 * H + H;
__host__ __device__ constexpr int p_we(int r) { return P_R0 + r * P_RSTRIDE; }
__host__ __device__ constexpr int p_be(int r) { return p_we(r) + H * FE; }
__host__ __device__ constexpr int p_w(int r) { return p_be(r) + H; }
__host__ __device__ constexpr int p_b(int r) { return p_w(r) + H * 2 * H; }
constexpr int P_WO = P_R0 + NR * P_RSTRIDE, P_BO = P_WO + H, P_WN = P_BO + 1, P_BN = P_WN + H;
constexpr int NPARAM = P_BN + 1;
static_assert(NPARAM + BLOB_HEADER == BLOB_SIZE, "parameter layout");

__device__ __forceinline__ float dsilu(float z) {
  const float sg = 1.0f / (1.0f + __expf(-z));
  return sg * (1.0f + z * (1.0f - sg));
}

constexpr int TB = 256;  // threads per block of the per-vertex training kernels

// input layer: z = W_in u + b_in, h = bf16(SiLU(z)); 8 threads per vertex,
// 8 channels each, persistent blocks with the weights in registers (weights
// loaded per vertex: 23 us at 40,962 vertices, now 12)
__global__ void __launch_bounds__(TB, 2) k_t_embed(int nv, const float* __restrict__ u, const float* __restrict__ th,
                                                   float* __restrict__ z, __nv_bfloat16* __restrict__ h) {
  const int sub = threadIdx.x & 7;
  const Embed8 emb(th + P_WIN, th + P_BIN, sub);
  for (int i = (blockIdx.x * TB + threadIdx.x) >> 3; i < nv; i += gridDim.x * (TB / 8)) {
    float x[FV], y[8], o[8];
#pragma unroll
    for (int k = 0; k < FV; ++k) x[k] = u[(size_t)FV * i + k];
    emb(x, y);
#pragma unroll
    for (int q = 0; q < 8; ++q) o[q] = silu(y[q]);
    float4* z4 = reinterpret_cast<float4*>(z + (size_t)H * i + 8 * sub);
    z4[0] = make_float4(y[0], y[1], y[2], y[3]);
    z4[1] = make_float4(y[4], y[5], y[6], y[7]);
    reinterpret_cast<uint4*>(h)[(size_t)i * (H / 8) + sub] = pack8(o);
  }
}

// Sum of a per-thread value over the block's threads in thread order,
// through shared memory (deterministic); returns it in thread 0.
__device__ __forceinline__ float block_sum(float v, float* sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  const float r = sh[0];
  __syncthreads();
  return r;
}

// Sums of NVAL values a thread over the threads of a block with the same
// sub = threadIdx.x & (S - 1), written to out[sub * NVAL + k] for the caller's
// layout through put(sub, k, sum): the lanes of a warp by a fixed shuffle
// tree, then the warps in warp order.  One pass at the end of a persistent
// block instead of one per tile of vertices.
template <int S, int NVAL, class Put>
__device__ __forceinline__ void block_group_sum(float* v, float* sh, const Put& put) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NVAL; ++k) {
#pragma unroll
    for (int o = 16; o >= S; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  }
  if (lane < S)
#pragma unroll
    for (int k = 0; k < NVAL; ++k) sh[(warp * NVAL + k) * S + lane] = v[k];
  __syncthreads();
  for (int q = threadIdx.x; q < S * NVAL; q += TB) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < TB / 32; ++w) s += sh[w * S * NVAL + q];
    put(q % S, q / S, s);
  }
}

// output head, loss and dL/dF: 8 threads per vertex
__global__ void __launch_bounds__(TB) k_t_out(int nv, int D, const int* __restrict__ nbr,
                                              const float* __restrict__ dirs, const float* __restrict__ nrm,
                                              const float* __restrict__ tgt, const float* __restrict__ th, float fs,
                                              float inv_norm, const __nv_bfloat16* __restrict__ h,
                                              float* __restrict__ F, float* __restrict__ dF,
                                              float* __restrict__ lossp) {
  __shared__ float sh[TB];
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = g >> 3, sub = g & 7;
  const unsigned gmask = 0xffu << (threadIdx.x & 24);
  const bool act = i < nv;
  const int ii = act ? i : 0;
  const uint4* h4 = reinterpret_cast<const uint4*>(h);
  float hi[8], pi[8];
  unpack8(h4[(size_t)ii * (H / 8) + sub], hi);
  float cn = 0.f;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    pi[c] = th[P_WO + 8 * sub + c] * hi[c];
    cn += th[P_WN + 8 * sub + c] * hi[c];
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) cn += __shfl_xor_sync(gmask, cn, o);
  cn += th[P_BN];
  float Fx = cn * nrm[4 * (size_t)ii], Fy = cn * nrm[4 * (size_t)ii + 1], Fz = cn * nrm[4 * (size_t)ii + 2];
  const float bo = th[P_BO];
  // the eight lanes of a vertex share its ring, so they leave the loop together
  int j = nbr[ii];
  for (int m = 0; j >= 0; ++m) {
    const size_t o = (size_t)m * nv + ii;
    const int jn = m + 1 < D ? nbr[o + nv] : -1;
    const float ux = dirs[3 * o], uy = dirs[3 * o + 1], uz = dirs[3 * o + 2];
    float hj[8];
    unpack8(h4[(size_t)j * (H / 8) + sub], hj);
    float c = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) c += pi[q] * hj[q];
#pragma unroll
    for (int q = 1; q < 8; q <<= 1) c += __shfl_xor_sync(gmask, c, q);
    c += bo;
    Fx += c * ux;
    Fy += c * uy;
    Fz += c * uz;
    j = jn;
  }
  Fx *= fs;
  Fy *= fs;
  Fz *= fs;
  float l = 0.f;
  if (act && sub == 0) {
    const float ex = Fx - tgt[3 * (size_t)i], ey = Fy - tgt[3 * (size_t)i + 1], ez = Fz - tgt[3 * (size_t)i + 2];
    l = (ex * ex + ey * ey + ez * ez) * inv_norm;
    if (F) {
      F[3 * (size_t)i] = Fx;
      F[3 * (size_t)i + 1] = Fy;
      F[3 * (size_t)i + 2] = Fz;
    }
    dF[3 * (size_t)i] = 2.0f * inv_norm * ex;
    dF[3 * (size_t)i + 1] = 2.0f * inv_norm * ey;
    dF[3 * (size_t)i + 2] = 2.0f * inv_norm * ez;
  }
  const float s = block_sum(l, sh);
  if (threadIdx.x == 0) lossp[blockIdx.x] = s;
}

// Backward of the output head: dh of the last round (FP32) and the block
// partials of (w_o, b_o, w_n, b_n) (part: 130 floats per block).  Persistent
// blocks: the parameter sums stay in registers over the block's vertices.
__global__ void __launch_bounds__(TB) k_t_outback(int nv, int D, const int* __restrict__ nbr,
                                                  const float* __restrict__ dirs, const float* __restrict__ nrm,
                                                  const float* __restrict__ th, float fs,
                                                  const __nv_bfloat16* __restrict__ h, const float* __restrict__ dF,
                                                  float* __restrict__ dh, float* __restrict__ part) {
  __shared__ float sh[(TB / 32) * 18 * 8];
  const int sub = threadIdx.x & 7;
  const uint4* h4 = reinterpret_cast<const uint4*>(h);
  float wo[8], wn[8], sum[18];  // sum: w_o (8 channels), w_n (8), b_o, b_n
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    wo[q] = th[P_WO + 8 * sub + q];
    wn[q] = th[P_WN + 8 * sub + q];
  }
#pragma unroll
  for (int q = 0; q < 18; ++q) sum[q] = 0.f;
  for (int i = (blockIdx.x * TB + threadIdx.x) >> 3; i < nv; i += gridDim.x * (TB / 8)) {
    float hi[8], acc[8], t[8];
    int j = nbr[i];
    unpack8(h4[(size_t)i * (H / 8) + sub], hi);
    const float dfx = dF[3 * (size_t)i], dfy = dF[3 * (size_t)i + 1], dfz = dF[3 * (size_t)i + 2];
    const float dci = fs * (dfx * nrm[4 * (size_t)i] + dfy * nrm[4 * (size_t)i + 1] + dfz * nrm[4 * (size_t)i + 2]);
    float pbo = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      acc[q] = dci * wn[q];
      t[q] = 0.f;
    }
    for (int m = 0; j >= 0; ++m) {
      const size_t o = (size_t)m * nv + i;
      const int jn = m + 1 < D ? nbr[o + nv] : -1;
      const float ux = dirs[3 * o], uy = dirs[3 * o + 1], uz = dirs[3 * o + 2];
      float hj[8];
      unpack8(h4[(size_t)j * (H / 8) + sub], hj);
      const float dcij = fs * (dfx * ux + dfy * uy + dfz * uz);
      const float dcji = -fs * (dF[3 * (size_t)j] * ux + dF[3 * (size_t)j + 1] * uy + dF[3 * (size_t)j + 2] * uz);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        acc[q] += (dcij + dcji) * wo[q] * hj[q];
        t[q] += dcij * hj[q];
      }
      pbo += dcij;
      j = jn;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      sum[q] += t[q] * hi[q];
      sum[8 + q] += dci * hi[q];
    }
    sum[16] += pbo;
    sum[17] += dci;
    float4* d4 = reinterpret_cast<float4*>(dh + (size_t)H * i + 8 * sub);
    d4[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    d4[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
  }
  float* pb = part + 130 * (size_t)blockIdx.x;
  block_group_sum<8, 18>(sum, sh, [&](int sb, int k, float v) {
    if (k < 8) pb[8 * sb + k] = v;
    else if (k < 16) pb[65 + 8 * sb + k - 8] = v;
    else if (sb == 0) pb[k == 16 ? 64 : 129] = v;
  });
}

// Backward of dense layer r over tiles of 32 vertices (persistent blocks):
// dz = dh1 * SiLU'(z); dh0 = dh1 + dz W[:, :64]; dm = dz W[:, 64:];
// block partials of dW (64 x 128, row n, column k) and db (64).  Both are
// FP32 matrix products (the gradients keep FP32 operands), bound by shared
// memory and the FMA pipe: thread t owns rows rg + 8 q (vertices, q < 4) or
// 8 rg + q (channels, q < 8) and columns 4 kg .. + 3 of each product, so that
// 16 or 32 FMAs share two or three 16-byte shared loads without bank conflicts
// (four row groups and eight column groups a warp; sdz rows are padded by four
// floats).  40,962 vertices: one column and 32 rows a thread, one shared load
// per FMA, took 142 us a layer, tiles of 64 vertices with two blocks per SM
// 56; with 32 and three blocks the loads of one overlap the products of
// another (a step of 420 us then, 400 now).
constexpr int DT = 32;        // vertices per tile
constexpr int ZP = H + 4;     // padded row of sdz
constexpr int DENSE_BACK_SMEM = (DT * ZP + DT * 2 * H + H * 2 * H) * sizeof(float);
__global__ void __launch_bounds__(TB, 3) k_t_dense_back(int nv, const float* __restrict__ th, int r,
                                                        const float* __restrict__ z,
                                                        const __nv_bfloat16* __restrict__ h,
                                                        const __nv_bfloat16* __restrict__ mm,
                                                        const float* __restrict__ dh1, float* __restrict__ dh0,
                                                        float* __restrict__ dm, float* __restrict__ part) {
  extern __shared__ float4 sm4[];
  float* sdz = reinterpret_cast<float*>(sm4);  // [DT][ZP]
  float* sa = sdz + DT * ZP;                   // [DT][2H]: [h | m]
  float* sw = sa + DT * 2 * H;                 // [H][2H]: W rounded to bf16
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int rg = (warp & 1) * 4 + (lane & 3);         // row group 0 .. 7
  const int kc = 4 * ((warp >> 1) * 8 + (lane >> 2));  // first column, 0 .. 124
  for (int q = t; q < H * 2 * H / 4; q += TB) {
    const float4 w = reinterpret_cast<const float4*>(th + p_w(r))[q];
    reinterpret_cast<float4*>(sw)[q] =
        make_float4(__bfloat162float(__float2bfloat16_rn(w.x)), __bfloat162float(__float2bfloat16_rn(w.y)),
                    __bfloat162float(__float2bfloat16_rn(w.z)), __bfloat162float(__float2bfloat16_rn(w.w)));
  }
  float gw[8][4];
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int c = 0; c < 4; ++c) gw[q][c] = 0.f;
  float gb = 0.f;
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const int ntile = (nv + DT - 1) / DT;
  for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int v0 = tile * DT, nrow = min(DT, nv - v0);
    __syncthreads();  // the previous tile's reads are done (and sw is written)
    for (int q = t; q < DT * H / 4; q += TB) {
      const int vr = q / (H / 4), c = q % (H / 4);
      float4 d = zero4;
      if (vr < nrow) {
        const float4 zz = reinterpret_cast<const float4*>(z + (size_t)v0 * H)[q];
        d = reinterpret_cast<const float4*>(dh1 + (size_t)v0 * H)[q];
        d = make_float4(d.x * dsilu(zz.x), d.y * dsilu(zz.y), d.z * dsilu(zz.z), d.w * dsilu(zz.w));
      }
      *reinterpret_cast<float4*>(sdz + vr * ZP + 4 * c) = d;
    }
    for (int q = t; q < DT * 2 * H / 8; q += TB) {  // eight bf16 at a time: h, then m
      const int vr = q / (2 * H / 8), c = q % (2 * H / 8);
      float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (vr < nrow) {
        const size_t row = (size_t)(v0 + vr) * (H / 8);
        unpack8(c < H / 8 ? reinterpret_cast<const uint4*>(h)[row + c]
                          : reinterpret_cast<const uint4*>(mm)[row + c - H / 8], f);
      }
      float4* d = reinterpret_cast<float4*>(sa + vr * 2 * H + 8 * c);
      d[0] = make_float4(f[0], f[1], f[2], f[3]);
      d[1] = make_float4(f[4], f[5], f[6], f[7]);
    }
    __syncthreads();
    // d[h | m][v][k] = sum_n dz[v][n] W[n][k], vertices rg + 8 q
    {
      float o[DT / 8][4];
#pragma unroll
      for (int q = 0; q < DT / 8; ++q)
#pragma unroll
        for (int c = 0; c < 4; ++c) o[q][c] = 0.f;
#pragma unroll 2
      for (int n = 0; n < H; n += 4) {
        float4 w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) w[u] = *reinterpret_cast<const float4*>(sw + (n + u) * 2 * H + kc);
#pragma unroll
        for (int q = 0; q < DT / 8; ++q) {
          const float4 d = *reinterpret_cast<const float4*>(sdz + (rg + 8 * q) * ZP + n);
          const float dd[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            o[q][0] += dd[u] * w[u].x;
            o[q][1] += dd[u] * w[u].y;
            o[q][2] += dd[u] * w[u].z;
            o[q][3] += dd[u] * w[u].w;
          }
        }
      }
#pragma unroll
      for (int q = 0; q < DT / 8; ++q) {
        if (rg + 8 * q >= nrow) break;
        const size_t v = v0 + rg + 8 * q;
        float4 x = make_float4(o[q][0], o[q][1], o[q][2], o[q][3]);
        if (kc < H) {
          const float4 y = *reinterpret_cast<const float4*>(dh1 + v * H + kc);
          *reinterpret_cast<float4*>(dh0 + v * H + kc) = make_float4(y.x + x.x, y.y + x.y, y.z + x.z, y.w + x.w);
        } else {
          *reinterpret_cast<float4*>(dm + v * H + kc - H) = x;
        }
      }
    }
    // dW[n][k] += sum over the tile's vertices of dz[v][n] a[v][k], channels
    // n = 8 rg + q
#pragma unroll 4
    for (int vr = 0; vr < DT; ++vr) {
      const float4 a = *reinterpret_cast<const float4*>(sa + vr * 2 * H + kc);
      const float4 d0 = *reinterpret_cast<const float4*>(sdz + vr * ZP + 8 * rg);
      const float4 d1 = *reinterpret_cast<const float4*>(sdz + vr * ZP + 8 * rg + 4);
      const float dd[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        gw[q][0] += dd[q] * a.x;
        gw[q][1] += dd[q] * a.y;
        gw[q][2] += dd[q] * a.z;
        gw[q][3] += dd[q] * a.w;
      }
    }
    if (t < H)
      for (int vr = 0; vr < DT; ++vr) gb += sdz[vr * ZP + t];
  }
  float* pb = part + (size_t)(H * 2 * H + H) * blockIdx.x;
#pragma unroll
  for (int q = 0; q < 8; ++q)
    *reinterpret_cast<float4*>(pb + (8 * rg + q) * 2 * H + kc) = make_float4(gw[q][0], gw[q][1], gw[q][2], gw[q][3]);
  if (t < H) pb[H * 2 * H + t] = gb;
}

// Backward of the messages of round r, per vertex v (16 threads, 4
// channels each): as a sender dh[v] += sum_i (W_e e_iv + b_e) * dm_i over
// v's ring (e_iv is e_vi with the antisymmetric feature 2 negated); as a
// receiver the block partials of dW_e and db_e (320 floats per block), summed
// in registers over the vertices of a persistent block.
__global__ void __launch_bounds__(TB, 3) k_t_msg_back(int nv, int D, const int* __restrict__ nbr,
                                                      const float* __restrict__ ef, const float* __restrict__ th,
                                                      int r, const __nv_bfloat16* __restrict__ h,
                                                      const float* __restrict__ dm, float* __restrict__ dh,
                                                      float* __restrict__ part) {
  __shared__ float sh[(TB / 32) * 20 * 16];
  const int sub = threadIdx.x & 15;
  float4 w[4];
  float b[4], sum[20];  // sum[5 c + k]: dW_e (k < 4) and db_e of channel c
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    w[c] = *reinterpret_cast<const float4*>(th + p_we(r) + (4 * sub + c) * FE);
    b[c] = th[p_be(r) + 4 * sub + c];
  }
#pragma unroll
  for (int q = 0; q < 20; ++q) sum[q] = 0.f;
  const uint2* h2 = reinterpret_cast<const uint2*>(h);
  const float4* dm4 = reinterpret_cast<const float4*>(dm);
  for (int i = (blockIdx.x * TB + threadIdx.x) >> 4; i < nv; i += gridDim.x * (TB / 16)) {
    int j = nbr[i];
    const float4 di = dm4[(size_t)i * (H / 4) + sub];
    const float dmi[4] = {di.x, di.y, di.z, di.w};
    float add[4] = {0.f, 0.f, 0.f, 0.f};
    for (int m = 0; j >= 0; ++m) {
      const size_t o = (size_t)m * nv + i;
      const int jn = m + 1 < D ? nbr[o + nv] : -1;
      const float4 e = *reinterpret_cast<const float4*>(ef + FE * o);  // e_vj
      const uint2 hv = h2[(size_t)j * (H / 4) + sub];
      const float4 dmj = dm4[(size_t)j * (H / 4) + sub];
      const float2 h01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&hv.x));
      const float2 h23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&hv.y));
      const float hj[4] = {h01.x, h01.y, h23.x, h23.y};
      const float dj[4] = {dmj.x, dmj.y, dmj.z, dmj.w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        // receiver: m_v gathers (W_e e_vj + b_e) * h_j
        const float q = dmi[c] * hj[c];
        sum[5 * c] += q * e.x;
        sum[5 * c + 1] += q * e.y;
        sum[5 * c + 2] += q * e.z;
        sum[5 * c + 3] += q * e.w;
        sum[5 * c + 4] += q;
        // sender: m_j gathers (W_e e_jv + b_e) * h_v, e_jv = e_vj with feature 2 negated
        add[c] += (b[c] + w[c].x * e.x + w[c].y * e.y - w[c].z * e.z + w[c].w * e.w) * dj[c];
      }
      j = jn;
    }
    float4* d4 = reinterpret_cast<float4*>(dh + (size_t)H * i + 4 * sub);
    float4 cur = *d4;
    cur.x += add[0];
    cur.y += add[1];
    cur.z += add[2];
    cur.w += add[3];
    *d4 = cur;
  }
  float* pb = part + (H * FE + H) * (size_t)blockIdx.x;
  block_group_sum<16, 20>(sum, sh, [&](int sb, int k, float v) {
    const int ch = 4 * sb + k / 5;
    if (k % 5 < FE)
      pb[ch * FE + k % 5] = v;
    else
      pb[H * FE + ch] = v;
  });
}

// Backward of the input layer: dz = dh * SiLU'(z), block partials of
// dW_in (64 x 8) and db_in (576 floats per block); 8 threads per vertex,
// persistent blocks
__global__ void __launch_bounds__(TB, 2) k_t_embed_back(int nv, const float* __restrict__ u,
                                                        const float* __restrict__ z, const float* __restrict__ dh,
                                                        float* __restrict__ part) {
  __shared__ float sh[(TB / 32) * 72 * 8];
  const int sub = threadIdx.x & 7;
  float sum[72];  // sum[9 q + k]: dW_in (k < 8) and db_in of channel 8 sub + q
#pragma unroll
  for (int q = 0; q < 72; ++q) sum[q] = 0.f;
  for (int i = (blockIdx.x * TB + threadIdx.x) >> 3; i < nv; i += gridDim.x * (TB / 8)) {
    float x[FV];
#pragma unroll
    for (int k = 0; k < FV; ++k) x[k] = u[(size_t)FV * i + k];
    const float4* z4 = reinterpret_cast<const float4*>(z + (size_t)H * i + 8 * sub);
    const float4* d4 = reinterpret_cast<const float4*>(dh + (size_t)H * i + 8 * sub);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const float4 zz = z4[p], dd = d4[p];
      const float dz[4] = {dd.x * dsilu(zz.x), dd.y * dsilu(zz.y), dd.z * dsilu(zz.z), dd.w * dsilu(zz.w)};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int k = 0; k < FV; ++k) sum[9 * (4 * p + q) + k] += dz[q] * x[k];
        sum[9 * (4 * p + q) + FV] += dz[q];
      }
    }
  }
  float* pb = part + (H * FV + H) * (size_t)blockIdx.x;
  block_group_sum<8, 72>(sum, sh, [&](int sb, int k, float v) {
    const int ch = 8 * sb + k / 9;
    if (k % 9 < FV)
      pb[ch * FV + k % 9] = v;
    else
      pb[H * FV + ch] = v;
  });
}

// All parameter gradients of a pass in one launch: group g's column k is the
// sum over its nb block partials part[b * stride + k], written to grad[dst + k]
// (32 columns a block, eight threads a column, each every eighth partial in
// order, then the eight in order).  The last block sums the loss partials.
// With ADAM the parameter is updated where its gradient is (Kingma & Ba 2015,
// with bias correction) and the dense weights' bf16 copies (what the forward
// reads) are refreshed from the FP32 master.  One thread a column over all
// partials, a launch per group, took 718 us of the 1,265 us step at 40,962
// vertices; with it, persistent blocks, the tiled products and k_layer the step
// is 400.
struct RedGroup {
  const float* part;
  int nb, n, dst, blk0;  // partials, columns (= stride), first parameter, first block
};
struct RedArgs {
  RedGroup g[2 + 2 * NR];
  int ng;
  const float* lossp;
  int nl;
  float *loss, *grad;
};
struct AdamArgs {
  float *th, *m1, *m2;
  float lr, b1, b2, eps, c1, c2;
  __nv_bfloat16* wd;
};
template <bool ADAM>
__global__ void __launch_bounds__(256) k_t_reduce(const __grid_constant__ RedArgs R, const __grid_constant__ AdamArgs A) {
  __shared__ float sh[256];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  if (blockIdx.x + 1 == gridDim.x) {
    float s = 0.f;
    for (int b = threadIdx.x; b < R.nl; b += 256) s += R.lossp[b];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) *R.loss = s;
    return;
  }
  int gi = 0;
  while (gi + 1 < R.ng && (int)blockIdx.x >= R.g[gi + 1].blk0) ++gi;
  const RedGroup G = R.g[gi];
  const int k = ((int)blockIdx.x - G.blk0) * 32 + x;
  float s = 0.f;
  if (k < G.n) {
#pragma unroll 8
    for (int b = y; b < G.nb; b += 8) s += G.part[(size_t)b * G.n + k];
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  if (y || k >= G.n) return;
  s = 0.f;
#pragma unroll
  for (int q = 0; q < 8; ++q) s += sh[32 * q + x];
  const int p = G.dst + k;
  R.grad[p] = s;
  if (ADAM) {
    const float a = A.b1 * A.m1[p] + (1.0f - A.b1) * s;
    const float b = A.b2 * A.m2[p] + (1.0f - A.b2) * s * s;
    A.m1[p] = a;
    A.m2[p] = b;
    const float v = A.th[p] - A.lr * (a * A.c1) / (sqrtf(b * A.c2) + A.eps);
    A.th[p] = v;
    for (int r = 0; r < NR; ++r)
      if (p >= p_w(r) && p < p_w(r) + H * 2 * H) A.wd[(size_t)r * H * 2 * H + (p - p_w(r))] = __float2bfloat16_rn(v);
  }
}

}  // namespace

struct tm_strain {
  int nv = 0, D = 0;
  float lbar = 1.f, abar = 1.f, fscale = 1.f;
  long long step = 0;
  DevBuf<float> th, grad, m1, m2, loss;
  DevBuf<__nv_bfloat16> wd;      // [NR][H][2H]
  DevBuf<float> z;               // [NR + 1][nv][H]: input layer, then the dense layers
  DevBuf<__nv_bfloat16> hb;      // [NR + 1][nv][H]
  DevBuf<__nv_bfloat16> mb;      // [NR][nv][H]
  DevBuf<float> dha, dhb, dm, dF, part, lossp;
  DevBuf<int> status;
  // persistent blocks of the backward kernels (at most one per tile)
  int nb_dense = 0, nb_msg = 0, nb_out = 0, nb_emb = 0;
  alignas(64) CUtensorMap map_h[NR + 1];
  alignas(64) CUtensorMap map_m[NR];
  alignas(64) CUtensorMap map_w[NR];
};

namespace {

// blocks of kernel k that fit on the GPU at once
template <class K>
int resident_blocks(K* k, int smem) {
  int per_sm = 0, nsm = 0, dev = 0;
  if (smem > 48 * 1024) allow_smem(k, smem);
  TM_CUDA(cudaGetDevice(&dev));
  TM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  TM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, TB, smem));
  return std::max(1, per_sm) * nsm;
}

// floats of nb partials of n columns, each group's on a 16-byte boundary
size_t part_floats(int nb, int n) { return ((size_t)nb * n + 3) & ~(size_t)3; }

struct TrainInputs {
  const float *u, *nrm, *ef, *dirs, *tgt;
  const int* nbr;
  int D;  // ring slots of the exported arrays ([D][n])
};

// forward pass (kept intermediates) and, with want_grad, the backward pass
// and the gradient into st->grad, with the update of adam when it is given;
// F (n x 3, may be NULL) receives the force
void train_pass(tm_strain* st, const TrainInputs& in, float inv_norm, bool want_grad, float* F, const AdamArgs* adam,
                cudaStream_t s) {
  const int nv = st->nv, D = in.D;
  const size_t NH = (size_t)nv * H;
  const float* th = st->th.get();
  const int nb8 = nblk((long)nv * 8, TB);
  k_t_embed<<<st->nb_emb, TB, 0, s>>>(nv, in.u, th, st->z.get(), st->hb.get());
  TM_LAUNCH();
  LayerIn q{};
  q.nbr = in.nbr;
  q.ef = reinterpret_cast<const float4*>(in.ef);
  q.D = D;
  q.M = nv;
  q.status = st->status.get();
  for (int r = 0; r < NR; ++r) {
    q.we = th + p_we(r);
    q.be = th + p_be(r);
    q.bias = th + p_b(r);
    q.h = reinterpret_cast<const uint4*>(st->hb.get() + r * NH);
    q.z = st->z.get() + (r + 1) * NH;
    layer_launch<true>(st->map_h[r], st->map_w[r], st->map_h[r + 1], st->map_m[r], q, s);
  }
  k_t_out<<<nb8, TB, 0, s>>>(nv, D, in.nbr, in.dirs, in.nrm, in.tgt, th, st->fscale, inv_norm,
                              st->hb.get() + NR * NH, F, st->dF.get(), st->lossp.get());
  TM_LAUNCH();
  RedArgs R{};
  int nblocks = 0;
  float* part = st->part.get();
  auto group = [&](int nb, int n, int dst) {  // partials of the next parameter group
    R.g[R.ng++] = RedGroup{part, nb, n, dst, nblocks};
    nblocks += nblk(n, 32);
    float* p = part;
    part += part_floats(nb, n);
    return p;
  };
  R.lossp = st->lossp.get();
  R.nl = nb8;
  R.loss = st->loss.get();
  R.grad = st->grad.get();
  if (want_grad) {
    // output head
    k_t_outback<<<st->nb_out, TB, 0, s>>>(nv, D, in.nbr, in.dirs, in.nrm, th, st->fscale, st->hb.get() + NR * NH,
                                           st->dF.get(), st->dha.get(), group(st->nb_out, 130, P_WO));
    TM_LAUNCH();
    // rounds, last to first: dense layer, then messages
    float* dcur = st->dha.get();
    float* dnext = st->dhb.get();
    for (int r = NR - 1; r >= 0; --r) {
      k_t_dense_back<<<st->nb_dense, TB, DENSE_BACK_SMEM, s>>>(
          nv, th, r, st->z.get() + (r + 1) * NH, st->hb.get() + r * NH, st->mb.get() + r * NH, dcur, dnext,
          st->dm.get(), group(st->nb_dense, H * 2 * H + H, p_w(r)));
      TM_LAUNCH();
      k_t_msg_back<<<st->nb_msg, TB, 0, s>>>(nv, D, in.nbr, in.ef, th, r, st->hb.get() + r * NH, st->dm.get(), dnext,
                                              group(st->nb_msg, H * FE + H, p_we(r)));
      TM_LAUNCH();
      std::swap(dcur, dnext);
    }
    // input layer
    k_t_embed_back<<<st->nb_emb, TB, 0, s>>>(nv, in.u, st->z.get(), dcur, group(st->nb_emb, H * FV + H, P_WIN));
    TM_LAUNCH();
  }
  if (adam)
    k_t_reduce<true><<<nblocks + 1, 256, 0, s>>>(R, *adam);
  else
    k_t_reduce<false><<<nblocks + 1, 256, 0, s>>>(R, AdamArgs{});
  TM_LAUNCH();
}

TrainInputs check_inputs(tm_strain* st, int64_t nv, int32_t D, const float* u, const float* nrm, const int32_t* nbr,
                         const float* ef, const float* dirs, const float* tgt) {
  if (!st || !u || !nrm || !nbr || !ef || !dirs || !tgt) fail(TM_ERR_ARG, "NULL argument");
  if (nv != st->nv) fail(TM_ERR_ARG, "training state built for " + std::to_string(st->nv) + " vertices");
  if (D < 1 || D > st->D) fail(TM_ERR_ARG, "max_valence out of the training state's range");
  if ((reinterpret_cast<uintptr_t>(ef) & 15) != 0) fail(TM_ERR_ARG, "edge features not 16-byte aligned");
  TrainInputs in{u, nrm, ef, dirs, tgt, nbr, (int)D};
  return in;
}

}  // namespace

extern "C" {

int tm_surrogate_create(tm_mesh* m, const float* weights, int64_t n_weights, tm_surrogate** out) {
  TM_API_BEGIN
  if (!m || !weights || !out) fail(TM_ERR_ARG, "NULL argument");
  *out = nullptr;
  std::unique_ptr<tm_surrogate> sg(new tm_surrogate());
  allow_smem(k_layer<false>, LAYER_SMEM);
  std::vector<__nv_bfloat16> wd;
  parse_blob(weights, n_weights, sg->hw, wd);
  int nv = m->nv;
  sg->nv = nv;
  size_t n = std::max(nv, 1);
  sg->w.ensure(1);
  sg->wd.ensure(wd.size());
  sg->nrm.ensure(4 * n);
  sg->hb[0].ensure(H * n);
  sg->hb[1].ensure(H * n);
  sg->gloc.ensure(3 * n);
  sg->status.ensure(1);
  TM_CUDA(cudaMemcpy(sg->w.get(), &sg->hw, sizeof(SurW), cudaMemcpyHostToDevice));
  TM_CUDA(cudaMemcpy(sg->wd.get(), wd.data(), sizeof(__nv_bfloat16) * wd.size(), cudaMemcpyHostToDevice));
  TM_CUDA(cudaMemset(sg->status.get(), 0, sizeof(int)));
  if (nv > 0)
    for (int k = 0; k < 2; ++k) make_map(&sg->map_h[k], sg->hb[k].get(), nv, H, BM);
  for (int r = 0; r < NR; ++r) make_map(&sg->map_w[r], sg->wd.get() + (size_t)r * H * 2 * H, H, 2 * H, H);
  *out = sg.release();
  TM_API_END
}

int tm_surrogate_destroy(tm_surrogate* sg) {
  delete sg;
  return TM_OK;
}

int tm_surrogate_gradient_device(tm_surrogate* sg, tm_energy* e, tm_mesh* m, const double* d_points, double* d_grad,
                                 void* stream) {
  TM_API_BEGIN
  if (!sg || !e || !m || !d_points || !d_grad) fail(TM_ERR_ARG, "NULL argument");
  cudaStream_t s = stream ? (cudaStream_t)stream : e->stream;
  surrogate_grad(sg, e, m, d_points, d_grad, s);
  int st = 0;
  TM_CUDA(cudaMemcpyAsync(&st, sg->status.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
  TM_CUDA(cudaStreamSynchronize(s));
  if (st) fail(TM_ERR_TIMEOUT, "tensor-core layer wait timed out (" + std::to_string(st) + ")");
  TM_API_END
}

int tm_surrogate_inputs_device(tm_surrogate* sg, tm_energy* e, tm_mesh* m, const double* d_points, int32_t max_valence,
                               float* d_u, float* d_normals, int32_t* d_nbr, float* d_edge_feat, float* d_dirs,
                               double* d_grad_local, void* stream) {
  TM_API_BEGIN
  if (!sg || !e || !m || !d_points || !d_u || !d_normals || !d_nbr || !d_edge_feat || !d_dirs || !d_grad_local)
    fail(TM_ERR_ARG, "NULL argument");
  if (m->nv != sg->nv) fail(TM_ERR_ARG, "surrogate built for another mesh size");
  if (max_valence < 1 || max_valence > TM_MAXVAL) fail(TM_ERR_ARG, "max_valence out of range");
  cudaStream_t s = stream ? (cudaStream_t)stream : e->stream;
  int nv = m->nv;
  if (nv == 0) return TM_OK;
  std::vector<int> val(nv);
  TM_CUDA(cudaMemcpyAsync(val.data(), m->d_val.get(), sizeof(int) * nv, cudaMemcpyDeviceToHost, s));
  TM_CUDA(cudaStreamSynchronize(s));
  int dmax = *std::max_element(val.begin(), val.end());
  if (dmax > max_valence) fail(TM_ERR_ARG, "a vertex valence exceeds max_valence (" + std::to_string(dmax) + ")");
  energy_eval32_local(e, m, d_points, d_grad_local, s);
  Topo t = m->topo();
  const FaceF* fd = reinterpret_cast<const FaceF*>(e->face.get());
  const EdgeF* ed = reinterpret_cast<const EdgeF*>(e->edge.get());
  const float* rho = reinterpret_cast<const float*>(e->rho.get());
  Split S{e->posdw.get()};
  k_sfeat<<<nblk(nv, SFB), SFB, 0, s>>>(t, fd, ed, rho, sg->w.get(), d_u, sg->nrm.get(), sg->hb[0].get());
  TM_LAUNCH();
  TM_CUDA(cudaMemcpyAsync(d_normals, sg->nrm.get(), sizeof(float) * 4 * nv, cudaMemcpyDeviceToDevice, s));
  k_export<<<nblk(nv, 128), 128, 0, s>>>(t, S, ed, rho, sg->w.get(), max_valence, d_nbr, d_edge_feat, d_dirs);
  TM_LAUNCH();
  TM_CUDA(cudaStreamSynchronize(s));
  TM_API_END
}

int tm_dense_silu_bf16(const void* d_h, const void* d_m, const void* d_w, const float* d_bias, void* d_out,
                       int64_t rows, void* stream) {
  return tm_dense_silu_bf16_bounded(d_h, d_m, d_w, d_bias, d_out, rows, WAIT_POLLS, stream);
}

int tm_dense_silu_bf16_bounded(const void* d_h, const void* d_m, const void* d_w, const float* d_bias, void* d_out,
                               int64_t rows, int wait_polls, void* stream) {
  TM_API_BEGIN
  if (wait_polls < 0) fail(TM_ERR_ARG, "wait_polls must be >= 0");
  if (!d_h || !d_m || !d_w || !d_bias || !d_out) fail(TM_ERR_ARG, "NULL argument");
  if (rows < 0 || rows > (1LL << 30)) fail(TM_ERR_ARG, "rows out of range");
  cudaStream_t s = (cudaStream_t)stream;
  alignas(64) CUtensorMap mh, mm, mw;
  if (rows == 0) return TM_OK;
  make_map(&mh, d_h, rows, H, BM);
  make_map(&mm, d_m, rows, H, BM);
  make_map(&mw, d_w, H, 2 * H, H);
  DevBuf<int> st;
  st.ensure(1);
  TM_CUDA(cudaMemsetAsync(st.get(), 0, sizeof(int), s));
  dense_launch(mh, mm, mw, d_bias, static_cast<__nv_bfloat16*>(d_out), (int)rows, st.get(), s, wait_polls);
  int hs = 0;
  TM_CUDA(cudaMemcpyAsync(&hs, st.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
  TM_CUDA(cudaStreamSynchronize(s));
  if (hs) fail(TM_ERR_TIMEOUT, "tensor-core layer wait timed out (" + std::to_string(hs) + ")");
  TM_API_END
}


int tm_surrogate_train_create(int64_t n_vertices, int32_t max_valence, const float* weights, int64_t n_weights,
                              tm_strain** out) {
  TM_API_BEGIN
  if (!weights || !out) fail(TM_ERR_ARG, "NULL argument");
  *out = nullptr;
  if (n_vertices < 1 || n_vertices > (1LL << 26)) fail(TM_ERR_ARG, "n_vertices out of range");
  if (max_valence < 1 || max_valence > TM_MAXVAL) fail(TM_ERR_ARG, "max_valence out of range");
  SurW hw{};
  std::vector<__nv_bfloat16> wd;
  parse_blob(weights, n_weights, hw, wd);  // validates the layout
  std::unique_ptr<tm_strain> st(new tm_strain());
  const int nv = (int)n_vertices;
  st->nv = nv;
  st->D = max_valence;
  st->lbar = weights[5];
  st->abar = weights[6];
  st->fscale = weights[7];
  const size_t NH = (size_t)nv * H;
  st->th.ensure(NPARAM);
  st->grad.ensure(NPARAM);
  st->m1.ensure(NPARAM);
  st->m2.ensure(NPARAM);
  st->loss.ensure(1);
  st->wd.ensure((size_t)NR * H * 2 * H);
  st->z.ensure((NR + 1) * NH);
  st->hb.ensure((NR + 1) * NH);
  st->mb.ensure(NR * NH);
  st->dha.ensure(NH);
  st->dhb.ensure(NH);
  st->dm.ensure(NH);
  st->dF.ensure(3 * (size_t)nv);
  const int nb8 = nblk((long)nv * 8, TB), nb16 = nblk((long)nv * 16, TB);
  allow_smem(k_layer<true>, LAYER_SMEM);
  st->nb_dense = std::min(resident_blocks(k_t_dense_back, DENSE_BACK_SMEM), nblk(nv, DT));
  st->nb_msg = std::min(resident_blocks(k_t_msg_back, 0), nb16);
  st->nb_out = std::min(resident_blocks(k_t_outback, 0), nb8);
  st->nb_emb = std::min(resident_blocks(k_t_embed_back, 0), nb8);
  st->part.ensure(part_floats(st->nb_out, 130) + NR * part_floats(st->nb_dense, H * 2 * H + H) +
                  NR * part_floats(st->nb_msg, H * FE + H) + part_floats(st->nb_emb, H * FV + H));
  st->lossp.ensure(nb8);
  st->status.ensure(1);
  TM_CUDA(cudaMemcpy(st->th.get(), weights + BLOB_HEADER, sizeof(float) * NPARAM, cudaMemcpyHostToDevice));
  TM_CUDA(cudaMemcpy(st->wd.get(), wd.data(), sizeof(__nv_bfloat16) * wd.size(), cudaMemcpyHostToDevice));
  TM_CUDA(cudaMemset(st->m1.get(), 0, sizeof(float) * NPARAM));
  TM_CUDA(cudaMemset(st->m2.get(), 0, sizeof(float) * NPARAM));
  TM_CUDA(cudaMemset(st->status.get(), 0, sizeof(int)));
  for (int r = 0; r < NR; ++r) {
    make_map(&st->map_h[r], st->hb.get() + r * NH, nv, H, BM);
    make_map(&st->map_m[r], st->mb.get() + r * NH, nv, H, BM);
    make_map(&st->map_w[r], st->wd.get() + (size_t)r * H * 2 * H, H, 2 * H, H);
  }
  make_map(&st->map_h[NR], st->hb.get() + NR * NH, nv, H, BM);
  *out = st.release();
  TM_API_END
}

int tm_surrogate_train_destroy(tm_strain* st) {
  delete st;
  return TM_OK;
}

int tm_surrogate_train_get_weights(tm_strain* st, float* weights, int64_t n_weights) {
  TM_API_BEGIN
  if (!st || !weights) fail(TM_ERR_ARG, "NULL argument");
  if (n_weights != BLOB_SIZE) fail(TM_ERR_ARG, "weights: expected " + std::to_string(BLOB_SIZE) + " floats");
  const float head[BLOB_HEADER] = {1.0f, (float)FV, (float)FE, (float)H, (float)NR, st->lbar, st->abar, st->fscale};
  std::memcpy(weights, head, sizeof head);
  TM_CUDA(cudaDeviceSynchronize());
  TM_CUDA(cudaMemcpy(weights + BLOB_HEADER, st->th.get(), sizeof(float) * NPARAM, cudaMemcpyDeviceToHost));
  TM_API_END
}

int tm_surrogate_train_grad(tm_strain* st, const float* d_u, const float* d_nrm, const int32_t* d_nbr,
                            const float* d_ef, const float* d_dirs, const float* d_target, int64_t n_vertices,
                            int32_t max_valence, float target_rms, float* d_force, float* d_loss, float* d_grad,
                            void* stream) {
  TM_API_BEGIN
  const TrainInputs in = check_inputs(st, n_vertices, max_valence, d_u, d_nrm, d_nbr, d_ef, d_dirs, d_target);
  if (!(target_rms > 0.0f)) fail(TM_ERR_ARG, "target_rms must be positive");
  cudaStream_t s = (cudaStream_t)stream;
  TM_CUDA(cudaMemsetAsync(st->status.get(), 0, sizeof(int), s));
  const float inv_norm = 1.0f / (3.0f * (float)st->nv * target_rms * target_rms);
  train_pass(st, in, inv_norm, d_grad != nullptr, d_force, nullptr, s);
  if (d_loss) TM_CUDA(cudaMemcpyAsync(d_loss, st->loss.get(), sizeof(float), cudaMemcpyDeviceToDevice, s));
  if (d_grad)
    TM_CUDA(cudaMemcpyAsync(d_grad, st->grad.get(), sizeof(float) * NPARAM, cudaMemcpyDeviceToDevice, s));
  int hs = 0;
  TM_CUDA(cudaMemcpyAsync(&hs, st->status.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
  TM_CUDA(cudaStreamSynchronize(s));
  if (hs) fail(TM_ERR_TIMEOUT, "tensor-core layer wait timed out (" + std::to_string(hs) + ")");
  TM_API_END
}

int tm_surrogate_train_step(tm_strain* st, const float* d_u, const float* d_nrm, const int32_t* d_nbr,
                            const float* d_ef, const float* d_dirs, const float* d_target, int64_t n_vertices,
                            int32_t max_valence, float target_rms, float lr, float beta1, float beta2, float eps,
                            float* d_loss, void* stream) {
  TM_API_BEGIN
  const TrainInputs in = check_inputs(st, n_vertices, max_valence, d_u, d_nrm, d_nbr, d_ef, d_dirs, d_target);
  if (!(target_rms > 0.0f) || !(lr >= 0.0f) || !(beta1 >= 0.0f && beta1 < 1.0f) ||
      !(beta2 >= 0.0f && beta2 < 1.0f) || !(eps > 0.0f))
    fail(TM_ERR_ARG, "invalid training hyperparameters");
  cudaStream_t s = (cudaStream_t)stream;
  const float inv_norm = 1.0f / (3.0f * (float)st->nv * target_rms * target_rms);
  // the step counts once the pass is queued, as its update does
  const double k = (double)(st->step + 1);
  const AdamArgs adam{st->th.get(), st->m1.get(), st->m2.get(), lr, beta1, beta2, eps,
                      (float)(1.0 / (1.0 - std::pow((double)beta1, k))),
                      (float)(1.0 / (1.0 - std::pow((double)beta2, k))), st->wd.get()};
  train_pass(st, in, inv_norm, true, nullptr, &adam, s);
  st->step += 1;
  if (d_loss) TM_CUDA(cudaMemcpyAsync(d_loss, st->loss.get(), sizeof(float), cudaMemcpyDeviceToDevice, s));
  TM_API_END
}

int tm_surrogate_train_status(tm_strain* st) {
  TM_API_BEGIN
  if (!st) fail(TM_ERR_ARG, "NULL argument");
  int hs = 0;
  TM_CUDA(cudaDeviceSynchronize());
  TM_CUDA(cudaMemcpy(&hs, st->status.get(), sizeof(int), cudaMemcpyDeviceToHost));
  if (hs) fail(TM_ERR_TIMEOUT, "tensor-core layer wait timed out (" + std::to_string(hs) + ")");
  TM_API_END
}

}  // extern "C"
