// FP32 element records and float helpers shared by the FP32-stencil
// evaluation and the surrogate force model.
#pragma once
#include "tm_dw.cuh"
#include "tm_internal.h"

namespace tmg {

// unit normal and a cotangent, then (A, V) and the other cotangents: one
// 16-byte or one 8-byte load for what the edge and vertex stages gather
struct __align__(32) FaceF {
  float nx, ny, nz, c0, A, V, c1, c2;
};
// l: length, with the sign bit set on boundary edges (length() and
// interior()); bond: the bond's value
struct __align__(16) EdgeF {
  float l, th, db, bond;
  __device__ __forceinline__ float length() const { return fabsf(l); }
  __device__ __forceinline__ bool interior() const { return __float_as_int(l) >= 0; }
};

namespace fp32 {

struct f3 {
  float x, y, z;
};
__device__ __forceinline__ f3 operator+(f3 a, f3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ f3 operator-(f3 a, f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ f3 operator*(float s, f3 a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ f3& operator+=(f3& a, f3 b) {
  a.x += b.x;
  a.y += b.y;
  a.z += b.z;
  return a;
}
__device__ __forceinline__ float fdot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ f3 fcross(f3 a, f3 b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ float fnorm(f3 a) { return sqrtf(fdot(a, a)); }
__device__ __forceinline__ float fipow(float x, int n) {
  int a = n < 0 ? -n : n;
  float r = 1.0f;
  for (int k = 0; k < a; ++k) r *= x;
  return n < 0 ? 1.0f / r : r;
}

// Split positions, one 32-byte sector per vertex: hi parts (x, y, z, rho), lo
// parts (x, y, z, .), with rho = c/a written by the vertex stage, so that a
// gather of a neighbour is one load instruction where separate hi, lo and rho
// arrays took seven.
struct Pos32 {
  f3 hi, lo;
  float rho;
};
struct Split {
  const float4* X;
  __device__ __forceinline__ Pos32 at(int v) const {
    float4 h, l;
    ld32(X + 2 * (size_t)v, h, l);
    return {{h.x, h.y, h.z}, {l.x, l.y, l.z}, h.w};
  }
};
// x_b - x_a with FP32 relative accuracy
__device__ __forceinline__ f3 diff(const Pos32& b, const Pos32& a) {
  return {(b.hi.x - a.hi.x) + (b.lo.x - a.lo.x), (b.hi.y - a.hi.y) + (b.lo.y - a.lo.y),
          (b.hi.z - a.hi.z) + (b.lo.z - a.lo.z)};
}

}  // namespace fp32
}  // namespace tmg
