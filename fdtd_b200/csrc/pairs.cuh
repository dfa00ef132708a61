// Packed pairs of FP32 values, two neighbouring columns of a 2D grid held by
// one lane: the operations of the windows (kernels_window.cu,
// kernels_adjoint.cu).
#pragma once
#include "internal.h"

namespace fdtdb {
namespace pairs {

constexpr unsigned kAll = 0xffffffffu;

// a packed pair of FP32 values (two columns), each half rounded as the
// scalar operation
typedef unsigned long long pair_t;
__device__ __forceinline__ pair_t pack(float x, float y) {
  pair_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack(pair_t p) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
  return r;
}
__device__ __forceinline__ pair_t fma2(pair_t a, pair_t b, pair_t c) {
  pair_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ pair_t mul2(pair_t a, pair_t b) {
  pair_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair_t add2(pair_t a, pair_t b) {
  pair_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair_t both(float x) { return pack(x, x); }
// a - b, one rounding
__device__ __forceinline__ pair_t sub2(pair_t a, pair_t b) { return fma2(b, both(-1.f), a); }
// a*b + c*d with the first product folded
__device__ __forceinline__ pair_t dot2(pair_t a, pair_t b, pair_t c, pair_t d) { return fma2(a, b, mul2(c, d)); }
__device__ __forceinline__ pair_t load_pair(const float* p) { return *reinterpret_cast<const pair_t*>(p); }
// state of the launch before: read through L2 (each value is read once)
__device__ __forceinline__ pair_t load_l2(const float* p) { return __ldcg(reinterpret_cast<const pair_t*>(p)); }
__device__ __forceinline__ void store_pair(float* p, pair_t v) { *reinterpret_cast<pair_t*>(p) = v; }
// v in the halves of the pair that the mask takes, 0 in the others
__device__ __forceinline__ pair_t masked(float v, bool k0, bool k1) { return pack(k0 ? v : 0.f, k1 ? v : 0.f); }

// the columns c, c + 1 of a lane within lo..hi
struct Cols {
  bool k0, k1;
  __device__ __forceinline__ Cols(int c, int lo, int hi) : k0(c >= lo && c <= hi), k1(c + 1 >= lo && c + 1 <= hi) {}
};

}  // namespace pairs
}  // namespace fdtdb
