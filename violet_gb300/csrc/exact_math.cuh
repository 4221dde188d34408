// Arithmetic policies for passes with many divisions and square roots.
//
// A pass is written once over one of two policies:
//   Ieee    the language's operations; ok() is always true;
//   Ranged  the branch-free forms of vlt_math.cuh, which give the same bits for operands
//           in [2^-60, 2^60], and for roots of any finite number of at least 2^-100. The pass
//           states each operand whose range does not follow from what it is (see; for a
//           squared length its reciprocal root, see_rsqrt), and where ok() is false at its
//           end throws its results away and runs again over Ieee.
// One test at the end replaces one per operation: the compiler's IEEE division and root
// each end in a test for rare operands and a call, so that twenty of them made one serial
// chain of basic blocks in which nothing overlapped.
#pragma once

#include "vlt_math.cuh"

namespace vlt {

struct Ieee {
  __device__ __forceinline__ void see(float) {}
  __device__ __forceinline__ void see_rsqrt(float) {}
  __device__ __forceinline__ void see_unless(bool, float) {}
  __device__ __forceinline__ bool ok() const { return true; }
  static __device__ __forceinline__ float rcp(float b) { return 1.0f / b; }
  static __device__ __forceinline__ float div(float a, float b) { return a / b; }
  static __device__ __forceinline__ float sqrt(float x) { return sqrt_(x); }
  static __device__ __forceinline__ float rsqrt(float x) { return rsqrt_(x); }
  // lcg_rand(s) < a / b, for a divisor that was seen or is 0
  __device__ __forceinline__ bool select(uint32_t& s, float a, float b) { return lcg_select(s, a, b); }
};

struct Ranged {
  // Largest (bits - bits of 2^-60) seen: one fused add and maximum per operand. Operands
  // below the range, negative ones and NaN wrap to large values.
  uint32_t span = 0u;
  static constexpr uint32_t kLow = (127u - 60u) << 23, kSpan = 120u << 23;
  __device__ __forceinline__ void see(float x) { span = __viaddmax_u32(as_uint(x), 0u - kLow, span); }
  __device__ __forceinline__ void see_unless(bool skip, float x) { see(skip ? 1.0f : x); }
  // r = rsqrt(x) of an x that was not seen: r is in [2^-64, 2^50] for finite x >= 2^-100, above
  // for smaller ones, NaN for 0, infinity and NaN; accepted up to 2^50. A hit may then lie as
  // far as a renderer likes (a miss on a sky sphere): with x itself in see(), hits beyond
  // 2^30 sent their whole warps through the pass twice (two specular passes at 1920x1080 over
  // hits at 1e10, 1 % of them: 349 us and 213; all: 473 and 213).
  __device__ __forceinline__ void see_rsqrt(float r) {
    span = __viaddmax_u32(as_uint(r), (10u << 23) - kLow, span);
  }
  __device__ __forceinline__ bool ok() const { return span <= kSpan; }
  __device__ __forceinline__ void fail() { span = 0xFFFFFFFFu; }
  static __device__ __forceinline__ float rcp(float b) { return rcp_ranged(b); }
  static __device__ __forceinline__ float div(float a, float b) { return div_ranged(a, b); }
  static __device__ __forceinline__ float sqrt(float x) { return sqrt_ranged(x); }
  static __device__ __forceinline__ float rsqrt(float x) { return rsqrt_ranged(x); }
  // As lcg_select; what that leaves to the division is left to the IEEE policy. Both
  // operands 0 (a NaN quotient, below which no draw lies) gives d = 0, which refuses.
  __device__ __forceinline__ bool select(uint32_t& s, float a, float b) {
    const float d = fma_(-lcg_rand(s), b, a);
    const bool take = d > b * 0x1p-22f;
    if (!(take | (d <= 0.0f))) fail();
    return take;
  }
};

}  // namespace vlt
