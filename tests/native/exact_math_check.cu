// Device arithmetic that claims the bits of the IEEE operations, against them: each check
// counts the operands on which it differs and keeps one of them.
#include <cuda_runtime.h>
#include <stdint.h>

#include "exact_math.cuh"

using namespace vlt;

namespace {

struct Result {
  unsigned long long checked, bad;
  uint32_t a, b;
};

__device__ void count(Result* r, bool ok, uint32_t a, uint32_t b, unsigned long long& n) {
  ++n;
  if (ok) return;
  atomicAdd(&r->bad, 1ull);
  r->a = a;
  r->b = b;
}

__device__ bool same(float x, float y) { return as_uint(x) == as_uint(y) || (is_nan(x) && is_nan(y)); }

__device__ uint32_t mix(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return (uint32_t)((x ^ (x >> 31)) >> 16);
}

// A number of random mantissa (all ones and zeros among them) and exponent in [-range, range].
__device__ float number(uint32_t h, uint32_t e, int range) {
  uint32_t m = h & 0x7FFFFFu;
  if ((h >> 23) == 0u) m = 0u;
  if ((h >> 23) == 1u) m = 0x7FFFFFu;
  if ((h >> 23) == 2u) m &= 7u;
  if ((h >> 23) == 3u) m |= 0x7FFFF8u;
  return as_float((uint32_t)(127 - range + (int)(e % (uint32_t)(2 * range + 1))) << 23 | m);
}

// The encoder as comparisons and integer rounding.
__device__ uint32_t ufloat_by_cases(float f, uint32_t mb) {
  const uint32_t x = as_uint(f), top = (30u << mb) | ((1u << mb) - 1u);
  if ((x & 0x80000000u) || x > 0x7F800000u) return 0u;
  if (x >= 0x47800000u) return top;
  const uint32_t e = x >> 23;
  uint32_t m = (x & 0x7FFFFFu) | 0x800000u, shift, base;
  if (e < 113u) {
    if (e == 0u) return 0u;
    shift = 136u - mb - e;
    base = 0u;
    if (shift >= 32u) return 0u;
  } else {
    shift = 23u - mb;
    base = (e - 113u) << mb;
  }
  uint32_t c = base + (m >> shift);
  const uint32_t rem = m & ((1u << shift) - 1u), half = 1u << (shift - 1u);
  if (rem > half || (rem == half && (c & 1u))) c += 1u;
  return c > top ? top : c;
}

enum { kRcp, kRoots, kDiv, kDivHalfway, kNinths, kEncode, kDecode, kSelect, kSee, kChecks };

__global__ void k_check(int which, Result* res) {
  const uint64_t first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
  unsigned long long n = 0;
  if (which == kRcp) {  // every b of either sign in [2^-100, 2^100]
    for (uint64_t i = first; i <= 200ull << 23; i += step) {
      const uint32_t u = (uint32_t)(i + (27ull << 23));
      const float b = as_float(u);
      count(res, same(rcp_ranged(b), 1.0f / b) && same(rcp_ranged(-b), 1.0f / -b), u, 0u, n);
    }
  } else if (which == kRoots) {  // every finite x >= 2^-100
    for (uint64_t i = first; i < (255ull - 27ull) << 23; i += step) {
      const uint32_t u = (uint32_t)(i + (27ull << 23));
      const float x = as_float(u);
      count(res, same(sqrt_ranged(x), sqrtf(x)) && same(rsqrt_ranged(x), 1.0f / sqrtf(x)), u, 0u, n);
    }
  } else if (which == kDiv) {
    for (uint64_t i = first; i < 1ull << 32; i += step) {
      float a = number(mix(4 * i), mix(4 * i + 1), 60), b = number(mix(4 * i + 2), mix(4 * i + 3), 60);
      if (i & 1u) a = -a;
      if (i & 2u) b = -b;
      count(res, same(div_ranged(a, b), a / b), as_uint(a), as_uint(b), n);
    }
  } else if (which == kDivHalfway) {  // quotients next to the middle of two neighbours
    for (uint64_t i = first; i < 1ull << 30; i += step) {
      const float b = number(mix(3 * i), mix(3 * i + 1), 30);
      const uint32_t q = 0x800000u | (mix(3 * i + 2) & 0x7FFFFFu);
      const double mid = ((double)q + 0.5) * (double)b;  // exact: 25 + 24 bits
      const float a0 = (float)mid;
      for (int d = -1; d <= 1; ++d) {
        const float a = as_float(as_uint(a0) + (uint32_t)d);
        count(res, same(div_ranged(a, b), a / b), as_uint(a), as_uint(b), n);
      }
    }
  } else if (which == kNinths) {  // the shared reciprocal of 9
    for (uint64_t i = first; i <= 120ull << 23; i += step) {
      const uint32_t u = (uint32_t)(i + (67ull << 23));
      count(res, same(div_shared(as_float(u), 9.0f, 1.0f / 9.0f), as_float(u) / 9.0f), u, 0u, n);
    }
  } else if (which == kEncode) {  // every binary32
    for (uint64_t i = first; i < 1ull << 32; i += step) {
      const float f = as_float((uint32_t)i);
      count(res, f32_to_ufloat(f, 5) == ufloat_by_cases(f, 5) && f32_to_ufloat(f, 6) == ufloat_by_cases(f, 6),
            (uint32_t)i, 0u, n);
    }
  } else if (which == kDecode) {  // every word
    for (uint64_t i = first; i < 1ull << 32; i += step) {
      const f3 x = unpack_r11g11b10((uint32_t)i), y = unpack_r11g11b10_int((uint32_t)i);
      count(res, same(x.x, y.x) && same(x.y, y.y) && same(x.z, y.z), (uint32_t)i, 0u, n);
    }
  } else if (which == kSelect) {  // quotients around the draw, zeros, and any
    for (uint64_t i = first; i < 1ull << 28; i += step) {
      const uint32_t seed = mix(5 * i) | 1u;
      uint32_t s0 = seed, s1 = seed, s2 = seed, s3 = seed;
      const float t = lcg_rand(s0);
      const float b = (i & 31u) == 7u ? 0.0f : number(mix(5 * i + 1), mix(5 * i + 2), 60);
      float a = (i & 1u) ? number(mix(5 * i + 3), mix(5 * i + 4), 60) : t * b;
      if (!(i & 1u)) a = as_float((uint32_t)max((int)as_uint(a) + (int)(mix(5 * i + 3) % 17u) - 8, 0));
      if ((i & 63u) == 11u) a = 0.0f;
      const bool want = t < a / b;
      Ranged r;
      const bool got = r.select(s1, a, b);
      Ieee e;
      // Ranged may decline, but then only next to the draw
      const bool close = fabsf(fma_(-t, b, a)) <= b * 0x1p-21f;
      count(res, lcg_select(s2, a, b) == want && e.select(s3, a, b) == want && (r.ok() ? got == want : close) &&
                     s1 == s0 && s2 == s0 && s3 == s0,
            as_uint(a), as_uint(b), n);
    }
  } else if (which == kSee) {  // every bit pattern of an operand, and of a squared length
    for (uint64_t i = first; i < 1ull << 32; i += step) {
      const float x = as_float((uint32_t)i);
      Ranged r, q;
      r.see(1.0f);
      r.see(x);
      r.see(1.0f);
      count(res, r.ok() == (x >= 0x1p-60f && x <= 0x1p60f), (uint32_t)i, 0u, n);
      if (x < 0.0f) continue;  // a squared length is not
      const float y = rsqrt_ranged(x);
      q.see_rsqrt(y);
      // accepted roots are right, and everything from 2^-100 to infinity is accepted
      count(res, (!q.ok() || same(y, 1.0f / sqrtf(x))) && (q.ok() || !(x >= 0x1p-100f && x < INFINITY)), (uint32_t)i,
            1u, n);
    }
  }
  atomicAdd(&res->checked, n);
}

}  // namespace

extern "C" int exact_math_checks() { return kChecks; }

// {operands checked, mismatches, one of them (a, b)}; a CUDA error code, or 0.
extern "C" int exact_math_check(int which, unsigned long long out[4]) {
  Result* d = nullptr;
  Result h = {};
  cudaError_t e = cudaMalloc(&d, sizeof(Result));
  if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof(Result));
  if (e == cudaSuccess) {
    k_check<<<152 * 8, 256>>>(which, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(Result), cudaMemcpyDeviceToHost);
  cudaFree(d);
  out[0] = h.checked;
  out[1] = h.bad;
  out[2] = h.a;
  out[3] = h.b;
  return (int)e;
}
