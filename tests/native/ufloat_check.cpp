// The branch-free R11G11B10 encode against rounding done step by step in binary64, for
// every 61st binary32 (argv[1]: another stride), and the decode as its inverse on every
// finite code. Prints the mismatches.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include "../../violet_gb300/csrc/vlt_math.cuh"

using namespace vlt;

static uint32_t encode(float f, int mb) {
  const uint32_t top = (30u << mb) | ((1u << mb) - 1u);
  if (!(f > 0.0f)) return 0u;  // NaN too
  if (f >= 65536.0f) return top;
  int e;
  frexp((double)f, &e);  // f = m * 2^e, m in [1/2, 1)
  const int lowest = -14 - mb;
  const int unit = e - 1 - mb > lowest ? e - 1 - mb : lowest;
  double n = nearbyint(ldexp((double)f, -unit));  // ties to even
  const uint32_t base = unit == lowest ? 0u : (uint32_t)(unit - lowest) << mb;
  const uint32_t c = base + (uint32_t)n;
  return c > top ? top : c;
}

int main(int argc, char** argv) {
  const unsigned long long stride = argc > 1 ? strtoull(argv[1], nullptr, 10) : 61ull;
  long bad = 0;
  for (unsigned long long v = 0; v <= 0xFFFFFFFFull; v += stride) {
    const float f = as_float((uint32_t)v);
    if (f32_to_ufloat(f, 6) != encode(f, 6) || f32_to_ufloat(f, 5) != encode(f, 5)) ++bad;
  }
  // a step to either side of every code's value and of the midpoint to the next
  for (int mb = 5; mb <= 6; ++mb)
    for (uint32_t c = 0; c < (31u << mb); ++c) {
      const float at = ufloat_to_f32(c, (uint32_t)mb);
      if (f32_to_ufloat(at, (uint32_t)mb) != c) ++bad;
      const float mid = 0.5f * (at + ufloat_to_f32(c + 1 < (31u << mb) ? c + 1 : c, (uint32_t)mb));
      for (int k = -1; k <= 1; ++k) {
        const float a = as_float(as_uint(at) + (uint32_t)(at > 0.0f ? k : 1));
        const float m = as_float(as_uint(mid) + (uint32_t)(mid > 0.0f ? k : 1));
        if (f32_to_ufloat(a, (uint32_t)mb) != encode(a, mb)) ++bad;
        if (f32_to_ufloat(m, (uint32_t)mb) != encode(m, mb)) ++bad;
      }
    }
  printf("%ld mismatches\n", bad);
  return bad != 0;
}
