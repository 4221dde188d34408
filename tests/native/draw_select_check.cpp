// lcg_select(s, a, b) against lcg_rand(s) < a / b: random operands over many magnitudes,
// quotients at and around the draw, zeros, infinities and NaN. Prints the mismatches.
#include <stdio.h>
#include <stdlib.h>

#include "../../violet_gb300/csrc/vlt_math.cuh"

using namespace vlt;

static uint64_t state = 0x9E3779B97F4A7C15ull;
static uint32_t rnd() {
  state ^= state << 13;
  state ^= state >> 7;
  state ^= state << 17;
  return (uint32_t)(state >> 16);
}
static float any() { return as_float(rnd()); }
static float positive(int span) { return as_float(((uint32_t)(127 - span + (int)(rnd() % (2 * span + 1))) << 23) | (rnd() >> 9)); }

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  const float special[] = {0.0f, -0.0f, as_float(1u), as_float(0x007FFFFFu), as_float(0x00800000u), 1.0f, -1.0f,
                           0x1p-100f, 0x1.fffffep-101f, 3.4e38f, as_float(0x7F800000u), as_float(0xFF800000u),
                           as_float(0x7FC00000u)};
  const int ns = (int)(sizeof(special) / sizeof(special[0]));
  long bad = 0, seen = 0;
  auto check = [&](uint32_t seed, float a, float b) {
    uint32_t s1 = seed, s2 = seed;
    const bool want = lcg_rand(s1) < a / b;
    const bool got = lcg_select(s2, a, b);
    ++seen;
    if (want != got || s1 != s2) ++bad;
  };
  for (long i = 0; i < n; ++i) {
    const uint32_t seed = rnd() | 1u;
    check(seed, any(), any());
    const float b = positive(i & 1 ? 20 : 120);
    check(seed, positive(20), b);
    // a / b within a few steps of the draw
    uint32_t s = seed;
    const float t = lcg_rand(s), at = t * b;
    for (int k = -3; k <= 3; ++k) check(seed, as_float(as_uint(at) + (uint32_t)k), b);
    check(seed, special[rnd() % ns], special[rnd() % ns]);
    check(seed, special[rnd() % ns], b);
    check(seed, b, special[rnd() % ns]);
  }
  printf("%ld of %ld\n", bad, seen);
  return bad != 0;
}
