// The scene tracer's march against the plain one: all 64 samples evaluated, the ground
// bisected before any sphere, shadow rays traced in full. Random rays of many shapes
// (grazing, climbing, descending, long, far from the origin) and special values. Prints
// the mismatches.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "../../violet_gb300/csrc/scene_gen.cuh"

using namespace vlt;
using namespace vlt::scene;

static Hit plain(const Object& o, f3 org, f3 dir) {
  Hit h;
  memset(&h, 0, sizeof(h));
  h.t = 1e30f;
  h.obj = -1;
  float before = 0.0f;
  for (int i = 1; i <= 64; ++i) {
    const float s = (float)i / 64.0f;
    const float t = VLT_SCENE_MAX_DIST * (s * sqrt_(s));
    const f3 p = org + t * dir;
    if (p.y - height(o, p.x, p.z) < 0.0f) {
      float lo = before, hi = t;
      for (int b = 0; b < 16; ++b) {
        const float mid = 0.5f * (lo + hi);
        const f3 q = org + mid * dir;
        if (q.y - height(o, q.x, q.z) < 0.0f) hi = mid;
        else lo = mid;
      }
      h.t = hi;
      h.obj = 0;
      break;
    }
    before = t;
  }
  for (int k = 0; k < 4; ++k) {
    const f3 oc = org - mk3(o.sc[k][0], o.sc[k][1], o.sc[k][2]);
    const float b = dot3(oc, dir), cc = dot3(oc, oc) - o.sc[k][3] * o.sc[k][3];
    const float disc = b * b - cc;
    if (!(disc > 0.0f)) continue;
    const float t = -b - sqrt_(disc);
    if (t > 0.05f && t < h.t) h.t = t, h.obj = 1 + k;
  }
  if (h.t > VLT_SCENE_MAX_DIST) h.obj = -1;
  return h;
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 100000;
  Rng r = {20241u};
  const float special[] = {0.0f, -0.0f, 1e-30f, 1.0f, -1.0f, 1e3f, 1e5f, -1e20f, as_float(0x7F800000u),
                           as_float(0xFF800000u), as_float(0x7FC00000u)};
  const int ns = (int)(sizeof(special) / sizeof(special[0]));
  long bad = 0, hits = 0;
  Object o = make_object(1);
  for (long i = 0; i < n; ++i) {
    if (i % 256 == 0) o = make_object((uint64_t)i * 7919u + 3u);
    const float reach = i % 5 == 0 ? 1000.0f : 20.0f;
    f3 org = mk3(reach * (2.0f * r.next() - 1.0f), 0.0f, reach * (2.0f * r.next() - 1.0f));
    const float ground = height(o, org.x, org.z);
    const float lift = i % 3 == 0 ? 1e-3f : i % 3 == 1 ? 0.02f : 4.0f;
    org.y = i % 11 == 0 ? o.top : ground + lift * r.next();
    f3 dir = mk3(2.0f * r.next() - 1.0f, 2.0f * r.next() - 1.0f, 2.0f * r.next() - 1.0f);
    if (i % 4 == 1) dir.y = dir.y * 0.1f;
    if (i % 7 == 2) dir.y = 0.0f;
    dir = normalize3(dir);
    if (i % 13 == 0) dir = 10.0f * dir;
    if (i % 17 == 0) {
      float* v[6] = {&org.x, &org.y, &org.z, &dir.x, &dir.y, &dir.z};
      *v[(int)(r.next() * 6.0f) % 6] = special[(int)(r.next() * (float)ns) % ns];
    }
    const Hit want = plain(o, org, dir);
    const Hit got = trace(o, org, dir);
    const bool same = want.obj == got.obj && (want.obj < 0 || as_uint(want.t) == as_uint(got.t));
    if (!same || occluded(o, org, dir) != (want.obj >= 0)) ++bad;
    hits += want.obj >= 0;
  }
  printf("%ld rays, %ld hits, %ld mismatches\n", n, hits, bad);
  return bad != 0 || hits < n / 10 || hits > n - n / 10;
}
