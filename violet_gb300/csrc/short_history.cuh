// The neighbourhood filters of the disocclusion fix (5x5) and the spatial fallback (7x7),
// which only pixels with a short history run.
//
// Such pixels lie along depth edges and the image border: about one pixel in 200 of a
// moving camera's frame, mostly a few in a tile. When each walked its own 25 or 49 taps
// (two dependent gathers, a division and an exponential per tap, the rest of its warp
// waiting), that walk was a small image's pass: at 320x180 6 us without short pixels and
// 20 (fix) or 27 us (fallback) with them. The block therefore evaluates its short
// pixels' weights together, one tap per thread, and each short pixel's thread then sums
// its taps in their order, so that the sums round as in the walk: 12 and 14 us; f32 frame
// 137 -> 125 us, reference-form denoiser passes at 1365x767 185 -> 174 us. At 1920x1080 and
// above other blocks hide the walk, and the passes stay as they were.
//
// A block of more than kShortChunk short pixels (an image edge, or every pixel after a
// reset) walks: its lanes are then mostly busy, and their loads coalesce. Staging 16 or
// more pixels served the small images as well, but the shared memory it asks for moves the
// L1 split against the kernels that run beside these (12-view batch 1,453 -> 1,480 us).
#pragma once

#include "vlt_device.cuh"

namespace vlt {

constexpr int kShortChunk = 8;  // short pixels that a block filters together

// What a tap's weight needs of the filtered pixel.
struct ShortPixel {
  f3 normal;
  float depth, fz_sigma;
  int x, y, stride;
};

template <int N>
struct ShortStage {
  static constexpr int kTaps = (2 * N + 1) * (2 * N + 1);
  ShortPixel px[kShortChunk];
  float w[kShortChunk * kTaps];
  int count;
};

// Filters the block's short pixels; every thread of the block calls it. tap(c, j, ox, oy)
// is the weight of the tap at pixel index j, offset (ox, oy) * stride, for the pixel c;
// add(w, j, inside) adds a tap of this thread's pixel to its sums (a tap outside the
// image comes with the centre's index and is not added, so that a row's loads overlap).
template <int N, class Tap, class Add>
__device__ __forceinline__ void filter_short_pixels(bool is_short, const ShortPixel& mine, int w, int h,
                                                    ShortStage<N>& st, const Tap& tap, const Add& add) {
  constexpr int D = 2 * N + 1, T = ShortStage<N>::kTaps;
  const int nt = (int)(blockDim.x * blockDim.y), tid = (int)(threadIdx.y * blockDim.x + threadIdx.x);
  if (tid == 0) st.count = 0;
  const int n = __syncthreads_count(is_short);
  if (n == 0) return;
  if (n > kShortChunk) {
    if (!is_short) return;
#pragma unroll 1
    for (int oy = -N; oy <= N; ++oy) {
#pragma unroll 1
      for (int ox = -N; ox <= N; ++ox) {
        const int cx = mine.x + ox * mine.stride, cy = mine.y + oy * mine.stride;
        if (!inb(cx, cy, w, h)) continue;
        const size_t j = (size_t)cy * w + cx;
        add(tap(mine, j, ox, oy), j, true);
      }
    }
    return;
  }
  int slot = 0;
  if (is_short) {
    slot = atomicAdd(&st.count, 1);  // any order: each pixel's sums are its own
    st.px[slot] = mine;
  }
  __syncthreads();
  for (int k = tid; k < n * T; k += nt) {
    const ShortPixel c = st.px[k / T];
    const int t = k % T, oy = t / D - N, ox = t % D - N;
    const int cx = c.x + ox * c.stride, cy = c.y + oy * c.stride;
    if (inb(cx, cy, w, h)) st.w[k] = tap(c, (size_t)cy * w + cx, ox, oy);
  }
  __syncthreads();
  if (is_short) {
    const float* ws = st.w + slot * T;
    const size_t centre = (size_t)mine.y * w + mine.x;
#pragma unroll 1
    for (int oy = -N; oy <= N; ++oy) {
#pragma unroll
      for (int ox = -N; ox <= N; ++ox) {
        const int cx = mine.x + ox * mine.stride, cy = mine.y + oy * mine.stride;
        const bool inside = inb(cx, cy, w, h);
        add(ws[(oy + N) * D + ox + N], inside ? (size_t)cy * w + cx : centre, inside);
      }
    }
  }
}

}  // namespace vlt
