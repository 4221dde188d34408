// ReLAX/SVGF denoiser passes: temporal accumulation (with dual-source virtual
// reprojection for specular), disocclusion fix, fast-history clamp, spatial
// fallback / variance estimation, and the edge-stopping a-trous filter.
// Colour history is a packed uint2 {diffuse, specular} of R11G11B10 words (one
// 64-bit access per tap), moments/variance are half2, history length is R8_UNORM.
// Kernels are templated on the geometry source (GeoRaw / GeoSurface).
#include "short_history.cuh"
#include "vlt_internal.h"

namespace vlt {

__device__ __forceinline__ f3 col_diff(uint2 c) { return unpack_r11g11b10(c.x); }
__device__ __forceinline__ f3 col_spec(uint2 c) { return unpack_r11g11b10(c.y); }
__device__ __forceinline__ f2 unpack_half2(uint32_t u) { return mk2(f16tof32(u & 0xFFFFu), f16tof32(u >> 16)); }

// EdgeStoppingFunc (svgf.inc.hlsl:6-84), with the per-centre reciprocals of the
// luminance deviation, rcp(sigma_l * std + eps), computed once per pixel.
struct EdgeStop {
  float depth_center, fwidth_z;
  f3 normal_center;
  f2 lumi_center;
  f2 lumi_rcp;
  float sigma_z;
  int sigma_n_log2;  // sigma_n = 2^k (128 -> 7, 32 -> 5)

  __device__ __forceinline__ void set_lumi(f2 lumi, f2 var) {
    const float sigma_l = 4.0f;
    const float eps = 1e-8f;
    lumi_center = lumi;
    f2 sd = mk2(sqrt_(var.x), sqrt_(var.y));
    lumi_rcp = mk2(1.0f / (sigma_l * sd.x + eps), 1.0f / (sigma_l * sd.y + eps));
  }

  __device__ __forceinline__ f2 weight(float tap_dist, float depth, f3 normal, f2 lumi) const {
    const float eps = 1e-8f;
    float dist_z = fabs_(depth - depth_center);
    float wz = -dist_z / ((sigma_z * fwidth_z) * tap_dist + eps);
    float n_dot = saturate(dot3(normal_center, normal));
    float wn = pow_2k(n_dot, sigma_n_log2);
    f2 dl = mk2(fabs_(lumi.x - lumi_center.x), fabs_(lumi.y - lumi_center.y));
    f2 wl = mk2(-dl.x * lumi_rcp.x, -dl.y * lumi_rcp.y);
    return mk2(wn * exp_(wl.x + wz), wn * exp_(wl.y + wz));
  }
};

__device__ __forceinline__ EdgeStop make_edge_stop(float depth, float fwidth_z, f3 normal) {
  EdgeStop e;
  e.depth_center = depth;
  e.fwidth_z = fwidth_z;
  e.normal_center = normal;
  e.lumi_center = mk2(0.0f, 0.0f);
  e.lumi_rcp = mk2(0.0f, 0.0f);
  e.sigma_z = 1.0f;
  e.sigma_n_log2 = 7;
  return e;
}

// dsr_weight (svgf_temporal_filter.hlsl:89-93).
__device__ __forceinline__ float dsr_weight(f3 color, f3 mean, f3 dev) {
  float dist = luminance(abs3(color - mean) / dev);
  return exp2_(-10.0f * dist);
}

// --------------------------------------------------------------- temporal

// svgf_temporal_filter.hlsl:96-362.
// FAST: the fast history (fast_history_clamp) is kept; the launcher picks the
// instantiation from the knob, so a frame without it carries none of its registers.
template <class Geo, bool FAST>
struct DnTemporalF {
  // 64 registers. Denoiser passes at 1365x767 with the fast history: 134.2 us, at 48 registers
  // (which spill 276 bytes) 136.1, at 80 134.5, at 40 137.2, uncapped 141.8; a 1280x720 frame
  // without it is the same at all of them.
  static constexpr int kMinBlocks = 4;
  static __device__ __forceinline__ void run(int x0, int y0, vlt_frame_params fp, int w, int h, DenoiseKnobs kn, Geo geo, Geo prev_geo, const uint32_t* __restrict__ gbuf, const uint32_t* __restrict__ diff_src, const uint32_t* __restrict__ spec_src, const uint16_t* __restrict__ ray_len_tex, const float* __restrict__ prev_depth, const uint2* __restrict__ color_hist, const uint32_t* __restrict__ mom_hist, const uint8_t* __restrict__ len_hist, const uint2* __restrict__ fast_hist, uint2* __restrict__ out_color, uint32_t* __restrict__ out_mom, uint8_t* __restrict__ out_len, uint2* __restrict__ out_fast, uint32_t has_history) {
  int x = x0 + (int)threadIdx.x, y = y0 + (int)threadIdx.y;
  if (!inb(x, y, w, h)) return;
  size_t i = (size_t)y * w + x;
  float depth = geo.dep(i);
  if (depth == 0.0f) {
    out_len[i] = 0;
    out_color[i] = make_uint2(0u, 0u);
    out_mom[i] = 0u;
    if (FAST) out_fast[i] = make_uint2(0u, 0u);
    return;
  }
  const float bw = (float)w, bh = (float)h;
  f2 screen_uv = pixel_uv(x, y, w, h);
  const f3 gnormal = geo.normal(i);
  const float grough = geo.rough(i);
  const float fwz = geo.fwz(i);
  const float fwn = f16tof32(gbuf[2 * (size_t)w * h + i] >> 16);

  // 3x3 specular moments (x outer, y inner as in the shader).
  f3 m1 = mk3(0.0f), m2 = mk3(0.0f);
#pragma unroll
  for (int dx = -1; dx <= 1; ++dx) {
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy) {
      int px = x + dx, py = y + dy;
      px = px < 0 ? 0 : (px > w - 1 ? w - 1 : px);
      py = py < 0 ? 0 : (py > h - 1 ? h - 1 : py);
      f3 s = unpack_r11g11b10(spec_src[(size_t)py * w + px]);
      m1 = m1 + s;
      m2 = m2 + s * s;
    }
  }
  m1 = m1 * (1.0f / 9.0f);
  m2 = m2 * (1.0f / 9.0f);

  // The shader reconstructs the position from depth twice; both equal cs_depth_to_position.
  const f3 position = geo.pos(x, y, i);

  // Virtual (hit-point) reprojection for specular.
  f3 vsh = mk3(0.0f), vsfh = mk3(0.0f);
  {
    f3 vdir = normalize3(position - vpos3(fp.view_pos));
    float ray_len = f16tof32(ray_len_tex[i]);
    f3 vp = position + vdir * ray_len;
    f4 hr = mul44(fp.prev_view_proj, mk4(vp.x, vp.y, vp.z, 1.0f));
    f2 ndc = mk2(hr.x / hr.w - fp.jitter[2], hr.y / hr.w - fp.jitter[3]);
    f2 vuv = mk2((ndc.x + fp.jitter[0]) * 0.5f + 0.5f, (ndc.y + fp.jitter[1]) * 0.5f + 0.5f);
    bool valid = vuv.x == saturate(vuv.x) && vuv.y == saturate(vuv.y) && has_history;
    if (valid) {
      BilinearTaps t = bilinear_taps(vuv, w, h);
      uint2 a = color_hist[(size_t)t.y0 * w + t.x0], b = color_hist[(size_t)t.y0 * w + t.x1];
      uint2 c = color_hist[(size_t)t.y1 * w + t.x0], d = color_hist[(size_t)t.y1 * w + t.x1];
      vsh = bilerp3(col_spec(a), col_spec(b), col_spec(c), col_spec(d), t.fx, t.fy);
      if (FAST) {
        uint2 fa = fast_hist[(size_t)t.y0 * w + t.x0], fb = fast_hist[(size_t)t.y0 * w + t.x1];
        uint2 fc = fast_hist[(size_t)t.y1 * w + t.x0], fd = fast_hist[(size_t)t.y1 * w + t.x1];
        vsfh = bilerp3(col_spec(fa), col_spec(fb), col_spec(fc), col_spec(fd), t.fx, t.fy);
      }
    }
  }

  // Surface reprojection.
  f2 mv;
  float reproj_depth;
  {
    f4 hp = mul44(fp.view_proj, mk4(position.x, position.y, position.z, 1.0f));
    f2 ndc = mk2(hp.x / hp.w - fp.jitter[0], hp.y / hp.w - fp.jitter[1]);
    f4 hr = mul44(fp.prev_view_proj, mk4(position.x, position.y, position.z, 1.0f));
    f2 ndc_r = mk2(hr.x / hr.w - fp.jitter[2], hr.y / hr.w - fp.jitter[3]);
    mv = mk2((ndc.x - ndc_r.x) * 0.5f, (ndc.y - ndc_r.y) * 0.5f);
    reproj_depth = hr.z / hr.w;
  }
  f2 huv = mk2(screen_uv.x - mv.x, screen_uv.y - mv.y);

  f3 dh = mk3(0.0f), sh = mk3(0.0f), dfh = mk3(0.0f), sfh = mk3(0.0f);
  f2 smh = mk2(0.0f, 0.0f);
  float hl = 0.0f;
  bool valid = huv.x == saturate(huv.x) && huv.y == saturate(huv.y) && has_history;
  if (valid) {
    f2 pcc = mk2(huv.x * bw - 0.5f, huv.y * bh - 0.5f);
    f2 frac = mk2(pcc.x - floor_(pcc.x), pcc.y - floor_(pcc.y));
    int bx = f2i_rz(pcc.x), by = f2i_rz(pcc.y);
    float depth_tol = fwz * 4.0f + 1e-4f;
    float normal_tol = fwn * 16.0f + 1e-2f;
    float normal_tol_sq = normal_tol * normal_tol;
    float bb = frac.y, rr = frac.x, tt = 1.0f - bb, ll = 1.0f - rr;
    float wts[2][2] = {{tt * ll, tt * rr}, {bb * ll, bb * rr}};
    f3 ds = mk3(0.0f), ss = mk3(0.0f), dfs = mk3(0.0f), sfs = mk3(0.0f);
    f2 ms = mk2(0.0f, 0.0f);
    float hs = 0.0f, wsum = 0.0f;
#pragma unroll
    for (int ox = 0; ox < 2; ++ox) {
#pragma unroll
      for (int oy = 0; oy < 2; ++oy) {
        int px = bx + ox, py = by + oy;
        bool cv = px >= 0 && py >= 0 && px <= w - 1 && py <= h - 1;
        if (!cv) continue;
        size_t j = (size_t)py * w + px;
        // History loads ahead of the geometry test (their latency overlaps its loads).
        const uint2 c = color_hist[j];
        const uint32_t mj = mom_hist[j];
        const uint8_t lj = len_hist[j];
        f3 n = prev_geo.normal(j);
        f3 nd = n - gnormal;
        bool ok = fabs_(prev_depth[j] - reproj_depth) < depth_tol && dot3(nd, nd) < normal_tol_sq;
        if (!ok) continue;
        float wt = wts[oy][ox];
        wsum = wsum + wt;
        ds = ds + wt * col_diff(c);
        ss = ss + wt * col_spec(c);
        ms = ms + wt * unpack_half2(mj);
        hs = hs + wt * unorm8_load(lj);
        if (FAST) {
          uint2 f = fast_hist[j];
          dfs = dfs + wt * col_diff(f);
          sfs = sfs + wt * col_spec(f);
        }
      }
    }
    valid = wsum > 0.00390625f;
    if (valid) {
      float inv = 1.0f / wsum;
      dh = ds * inv;
      sh = ss * inv;
      smh = ms * inv;
      hl = hs * inv;
      dfh = dfs * inv;
      sfh = sfs * inv;
    }
  }
  if (!valid) {
    dh = sh = dfh = sfh = mk3(0.0f);
    smh = mk2(0.0f, 0.0f);
    hl = 0.0f;
  }
  hl = hl + VLT_HISTORY_LEN_UNIT;

  f3 dsrc = unpack_r11g11b10(diff_src[i]);
  f3 ssrc = unpack_r11g11b10(spec_src[i]);
  f2 lsrc = mk2(luminance(dsrc), luminance(ssrc));
  f2 smsrc = lsrc * lsrc;

  const float bfd = kn.blend_diff;
  const float bff = 1.0f / 3.0f;
  float blurness = sqrt_(saturate(grough * 6.0f));
  const float bfs = lerpf(7.0f / 8.0f, bfd, blurness);
  const float bfsf = lerpf(1.0f, bff, blurness);
  float ratio = VLT_HISTORY_LEN_UNIT / hl;
  f2 alpha = mk2(fmax_(bfd, ratio), fmax_(bfs, ratio));
  f3 df = lerp3(dh, dsrc, alpha.x);
  f3 sf;
  f2 smf = mk2(lerpf(smh.x, smsrc.x, alpha.x), lerpf(smh.y, smsrc.y, alpha.y));
  f2 alpha_f = mk2(fmax_(bff, ratio), fmax_(bfsf, ratio));
  f3 dff = lerp3(dfh, dsrc, alpha_f.x);
  f3 sff = lerp3(sfh, ssrc, alpha_f.y);
  {
    f3 mean = m1;
    f3 dev = sqrt3(abs3(m2 - mean * mean));
    dev = mk3(fmax_(dev.x, 1e-19f), fmax_(dev.y, 1e-19f), fmax_(dev.z, 1e-19f));
    float wv = dsr_weight(vsh, mean, dev);
    float wh = dsr_weight(sh, mean, dev);
    f3 dual = wv * vsh + wh * sh;
    float ws = wv + wh;
    dual = dual / fmax_(ws, 1e-37f);
    sf = lerp3(dual, ssrc, alpha.y);
    if (FAST) {
      float wv2 = dsr_weight(vsfh, mean, dev);
      float wh2 = dsr_weight(sfh, mean, dev);
      f3 dual2 = wv2 * vsfh + wh2 * sfh;
      float ws2 = wv2 + wh2;
      dual2 = dual2 / fmax_(ws2, 1e-37f);
      sff = lerp3(dual2, ssrc, alpha_f.y);
    }
  }
  out_color[i] = make_uint2(pack_r11g11b10(df), pack_r11g11b10(sf));
  out_mom[i] = pack_half2(smf);
  out_len[i] = (uint8_t)unorm8_store(hl);
  if (FAST) out_fast[i] = make_uint2(pack_r11g11b10(dff), pack_r11g11b10(sff));
}
};

// Max history length over the aligned 2x2 quad (QuadReadAcrossX/Y of the
// quad-remapped 8x8 groups); out-of-range quad members read as 0.
__device__ __forceinline__ float quad_max_len(const uint8_t* __restrict__ len, int x, int y, int w, int h) {
  int x0 = x & ~1, y0 = y & ~1;
  float m = 0.0f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    int px = x0 + (k & 1), py = y0 + (k >> 1);
    float v = inb(px, py, w, h) ? unorm8_load(len[(size_t)py * w + px]) : 0.0f;
    m = fmax_(m, v);
  }
  return m;
}

// --------------------------------------------------------- disocclusion fix

namespace {

// Sums of the short-history filters (the weight without luminance terms is the same for
// both channels), and that weight.
struct FilterSums {
  float w = 0.0f;
  f3 d = mk3(0.0f), s = mk3(0.0f);
  f2 m = mk2(0.0f, 0.0f);
  __device__ __forceinline__ void add(float wt, uint2 c, uint32_t mom) {
    w = w + wt;
    d = d + col_diff(c) * wt;
    s = s + col_spec(c) * wt;
    m = m + unpack_half2(mom) * wt;
  }
};
template <class Geo>
__device__ __forceinline__ float short_weight(const ShortPixel& c, const Geo& geo, size_t j, float tap_dist,
                                              int sigma_n_log2) {
  const float wz = -fabs_(geo.dep(j) - c.depth) / (c.fz_sigma * tap_dist + 1e-8f);
  return pow_2k(saturate(dot3(c.normal, geo.normal(j))), sigma_n_log2) * exp_(wz);
}

}  // namespace

// relax_disocclusion_fix.hlsl:27-122. Pixels without geometry (history 0) are not
// written by the shader; here they get zeros.
template <class Geo>
struct DnFixF {
  static constexpr int kMinBlocks = 5;  // 48 registers: most pixels only copy their record
  static __device__ __forceinline__ void run(int x0, int y0, int w, int h, Geo geo, const uint8_t* __restrict__ len_tex, const uint2* __restrict__ color, const uint32_t* __restrict__ mom, uint2* __restrict__ out_color, uint32_t* __restrict__ out_mom) {
  __shared__ ShortStage<2> st;
  const int x = x0 + (int)threadIdx.x, y = y0 + (int)threadIdx.y;
  const bool inside = inb(x, y, w, h);
  const size_t i = inside ? (size_t)y * w + x : 0;
  const float hl = inside ? unorm8_load(len_tex[i]) : 0.0f;
  const float qmax = inside ? quad_max_len(len_tex, x, y, w, h) : 0.0f;
  const bool is_short = hl != 0.0f && qmax < 4.0f * VLT_HISTORY_LEN_UNIT;
  ShortPixel c = {mk3(0.0f), 0.0f, 0.0f, x, y, 0};
  if (is_short) {
    c.stride = f2i_rz((14.0f * VLT_HISTORY_LEN_UNIT) / qmax);
    c.depth = geo.dep(i);
    c.fz_sigma = 5.0f * geo.fwz(i);
    c.normal = geo.normal(i);
  } else if (inside) {
    out_color[i] = hl == 0.0f ? make_uint2(0u, 0u) : color[i];
    out_mom[i] = hl == 0.0f ? 0u : mom[i];
  }
  FilterSums t;
  filter_short_pixels<2>(
      is_short, c, w, h, st,
      [&](const ShortPixel& cc, size_t j, int ox, int oy) {
        return short_weight(cc, geo, j, length2(mk2((float)(ox * cc.stride), (float)(oy * cc.stride))), 5);
      },
      [&](float wt, size_t j, bool ok) {
        const uint2 cj = color[j];
        const uint32_t mj = mom[j];
        if (ok) t.add(wt, cj, mj);
      });
  if (is_short) {
    out_color[i] = make_uint2(pack_r11g11b10(t.d / t.w), pack_r11g11b10(t.s / t.w));
    out_mom[i] = pack_half2(mk2(t.m.x / t.w, t.m.y / t.w));
  }
}
};

// ------------------------------------------------------ fast history clamp

__device__ __forceinline__ f3 rgb_to_ycocg(f3 c) {
  return mk3(c.x * 0.25f + c.y * 0.5f + c.z * 0.25f, c.x * 0.5f - c.z * 0.5f, c.x * -0.25f + c.y * 0.5f - c.z * 0.25f);
}
__device__ __forceinline__ f3 ycocg_to_rgb(f3 c) {
  float tmp = c.x - c.z;
  return mk3(tmp + c.y, c.x + c.z, tmp - c.y);
}

// relax_fast_history_clamp.hlsl:11-75 (in place on the slow colour). A block decodes its
// tile and a pixel around it into YCoCg once (each pixel decoded its nine neighbours: 18
// R11G11B10 words); the twelve means share the reciprocal of 9: they are multiples of
// 2^-48 within 2^36, and a special code makes the clamp's bounds NaN either way.
// 1365x767: 45 -> 30 us, 1280x720 reference frame with the clamp 595 -> 579 us.
struct DnFastClampF {
  // single views run 32x4 tiles, which are among the candidates of the batches
  static constexpr int kStage = max_staged_tile(1);
  static __device__ __forceinline__ void run(int x0, int y0, int w, int h, const uint2* __restrict__ fast, uint2* __restrict__ color) {
  struct Px {
    float2 y, co, cg;  // diffuse, specular
  };
  __shared__ Px tile[kStage];
  const int bx = (int)blockDim.x, by = (int)blockDim.y, pw = bx + 2;
  const int tid = (int)threadIdx.y * bx + (int)threadIdx.x;
  __syncthreads();  // a persistent block's previous tile is done with the stage
  for (int k = tid; k < pw * (by + 2); k += bx * by) {
    const int r = k / pw;
    int cx = x0 + k - r * pw - 1, cy = y0 + r - 1;
    cx = cx < 0 ? 0 : (cx > w - 1 ? w - 1 : cx);
    cy = cy < 0 ? 0 : (cy > h - 1 ? h - 1 : cy);
    const uint2 f = fast[(size_t)cy * w + cx];
    const f3 d = rgb_to_ycocg(col_diff(f)), s = rgb_to_ycocg(col_spec(f));
    tile[k].y = make_float2(d.x, s.x);
    tile[k].co = make_float2(d.y, s.y);
    tile[k].cg = make_float2(d.z, s.z);
  }
  __syncthreads();
  const int x = x0 + (int)threadIdx.x, y = y0 + (int)threadIdx.y;
  if (!inb(x, y, w, h)) return;
  size_t i = (size_t)y * w + x;
  f3 dm1 = mk3(0.0f), dm2 = mk3(0.0f), sm1 = mk3(0.0f), sm2 = mk3(0.0f);
#pragma unroll
  for (int oy = 0; oy <= 2; ++oy) {
#pragma unroll
    for (int ox = 0; ox <= 2; ++ox) {
      const Px t = tile[((int)threadIdx.y + oy) * pw + (int)threadIdx.x + ox];
      const f3 d = mk3(t.y.x, t.co.x, t.cg.x), s = mk3(t.y.y, t.co.y, t.cg.y);
      dm1 = dm1 + d;
      dm2 = dm2 + d * d;
      sm1 = sm1 + s;
      sm2 = sm2 + s * s;
    }
  }
  const auto mean = [](f3 v) {
    const float r = 1.0f / 9.0f;
    return mk3(div_shared(v.x, 9.0f, r), div_shared(v.y, 9.0f, r), div_shared(v.z, 9.0f, r));
  };
  const auto root = [](f3 v) {
    return mk3(v.x == 0.0f ? 0.0f : sqrt_ranged(v.x), v.y == 0.0f ? 0.0f : sqrt_ranged(v.y),
               v.z == 0.0f ? 0.0f : sqrt_ranged(v.z));
  };
  dm1 = mean(dm1);
  dm2 = mean(dm2);
  sm1 = mean(sm1);
  sm2 = mean(sm2);
  f3 ddev = root(dm2 - dm1 * dm1) * 0.75f;
  f3 sdev = root(sm2 - sm1 * sm1) * 0.75f;
  uint2 c = color[i];
  f3 d = rgb_to_ycocg(col_diff(c));
  f3 s = rgb_to_ycocg(col_spec(c));
  d = clamp3(d, dm1 - ddev, dm1 + ddev);
  s = clamp3(s, sm1 - sdev, sm1 + sdev);
  color[i] = make_uint2(pack_r11g11b10(ycocg_to_rgb(d)), pack_r11g11b10(ycocg_to_rgb(s)));
}
};

// ---------------------------------------------------------- spatial fallback

// svgf_spatial_fallback_filter.hlsl:25-125. History-0 pixels get zeros.
template <class Geo>
struct DnFallbackF {
  static constexpr int kMinBlocks = 5;  // 48 registers: most pixels only copy their record
  static __device__ __forceinline__ void run(int x0, int y0, int w, int h, Geo geo, const uint8_t* __restrict__ len_tex, const uint2* __restrict__ color, const uint32_t* __restrict__ mom, uint2* __restrict__ out_color, uint32_t* __restrict__ out_var) {
  __shared__ ShortStage<3> st;
  const int x = x0 + (int)threadIdx.x, y = y0 + (int)threadIdx.y;
  const bool inside = inb(x, y, w, h);
  const size_t i = inside ? (size_t)y * w + x : 0;
  const float own = inside ? unorm8_load(len_tex[i]) : 0.0f;
  const float hl = inside ? quad_max_len(len_tex, x, y, w, h) : 0.0f;
  const bool is_short = own != 0.0f && hl < 4.0f * VLT_HISTORY_LEN_UNIT;
  ShortPixel c = {mk3(0.0f), 0.0f, 0.0f, x, y, 1};
  if (is_short) {
    c.depth = geo.dep(i);
    c.fz_sigma = 1.0f * (geo.fwz(i) * 3.0f);
    c.normal = geo.normal(i);
  }
  const auto finish = [&](f3 dd, f3 sd, f2 md) {
    f2 fst = mk2(luminance(dd), luminance(sd));
    f2 var = mk2(fmax_(md.x - fst.x * fst.x, 0.0f), fmax_(md.y - fst.y * fst.y, 0.0f));
    float boost = fmax_(1.0f, (4.0f * VLT_HISTORY_LEN_UNIT) / hl);
    var = var * boost;
    out_color[i] = make_uint2(pack_r11g11b10(dd), pack_r11g11b10(sd));
    out_var[i] = pack_half2(var);
  };
  if (inside && !is_short) {
    if (own == 0.0f) {
      out_color[i] = make_uint2(0u, 0u);
      out_var[i] = 0u;
    } else {
      const uint2 cc = color[i];
      finish(col_diff(cc), col_spec(cc), unpack_half2(mom[i]));
    }
  }
  FilterSums t;
  filter_short_pixels<3>(
      is_short, c, w, h, st,
      [&](const ShortPixel& cc, size_t j, int ox, int oy) {
        return short_weight(cc, geo, j, length2(mk2((float)ox, (float)oy)), 7);
      },
      [&](float wt, size_t j, bool ok) {
        const uint2 cj = color[j];
        const uint32_t mj = mom[j];
        if (ok) t.add(wt, cj, mj);
      });
  if (is_short) finish(t.d / t.w, t.s / t.w, mk2(t.m.x / t.w, t.m.y / t.w));
}
};

// --------------------------------------------------------------- a-trous

// length(float2(coord_offset)) of the 16 off-axis taps at one step size,
// tabulated once per launch (tap k = (oy+2)*4 + ox' over the non-zero offsets).
struct AtrousTaps {
  float dist[16];
};

// svgf_atrous_filter.hlsl:23-88: 5x5 taps at step 2^i, kernel {1, 2/3, 1/6}, only
// the 16 taps off both centre axes (the shader's `(x != 0) && (y != 0)`).
template <class Geo>
__device__ __forceinline__ void atrous_px(int x, int y, int w, int h, const Geo& geo, const AtrousTaps& taps, const uint2* __restrict__ color, const uint32_t* __restrict__ var_tex, uint2* __restrict__ out_color, uint32_t* __restrict__ out_var, uint32_t* __restrict__ out_diff, uint32_t* __restrict__ out_spec, int step) {
  size_t i = (size_t)y * w + x;
  uint2 cc = color[i];
  f3 diff_c = col_diff(cc), spec_c = col_spec(cc);
  f2 lumi_c = mk2(luminance(diff_c), luminance(spec_c));
  f2 var_c = unpack_half2(var_tex[i]);
  EdgeStop es = make_edge_stop(geo.dep(i), geo.fwz(i), geo.normal(i));
  es.set_lumi(lumi_c, var_c);
  const float kw[3] = {1.0f, 2.0f / 3.0f, 1.0f / 6.0f};
  f3 dsum = diff_c, ssum = spec_c;
  f2 vsum = var_c;
  f2 wsum = mk2(1.0f, 1.0f);
  int tap = 0;
#pragma unroll
  for (int oy = -2; oy <= 2; ++oy) {
    if (oy == 0) continue;
    const float kwy = kw[oy < 0 ? -oy : oy];
#pragma unroll
    for (int ox = -2; ox <= 2; ++ox) {
      if (ox == 0) continue;
      const float tap_dist = taps.dist[tap++];
      int cx = x + ox * step, cy = y + oy * step;
      bool cv = cx >= 0 && cy >= 0 && cx <= w - 1 && cy <= h - 1;
      if (!cv) continue;
      float k = kwy * kw[ox < 0 ? -ox : ox];
      size_t j = (size_t)cy * w + cx;
      uint2 c = color[j];
      f3 d = col_diff(c), s = col_spec(c);
      f2 lumi = mk2(luminance(d), luminance(s));
      f2 e = es.weight(tap_dist, geo.dep(j), geo.normal(j), lumi);
      f2 wt = mk2(k * e.x, k * e.y);
      f2 wv = wt * wt;
      dsum = dsum + wt.x * d;
      ssum = ssum + wt.y * s;
      vsum = vsum + wv * unpack_half2(var_tex[j]);
      wsum = wsum + wt;
    }
  }
  f3 dd = dsum / wsum.x;
  f3 sd = ssum / wsum.y;
  f2 vd = vsum / (wsum * wsum);
  uint32_t pd = pack_r11g11b10(dd), ps = pack_r11g11b10(sd);
  if (out_color) out_color[i] = make_uint2(pd, ps);
  if (out_var) out_var[i] = pack_half2(vd);
  if (out_diff) out_diff[i] = pd;
  if (out_spec) out_spec[i] = ps;
}

template <class Geo>
struct DnAtrousF {
  static __device__ __forceinline__ void run(int x0, int y0, int w, int h, Geo geo, AtrousTaps taps, const uint2* __restrict__ color, const uint32_t* __restrict__ var_tex, uint2* __restrict__ out_color, uint32_t* __restrict__ out_var, uint32_t* __restrict__ out_diff, uint32_t* __restrict__ out_spec, int step) {
  int x = x0 + (int)threadIdx.x, y = y0 + (int)threadIdx.y;
  if (!inb(x, y, w, h)) return;
  atrous_px(x, y, w, h, geo, taps, color, var_tex, out_color, out_var, out_diff, out_spec, step);
}
};

// The a-trous iteration over tiles staged in shared memory, for steps up to
// kAtrousTileMaxStep. The per-pixel form above decodes every tap anew: two R11G11B10
// words, two luminances, and from the raw G-buffer an octahedral normal, 16 times per
// pixel (235 warp instructions per tap, and a third of the stalls instruction fetch).
// Here a block decodes each pixel of its tile and halo once. The tile is 64
// consecutive columns of 8 rows that lie `step` apart, so that at every step the halo
// is four rows and 4 * step columns, loads stay coalesced and 1.6 (step 1) to 3 (step
// 16) pixels are decoded per output pixel.
//
// A staged pixel is 48 bytes, diffuse and specular channel interleaved (a stride of 12
// words: the eight lanes of each phase of a 128-bit load fall on distinct banks), plus
// the two variances. The interleaving gives both channels' arithmetic as register
// pairs, and the paired binary32 instructions (one IEEE operation per component, the
// same bits) halve the issue slots of the parts that run per channel.
//
// What the per-pixel form guards per tap is settled per block and pixel. The depths are
// `tame` when every one is 0 or of a magnitude in [2^-70, 2^70]; with a fwidth_z that is
// finite and not negative, the depth terms' quotients may be formed with a shared
// reciprocal (div_shared) and no weight exponent is positive. Blocks of other depths and
// pixels of other fwidth_z run the per-pixel form. The values are `ordinary` when every
// staged colour and variance is finite and no variance is negative. Then the per-pixel
// roots and quotients are the branch-free ones (three iterations at 1080p 379 -> 365 us
// against the IEEE operations); blocks with other values take those few operations as IEEE
// ones, and the rest of the arithmetic is the same for infinities and NaN: an overflowed
// variance, which the iterations spread over ever more blocks (0.9 % of them in the first,
// 31 % in the fifth in a walk at 1080p), does not take a block off the tile. An iteration
// at 1080p over one special variance per tile, steps 1 / 4 / 16: 337 / 201 / 195 us in the
// per-pixel form, 148 / 138 / 140 so; all variances infinite at step 16: 398 (328 in the
// per-pixel form alone) and 154; all depths extreme: 441 with 256 threads, 322 with 512 (355
// alone), so that no input is slower than without the tiles by more than the 5-8 % of step 8.
// The normal weight's seven squarings run for two taps of a row as a pair (reference-form
// frame at 1280x720 549 -> 544 us; in the float forms, which wait for loads, it gained
// nothing).
//
// Bound by binary32 arithmetic: 1,452 warp instructions per 32 pixels (3,770 in the
// per-pixel form) at 67 % issue, FMA pipe 66 % (the paired instructions take two of its
// cycles). 1920x1080 from the raw G-buffer: 337 -> 118 us per iteration; from the surface
// planes at 1280x720: 124 -> 60 us. Measured and not kept, when three iterations took 398
// us (356 now): a loop over the four tap rows instead of unrolled taps (416), 3 or 2 blocks
// per SM (423, 534), 16 rows by 512 threads (416), 4 rows by 128 (446), staging unrolled by
// two (408). Above kAtrousTileMaxStep the halo outgrows the tile and the per-pixel form
// runs; recorded (batched) jobs, whose tile shape the batch chooses, run it too.
constexpr int kAtrousTileMaxStep = 16;
constexpr int kAtrousTileX = 64, kAtrousTileRows = 8;
constexpr size_t kSharedPerSM = 228 * 1024, kSharedPerBlock = 1024;  // the latter reserved by the system

struct AtrousPx {
  float4 a;  // diffuse.r, specular.r, diffuse.g, specular.g
  float4 b;  // diffuse.b, specular.b, diffuse and specular luminance
  float4 c;  // normal, depth
};

__device__ __forceinline__ float2 bc2(float v) { return make_float2(v, v); }
// a * b + c per component with the product rounded before the sum. The compiler fuses a
// paired multiply and a paired add (also the explicitly rounded intrinsics, and a
// fused multiply-add by a literal 1) into one fused multiply-add, which rounds once.
// A factor of 1 that only the host knows, a kernel argument, keeps the two apart.
__device__ __forceinline__ float2 madd2(float2 a, float2 b, float2 c, float one) {
  return __ffma2_rn(__fmul2_rn(a, b), bc2(one), c);
}

struct AtrousOut {
  uint2* __restrict__ color;
  uint32_t* __restrict__ var;
  uint32_t* __restrict__ diff;
  uint32_t* __restrict__ spec;
};

// max(a, b), NaN where a is.
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// One output pixel of a block of tame depths and ordinary fwidth_z; s is the staged tile, li the pixel's place
// in it, pw the tile's row pitch. CHECK: the footprint may leave the image.
template <bool CHECK, bool ORDINARY>
__device__ __forceinline__ void atrous_tile_px(const AtrousPx* s, const float2* sv, int li, int pw, int x, int y,
                                               int w, int h, float fwz, float3 td, int step, const AtrousOut& o, float one) {
  const float4 ca = s[li].a, cb = s[li].b, cc = s[li].c;
  const float2 cv = sv[li];
  const float eps = 1e-8f;
  const float2 neg_lum = make_float2(-cb.z, -cb.w);
  // Ordinary operands are in the branch-free forms' ranges: a variance is 0 or a half of at
  // least 2^-24, the denominators lie in [1e-8, 1e8], the weight sum in [1, 17].
  float2 rcp_l;
  if (ORDINARY) {
    const float2 sd = make_float2(cv.x > 0.0f ? sqrt_ranged(cv.x) : 0.0f, cv.y > 0.0f ? sqrt_ranged(cv.y) : 0.0f);
    rcp_l = make_float2(rcp_ranged(4.0f * sd.x + eps), rcp_ranged(4.0f * sd.y + eps));
  } else {
    rcp_l = make_float2(1.0f / (4.0f * sqrt_(cv.x) + eps), 1.0f / (4.0f * sqrt_(cv.y) + eps));
  }
  const float den[3] = {fwz * td.x + eps, fwz * td.y + eps, fwz * td.z + eps};
  const float rden[3] = {rcp_ranged(den[0]), rcp_ranged(den[1]), rcp_ranged(den[2])};
  float2 r = make_float2(ca.x, ca.y), g = make_float2(ca.z, ca.w), b = make_float2(cb.x, cb.y), v = cv,
         ws = bc2(1.0f);
  const float kw[3] = {1.0f, 2.0f / 3.0f, 1.0f / 6.0f};
  const float M = 12582912.0f;  // 1.5 * 2^23: the shifter of exp2_select
#pragma unroll
  for (int oy = -2; oy <= 2; ++oy) {
    if (oy == 0) continue;
    if (CHECK && !inb(0, y + oy * step, 1, h)) continue;
#pragma unroll
    for (int side = -1; side <= 1; side += 2) {
      const int j1 = li + oy * pw + side * step, j2 = j1 + side * step;
      const bool in1 = !CHECK || inb(x + side * step, 0, w, 1), in2 = !CHECK || inb(x + 2 * side * step, 0, w, 1);
      const auto cosine = [&](int j) {
        const float4 tc = s[j].c;
        const float2 nxy = __fmul2_rn(make_float2(cc.x, cc.y), make_float2(tc.x, tc.y));
        return __saturatef(nxy.x + nxy.y + cc.z * tc.z);
      };
      const auto tap = [&](int j, int ax, float wn) {
        const int ay = oy < 0 ? -oy : oy, cls = ax + ay - 2;
        const float4 ta = s[j].a, tb = s[j].b, tc = s[j].c;
        const float2 tv = sv[j];
        const float q = div_shared(fabsf(tc.w - cc.w), den[cls], rden[cls]);
        // exponent -(|dl| rcp_l + q): every term is non-negative or NaN, q finite
        const float2 dl = __fmul2_rn(__fadd2_rn(make_float2(tb.z, tb.w), neg_lum), rcp_l);
        float2 e = __ffma2_rn(make_float2(fabsf(dl.x), fabsf(dl.y)), bc2(one), bc2(q));
        e = __fmul2_rn(e, bc2(-VLT_LOG2E));
        // exp2_select<false> for arguments <= 0 or NaN: below -151 the clamp itself gives 0
        e = ORDINARY ? make_float2(fmax_(e.x, -151.0f), fmax_(e.y, -151.0f))
                     : make_float2(max_nan(e.x, -151.0f), max_nan(e.y, -151.0f));
        const float2 t = __fadd2_rn(e, bc2(M));
        const float2 f = __fadd2_rn(e, __ffma2_rn(t, bc2(-1.0f), bc2(M)));
        float2 p = madd2(bc2(VLT_EXP2_C6), f, bc2(VLT_EXP2_C5), one);
        p = madd2(p, f, bc2(VLT_EXP2_C4), one);
        p = madd2(p, f, bc2(VLT_EXP2_C3), one);
        p = madd2(p, f, bc2(VLT_EXP2_C2), one);
        p = madd2(p, f, bc2(VLT_EXP2_C1), one);
        p = madd2(p, f, bc2(VLT_EXP2_C0), one);
        // 2^n as 2^max(n, -126) 2^min(n + 126, 0): the integers sit in the shifted sums' low bits.
        // (With the second exponent as n - max(n, -126) the compiled kernel takes it as 0.)
        const int tx = (int)as_uint(t.x), ty = (int)as_uint(t.y);
        const int lo = 0x4B400000 - 126;
        const uint32_t one2 = 0x3F800000u - ((uint32_t)lo << 23);
        const float2 s1 = make_float2(as_float(((uint32_t)max(tx, lo) << 23) + 0x3F800000u),
                                      as_float(((uint32_t)max(ty, lo) << 23) + 0x3F800000u));
        const float2 s2 = make_float2(as_float(((uint32_t)min(tx, lo) << 23) + one2),
                                      as_float(((uint32_t)min(ty, lo) << 23) + one2));
        p = __fmul2_rn(__fmul2_rn(p, s1), s2);
        const float2 wt = __fmul2_rn(bc2(kw[ay] * kw[ax]), __fmul2_rn(bc2(wn), p));
        r = madd2(wt, make_float2(ta.x, ta.y), r, one);
        g = madd2(wt, make_float2(ta.z, ta.w), g, one);
        b = madd2(wt, make_float2(tb.x, tb.y), b, one);
        v = madd2(__fmul2_rn(wt, wt), tv, v, one);
        ws = __ffma2_rn(wt, bc2(one), ws);
      };
      // The two taps' powers as a pair; the sums take the taps from left to right.
      float2 nn = make_float2(in1 ? cosine(j1) : 0.0f, in2 ? cosine(j2) : 0.0f);
#pragma unroll
      for (int k = 0; k < 7; ++k) nn = __fmul2_rn(nn, nn);
      if (side < 0) {
        if (in2) tap(j2, 2, nn.y);
        if (in1) tap(j1, 1, nn.x);
      } else {
        if (in1) tap(j1, 1, nn.x);
        if (in2) tap(j2, 2, nn.y);
      }
    }
  }
  const float2 w2 = __fmul2_rn(ws, ws);
  f3 d, sp;
  f2 vd;
  if (ORDINARY) {
    // 1 <= ws <= 17; a sum too small for div_shared is stored as 0 either way, and a variance
    // of -0 beside no tap keeps its sign
    const float2 rw = make_float2(rcp_ranged(ws.x), rcp_ranged(ws.y));
    d = mk3(div_shared(r.x, ws.x, rw.x), div_shared(g.x, ws.x, rw.x), div_shared(b.x, ws.x, rw.x));
    sp = mk3(div_shared(r.y, ws.y, rw.y), div_shared(g.y, ws.y, rw.y), div_shared(b.y, ws.y, rw.y));
    vd = mk2(v.x > 0.0f ? div_ranged(v.x, w2.x) : v.x, v.y > 0.0f ? div_ranged(v.y, w2.y) : v.y);
  } else {
    d = mk3(r.x, g.x, b.x) / ws.x;
    sp = mk3(r.y, g.y, b.y) / ws.y;
    vd = mk2(v.x / w2.x, v.y / w2.y);
  }
  const uint32_t pd = pack_r11g11b10(d), ps = pack_r11g11b10(sp);
  const size_t i = (size_t)y * w + x;
  if (o.color) o.color[i] = make_uint2(pd, ps);
  if (o.var) o.var[i] = pack_half2(vd);
  if (o.diff) o.diff[i] = pd;
  if (o.spec) o.spec[i] = ps;
}

// Bytes of a block's staged tile at a step.
static inline size_t atrous_tile_bytes(int step) {
  return (size_t)(kAtrousTileX + 4 * step) * (kAtrousTileRows + 4) * (sizeof(AtrousPx) + sizeof(float2));
}

template <class Geo, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT)  // 64 registers
    k_atrous_tile(int w, int h, Geo geo, AtrousTaps taps, const uint2* __restrict__ color,
                  const uint32_t* __restrict__ var_tex, AtrousOut o, int step, uint32_t pitch_inv, float one) {
  extern __shared__ float4 smem[];
  const int pw = kAtrousTileX + 4 * step, np = pw * (kAtrousTileRows + 4);
  AtrousPx* s = reinterpret_cast<AtrousPx*>(smem);
  float2* sv = reinterpret_cast<float2*>(s + np);
  const int tid = (int)threadIdx.x;
  // Tile rows: blockIdx.y counts (group of 8 * step image rows, phase within it).
  const int group = (int)blockIdx.y / step, phase = (int)blockIdx.y - group * step;
  const int x0 = (int)blockIdx.x * kAtrousTileX, y0 = group * (kAtrousTileRows * step) + phase;
  uint32_t odd = 0u;  // 1: a value, 2: a depth
  const auto tame_depth = [](float d) { return d == 0.0f || (fabsf(d) >= 0x1p-70f && fabsf(d) <= 0x1p70f); };
  for (int k = tid; k < np; k += NT) {
    const int row = (int)__umulhi((uint32_t)k, pitch_inv), col = k - row * pw;  // k / pw (host: exact for k < np)
    const int gx = x0 + col - 2 * step, gy = y0 + (row - 2) * step;
    if (!inb(gx, gy, w, h)) continue;  // never read: the border form checks every tap
    const size_t i = (size_t)gy * w + gx;
    const uint2 cw = color[i];
    const uint32_t vw = var_tex[i];
    const f3 n = geo.normal(i);
    const float dep = geo.dep(i);
    const f3 d = col_diff(cw), sp = col_spec(cw);
    AtrousPx px;
    px.a = make_float4(d.x, sp.x, d.y, sp.y);
    px.b = make_float4(d.z, sp.z, luminance(d), luminance(sp));
    px.c = make_float4(n.x, n.y, n.z, dep);
    s[k] = px;
    const f2 v = unpack_half2(vw);
    sv[k] = make_float2(v.x, v.y);
    // a luminance is finite where its channels are
    if (!(px.b.z < 1e6f && px.b.w < 1e6f && v.x >= 0.0f && v.y >= 0.0f && v.x < 1e6f && v.y < 1e6f)) odd |= 1u;
    if (!tame_depth(dep)) odd |= 2u;
  }
  const bool ordinary = __syncthreads_and(odd == 0u);
  const bool tame = ordinary || __syncthreads_and(odd < 2u);
  const float3 td = make_float3(taps.dist[5], taps.dist[4], taps.dist[0]);
  const bool interior = x0 - 2 * step >= 0 && x0 + kAtrousTileX - 1 + 2 * step <= w - 1 && y0 - 2 * step >= 0 &&
                        y0 + (kAtrousTileRows + 1) * step <= h - 1;
  const int tx = tid & (kAtrousTileX - 1), ty = tid / kAtrousTileX;
#pragma unroll 1
  for (int row = ty; row < kAtrousTileRows; row += NT / kAtrousTileX) {
    const int x = x0 + tx, y = y0 + row * step;
    if (!inb(x, y, w, h)) return;
    const float fwz = geo.fwz((size_t)y * w + x);
    if (!(tame && fwz >= 0.0f && fwz < 1e6f)) {
      atrous_px(x, y, w, h, geo, taps, color, var_tex, o.color, o.var, o.diff, o.spec, step);
      continue;
    }
    const int li = (row + 2) * pw + tx + 2 * step;
    if (!ordinary) atrous_tile_px<true, false>(s, sv, li, pw, x, y, w, h, fwz, td, step, o, one);
    else if (interior) atrous_tile_px<false, true>(s, sv, li, pw, x, y, w, h, fwz, td, step, o, one);
    else atrous_tile_px<true, true>(s, sv, li, pw, x, y, w, h, fwz, td, step, o, one);
  }
}

struct SplitColorF {
  static __device__ __forceinline__ void run(int x0, int y0, int n, const uint2* __restrict__ color, uint32_t* __restrict__ d, uint32_t* __restrict__ s) {
  int i = x0 + (int)threadIdx.x;
  if (i >= n) return;
  uint2 c = color[i];
  if (d) d[i] = c.x;
  if (s) s[i] = c.y;
}
};

// ------------------------------------------------------------- launchers

static GeoRaw raw_geo(const GeoArgs& a, int w, int h) {
  GeoRaw g = make_geo_raw(a.depth, a.gbuf, a.inv_vp, w, h);
  return g;
}
static GeoSurface surf_geo(const GeoArgs& a, int w, int h) {
  GeoSurface g = {a.nd, a.pr, a.fz, w, h};
  return g;
}

void launch_dn_temporal(const Exec& ex, const vlt_frame_params& fp, int w, int h, const DenoiseKnobs& kn,
                        const GeoArgs& ga, const GeoArgs& prev_ga, const uint32_t* diff_src, const uint32_t* spec_src,
                        const uint16_t* ray_len, const float* prev_depth, const uint32_t* color_hist,
                        const uint32_t* mom_hist, const uint8_t* len_hist, const uint32_t* fast_hist,
                        uint32_t* out_color, uint32_t* out_mom, uint8_t* out_len, uint32_t* out_fast,
                        uint32_t has_history) {
#define VLT_DN_TEMPORAL(GEO, G, PG, FASTV)                                                                 \
  launch2d<DnTemporalF<GEO, FASTV>>(ex, "dn_temporal", w, h, fp, w, h, kn, G, PG, ga.gbuf, diff_src, spec_src,     \
                                    ray_len, prev_depth, (const uint2*)color_hist, mom_hist, len_hist,             \
                                    (const uint2*)fast_hist, (uint2*)out_color, out_mom, out_len, (uint2*)out_fast, \
                                    has_history)
  if (ga.nd) {
    if (kn.fast_history) VLT_DN_TEMPORAL(GeoSurface, surf_geo(ga, w, h), surf_geo(prev_ga, w, h), true);
    else VLT_DN_TEMPORAL(GeoSurface, surf_geo(ga, w, h), surf_geo(prev_ga, w, h), false);
  } else {
    if (kn.fast_history) VLT_DN_TEMPORAL(GeoRaw, raw_geo(ga, w, h), raw_geo(prev_ga, w, h), true);
    else VLT_DN_TEMPORAL(GeoRaw, raw_geo(ga, w, h), raw_geo(prev_ga, w, h), false);
  }
#undef VLT_DN_TEMPORAL
}

void launch_dn_fix(const Exec& ex, int w, int h, const GeoArgs& ga, const uint8_t* len, const uint32_t* color,
                   const uint32_t* mom, uint32_t* out_color, uint32_t* out_mom) {
  if (ga.nd)
    launch2d<DnFixF<GeoSurface>>(ex, "dn_fix", w, h, w, h, surf_geo(ga, w, h), len, (const uint2*)color, mom,
                                 (uint2*)out_color, out_mom);
  else
    launch2d<DnFixF<GeoRaw>>(ex, "dn_fix", w, h, w, h, raw_geo(ga, w, h), len, (const uint2*)color, mom,
                             (uint2*)out_color, out_mom);
}

void launch_dn_fast_clamp(const Exec& ex, int w, int h, const uint32_t* fast, uint32_t* color) {
  launch2d<DnFastClampF>(ex, "dn_fast_clamp", w, h, w, h, (const uint2*)fast, (uint2*)color);
}

void launch_dn_fallback(const Exec& ex, int w, int h, const GeoArgs& ga, const uint8_t* len, const uint32_t* color,
                        const uint32_t* mom, uint32_t* out_color, uint32_t* out_var) {
  if (ga.nd)
    launch2d<DnFallbackF<GeoSurface>>(ex, "dn_fallback", w, h, w, h, surf_geo(ga, w, h), len, (const uint2*)color,
                                      mom, (uint2*)out_color, out_var);
  else
    launch2d<DnFallbackF<GeoRaw>>(ex, "dn_fallback", w, h, w, h, raw_geo(ga, w, h), len, (const uint2*)color, mom,
                                  (uint2*)out_color, out_var);
}

template <class Geo>
static void launch_atrous_tile(const Exec& ex, int w, int h, const Geo& geo, const AtrousTaps& taps,
                               const uint32_t* color, const uint32_t* var, uint32_t* out_color, uint32_t* out_var,
                               uint32_t* out_diff, uint32_t* out_spec, int step) {
  if (w <= 0 || h <= 0) return;
  if (ex.launches) ++*ex.launches;
  const int pw = kAtrousTileX + 4 * step;
  const unsigned groups = (unsigned)((h + kAtrousTileRows * step - 1) / (kAtrousTileRows * step));
  const dim3 grid((unsigned)((w + kAtrousTileX - 1) / kAtrousTileX), groups * (unsigned)step, 1);
  // floor(2^32 / pw) + 1: the high word of k * pitch_inv is k / pw for k below 2^16
  const uint32_t pitch_inv = (uint32_t)(((uint64_t)1 << 32) / (uint32_t)pw + 1u);
  const AtrousOut o = {(uint2*)out_color, out_var, out_diff, out_spec};
  const size_t bytes = atrous_tile_bytes(step);
  auto run = [&](auto kernel, int threads) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)atrous_tile_bytes(kAtrousTileMaxStep));
    kernel<<<grid, threads, bytes, ex.stream>>>(w, h, geo, taps, (const uint2*)color, var, o, step, pitch_inv, 1.0f);
  };
  // One output row per thread while there are few tiles per SM (a block's own latency is
  // then the pass), two rows on fewer threads for more. Five iterations, 256 / 512
  // threads: 320x180 61 / 50 us, 640x360 111 / 102 us, 854x480 163 / 156 us, 1280x720 299 /
  // 304 us; three at 1920x1080 355 / 385 us.
  // One row per thread also where shared memory leaves room for two blocks per SM only
  // (steps above 12): 256 threads are then 16 warps, and step 16 at 1920x1080 takes 152 us
  // instead of 135 (at step 8, where three blocks fit, 125 instead of 129).
  if ((int)(grid.x * grid.y) <= 8 * device_sm_count() || 3 * (bytes + kSharedPerBlock) > kSharedPerSM)
    run(k_atrous_tile<Geo, 512>, 512);
  else run(k_atrous_tile<Geo, 256>, 256);
}

void launch_dn_atrous(const Exec& ex, int w, int h, const GeoArgs& ga, const uint32_t* color, const uint32_t* var,
                      uint32_t* out_color, uint32_t* out_var, uint32_t* out_diff, uint32_t* out_spec, int step) {
  AtrousTaps taps;
  int k = 0;
  for (int oy = -2; oy <= 2; ++oy) {
    if (oy == 0) continue;
    for (int ox = -2; ox <= 2; ++ox) {
      if (ox == 0) continue;
      float fx = (float)(ox * step), fy = (float)(oy * step);
      taps.dist[k++] = sqrtf(fx * fx + fy * fy);  // correctly rounded, == device sqrt.rn
    }
  }
  if (!ex.rec && step <= kAtrousTileMaxStep) {
    if (ga.nd)
      launch_atrous_tile(ex, w, h, surf_geo(ga, w, h), taps, color, var, out_color, out_var, out_diff, out_spec, step);
    else
      launch_atrous_tile(ex, w, h, raw_geo(ga, w, h), taps, color, var, out_color, out_var, out_diff, out_spec, step);
    return;
  }
  if (ga.nd)
    launch2d<DnAtrousF<GeoSurface>>(ex, "dn_atrous", w, h, w, h, surf_geo(ga, w, h), taps, (const uint2*)color, var,
                                    (uint2*)out_color, out_var, out_diff, out_spec, step);
  else
    launch2d<DnAtrousF<GeoRaw>>(ex, "dn_atrous", w, h, w, h, raw_geo(ga, w, h), taps, (const uint2*)color, var,
                                (uint2*)out_color, out_var, out_diff, out_spec, step);
}

void launch_split_color(const Exec& ex, int w, int h, const uint32_t* color, uint32_t* diff, uint32_t* spec) {
  int n = w * h;
  launch1d<SplitColorF>(ex, "split_color", (uint32_t)n, n, (const uint2*)color, diff, spec);
}

}  // namespace vlt
