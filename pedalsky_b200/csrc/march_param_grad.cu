// Gradient of the procedural march's image loss with respect to one cloud
// layer's parameters: coverage, shape_bias, detail_bias, density_scale,
// base_m and top_m.
//
// The first four enter the march only through sample_density
// (cloud_march.wgsl:432-530; march_plain.cuh:density_at): the coverage gate
// and remap (eff = clamp(weather.r * coverage, 0, 1)), the low-frequency
// erosion (lf = clamp(fbm + shape_bias * diurnal / 2, 0, 1)), the detail
// erosion (clamp(detail_strength + detail_bias * diurnal, 0, 1)) and the
// final scale.  The layer's base and top enter geometrically: the ray's
// entry and exit distances are its intersections with the spheres at planet
// radius + base and + top, the primary samples are spread over that
// interval, the normalised height h = (alt - base) / (top - base) drives the
// profile, the height-scaled skew (skew_thickness = (top - base) * skew
// strength) and the detail polarity, the wind offset is the wind field at the
// layer's mid-altitude, the light path runs to the top, and the ambient
// gradient uses h.  Every quantity of the per-ray march is carried here as a
// value with its six derivatives (forward mode), one thread per ray, in the
// PLAIN march's FP32 arithmetic and order with exact (FP32-weight)
// filtering: sample positions and altitudes, the weather, base, curl and
// detail taps (their filter weights' derivatives with respect to the
// position), the density, the light march's optical depth, Beer-powder and
// the multi-scatter octaves, the sun transmittance and sky-view lookups, the
// in-scattered step integral, the transmittance, the luminance-weighted
// cloud distance and the aerial-perspective blend it selects.  The branch
// decisions (the 1e-3 density threshold, the 0.01 coverage gate, the early
// exits, the layer hits and their order) are taken on the values and are
// constant under the derivative, as for any tangent of the march.  With the
// Kahan option the carried layer's values and the transmittance are summed
// plainly.
//
// Only the derivatives a quantity has are carried (DV's mask): positions,
// heights, taps and LUT lookups move with base and top only, a light tap's
// density has no detail slot, and a layer other than the carried one is
// marched in plain values that meet the six derivatives where they multiply
// the transmittance.  480x270, three layers, 128 + 6 steps: 8.44 -> 3.05 ms
// (2506 M to 1308 M warp instructions, 243 to 168 registers).  What bounds it
// is the size of the loop body: 1.5 of 5 stalled warps per issue wait for
// instructions (three channels unrolled: 3.26 ms; four CTAs per SM at 128
// registers: 3.46 ms; 64-thread CTAs: 3.20 ms).
//
// The loss is the adjoint's: sum((I - target)^2) / (3 * viewport pixels),
// I = L + background * T per pixel and channel, over the view's rectangle;
// each ray adds its 2 (I - target) / N . dI to the six results.
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "march_common.cuh"
#include "march_plain.cuh"
#include "march_ray.cuh"
#include "psc_internal.h"

namespace psc {
namespace {

constexpr int kTileW = 16;
constexpr int kTileH = 8;
constexpr int kThreads = 128;
// derivative slots: coverage, shape_bias, detail_bias, density_scale, base_m, top_m
constexpr int kP = 6;
constexpr int kBase = 4, kTop = 5;

// A value and its derivatives in the slots of M (bit i: slot i); the others
// are 0 and neither stored nor computed, so what moves with the layer's range
// only (every position) carries two derivatives and a constant none.
constexpr unsigned kCov = 1u, kShape = 2u, kDetail = 4u, kScale = 8u, kRange = 48u, kAll = 63u;

template <unsigned M>
struct DV {
  float v;
  float d[kP];
};
// f(Slot<i>{}) for each slot i of M
template <int I>
struct Slot {
  static constexpr int n = I;
};
template <unsigned M, class F>
__device__ __forceinline__ void each(F f) {
  if constexpr (M & 1u) f(Slot<0>{});
  if constexpr (M & 2u) f(Slot<1>{});
  if constexpr (M & 4u) f(Slot<2>{});
  if constexpr (M & 8u) f(Slot<3>{});
  if constexpr (M & 16u) f(Slot<4>{});
  if constexpr (M & 32u) f(Slot<5>{});
}
// a value whose derivatives are 0
template <unsigned M>
__device__ __forceinline__ DV<M> flat(float v) {
  DV<M> r;
  r.v = v;
  each<M>([&](auto i) {
    constexpr int j = decltype(i)::n;
    r.d[j] = 0.0f;
  });
  return r;
}
__device__ __forceinline__ DV<0> dc(float v) { return flat<0>(v); }
// the same value with room for more slots
template <unsigned N, unsigned M>
__device__ __forceinline__ DV<N> widen(const DV<M>& x) {
  static_assert((M & ~N) == 0u, "widen keeps every slot");
  DV<N> r = flat<N>(x.v);
  each<M>([&](auto i) {
    constexpr int j = decltype(i)::n;
    r.d[j] = x.d[j];
  });
  return r;
}
// a value with slope k along another value's derivatives
template <unsigned M>
__device__ __forceinline__ DV<M> along(float v, float k, const DV<M>& x) {
  DV<M> r;
  r.v = v;
  each<M>([&](auto i) {
    constexpr int j = decltype(i)::n;
    r.d[j] = k * x.d[j];
  });
  return r;
}
template <unsigned A, unsigned B>
__device__ __forceinline__ DV<A | B> operator+(const DV<A>& x, const DV<B>& y) {
  DV<A | B> r;
  r.v = x.v + y.v;
  each<A | B>([&](auto i) {
    constexpr int j = decltype(i)::n;
    if constexpr (((A & B) >> j) & 1u) r.d[j] = x.d[j] + y.d[j];
    else if constexpr ((A >> j) & 1u) r.d[j] = x.d[j];
    else r.d[j] = y.d[j];
  });
  return r;
}
template <unsigned A, unsigned B>
__device__ __forceinline__ DV<A | B> operator-(const DV<A>& x, const DV<B>& y) {
  DV<A | B> r;
  r.v = x.v - y.v;
  each<A | B>([&](auto i) {
    constexpr int j = decltype(i)::n;
    if constexpr (((A & B) >> j) & 1u) r.d[j] = x.d[j] - y.d[j];
    else if constexpr ((A >> j) & 1u) r.d[j] = x.d[j];
    else r.d[j] = -y.d[j];
  });
  return r;
}
template <unsigned M>
__device__ __forceinline__ DV<M> operator+(const DV<M>& x, float s) {
  DV<M> r = x;
  r.v = x.v + s;
  return r;
}
template <unsigned M>
__device__ __forceinline__ DV<M> operator+(float s, const DV<M>& x) { return x + s; }
template <unsigned M>
__device__ __forceinline__ DV<M> operator-(const DV<M>& x, float s) {
  DV<M> r = x;
  r.v = x.v - s;
  return r;
}
template <unsigned M>
__device__ __forceinline__ DV<M> operator-(float s, const DV<M>& x) { return along(s - x.v, -1.0f, x); }
template <unsigned M>
__device__ __forceinline__ DV<M> operator-(const DV<M>& x) { return 0.0f - x; }
template <unsigned M>
__device__ __forceinline__ DV<M> operator*(const DV<M>& x, float s) { return along(x.v * s, s, x); }
template <unsigned M>
__device__ __forceinline__ DV<M> operator*(float s, const DV<M>& x) { return along(s * x.v, s, x); }
template <unsigned A, unsigned B>
__device__ __forceinline__ DV<A | B> operator*(const DV<A>& x, const DV<B>& y) {
  DV<A | B> r;
  r.v = x.v * y.v;
  each<A | B>([&](auto i) {
    constexpr int j = decltype(i)::n;
    if constexpr (((A & B) >> j) & 1u) r.d[j] = fmaf(x.d[j], y.v, x.v * y.d[j]);
    else if constexpr ((A >> j) & 1u) r.d[j] = x.d[j] * y.v;
    else r.d[j] = x.v * y.d[j];
  });
  return r;
}
template <unsigned A, unsigned B>
__device__ __forceinline__ DV<A | B> operator/(const DV<A>& x, const DV<B>& y) {
  const float iy = rcp_near(y.v), q = div_by(x.v, y.v, iy);  // no divisor here is 0 or subnormal
  DV<A | B> r;
  r.v = q;
  each<A | B>([&](auto i) {
    constexpr int j = decltype(i)::n;
    if constexpr (((A & B) >> j) & 1u) r.d[j] = (x.d[j] - q * y.d[j]) * iy;
    else if constexpr ((A >> j) & 1u) r.d[j] = x.d[j] * iy;
    else r.d[j] = -(q * y.d[j]) * iy;
  });
  return r;
}
template <unsigned M>
__device__ __forceinline__ DV<M> over(const DV<M>& x, float s, float inv) {  // x / s, inv = 1 / s
  return along(div_by(x.v, s, inv), inv, x);
}
template <unsigned M>
__device__ __forceinline__ DV<M> operator/(const DV<M>& x, float s) { return over(x, s, 1.0f / s); }
template <unsigned M>
__device__ __forceinline__ DV<M> dexp(const DV<M>& x) {
  const float e = expf(x.v);
  return along(e, e, x);
}
template <unsigned M>
__device__ __forceinline__ DV<M> dlog(const DV<M>& x) { return along(logf(x.v), 1.0f / x.v, x); }
template <unsigned M>
__device__ __forceinline__ DV<M> dsqrt(const DV<M>& x) {
  const float r = sqrt_near(fmaxf(x.v, 0.0f));
  return along(r, r > 1e-19f ? 0.5f * rcp_near(r) : 0.0f, x);
}
template <unsigned M>
__device__ __forceinline__ DV<M> dmax(const DV<M>& x, float m) { return x.v > m ? x : flat<M>(fmaxf(x.v, m)); }
template <unsigned M>
__device__ __forceinline__ DV<M> dmin(const DV<M>& x, float m) { return x.v < m ? x : flat<M>(fminf(x.v, m)); }
template <unsigned M>
__device__ __forceinline__ DV<M> dclamp(const DV<M>& x, float lo, float hi) {
  return (x.v > lo && x.v < hi) ? x : flat<M>(clampf(x.v, lo, hi));
}
template <unsigned M>
__device__ __forceinline__ DV<M> dclamp01(const DV<M>& x) { return dclamp(x, 0.0f, 1.0f); }
// mixf(a, b, t) = a (1 - t) + b t
template <unsigned A, unsigned B>
__device__ __forceinline__ DV<A | B> dmix(const DV<A>& a, const DV<B>& b, float t) { return a * (1.0f - t) + b * t; }
template <unsigned A, unsigned B, unsigned T>
__device__ __forceinline__ DV<A | B | T> dmix(const DV<A>& a, const DV<B>& b, const DV<T>& t) {
  return a * (1.0f - t) + b * t;
}
template <unsigned T>
__device__ __forceinline__ DV<T> dmix(float a, float b, const DV<T>& t) { return along(mixf(a, b, t.v), b - a, t); }
// remapf(v, a, 1, 0, 1) = 0 + ((v - a) * 1) / max(1 - a, 1e-5)
template <unsigned V, unsigned A>
__device__ __forceinline__ DV<V | A> dremap01(const DV<V>& v, const DV<A>& a) {
  return (v - a) * 1.0f / dmax(1.0f - a, 1e-5f);
}
// smoothstepf(e0, e1, x), reversed ramps included
template <unsigned M>
__device__ __forceinline__ DV<M> dsmooth(float e0, float e1, const DV<M>& x) {
  const float inv = 1.0f / (e1 - e0);
  const float t = clamp01(div_by(x.v - e0, e1 - e0, inv));
  const float k = (t > 0.0f && t < 1.0f) ? div_by(6.0f * t * (1.0f - t), e1 - e0, inv) : 0.0f;
  return along(t * t * (3.0f - 2.0f * t), k, x);
}
// atan2(y, x): d = (x dy - y dx) / (x^2 + y^2)
template <unsigned M>
__device__ __forceinline__ DV<M> datan2(const DV<M>& y, const DV<M>& x) {
  const float n = fmaf(x.v, x.v, y.v * y.v), k = n > 0.0f ? 1.0f / n : 0.0f;
  DV<M> r;
  r.v = atan2f(y.v, x.v);
  each<M>([&](auto i) {
    constexpr int j = decltype(i)::n;
    r.d[j] = (x.v * y.d[j] - y.v * x.d[j]) * k;
  });
  return r;
}
template <unsigned M>
__device__ __forceinline__ DV<M> dasin(const DV<M>& x) {
  const float q = fmaf(-x.v, x.v, 1.0f);
  return along(asinf(x.v), q > 0.0f ? rsqrtf(q) : 0.0f, x);
}
// Everything that moves with the layer's base and top only.
using DR = DV<kRange>;
struct DR3 {
  DR x, y, z;
};
struct DR4 {
  DR x, y, z, w;
};
// value v + gradient g along coordinates (a, b, c): v + g . d(a, b, c)
__device__ __forceinline__ DR chain3(float v, float ga, float gb, float gc, const DR& a, const DR& b, const DR& c) {
  DR r;
  r.v = v;
  each<kRange>([&](auto i) {
    constexpr int j = decltype(i)::n;
    r.d[j] = fmaf(ga, a.d[j], fmaf(gb, b.d[j], gc * c.d[j]));
  });
  return r;
}
__device__ __forceinline__ DR chain2(float v, float ga, float gb, const DR& a, const DR& b) {
  DR r;
  r.v = v;
  each<kRange>([&](auto i) {
    constexpr int j = decltype(i)::n;
    r.d[j] = fmaf(ga, a.d[j], gb * b.d[j]);
  });
  return r;
}

// ------------------------------------------------ filters with gradients
// trilinear_repeat (march_common.cuh) and its gradient with respect to the
// normalised coordinates (texel weights w = u N - 0.5 - floor: dw/du = N).
template <int ST, int N>
__device__ __forceinline__ DR4 trilinear_d(const void* vol, const DR& u, const DR& v, const DR& w, float vscale) {
  const float x = u.v * (float)N - 0.5f, y = v.v * (float)N - 0.5f, z = w.v * (float)N - 0.5f;
  const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
  const int ix = (int)fx, iy = (int)fy, iz = (int)fz;
  const float wx = x - fx, wy = y - fy, wz = z - fz;
  const uint32_t x0 = (uint32_t)ix & (N - 1), x1 = (uint32_t)(ix + 1) & (N - 1);
  const uint32_t y0 = (uint32_t)iy & (N - 1), y1 = (uint32_t)(iy + 1) & (N - 1);
  const uint32_t z0 = (uint32_t)iz & (N - 1), z1 = (uint32_t)(iz + 1) & (N - 1);
  const uint32_t r00 = (z0 * N + y0) * N, r10 = (z0 * N + y1) * N;
  const uint32_t r01 = (z1 * N + y0) * N, r11 = (z1 * N + y1) * N;
  const float4 c[8] = {load_texel<ST>(vol, r00 + x0), load_texel<ST>(vol, r00 + x1),
                       load_texel<ST>(vol, r10 + x0), load_texel<ST>(vol, r10 + x1),
                       load_texel<ST>(vol, r01 + x0), load_texel<ST>(vol, r01 + x1),
                       load_texel<ST>(vol, r11 + x0), load_texel<ST>(vol, r11 + x1)};
  const float s = storage_scale<ST>(vscale);
  float val[4], gx[4], gy[4], gz[4];
#pragma unroll
  for (int ch = 0; ch < 4; ++ch) {
    auto C = [&](int k) {
      const float4 t = c[k];
      return ch == 0 ? t.x : (ch == 1 ? t.y : (ch == 2 ? t.z : t.w));
    };
    // the value exactly as trilinear_repeat forms it
    const float a = lerpf(lerpf(C(0), C(1), wx), lerpf(C(2), C(3), wx), wy);
    const float b = lerpf(lerpf(C(4), C(5), wx), lerpf(C(6), C(7), wx), wy);
    val[ch] = lerpf(a, b, wz) * s;
    const float dx0 = lerpf(C(1) - C(0), C(3) - C(2), wy), dx1 = lerpf(C(5) - C(4), C(7) - C(6), wy);
    gx[ch] = lerpf(dx0, dx1, wz) * s * (float)N;
    const float dy0 = lerpf(C(2), C(3), wx) - lerpf(C(0), C(1), wx);
    const float dy1 = lerpf(C(6), C(7), wx) - lerpf(C(4), C(5), wx);
    gy[ch] = lerpf(dy0, dy1, wz) * s * (float)N;
    gz[ch] = (b - a) * s * (float)N;
  }
  return {chain3(val[0], gx[0], gy[0], gz[0], u, v, w), chain3(val[1], gx[1], gy[1], gz[1], u, v, w),
          chain3(val[2], gx[2], gy[2], gz[2], u, v, w), chain3(val[3], gx[3], gy[3], gz[3], u, v, w)};
}

// curl_sample (128^2 RG8, repeat, bilinear) with its gradient
__device__ __forceinline__ void curl_d(const uint8_t* curl, const DR& u, const DR& v, DR& r, DR& g) {
  const float x = u.v * 128.0f - 0.5f, y = v.v * 128.0f - 0.5f;
  const float fx = floorf(x), fy = floorf(y);
  const int ix = (int)fx, iy = (int)fy;
  const float wx = x - fx, wy = y - fy;
  const uint32_t x0 = (uint32_t)ix & 127u, x1 = (uint32_t)(ix + 1) & 127u;
  const uint32_t y0 = (uint32_t)iy & 127u, y1 = (uint32_t)(iy + 1) & 127u;
  const uint16_t* c = reinterpret_cast<const uint16_t*>(curl);
  const uint32_t t00 = __ldg(c + y0 * 128 + x0), t10 = __ldg(c + y0 * 128 + x1);
  const uint32_t t01 = __ldg(c + y1 * 128 + x0), t11 = __ldg(c + y1 * 128 + x1);
  DR out[2];
#pragma unroll
  for (int ch = 0; ch < 2; ++ch) {
    const uint32_t sel = ch ? 0x7541u : 0x7540u;
    const float a00 = byte_to_float(t00, sel), a10 = byte_to_float(t10, sel);
    const float a01 = byte_to_float(t01, sel), a11 = byte_to_float(t11, sel);
    const float val = lerpf(lerpf(a00, a10, wx), lerpf(a01, a11, wx), wy) * (1.0f / 255.0f);
    const float gxv = lerpf(a10 - a00, a11 - a01, wy) * (128.0f / 255.0f);
    const float gyv = (lerpf(a01, a11, wx) - lerpf(a00, a10, wx)) * (128.0f / 255.0f);
    out[ch] = chain2(val, gxv, gyv, u, v);
  }
  r = out[0];
  g = out[1];
}

// weather_sample (R channel, W x H floats, repeat, bilinear) with its gradient
__device__ __forceinline__ DR weather_d(const float* wm, uint32_t W, uint32_t H, const DR& u, const DR& v) {
  const float x = u.v * (float)W - 0.5f, y = v.v * (float)H - 0.5f;
  const float fx = floorf(x), fy = floorf(y);
  const int ix = (int)fx, iy = (int)fy;
  const float wx = x - fx, wy = y - fy;
  const int x0 = wrap_mod(ix, (int)W), x1 = wrap_mod(ix + 1, (int)W);
  const int y0 = wrap_mod(iy, (int)H), y1 = wrap_mod(iy + 1, (int)H);
  const float a00 = __ldg(wm + y0 * W + x0), a10 = __ldg(wm + y0 * W + x1);
  const float a01 = __ldg(wm + y1 * W + x0), a11 = __ldg(wm + y1 * W + x1);
  const float val = lerpf(lerpf(a00, a10, wx), lerpf(a01, a11, wx), wy);
  const float gxv = lerpf(a10 - a00, a11 - a01, wy) * (float)W;
  const float gyv = (lerpf(a01, a11, wx) - lerpf(a00, a10, wx)) * (float)H;
  return chain2(val, gxv, gyv, u, v);
}

// lut2d (RGBA, clamp-to-edge, bilinear) of the RGB channels with gradients
__device__ __forceinline__ DR3 lut2d_d(const float4* lut, int W, int H, const DR& u, const DR& v) {
  const float x = u.v * (float)W - 0.5f, y = v.v * (float)H - 0.5f;
  const float fx = floorf(x), fy = floorf(y);
  const int ix = (int)fx, iy = (int)fy;
  const float wx = x - fx, wy = y - fy;
  const int x0 = clamp_idx(ix, W), x1 = clamp_idx(ix + 1, W);
  const int y0 = clamp_idx(iy, H), y1 = clamp_idx(iy + 1, H);
  const float4 t00 = __ldg(lut + y0 * W + x0), t10 = __ldg(lut + y0 * W + x1);
  const float4 t01 = __ldg(lut + y1 * W + x0), t11 = __ldg(lut + y1 * W + x1);
  const float c00[3] = {t00.x, t00.y, t00.z}, c10[3] = {t10.x, t10.y, t10.z};
  const float c01[3] = {t01.x, t01.y, t01.z}, c11[3] = {t11.x, t11.y, t11.z};
  DR out[3];
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) {
    const float a = lerpf(c00[ch], c10[ch], wx), b = lerpf(c01[ch], c11[ch], wx);
    const float gxv = lerpf(c10[ch] - c00[ch], c11[ch] - c01[ch], wy) * (float)W;
    out[ch] = chain2(lerpf(a, b, wy), gxv, (b - a) * (float)H, u, v);
  }
  return {out[0], out[1], out[2]};
}

// Aerial-perspective LUT (lut_ap) and its derivative along the distance
// coordinate w (trilinear: d/dw = 64 (upper - lower z plane)).
__device__ __forceinline__ void lut_ap_dw(const float4* lut, float u, float v, float w, float4& val, float4& dw) {
  const float x = u * 32.0f - 0.5f, y = v * 32.0f - 0.5f, z = w * 64.0f - 0.5f;
  const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
  const int ix = (int)fx, iy = (int)fy, iz = (int)fz;
  const float wx = x - fx, wy = y - fy, wz = z - fz;
  const int x0 = clamp_idx(ix, 32), x1 = clamp_idx(ix + 1, 32);
  const int y0 = clamp_idx(iy, 32), y1 = clamp_idx(iy + 1, 32);
  const int z0 = clamp_idx(iz, 64), z1 = clamp_idx(iz + 1, 64);
  auto at = [&](int xx, int yy, int zz) { return __ldg(lut + (zz * 32 + yy) * 32 + xx); };
  const float4 a = lerp4(lerp4(at(x0, y0, z0), at(x1, y0, z0), wx), lerp4(at(x0, y1, z0), at(x1, y1, z0), wx), wy);
  const float4 b = lerp4(lerp4(at(x0, y0, z1), at(x1, y0, z1), wx), lerp4(at(x0, y1, z1), at(x1, y1, z1), wx), wy);
  val = lerp4(a, b, wz);
  dw = make_float4((b.x - a.x) * 64.0f, (b.y - a.y) * 64.0f, (b.z - a.z) * 64.0f, (b.w - a.w) * 64.0f);
}

// ------------------------------------------------ march pieces, carried
// ndf (cloud_density_common.wgsl:49-91) of a carried height
__device__ __forceinline__ DR ndf_d(const DR& h, uint32_t t, float anvil_bias) {
  switch (t) {
    case 0: return dsmooth(0.0f, 0.07f, h) * dsmooth(1.0f, 0.2f, h);
    case 1: return dsmooth(0.0f, 0.10f, h) * (1.0f - dsmooth(0.6f, 1.0f, h));
    case 2: return dsmooth(0.0f, 0.15f, h) * dsmooth(1.0f, 0.4f, h);
    case 3: return dsmooth(0.0f, 0.20f, h) * dsmooth(1.0f, 0.3f, h);
    case 4: return dsmooth(0.0f, 0.30f, h) * (1.0f - dsmooth(0.7f, 1.0f, h));
    case 5: return dsmooth(0.0f, 0.40f, h) * (1.0f - dsmooth(0.6f, 1.0f, h));
    case 6: return dsmooth(0.0f, 0.50f, h) * (1.0f - dsmooth(0.8f, 1.0f, h));
    case 7: {
      const DR base = dsmooth(0.0f, 0.05f, h);
      const DR mid = dsmooth(0.95f, 0.5f, h);
      const DR anvil = dsmooth(0.7f, 0.9f, h) * (1.5f * clampf(anvil_bias, 0.0f, 2.0f));
      const DR mt = dsmooth(0.65f, 0.8f, h);
      return base * dmix(mid, anvil, mt);
    }
    default: return flat<kRange>(0.0f);
  }
}

// altitude_from_entry (march_plain.cuh) of a carried point and distance
template <unsigned M>
__device__ __forceinline__ DR altitude_d(const MarchUniforms& u, const DR3& p, const DV<M>& r0, const DV<M>& cv,
                                         const DV<M>& h0, const DR& t) {
  const DR yy = p.y + u.planet_r;
  const DR len = dsqrt((p.x * p.x + yy * yy) + p.z * p.z);
  const DR num = 2.0f * t * r0 * cv + t * t;
  return h0 + num / (dmax(r0, 1.0f) + len);
}

// The carried layer's own record: its parameters with their slots, and the
// wind-cache quantities that move with its base and top.
struct LayerD {
  DR base, top;
  DV<kCov> coverage;
  DV<kShape> lf_bias;
  DV<kDetail> layer_detail;
  DV<kScale> density_scale;
  DR wind_x, wind_z, skew_x, skew_z, skew_thickness;
};
constexpr unsigned kEff = kCov | kRange;                      // eff = clamp(weather * coverage)
constexpr unsigned kLight = kCov | kShape | kScale | kRange;  // a light tap's density: no detail erosion

// density_at of the carried layer.  Samples and taps whose value the profile
// rules out (can_be_dense; exactly 0 for a light tap) have no derivative
// either: the branches are taken on the values.
template <int ST, bool LIGHT>
__device__ __forceinline__ DV<LIGHT ? kLight : kAll> density_d(const MarchUniforms& u, const LayerConst& L,
                                                               const LayerD& D, const DR3& p, const DR& alt,
                                                               const DV<kEff>& eff, uint32_t type) {
  constexpr unsigned kOut = LIGHT ? kLight : kAll;
  const DR h = (alt - D.base) / dmax(D.top - D.base, 1.0f);
  if (h.v < 0.0f || h.v > 1.0f) return flat<kOut>(0.0f);
  if (eff.v < 0.01f) return flat<kOut>(0.0f);
  const DR nd = ndf_d(h, type, L.anvil_bias);
  if (LIGHT ? !(nd.v * 1.000001f > 1.0f - eff.v) : !can_be_dense(L, nd.v, 1.0f - eff.v)) return flat<kOut>(0.0f);
  const DR sk = h * D.skew_thickness;
  const DR ax = (p.x - D.wind_x) - D.skew_x * sk;
  const DR ay = p.y;
  const DR az = (p.z - D.wind_z) - D.skew_z * sk;
  const float bs = u.base_scale, ibs = u.inv_base_scale;
  const DR4 b = trilinear_d<ST, 128>(u.noise_base, over(ax, bs, ibs), over(ay, bs, ibs), over(az, bs, ibs),
                                     u.noise_scale);
  const auto lf = dclamp01(((b.y * 0.625f + b.z * 0.25f) + b.w * 0.125f) + D.lf_bias);
  const auto base_cloud = dremap01(b.x, -(1.0f - lf));
  const auto shaped = base_cloud * nd;
  const auto cloud = dremap01(shaped, 1.0f - eff) * eff;
  if constexpr (LIGHT) {
    return dclamp01(cloud) * D.density_scale;
  } else {
    if (!(cloud.v > 0.0f)) return widen<kAll>(dclamp01(cloud) * D.density_scale);
    const float ds = u.detail_scale, ids = u.inv_detail_scale;
    DR c2x, c2y;
    curl_d(u.curl, over(ax, ds, ids), over(az, ds, ids), c2x, c2y);
    const DR cx = c2x * 2.0f - 1.0f, cz = c2y * 2.0f - 1.0f;
    const DR dx = ax + (cx * u.curl_strength) * u.detail_scale;
    const DR dz = az + (cz * u.curl_strength) * u.detail_scale;
    const DR4 det = trilinear_d<ST, 32>(u.noise_detail, over(dx, ds, ids), over(ay, ds, ids), over(dz, ds, ids),
                                        u.noise_scale);
    const DR hf = (det.x * 0.625f + det.y * 0.25f) + det.z * 0.125f;
    const DR dmod = dmix(hf, 1.0f - hf, dclamp01(h * 10.0f));
    return dclamp01(dremap01(cloud, dmod * D.layer_detail)) * D.density_scale;
  }
}

__constant__ float kCone[6][3] = {{0.38051305f, 0.92453449f, -0.02111345f}, {-0.50625799f, -0.03590792f, -0.86163418f},
                                  {-0.32509218f, -0.94557439f, 0.01428793f}, {0.09026238f, -0.27376545f, 0.95755165f},
                                  {0.28128598f, 0.42443639f, -0.86065785f},  {-0.16852403f, 0.14748697f, 0.97460106f}};

// march_to_light (march_plain.cuh) of the carried layer
template <int ST>
__device__ __forceinline__ DV<kLight> light_od_d(const MarchUniforms& u, const LayerConst& L, const LayerD& D,
                                                 const DR3& p, const DR& alt, const DV<kEff>& eff, uint32_t type) {
  const float sx = u.sun[0], sy = u.sun[1], sz = u.sun[2];
  const DR r0 = alt + u.planet_r;
  const DR inv = dc(1.0f) / dmax(r0, 1.0f);
  const DR cv = ((p.x * inv) * sx + ((p.y + u.planet_r) * inv) * sy) + (p.z * inv) * sz;
  const float cos_sun = fmaxf(sy, 0.05f);
  const DR dist = dmax(over(D.top - alt, cos_sun, u.inv_cos_sun), 1.0f);
  const uint32_t n = u.cone ? 6u : u.light_steps;
  const DR step = dist / (u.cone ? 5.0f : (float)u.light_steps);
  DV<kLight> od = flat<kLight>(0.0f);
#pragma unroll 1
  for (uint32_t i = 0; i < n; ++i) {
    const bool last = u.cone && i == 5u;  // the cone's sixth tap reaches out to three times the path
    const DR t = last ? dist * 3.0f : ((float)i + 0.5f) * step;
    DR3 q = {t * sx + p.x, t * sy + p.y, t * sz + p.z};
    if (u.cone) {  // cloud_march.wgsl:599-666
      const DR sc = last ? step * 3.0f : step * ((float)i + 1.0f) / 5.0f;
      q = {q.x + kCone[i][0] * sc, q.y + kCone[i][1] * sc, q.z + kCone[i][2] * sc};
    }
    const DR a = altitude_d(u, q, r0, cv, alt, t);
    const auto part = density_d<ST, true>(u, L, D, q, a, eff, type) * step;
    od = od + (last ? part * 3.0f : part);
  }
  return od;
}

// sun_and_sky_at (march_plain.cuh) of a carried point
struct SunSkyD {
  DR3 sun, sky;
};
__device__ __forceinline__ SunSkyD sun_and_sky_d(const MarchUniforms& u, const DR3& p, float sun_az) {
  SunSkyD out;
  const float R = u.planet_r;
  const DR ay = p.y + R;
  const DR len = dsqrt((p.x * p.x + ay * ay) + p.z * p.z);
  const DR r = dmax(len, R + 1.0f);
  const DR mu = dclamp(((p.x / r) * u.sun[0] + (ay / r) * u.sun[1]) + (p.z / r) * u.sun[2], -1.0f, 1.0f);
  const DR ratio = dc(R) / r;
  const DR sin_h = -dsqrt(dmax(1.0f - ratio * ratio, 0.0f));
  if (mu.v <= sin_h.v) {
    out.sun = {flat<kRange>(0.0f), flat<kRange>(0.0f), flat<kRange>(0.0f)};
  } else {
    const float ht = u.atmo_top;
    const float bh = sqrtf(fmaxf(ht * ht - R * R, 0.0f));
    const DR rho = dsqrt(dmax(r * r - R * R, 0.0f));
    const DR disc = r * r * (mu * mu - 1.0f) + ht * ht;
    const DR d = dmax(-r * mu + dsqrt(dmax(disc, 0.0f)), 0.0f);
    const DR d_min = ht - r, d_max = rho + bh;
    const DR xm = dclamp01((d - d_min) / dmax(d_max - d_min, 1.0f));
    const DR xr = rho / fmaxf(bh, 1.0f);
    out.sun = lut2d_d(u.lut_trans, 256, 64, xm, xr);
  }
  const DR ux = p.x / len, uy = ay / len, uz = p.z / len;
  const DR vza = datan2(dsqrt(ux * ux + uz * uz), uy);
  const DR sin_z = dclamp01(dc(R) / len);
  const DR zha = kPi - dasin(sin_z);
  DR vv;
  if (vza.v < zha.v) {
    vv = dsqrt(dclamp01(vza / dmax(zha, 1e-6f))) * 0.5f;
  } else {
    const DR br = dmax(kPi - zha, 1e-6f);
    vv = 0.5f + dsqrt(dclamp01((vza - zha) / br)) * 0.5f;
  }
  const DR vaz = datan2(ux, uz);
  DR du = (vaz - sun_az) / (2.0f * kPi);
  du = du - floorf(du.v);
  const DR3 s = lut2d_d(u.lut_sky, 192, 108, du, vv);
  out.sky = {s.x * u.sun_illum[0], s.y * u.sun_illum[1], s.z * u.sun_illum[2]};
  return out;
}

// The distance t of a shell crossing with its derivatives with respect to the
// carried layer's base and top: a t on the sphere at planet radius + base
// (or + top) moves by dt/dr = r / (t + b), b = o.d; t = 0 (inside the layer)
// or a depth clip does not move.
__device__ DR shell_distance_d(const MarchUniforms& u, const LayerConst& L, const double oc[3], const double d[3],
                               float t) {
  DR r = flat<kRange>(t);
  if (!(t > 0.0f)) return r;
  const double td = (double)t;
  const double px = oc[0] + d[0] * td, py = oc[1] + d[1] * td, pz = oc[2] + d[2] * td;
  const double rr = sqrt(px * px + py * py + pz * pz);
  const double b = oc[0] * d[0] + oc[1] * d[1] + oc[2] * d[2];
  const double eb = fabs(rr - L.r_bottom), et = fabs(rr - L.r_top);
  const double tol = 0.1 + 1e-6 * td;  // float rounding of t
  if (fmin(eb, et) > tol || fabs(td + b) < 1e-9) return r;
  const double k = (eb <= et ? L.r_bottom : L.r_top) / (td + b);
  r.d[eb <= et ? kBase : kTop] = (float)k;
  return r;
}

// What the march accumulates along a ray, radiance and transmittance per
// channel and the distance weights, with all derivatives: touched once per
// dense sample and so kept in shared memory, [word][thread], out of the
// registers a sample needs (56 words).  The transmittances' values are kept in
// registers too, for the exits.
struct Path {
  float* s;  // this thread's column
  float T[3];
  enum : uint32_t { kL = 0, kT = 3, kTw = 6, kTwn = 7, kCount = 8 };
  __device__ __forceinline__ DV<kAll> get(uint32_t what) const {
    DV<kAll> r;
    const float* const w = s + what * (kP + 1) * kThreads;
    r.v = w[0];
    each<kAll>([&](auto i) {
      constexpr int j = decltype(i)::n;
      r.d[j] = w[(j + 1) * kThreads];
    });
    return r;
  }
  __device__ __forceinline__ void put(uint32_t what, const DV<kAll>& x) {
    float* const w = s + what * (kP + 1) * kThreads;
    w[0] = x.v;
    each<kAll>([&](auto i) {
      constexpr int j = decltype(i)::n;
      w[(j + 1) * kThreads] = x.d[j];
    });
  }
  __device__ __forceinline__ bool opaque() const { return fmaxf(T[0], fmaxf(T[1], T[2])) < 0.01f; }
};
// Adds channel c of a dense sample, its in-scattered radiance integral (before
// T) and its transmittance; returns what L gained.
template <unsigned S, unsigned M>
__device__ __forceinline__ DV<kAll> add_channel(Path& path, uint32_t c, const DV<S>& in, const DV<M>& through) {
  const DV<kAll> before = path.get(Path::kT + c);
  const DV<kAll> gain = before * in, after = before * through;
  path.put(Path::kL + c, path.get(Path::kL + c) + gain);
  path.put(Path::kT + c, after);
  if (c == 0) path.T[0] = after.v;
  if (c == 1) path.T[1] = after.v;
  if (c == 2) path.T[2] = after.v;
  return gain;
}
template <unsigned T>
__device__ __forceinline__ void add_weight(Path& path, const DV<kAll>& w, const DV<T>& t) {
  path.put(Path::kTw, path.get(Path::kTw) + w * t);
  path.put(Path::kTwn, path.get(Path::kTwn) + w);
}
__device__ __forceinline__ float luminance_weight(uint32_t c) { return c == 0 ? 0.2126f : (c == 1 ? 0.7152f : 0.0722f); }

constexpr uint32_t kPhaseOctaves = 8;  // octaves whose phase values are kept per ray and layer

// The octaves' phase value at one sample: kept, or evaluated (octaves past
// the kept ones, and the blend band of a Cumulonimbus layer's droplet size).
struct PhaseAt {
  const float* kept;
  PhaseConst pc;
  bool own;
  __device__ __forceinline__ float operator()(const MarchUniforms& u, float cos_theta, uint32_t o, float cc) const {
    return (own || o >= kPhaseOctaves) ? phase_with(u, cos_theta, cc, pc) : kept[o * kThreads];
  }
};

// One dense sample of a layer that is not the carried one: no derivative of
// its own, so plain values (march.cu's k_march_plain).
template <int ST>
__device__ __forceinline__ void plain_sample(const MarchUniforms& u, const LayerConst& L, Path& path, float px, float py,
                                             float pz, float alt, float t, float step, float density, const Cover& cov,
                                             uint32_t type, float cos_theta, float fwd, float sun_az, float bh,
                                             float inv_bh, const float* s_ph) {
  const float od = march_to_light<ST, PSC_FILTER_EXACT>(u, L, px, py, pz, alt, cov, type, nullptr);
  const float hn = clamp01(layer_height(L, alt));
  PhaseAt phase{s_ph, PhaseConst{L.g_hg, L.g_d, L.alpha, L.w_d, L.ice}, L.cloud_type == 7u};
  if (L.cloud_type == 7u)
    phase.pc = phase_consts_from_d(mixf(L.droplet_um, 50.0f, smoothstepf(0.60f, 0.85f, hn)), u.droplet_bias);
  const SunSky ss = sun_and_sky_at(u, px, py, pz, sun_az, bh, inv_bh, nullptr);
  const float ts[3] = {ss.sun.x, ss.sun.y, ss.sun.z}, sky[3] = {ss.sky.x, ss.sky.y, ss.sky.z};
  const float ag = mixf(0.3f, 1.0f, hn) * u.ambient;
  float lw = 0.0f;
  if (u.lightning_radius > 0.0f) {
    const float ddx = px - u.lightning_origin_x, ddz = pz - u.lightning_origin_z;
    const float fo = clamp01(1.0f - sqrtf(ddx * ddx + ddz * ddz) / u.lightning_radius);
    lw = fo * fo * (3.0f - 2.0f * fo);
  }
  float S[3] = {0.0f, 0.0f, 0.0f}, beer[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) beer[c] = expf(od * -L.sigma_t[c]);
  float a = 1.0f, b = 1.0f, cc = 1.0f;
#pragma unroll 1
  for (uint32_t o = 0; o < u.octaves; ++o) {
    const float ph = phase(u, cos_theta, o, cc);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float e = o ? expf((od * -L.sigma_t[c]) * b) : beer[c];
      S[c] = S[c] + e * ts[c] * ((a * u.sun_illum[c]) * ph);
    }
    a *= u.ms_a;
    b *= u.ms_b;
    cc *= u.ms_c;
  }
  const float f = u.forward_bias > 0.0f ? 1.0f + u.forward_bias * fwd : 1.0f;
  DV<kAll> w = flat<kAll>(0.0f);
#pragma unroll
  for (uint32_t c = 0; c < 3; ++c) {
    const float st = L.sigma_t[c];
    const float pw = 1.0f - expf(od * (-2.0f * st));
    const float e = mixf(beer[c], beer[c] * pw * 2.0f, u.powder);
    if (u.forward_bias > 0.0f) S[c] = S[c] * f;
    const float is = (density * u.sigma_s[c]) * ((S[c] * e + sky[c] * ag) + lw * u.lightning_rgb[c]);
    const float ls = fmaxf(density * st, 1e-6f);
    const float sm = expf(ls * step * -1.0f);
    w = w + add_channel(path, c, dc((is - is * sm) / ls), dc(sm)) * luminance_weight(c);
  }
  add_weight(path, w, dc(t));
}

// One dense sample of the carried layer.
template <int ST>
__device__ __forceinline__ void carried_sample(const MarchUniforms& u, const LayerConst& L, const LayerD& D, Path& path,
                                               const DR3& p, const DR& alt, const DR& t, const DR& step,
                                               const DV<kAll>& density, const DV<kEff>& eff, uint32_t type,
                                               float cos_theta, float fwd, float sun_az, const float* s_ph) {
  const DV<kLight> od = light_od_d<ST>(u, L, D, p, alt, eff, type);
  const DR hn = dclamp01((alt - D.base) / dmax(D.top - D.base, 1.0f));
  // not Cumulonimbus under approx-Mie: the phase does not depend on the height
  const PhaseAt phase{s_ph, PhaseConst{L.g_hg, L.g_d, L.alpha, L.w_d, L.ice}, false};
  const SunSkyD ss = sun_and_sky_d(u, p, sun_az);
  const DR ag = dmix(0.3f, 1.0f, hn) * u.ambient;
  DR lw = flat<kRange>(0.0f);
  if (u.lightning_radius > 0.0f) {
    const DR ddx = p.x - u.lightning_origin_x, ddz = p.z - u.lightning_origin_z;
    const DR fo = dclamp01(1.0f - dsqrt(ddx * ddx + ddz * ddz) / u.lightning_radius);
    lw = fo * fo * (3.0f - 2.0f * fo);
  }
  const float f = u.forward_bias > 0.0f ? 1.0f + u.forward_bias * fwd : 1.0f;
  // one channel at a time: the body of all three together is larger than the
  // instruction cache
  DV<kAll> w = flat<kAll>(0.0f);
#pragma unroll 1
  for (uint32_t c = 0; c < 3; ++c) {
    const float st = L.sigma_t[c];
    const DR ts = c == 0 ? ss.sun.x : (c == 1 ? ss.sun.y : ss.sun.z), sky = c == 0 ? ss.sky.x : (c == 1 ? ss.sky.y : ss.sky.z);
    const auto bb = dexp(od * -st);
    const auto pw = 1.0f - dexp(od * (-2.0f * st));
    const auto e = dmix(bb, bb * pw * 2.0f, u.powder);
    DV<kLight> S = flat<kLight>(0.0f);
    float a = 1.0f, b = 1.0f, cc = 1.0f;
#pragma unroll 1
    for (uint32_t o = 0; o < u.octaves; ++o) {
      S = S + (o ? dexp((od * -st) * b) : bb) * ts * ((a * u.sun_illum[c]) * phase(u, cos_theta, o, cc));
      a *= u.ms_a;
      b *= u.ms_b;
      cc *= u.ms_c;
    }
    if (u.forward_bias > 0.0f) S = S * f;
    const auto is = (density * u.sigma_s[c]) * ((S * e + sky * ag) + lw * u.lightning_rgb[c]);
    const auto ls = dmax(density * st, 1e-6f);
    const auto sm = dexp(ls * step * -1.0f);
    w = w + add_channel(path, c, (is - is * sm) / ls, sm) * luminance_weight(c);
  }
  add_weight(path, w, t);
}

// One ray of the PLAIN march (k_march_plain) with its tangents; adds this
// pixel's loss and d loss / d parameter (before the 1 / N) to `acc`.  `s_ph`
// and `s_path` are this thread's columns of kept phase values and of Path.
template <int ST>
__device__ void param_grad_pixel(const MarchUniforms& u, const ViewDev& v, const ParamGradDev& g, uint32_t px,
                                 uint32_t py, float* s_ph, float* s_path, float acc[kP + 1]) {
  RaySetup rs;
  setup_ray(u, v, px, py, rs);
  float* const s_t = s_ph + kPhaseOctaves * kThreads;  // entry and exit of each layer
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    s_t[j * kThreads] = rs.t0[j];
    s_t[(8 + j) * kThreads] = rs.t1[j];
  }
  const float dx = rs.dir[0], dy = rs.dir[1], dz = rs.dir[2];
  const float cx = u.cam[0], cy = u.cam[1], cz = u.cam[2];
  const float cos_theta = (dx * u.sun[0] + dy * u.sun[1]) + dz * u.sun[2];
  const float fwd = smoothstepf(0.0f, 1.0f, fmaxf(cos_theta, 0.0f));
  const float sun_az = atan2f(u.sun[0], u.sun[2]);
  const float bh = horizon_h(u), inv_bh = 1.0f / fmaxf(bh, 1.0f);
  uint32_t sx = (px + v.x_off) & 63u, sy = (py + v.y_off) & 63u;
  if (u.temporal_jitter) {
    const uint32_t ph = u.frame_index & 15u;
    sx = (sx ^ ((ph * 11u + 7u) & 63u)) & 63u;
    sy = (sy ^ ((ph * 23u + 13u) & 63u)) & 63u;
  }
  const float jitter = __ldg(u.blue + sy * 64u + sx);
  const double oc[3] = {(double)u.cam[0], (double)u.cam[1] + u.planet_r_d, (double)u.cam[2]};

  // the carried layer's parameters and wind quantities with their slots
  LayerD D;
  {
    const LayerConst& L = u.layers[g.layer];
    auto bt = [](float v0, float kb, float kt) {
      DR r;
      r.v = v0;
      r.d[kBase] = kb;
      r.d[kTop] = kt;
      return r;
    };
    D.base = bt(L.base_m, 1.0f, 0.0f);
    D.top = bt(L.top_m, 0.0f, 1.0f);
    D.coverage.v = L.coverage;
    D.coverage.d[0] = 1.0f;
    D.lf_bias.v = L.lf_bias;
    D.lf_bias.d[1] = g.dlf_dshape;
    D.layer_detail.v = L.layer_detail;
    D.layer_detail.d[2] = g.dld_ddetail;
    D.density_scale.v = L.density_scale;
    D.density_scale.d[3] = 1.0f;
    D.wind_x = bt(L.wind_off_x, g.dwind[0][0], g.dwind[0][1]);
    D.wind_z = bt(L.wind_off_z, g.dwind[1][0], g.dwind[1][1]);
    D.skew_x = bt(L.skew_x, g.dskew[0][0], g.dskew[0][1]);
    D.skew_z = bt(L.skew_z, g.dskew[1][0], g.dskew[1][1]);
    D.skew_thickness = bt(L.skew_thickness, g.dskew[2][0], g.dskew[2][1]);
  }

  Path path{s_path, {1.0f, 1.0f, 1.0f}};
#pragma unroll
  for (uint32_t w = 0; w < Path::kCount; ++w) path.put(w, flat<kAll>(w >= Path::kT && w < Path::kTw ? 1.0f : 0.0f));
  const DV<0> r0c = dc(rs.r0), cvc = dc(rs.cos_view), h0c = dc(rs.h0);
  for (uint32_t k = 0; k < u.layer_count; ++k) {
    if (path.opaque()) break;
    const uint32_t li = (rs.order >> (4u * k)) & 15u;
    if (!((rs.hit_mask >> li) & 1u) || li >= 8u) continue;
    const float t0f = s_t[li * kThreads], t1f = s_t[(8u + li) * kThreads];
    const LayerConst& L = u.layers[li];
    const bool carried = li == g.layer;
    if (t1f - t0f <= 0.0f) continue;
    const float stepf = (t1f - t0f) / (float)u.cloud_steps;
    // the steps that can hold cloud, as in k_march_plain
    uint32_t s_begin = 0u, s_end = u.cloud_steps;
    if (!u.type_grid) {
      if (!(L.live_lo <= L.live_hi)) continue;
      if (!live_step_range(rs.r0, 2.0f * rs.r0 * rs.cos_view, L, u.planet_r, t0f, t1f, stepf, jitter, u.cloud_steps,
                           s_begin, s_end))
        continue;
    }
    {
      const PhaseConst pc{L.g_hg, L.g_d, L.alpha, L.w_d, L.ice};
#pragma unroll 1
      for (uint32_t o = 0; o < min(u.octaves, kPhaseOctaves); ++o)
        s_ph[o * kThreads] = phase_with(u, cos_theta, u.cpow[o], pc);
    }
    if (carried) {
      const DR t0 = shell_distance_d(u, L, oc, rs.dird, t0f), t1 = shell_distance_d(u, L, oc, rs.dird, t1f);
      const DR step = (t1 - t0) / (float)u.cloud_steps;
#pragma unroll 1
      for (uint32_t s = s_begin; s < s_end; ++s) {
        const DR t = t0 + step * ((float)s + jitter);
        const DR3 p = {t * dx + cx, t * dy + cy, t * dz + cz};
        const DR alt = altitude_d(u, p, r0c, cvc, h0c, t);
        const DR wsx = p.x - D.wind_x, wsz = p.z - D.wind_z;
        const DR wr = u.weather_uniform ? flat<kRange>(u.weather_value)
                                        : weather_d(u.weather, u.weather_w, u.weather_h, wsx / u.weather_scale + 0.5f,
                                                    wsz / u.weather_scale + 0.5f);
        const DV<kEff> eff = dclamp01(wr * D.coverage);
        const uint32_t type = effective_type(u, wsx.v, wsz.v, L.cloud_type);
        const DV<kAll> density = density_d<ST, false>(u, L, D, p, alt, eff, type);
        if (!(density.v > 1e-3f)) continue;
        carried_sample<ST>(u, L, D, path, p, alt, t, step, density, eff, type, cos_theta, fwd, sun_az, s_ph);
        if (path.opaque()) break;
      }
    } else {
      Cover cov = cover_of(L, u.weather_value);
#pragma unroll 1
      for (uint32_t s = s_begin; s < s_end; ++s) {
        const float t = t0f + stepf * ((float)s + jitter);
        const float px3 = t * dx + cx, py3 = t * dy + cy, pz3 = t * dz + cz;
        const float alt = altitude_from_entry(u, px3, py3, pz3, rs.r0, rs.cos_view, rs.h0, t);
        const float wsx = px3 - L.wind_off_x, wsz = pz3 - L.wind_off_z;
        if (!u.weather_uniform)
          cov = cover_of(L, weather_sample(u.weather, u.weather_w, u.weather_h, wsx / u.weather_scale + 0.5f,
                                           wsz / u.weather_scale + 0.5f));
        const uint32_t type = effective_type(u, wsx, wsz, L.cloud_type);
        const float density = density_primary_at<ST, PSC_FILTER_EXACT>(u, L, px3, py3, pz3, alt, cov, type, nullptr);
        if (!(density > 1e-3f)) continue;
        plain_sample<ST>(u, L, path, px3, py3, pz3, alt, t, stepf, density, cov, type, cos_theta, fwd, sun_az, bh,
                         inv_bh, s_ph);
        if (path.opaque()) break;
      }
    }
  }

  // aerial perspective (cloud_march.wgsl:1016-1048)
  const DV<kAll> T[3] = {path.get(Path::kT), path.get(Path::kT + 1), path.get(Path::kT + 2)};
  const DV<kAll> t_lum = (T[0] * 0.2126f + T[1] * 0.7152f) + T[2] * 0.0722f;
  const DV<kAll> opacity = 1.0f - t_lum;
  DV<kAll> O[3] = {path.get(Path::kL), path.get(Path::kL + 1), path.get(Path::kL + 2)};
  if (opacity.v > 1e-4f) {
    const DV<kAll> t_cloud = path.get(Path::kTw) / dmax(path.get(Path::kTwn), 1e-6f);
    const DV<kAll> ds = dmax(t_cloud, 50.0f);
    const DV<kAll> azd = dclamp01(dlog(ds * (1.0f / 50.0f)) * (1.0f / logf(100000.0f / 50.0f)));
    float4 ap, dap;
    lut_ap_dw(u.lut_ap, ((float)(px + v.x_off) + 0.5f) / u.vp_w, ((float)(py + v.y_off) + 0.5f) / u.vp_h, azd.v,
              ap, dap);
    const DV<kAll> apw = along(ap.w, dap.w, azd);
    const DV<kAll> apc[3] = {along(ap.x, dap.x, azd), along(ap.y, dap.y, azd), along(ap.z, dap.z, azd)};
#pragma unroll
    for (int c = 0; c < 3; ++c) O[c] = O[c] * apw + apc[c] * opacity;
  }
  const size_t idx = (size_t)py * v.width + px;
  const float4 bgp = __ldg(g.bg + idx), tg = __ldg(g.target + idx);
  const float bgc[3] = {bgp.x, bgp.y, bgp.z}, tgc[3] = {tg.x, tg.y, tg.z};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const DV<kAll> I = O[c] + T[c] * bgc[c];
    const float r = I.v - tgc[c];
    acc[0] = fmaf(r, r, acc[0]);
#pragma unroll
    for (int i = 0; i < kP; ++i) acc[1 + i] = fmaf(2.0f * r, I.d[i], acc[1 + i]);
  }
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// out[0..5] += d loss / d (coverage, shape_bias, detail_bias, density_scale,
// base_m, top_m); loss (nullable) += the loss.
template <int ST>
__global__ void __launch_bounds__(kThreads) k_march_param_grad(const __grid_constant__ MarchUniforms u,
                                                               const __grid_constant__ ViewDev v,
                                                               const __grid_constant__ ParamGradDev g, double* out,
                                                               double* loss) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t px = blockIdx.x * kTileW + (warp & 1u) * 8u + (lane & 7u);
  const uint32_t py = blockIdx.y * kTileH + (warp >> 1) * 4u + (lane >> 3);
  __shared__ float s_phase[(kPhaseOctaves + 16u) * kThreads];  // and the layers' entries and exits
  __shared__ float s_path[Path::kCount * (kP + 1) * kThreads];
  float acc[kP + 1];
#pragma unroll
  for (int i = 0; i < kP + 1; ++i) acc[i] = 0.0f;
  if (px < v.width && py < v.height) 
    param_grad_pixel<ST>(u, v, g, px, py, s_phase + threadIdx.x, s_path + threadIdx.x, acc);
  __shared__ double s_red[kP + 1][kThreads / 32];
#pragma unroll
  for (int i = 0; i < kP + 1; ++i) {
    const double w = warp_sum((double)acc[i] * (double)g.inv_n);
    if (lane == 0) s_red[i][warp] = w;
  }
  __syncthreads();
  if (threadIdx.x < kP + 1) {
    double a = 0.0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) a += s_red[threadIdx.x][w];
    if (threadIdx.x == 0) {
      if (loss) atomicAdd(loss, a);
    } else {
      atomicAdd(out + threadIdx.x - 1, a);
    }
  }
}

template <int ST>
cudaError_t launch_st(const MarchUniforms& u, const ViewDev& v, const ParamGradDev& g, double* out, double* loss,
                      cudaStream_t s) {
  const dim3 grid((v.width + kTileW - 1) / kTileW, (v.height + kTileH - 1) / kTileH);
  k_march_param_grad<ST><<<grid, kThreads, 0, s>>>(u, v, g, out, loss);
  return cudaGetLastError();
}

}  // namespace

int launch_march_param_grad(const MarchUniforms& u, const ViewDev& v, const ParamGradDev& g, uint32_t storage,
                            double* out, double* loss, cudaStream_t s) {
  if (g.layer >= u.layer_count || g.layer >= 8u) return PSC_ERR_INVALID_ARGUMENT;
  cudaError_t e;
  switch (storage) {
    case PSC_STORAGE_U8:
      e = u.far_texels ? launch_st<kStorageU8Far>(u, v, g, out, loss, s)
                       : launch_st<PSC_STORAGE_U8>(u, v, g, out, loss, s);
      break;
    case PSC_STORAGE_F32: e = launch_st<PSC_STORAGE_F32>(u, v, g, out, loss, s); break;
    case PSC_STORAGE_F16: e = launch_st<PSC_STORAGE_F16>(u, v, g, out, loss, s); break;
    case PSC_STORAGE_BF16: e = launch_st<PSC_STORAGE_BF16>(u, v, g, out, loss, s); break;
    case PSC_STORAGE_FP8: e = launch_st<PSC_STORAGE_FP8>(u, v, g, out, loss, s); break;
    default: return PSC_ERR_INVALID_ARGUMENT;
  }
  return e == cudaSuccess ? PSC_OK : PSC_ERR_CUDA;
}

}  // namespace psc
