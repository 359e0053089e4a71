// Device functions of the PLAIN march (march.cu) shared with its tangent
// form (march_param_grad.cu): the density kernel, the altitude along a ray,
// the light march, and the sun transmittance / sky-view ambient lookups.
// FP32 as the reference (cloud_march.wgsl, cloud_density_common.wgsl), in its
// order; divisions by what is fixed for the frame, the layer or the sample go
// through div_by.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "march_common.cuh"
#include "psc_internal.h"

namespace psc {
namespace {

// The coverage remap remap(cloud, 1 - eff, 1, 0, 1) * eff of one weather
// sample: its constants, shared by the primary sample and its light taps.
struct Cover {
  float eff, ome, den, inv_den;  // eff, 1 - eff, max(1 - (1 - eff), 1e-5) and its reciprocal
};
__device__ __forceinline__ Cover cover_of(const LayerConst& L, float wr) {
  Cover c;
  c.eff = clamp01(wr * L.coverage);
  c.ome = 1.0f - c.eff;
  c.den = fmaxf(1.0f - c.ome, 1e-5f);
  c.inv_den = rcp_near(c.den);
  return c;
}

// Normalised height of an altitude in the layer.
__device__ __forceinline__ float layer_height(const LayerConst& L, float alt) {
  return div_by(alt - L.base_m, fmaxf(L.top_m - L.base_m, 1.0f), L.inv_thickness);
}

// Whether a sample of profile value nd can be dense (density > 1e-3) for a
// coverage of which 1 - eff is at least `ome`: the base shape is at most 1,
// the remap of c takes at most c - (1 - eff) (to 2e-5) and the erosion only
// lowers that.  Where it cannot, the sample adds nothing and its noise taps
// are left out.
__device__ __forceinline__ bool can_be_dense(const LayerConst& L, float nd, float ome) {
  return fmaf(nd, 1.000001f, -ome) * L.density_scale > 0.999e-3f;
}

// Density (cloud_march.wgsl:432-530; light variant cloud_density_common.wgsl:266-305)
// of a sample inside the layer, h its normalised height, nd = ndf(h, type).
template <int ST, int FILT, bool LIGHT>
__device__ __forceinline__ float density_in(const MarchUniforms& u, const LayerConst& L, float px,
                                            float py, float pz, float h, float nd, const Cover& cov, int* chk) {
  const float sk = h * L.skew_thickness;
  const float ax = __fmaf_rn(-L.skew_x, sk, px - L.wind_off_x);
  const float ay = py;
  const float az = __fmaf_rn(-L.skew_z, sk, pz - L.wind_off_z);
  const float4 b = Noise<ST, FILT>::base(u, div_by(ax, u.base_scale, u.inv_base_scale),
                                         div_by(ay, u.base_scale, u.inv_base_scale),
                                         div_by(az, u.base_scale, u.inv_base_scale), chk);
  const float lf = clamp01((__fmaf_rn(b.y, 0.625f, __fmul_rn(b.z, 0.25f)) + b.w * 0.125f) + L.lf_bias);
  // remapf(b.x, -(1 - lf), 1, 0, 1)
  const float a = -(1.0f - lf), base_cloud = 0.0f + div_near(b.x - a, fmaxf(1.0f - a, 1e-5f));
  float cloud = base_cloud * nd;
  cloud = (0.0f + div_by(cloud - cov.ome, cov.den, cov.inv_den)) * cov.eff;
  if (!LIGHT && cloud > 0.0f) {
    const float inv = u.inv_detail_scale;
    const float2 c2 = Noise<ST, FILT>::curl(u, div_by(ax, u.detail_scale, inv), div_by(az, u.detail_scale, inv), chk);
    const float cx = c2.x * 2.0f - 1.0f, cz = c2.y * 2.0f - 1.0f;
    const float dx = ax + (cx * u.curl_strength) * u.detail_scale;
    const float dy = ay + (0.0f * u.curl_strength) * u.detail_scale;
    const float dz = az + (cz * u.curl_strength) * u.detail_scale;
    const float4 det = Noise<ST, FILT>::detail(u, div_by(dx, u.detail_scale, inv), div_by(dy, u.detail_scale, inv),
                                               div_by(dz, u.detail_scale, inv), chk);
    const float hf = __fmaf_rn(det.x, 0.625f, __fmul_rn(det.y, 0.25f)) + det.z * 0.125f;
    const float dmod = mixf(hf, 1.0f - hf, clamp01(h * 10.0f));
    const float lo = dmod * L.layer_detail;
    cloud = 0.0f + div_near(cloud - lo, fmaxf(1.0f - lo, 1e-5f));  // remapf(cloud, lo, 1, 0, 1)
  }
  return clamp01(cloud) * L.density_scale;
}

// Density of a light-march tap.  A tap whose profile value does not reach
// 1 - eff has density exactly 0 (the base shape is at most 1), and its noise
// tap is left out.
template <int ST, int FILT>
__device__ __forceinline__ float density_light_at(const MarchUniforms& u, const LayerConst& L, float px, float py,
                                                  float pz, float alt, const Cover& cov, uint32_t type, int* chk) {
  const float h = layer_height(L, alt);
  if (h < 0.0f || h > 1.0f) return 0.0f;
  if (cov.eff < 0.01f) return 0.0f;
  const float nd = ndf(h, type, L.anvil_bias);
  if (!(nd * 1.000001f > cov.ome)) return 0.0f;
  return density_in<ST, FILT, true>(u, L, px, py, pz, h, nd, cov, chk);
}

// Density of a primary sample; 0 where it cannot be dense.
template <int ST, int FILT>
__device__ __forceinline__ float density_primary_at(const MarchUniforms& u, const LayerConst& L, float px, float py,
                                                    float pz, float alt, const Cover& cov, uint32_t type, int* chk) {
  const float h = layer_height(L, alt);
  if (h < 0.0f || h > 1.0f) return 0.0f;
  if (cov.eff < 0.01f) return 0.0f;
  const float nd = ndf(h, type, L.anvil_bias);
  if (!can_be_dense(L, nd, cov.ome)) return 0.0f;
  return density_in<ST, FILT, false>(u, L, px, py, pz, h, nd, cov, chk);
}

__device__ __forceinline__ float altitude_from_entry(const MarchUniforms& u, float px, float py,
                                                     float pz, float r0, float cos_view, float h0,
                                                     float t) {
  // contractions written out: the last bit of the altitude moves the noise
  // coordinates, and left to the compiler it follows the code around the call
  const float yy = py + u.planet_r;
  const float len = sqrt_near(__fmaf_rn(pz, pz, __fmaf_rn(px, px, __fmul_rn(yy, yy))));
  const float num = __fmaf_rn(t, t, 2.0f * t * r0 * cos_view);
  return h0 + div_near(num, fmaxf(r0, 1.0f) + len);
}

template <int ST, int FILT>
__device__ float march_to_light(const MarchUniforms& u, const LayerConst& L, float px, float py,
                                float pz, float alt, const Cover& cov, uint32_t type, int* chk) {
  const float sx = u.sun[0], sy = u.sun[1], sz = u.sun[2];
  const float r0 = u.planet_r + alt;
  const float inv = rcp_near(fmaxf(r0, 1.0f));
  const float cv = ((px * inv) * sx + ((py + u.planet_r) * inv) * sy) + (pz * inv) * sz;
  const float cos_sun = fmaxf(sy, 0.05f);
  const float dist = fmaxf(div_by(L.top_m - alt, cos_sun, u.inv_cos_sun), 1.0f);
  float od = 0.0f, comp = 0.0f;
  if (u.cone) {  // cloud_march.wgsl:599-666
    const float K[6][3] = {{0.38051305f, 0.92453449f, -0.02111345f},
                           {-0.50625799f, -0.03590792f, -0.86163418f},
                           {-0.32509218f, -0.94557439f, 0.01428793f},
                           {0.09026238f, -0.27376545f, 0.95755165f},
                           {0.28128598f, 0.42443639f, -0.86065785f},
                           {-0.16852403f, 0.14748697f, 0.97460106f}};
    const float step = dist / 5.0f;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const float t = ((float)i + 0.5f) * step;
      const float sc = step * ((float)i + 1.0f) / 5.0f;
      const float qx = fmaf(sx, t, px) + K[i][0] * sc;
      const float qy = fmaf(sy, t, py) + K[i][1] * sc;
      const float qz = fmaf(sz, t, pz) + K[i][2] * sc;
      const float a = altitude_from_entry(u, qx, qy, qz, r0, cv, alt, t);
      od += density_light_at<ST, FILT>(u, L, qx, qy, qz, a, cov, type, chk) * step;
    }
    const float tf = dist * 3.0f;
    const float qx = fmaf(sx, tf, px) + K[5][0] * (step * 3.0f);
    const float qy = fmaf(sy, tf, py) + K[5][1] * (step * 3.0f);
    const float qz = fmaf(sz, tf, pz) + K[5][2] * (step * 3.0f);
    const float a = altitude_from_entry(u, qx, qy, qz, r0, cv, alt, tf);
    od += density_light_at<ST, FILT>(u, L, qx, qy, qz, a, cov, type, chk) * step * 3.0f;
    return od;
  }
  const float step = div_near(dist, (float)u.light_steps);
#pragma unroll 1
  for (uint32_t i = 0; i < u.light_steps; ++i) {
    const float t = ((float)i + 0.5f) * step;
    const float qx = fmaf(sx, t, px), qy = fmaf(sy, t, py), qz = fmaf(sz, t, pz);
    const float a = altitude_from_entry(u, qx, qy, qz, r0, cv, alt, t);
    const float term = density_light_at<ST, FILT>(u, L, qx, qy, qz, a, cov, type, chk) * step;
    if (u.kahan) {  // compensated sum
      const float y = term - comp;
      const float tt = od + y;
      comp = (tt - od) - y;
      od = tt;
    } else {
      od += term;
    }
  }
  return od;
}

// The two lookups of a dense sample: transmittance toward the sun
// (cloud_march.wgsl:328-354) and sky-view ambient (:672-700; the zenith angle
// uses atan2(|xz|, y), the well-conditioned form of acos(y) for directions
// near local up).  `bh` = sqrt(max(top^2 - R^2, 0)), `inv_bh` = 1 / max(bh, 1).
struct SunSky {
  float3 sun, sky;
};
__device__ __forceinline__ float horizon_h(const MarchUniforms& u) {
  const float R = u.planet_r, ht = u.atmo_top;
  return sqrtf(fmaxf(ht * ht - R * R, 0.0f));
}
__device__ __forceinline__ SunSky sun_and_sky_at(const MarchUniforms& u, float px, float py, float pz, float sun_az,
                                                 float bh, float inv_bh, int* chk) {
  SunSky out;
  const float R = u.planet_r;
  const float ay = py + R;
  const float len = sqrt_near(__fmaf_rn(pz, pz, __fmaf_rn(px, px, __fmul_rn(ay, ay))));
  const float r = fmaxf(len, R + 1.0f);
  const float inv_len = rcp_near(len), inv_r = r == len ? inv_len : rcp_near(r);
  const float mu = clampf((div_by(px, r, inv_r) * u.sun[0] + div_by(ay, r, inv_r) * u.sun[1]) +
                              div_by(pz, r, inv_r) * u.sun[2], -1.0f, 1.0f);
  const float ratio = div_by(R, r, inv_r);
  const float sin_h = -sqrt_near(fmaxf(1.0f - ratio * ratio, 0.0f));
  if (mu <= sin_h) {
    out.sun = make_float3(0.0f, 0.0f, 0.0f);
  } else {
    const float ht = u.atmo_top;
    const float rho = sqrt_near(fmaxf(r * r - R * R, 0.0f));
    const float disc = r * r * (mu * mu - 1.0f) + ht * ht;
    const float d = fmaxf(-r * mu + sqrt_near(fmaxf(disc, 0.0f)), 0.0f);
    const float d_min = ht - r, d_max = rho + bh;
    const float xm = clamp01(div_near(d - d_min, fmaxf(d_max - d_min, 1.0f)));
    const float xr = div_by(rho, fmaxf(bh, 1.0f), inv_bh);
    const float4 t = lut2d(u.lut_trans, 256, 64, xm, xr, chk, kChkTrans);
    out.sun = make_float3(t.x, t.y, t.z);
  }
  const float ux = div_by(px, len, inv_len), uy = div_by(ay, len, inv_len), uz = div_by(pz, len, inv_len);
  const float vza = atan2f(sqrt_near(ux * ux + uz * uz), uy);
  const float sin_z = clamp01(div_by(R, len, inv_len));
  const float zha = kPi - asinf(sin_z);
  float vv;
  if (vza < zha) {
    vv = sqrt_near(clamp01(div_near(vza, fmaxf(zha, 1e-6f)))) * 0.5f;
  } else {
    const float br = fmaxf(kPi - zha, 1e-6f);
    vv = 0.5f + sqrt_near(clamp01(div_near(vza - zha, br))) * 0.5f;
  }
  const float vaz = atan2f(ux, uz);
  float du = div_by(vaz - sun_az, 2.0f * kPi, 1.0f / (2.0f * kPi));
  du = du - floorf(du);
  const float4 s = lut2d(u.lut_sky, 192, 108, du, vv, chk, kChkSky);
  out.sky = make_float3(s.x * u.sun_illum[0], s.y * u.sun_illum[1], s.z * u.sun_illum[2]);
  return out;
}

}  // namespace
}  // namespace psc
