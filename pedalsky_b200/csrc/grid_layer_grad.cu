// Gradient of the voxel-grid form's image loss with respect to the layer's
// altitude range: d loss / d base_m and d loss / d top_m of layer 0.
//
// The layer parameters enter the grid march geometrically: the ray's entry
// and exit distances are its intersections with the spheres at planet
// radius + base and + top, the primary samples are spread over that
// interval, the grid spans base..top in altitude (its vertical cell size is
// (top - base) / ny), the light path runs to the layer top, and the ambient
// term depends on the normalised height in the layer.  Every quantity of the
// per-ray march (grid_march.cu) is therefore carried here as a value with its
// two derivatives (forward mode): the entry/exit distances from the FP64
// set-up (dt/dr = r / (t + b) for either root of |o + t d| = r, b = o.d),
// positions and altitudes, the trilinear grid weights, the light taps, the
// transmittance and sky-view LUT lookups (bilinear, FP32 weights, and the
// derivatives of their parameterisations), the octave source and the step
// integral.  Each ray adds 2 (I - target) / N . dI/dtheta to the result, the
// loss being sum((I - target)^2) / N over the viewport, I = L + background T.
// The other layer parameters do not enter the grid form (the grid replaces
// the procedural density that coverage and the shape/detail biases shape);
// d loss / d density_scale comes with the grid gradient from psc_adjoint.
#include <cuda_runtime.h>
#include <stdint.h>

#include "grid_common.cuh"

namespace psc {
namespace {

constexpr int kTileW = 16;
constexpr int kTileH = 8;
constexpr int kThreads = 128;

// A value and its derivatives with respect to the layer's base (a) and top (b).
struct D2 {
  float v, a, b;
};
__device__ __forceinline__ D2 dc(float v) { return {v, 0.0f, 0.0f}; }
__device__ __forceinline__ D2 operator+(D2 x, D2 y) { return {x.v + y.v, x.a + y.a, x.b + y.b}; }
__device__ __forceinline__ D2 operator-(D2 x, D2 y) { return {x.v - y.v, x.a - y.a, x.b - y.b}; }
__device__ __forceinline__ D2 operator-(D2 x) { return {-x.v, -x.a, -x.b}; }
__device__ __forceinline__ D2 operator+(D2 x, float s) { return {x.v + s, x.a, x.b}; }
__device__ __forceinline__ D2 operator-(D2 x, float s) { return {x.v - s, x.a, x.b}; }
__device__ __forceinline__ D2 operator-(float s, D2 x) { return {s - x.v, -x.a, -x.b}; }
__device__ __forceinline__ D2 operator*(D2 x, float s) { return {x.v * s, x.a * s, x.b * s}; }
__device__ __forceinline__ D2 operator*(float s, D2 x) { return {x.v * s, x.a * s, x.b * s}; }
__device__ __forceinline__ D2 operator*(D2 x, D2 y) {
  return {x.v * y.v, fmaf(x.a, y.v, x.v * y.a), fmaf(x.b, y.v, x.v * y.b)};
}
__device__ __forceinline__ D2 operator/(D2 x, D2 y) {
  const float iy = 1.0f / y.v, q = x.v * iy;
  return {q, (x.a - q * y.a) * iy, (x.b - q * y.b) * iy};
}
__device__ __forceinline__ D2 dsqrt(D2 x) {
  const float r = sqrtf(fmaxf(x.v, 0.0f)), k = r > 0.0f ? 0.5f / r : 0.0f;
  return {r, x.a * k, x.b * k};
}
__device__ __forceinline__ D2 dexp(D2 x) {
  const float e = __expf(x.v);
  return {e, x.a * e, x.b * e};
}
__device__ __forceinline__ D2 dmax(D2 x, float m) { return x.v > m ? x : dc(m); }
__device__ __forceinline__ D2 dmax(D2 x, D2 y) { return x.v >= y.v ? x : y; }
__device__ __forceinline__ D2 dmin(D2 x, float m) { return x.v < m ? x : dc(m); }
__device__ __forceinline__ D2 dclamp(D2 x, float lo, float hi) {
  return x.v < lo ? dc(lo) : (x.v > hi ? dc(hi) : x);
}
__device__ __forceinline__ D2 datan01(D2 x) {
  const float k = 1.0f / fmaf(x.v, x.v, 1.0f);
  return {atan01(x.v), x.a * k, x.b * k};
}
// d atan2(y, x) = (x dy - y dx) / (x^2 + y^2); `upper` for y >= 0 as atan2_upper
__device__ __forceinline__ D2 datan2(D2 y, D2 x, bool upper) {
  const float n = fmaf(x.v, x.v, y.v * y.v), k = n > 0.0f ? 1.0f / n : 0.0f;
  return {upper ? atan2_upper(y.v, x.v) : fast_atan2(y.v, x.v), (x.v * y.a - y.v * x.a) * k,
          (x.v * y.b - y.v * x.b) * k};
}
__device__ __forceinline__ D2 dlerp(D2 a, D2 b, D2 t) { return a + (b - a) * t; }

// alt_from (the altitude of a point at distance t along a ray that starts
// at radius r0 with cos(up, dir) = cv and altitude h0), every input carried.
__device__ __forceinline__ D2 alt_from_d(const MarchUniforms& u, D2 qx, D2 qy, D2 qz, D2 r0, D2 cv,
                                         D2 h0, D2 t) {
  const D2 yy = qy + u.planet_r;
  const D2 len = dsqrt(qx * qx + yy * yy + qz * qz);
  const D2 num = t * (2.0f * r0 * cv + t);
  return h0 + num / (r0 + len);
}

// Whether any of a cell's eight corners holds a value: without one the grid
// value and its derivatives are 0.
template <bool WIDE>
__device__ __forceinline__ bool cell_filled(const GridDev& g, const Cell<WIDE>& c) {
  const auto [a, b] = grid_rows<WIDE>(g, c);
  const uint32_t bits = __float_as_uint(a.x) | __float_as_uint(a.y) | __float_as_uint(a.z) | __float_as_uint(a.w) |
                        __float_as_uint(b.x) | __float_as_uint(b.y) | __float_as_uint(b.z) | __float_as_uint(b.w);
  return (bits << 1) != 0u;  // -0 is empty too
}

// Grid value and its slopes along the three cell coordinates.
struct GridSlopes {
  float v, x, y, z;
};
template <bool WIDE>
__device__ __forceinline__ GridSlopes grid_fetch_slopes(const GridDev& g, const GridPos& p) {
  const Cell<WIDE> c = grid_cell<WIDE>(g, p);
  const auto [a, b] = grid_rows<WIDE>(g, c);
  // the quad's lanes are (z, x): 00, 10, 01, 11
  const float a0 = fmaf(c.wz, a.y - a.x, a.x), a1 = fmaf(c.wz, a.w - a.z, a.z);
  const float b0 = fmaf(c.wz, b.y - b.x, b.x), b1 = fmaf(c.wz, b.w - b.z, b.z);
  const float ya = fmaf(c.wx, a1 - a0, a0), yb = fmaf(c.wx, b1 - b0, b0);
  GridSlopes s;
  s.v = fmaf(c.wy, yb - ya, ya);
  s.x = fmaf(c.wy, (b1 - b0) - (a1 - a0), a1 - a0);
  s.y = yb - ya;
  const float za = fmaf(c.wx, (a.w - a.z) - (a.y - a.x), a.y - a.x);
  const float zb = fmaf(c.wx, (b.w - b.z) - (b.y - b.x), b.y - b.x);
  s.z = fmaf(c.wy, zb - za, za);
  return s;
}

// Bilinear clamp-to-edge lookup of the RGB channels of a float4 LUT at
// carried (u, v): the value and, per channel, its derivatives through the
// bilinear weights.
__device__ __forceinline__ void lut2d_d(const float4* lut, int W, int H, D2 uu, D2 vv, D2 out[3]) {
  const D2 x = uu * (float)W - 0.5f, y = vv * (float)H - 0.5f;
  const float fx = floorf(x.v), fy = floorf(y.v);
  const int ix = (int)fx, iy = (int)fy;
  const int x0 = min(max(ix, 0), W - 1), x1 = min(max(ix + 1, 0), W - 1);
  const int y0 = min(max(iy, 0), H - 1), y1 = min(max(iy + 1, 0), H - 1);
  const D2 wx = x - fx, wy = y - fy;
  const float4 t00 = __ldg(lut + y0 * W + x0), t10 = __ldg(lut + y0 * W + x1);
  const float4 t01 = __ldg(lut + y1 * W + x0), t11 = __ldg(lut + y1 * W + x1);
  const float c00[3] = {t00.x, t00.y, t00.z}, c10[3] = {t10.x, t10.y, t10.z};
  const float c01[3] = {t01.x, t01.y, t01.z}, c11[3] = {t11.x, t11.y, t11.z};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const D2 a = dlerp(dc(c00[c]), dc(c10[c]), wx), b = dlerp(dc(c01[c]), dc(c11[c]), wx);
    out[c] = dlerp(a, b, wy);
  }
}

// lut_lookups (march_fast_body.cuh) with every quantity carried: the sun
// transmittance (earth shadow, Bruneton uv) and the sky-view ambient at the
// local up, times the sun illuminance.  Plain FP32-weight LUT loads.
__device__ __forceinline__ void lut_lookups_d(const MarchUniforms& u, D2 alt, D2 ux, D2 uy, D2 uz,
                                              D2 trans[3], D2 sky[3]) {
  const float R = u.planet_r;
  const D2 a0 = dmax(alt, 0.0f);
  const D2 rho0 = dsqrt(a0 * (a0 + 2.0f * R));
  const D2 a = dmax(alt, 1.0f);
  const D2 r = a + R;
  const D2 rho = alt.v >= 1.0f ? rho0 : dc(u.rho_1m);
  const D2 mu = dclamp(ux * u.sun[0] + uy * u.sun[1] + uz * u.sun[2], -1.0f, 1.0f);
  if (mu.v <= -rho.v / r.v) {
    trans[0] = trans[1] = trans[2] = dc(0.0f);
  } else {
    const float top = u.atmo_top;
    const D2 rm = r * mu;
    const D2 disc = rm * rm + (top - r) * (r + top);
    const D2 d = dmax(dsqrt(dmax(disc, 0.0f)) - rm, 0.0f);
    const D2 d_min = top - r, d_max = rho + u.big_h;
    const D2 xm = dclamp((d - d_min) / dmax(d_max - d_min, 1.0f), 0.0f, 1.0f);
    lut2d_d(u.lut_trans, 256, 64, xm, rho * u.inv_big_h, trans);
  }
  const D2 vza = datan2(dsqrt(ux * ux + uz * uz), uy, true);
  const D2 zha = datan01(dmin(rho0 * u.inv_planet_r, 1.0f)) + 1.57079632679f;
  const bool below = vza.v < zha.v;
  const D2 num = below ? vza : vza - zha;
  const D2 den = below ? zha : kPi - zha;
  const D2 vv = dsqrt(dclamp(num / dmax(den, 1e-6f), 0.0f, 1.0f)) * 0.5f + (below ? 0.0f : 0.5f);
  D2 du = (datan2(ux, uz, false) - u.sun_az) * (1.0f / (2.0f * kPi));
  du = du - floorf(du.v);
  lut2d_d(u.lut_sky, 192, 108, du, vv, sky);
#pragma unroll
  for (int c = 0; c < 3; ++c) sky[c] = sky[c] * u.sun_illum[c];
}

// 1 - exp(-x) for x >= 0 without cancellation, with d/dx = exp(-x).
__device__ __forceinline__ D2 one_minus_exp_neg_d(D2 x, float e) {
  const float v = x.v < 0.03f ? x.v * fmaf(x.v, fmaf(x.v, fmaf(x.v, -1.0f / 24.0f, 1.0f / 6.0f), -0.5f), 1.0f)
                              : 1.0f - e;
  return {v, x.a * e, x.b * e};
}

// d entry-or-exit distance / d (base, top) for a distance t of the FP64
// set-up: the sphere it lies on (radius + base or + top) gives
// dt/dr = r / (t + b), b = o.d; t = 0 (inside the layer) or a depth clip
// does not move with the layer.
__device__ __forceinline__ D2 shell_distance(const MarchUniforms& u, const LayerConst& L, const double oc[3],
                                             const double d[3], float t) {
  if (!(t > 0.0f)) return dc(t);
  const double td = (double)t;
  const double px = oc[0] + d[0] * td, py = oc[1] + d[1] * td, pz = oc[2] + d[2] * td;
  const double r = sqrt(px * px + py * py + pz * pz);
  const double b = oc[0] * d[0] + oc[1] * d[1] + oc[2] * d[2];
  const double eb = fabs(r - L.r_bottom), et = fabs(r - L.r_top);
  const double tol = 0.1 + 1e-6 * td;  // float rounding of t
  if (fmin(eb, et) > tol || fabs(td + b) < 1e-9) return dc(t);
  const double k = (eb <= et ? L.r_bottom : L.r_top) / (td + b);
  return eb <= et ? D2{t, (float)k, 0.0f} : D2{t, 0.0f, (float)k};
}

// One ray of the grid march (grid_pixel in grid_march.cu) carried with its
// derivatives; returns this pixel's d loss / d base and d loss / d top.
//
// A grid value's derivatives are its slopes along the three cell coordinates
// times theirs, so the eight weights are not carried.  Samples whose eight
// corners are empty add nothing and are passed over.  The sums cancel (a
// sample near the vertical through the world's origin turns its azimuth fast,
// and slopes jump at cell borders), so positions keep the operations of the
// carried form.  Bound by instructions (164 registers, 3 CTAs per SM): 512^2
// rays, 96 + 6 steps, 256x64x256 cells at 13 % fill 2951 -> 356 us; bounded
// to 128 or 96 registers it spills and takes 362 or 412 us.
template <bool WIDE>
__device__ __forceinline__ void layer_grad_pixel(const MarchUniforms& u, const ViewDev& v, const GridDev& g,
                                                 uint32_t px, uint32_t py, float& d_base, float& d_top) {
  d_base = d_top = 0.0f;
  RaySetup rs;
  setup_ray(u, v, px, py, rs);
  const LayerConst& L = u.layers[0];
  const float dx = rs.dir[0], dy = rs.dir[1], dz = rs.dir[2];
  const float cx = u.cam[0], cy = u.cam[1], cz = u.cam[2];
  const float cos_theta = fmaf(dx, u.sun[0], fmaf(dy, u.sun[1], dz * u.sun[2]));
  const float fwd_gain =
      u.forward_bias > 0.0f ? 1.0f + u.forward_bias * smoothstepf(0.0f, 1.0f, fmaxf(cos_theta, 0.0f))
                            : 1.0f;
  uint32_t sx = (px + v.x_off) & 63u, sy = (py + v.y_off) & 63u;
  if (u.temporal_jitter) {
    const uint32_t ph = u.frame_index & 15u;
    sx = (sx ^ ((ph * 11u + 7u) & 63u)) & 63u;
    sy = (sy ^ ((ph * 23u + 13u) & 63u)) & 63u;
  }
  const float jitter = __ldg(u.blue + sy * 64u + sx);
  float coef[kMaxOct];
  {
    const PhaseConst pc{L.g_hg, L.g_d, L.alpha, L.w_d, L.ice};
#pragma unroll
    for (int n = 0; n < kMaxOct; ++n) {
      float ph = 0.0f;
      if (n < (int)u.octaves)
        ph = u.phase_mode == PSC_PHASE_DUAL_LOBE_HG
                 ? mixf(hg_phase(cos_theta, u.hg_f * u.cpow[n]), hg_phase(cos_theta, u.hg_b * u.cpow[n]), u.hg_w)
                 : phase_with(u, cos_theta, u.cpow[n], pc);
      coef[n] = u.apow[n] * fwd_gain * ph;
    }
  }
  const float st[3] = {L.sigma_t[0], L.sigma_t[1], L.sigma_t[2]};
  const float ss[3] = {u.sigma_s[0], u.sigma_s[1], u.sigma_s[2]};
  const bool hit = (rs.hit_mask & 1u) && rs.t1[0] > rs.t0[0];

  // layer parameters as carried values
  const D2 base = {L.base_m, 1.0f, 0.0f}, top = {L.top_m, 0.0f, 1.0f};
  const D2 thick = top - base;
  const D2 inv_thick = dc(1.0f) / dmax(thick, 1.0f);
  // cells per metre of altitude, ny / (top - base)
  const D2 icy = dc((float)g.ny) / dmax(thick, 1.0f);
  const bool every = __ldg(g.nonfinite) != 0u;  // as in grid_pixel

  D2 Lc[3] = {dc(0.0f), dc(0.0f), dc(0.0f)}, T[3] = {dc(1.0f), dc(1.0f), dc(1.0f)};
  if (hit) {
    const double oc[3] = {(double)u.cam[0], (double)u.cam[1] + u.planet_r_d, (double)u.cam[2]};
    const D2 t0 = shell_distance(u, L, oc, rs.dird, rs.t0[0]);
    const D2 t1 = shell_distance(u, L, oc, rs.dird, rs.t1[0]);
    const D2 step = (t1 - t0) * (1.0f / (float)u.cloud_steps);
    const D2 r0 = dc(rs.r0), cvv = dc(rs.cos_view), h0 = dc(rs.h0);
    constexpr uint32_t kAhead = 4;  // steps whose cells are looked at together, as in grid_pixel
    bool done = false;
    for (uint32_t s0 = 0; s0 < u.cloud_steps && !done; s0 += kAhead) {
      uint32_t todo = 0;
#pragma unroll
      for (uint32_t k = 0; k < kAhead; ++k) {
        // the values of the carried position below, in the same operations:
        // a sample must be looked at in the cell it is evaluated in
        const float t = t0.v + step.v * ((float)(s0 + k) + jitter);
        const float x = t * dx + cx, y = t * dy + cy, z = t * dz + cz, yy = y + u.planet_r;
        const float num = t * (2.0f * rs.r0 * rs.cos_view + t), len = sqrtf(fmaxf(x * x + yy * yy + z * z, 0.0f));
        const float alt = rs.h0 + num * (1.0f / (rs.r0 + len));
        const GridPos q{(x - g.min_x) * g.inv_cell_x - 0.5f, (alt - base.v) * icy.v - 0.5f, (z - g.min_z) * g.inv_cell_z - 0.5f};
        const bool filled = cell_filled<WIDE>(g, grid_cell<WIDE>(g, q));
        todo |= (s0 + k < u.cloud_steps && (filled || every)) ? 1u << k : 0u;
      }
      while (todo) {
        const uint32_t s = s0 + (uint32_t)__ffs((int)todo) - 1u;
        todo &= todo - 1u;
        const D2 t = t0 + step * ((float)s + jitter);
        const D2 p3x = t * dx + cx, p3y = t * dy + cy, p3z = t * dz + cz;
        const D2 alt = alt_from_d(u, p3x, p3y, p3z, r0, cvv, h0, t);
        const D2 inv_r = dc(1.0f) / (alt + u.planet_r);
        const D2 ux = p3x * inv_r, uy = (p3y + u.planet_r) * inv_r, uz = p3z * inv_r;
        // grid value at a point whose altitude is `h`
        auto value = [&](D2 x, D2 h, D2 z) {
          const D2 y = (h - base) * icy - 0.5f;
          const GridSlopes f =
              grid_fetch_slopes<WIDE>(g, GridPos{(x.v - g.min_x) * g.inv_cell_x - 0.5f, y.v, (z.v - g.min_z) * g.inv_cell_z - 0.5f});
          const float kx = f.x * g.inv_cell_x, kz = f.z * g.inv_cell_z;
          return D2{f.v, fmaf(kx, x.a, fmaf(f.y, y.a, kz * z.a)), fmaf(kx, x.b, fmaf(f.y, y.b, kz * z.b))};
        };
        const D2 gv = value(p3x, alt, p3z);
        // light march toward the sun (light_geo / light_sum)
        const D2 lr0 = alt + u.planet_r;
        const D2 lcv = ux * u.sun[0] + uy * u.sun[1] + uz * u.sun[2];
        const D2 delta = dmax((top - alt) * u.inv_cos_sun, 1.0f) * (1.0f / (float)u.light_steps);
        D2 gl = dc(0.0f);
#pragma unroll 1
        for (uint32_t j = 0; j < u.light_steps; ++j) {
          const D2 tj = delta * ((float)j + 0.5f);
          const D2 qx = p3x + tj * u.sun[0], qy = p3y + tj * u.sun[1], qz = p3z + tj * u.sun[2];
          gl = gl + value(qx, alt_from_d(u, qx, qy, qz, lr0, lcv, alt, tj), qz);
        }
        gl = gl * delta;
        const D2 rho = gv * g.k, od = gl * g.k;
        // lighting: sun factor, ambient (+ lightning)
        D2 ts[3], sky[3];
        lut_lookups_d(u, alt, ux, uy, uz, ts, sky);
        const D2 h = dclamp((alt - base) * inv_thick, 0.0f, 1.0f);
        const D2 ag = (h * 0.7f + 0.3f) * u.ambient;
        float lgt[3] = {0.0f, 0.0f, 0.0f};
        D2 lw = dc(0.0f);
        if (u.lightning_radius > 0.0f) {
          const D2 ddx = p3x - u.lightning_origin_x, ddz = p3z - u.lightning_origin_z;
          const D2 fo = dclamp(1.0f - dsqrt(ddx * ddx + ddz * ddz) * (1.0f / u.lightning_radius), 0.0f, 1.0f);
          lw = fo * fo * (3.0f - 2.0f * fo);
          lgt[0] = u.lightning_rgb[0];
          lgt[1] = u.lightning_rgb[1];
          lgt[2] = u.lightning_rgb[2];
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          // source X(od) = sun * Beer-powder * octaves + ambient (grid_march.cu:source)
          D2 S = dc(0.0f), B = dc(1.0f);
#pragma unroll
          for (int n = 0; n < kMaxOct; ++n) {
            if (n < (int)u.octaves) {
              const D2 e = dexp(od * (-st[c] * u.bpow[n]));
              if (n == 0) B = e;
              S = S + e * coef[n];
            }
          }
          S = S * (ts[c] * u.sun_illum[c]);
          const D2 P = 1.0f - B * B;
          const D2 E = B + (B * P * 2.0f - B) * u.powder;
          const D2 X = S * E + sky[c] * ag + lw * lgt[c];
          const D2 x = rho * step * st[c];
          const float e = __expf(-x.v);
          const D2 om = one_minus_exp_neg_d(x, e);  // 1 - exp(-x)
          // the step integral rho ss X step (1 - e^-x) / x = ss X (1 - e^-x) / st
          Lc[c] = Lc[c] + T[c] * X * om * (ss[c] / st[c]);
          T[c] = T[c] * D2{e, -x.a * e, -x.b * e};
        }
        if (fmaxf(T[0].v, fmaxf(T[1].v, T[2].v)) < g.exit_t) {
          done = true;
          break;
        }
      }
    }
  }
  const size_t idx = (size_t)py * v.width + px;
  const float4 bgp = __ldg(g.bg + idx), tg = __ldg(g.target + idx);
  const float bgc[3] = {bgp.x, bgp.y, bgp.z}, tgc[3] = {tg.x, tg.y, tg.z};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const D2 I = Lc[c] + T[c] * bgc[c];
    const float gI = 2.0f * (I.v - tgc[c]) * g.inv_n;
    d_base = fmaf(gI, I.a, d_base);
    d_top = fmaf(gI, I.b, d_top);
  }
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

template <bool WIDE>
__global__ void __launch_bounds__(kThreads) k_grid_layer_grad(const __grid_constant__ MarchUniforms u,
                                                              const __grid_constant__ ViewDev v,
                                                              const __grid_constant__ GridDev g,
                                                              double* out) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t px = blockIdx.x * kTileW + (warp & 1u) * 8u + (lane & 7u);
  const uint32_t py = blockIdx.y * kTileH + (warp >> 1) * 4u + (lane >> 3);
  float db = 0.0f, dt = 0.0f;
  if (px < v.width && py < v.height) layer_grad_pixel<WIDE>(u, v, g, px, py, db, dt);
  __shared__ double s_red[2][kThreads / 32];
  const double sb = warp_sum((double)db), st = warp_sum((double)dt);
  if (lane == 0) {
    s_red[0][warp] = sb;
    s_red[1][warp] = st;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
      a += s_red[0][w];
      b += s_red[1][w];
    }
    atomicAdd(out, a);
    atomicAdd(out + 1, b);
  }
}

}  // namespace

int launch_grid_layer_grad(const MarchUniforms& u, const ViewDev& v, const GridDev& g, double* out,
                           cudaStream_t s) {
  if (!g.quads) return PSC_ERR_INVALID_ARGUMENT;
  if (u.octaves == 0 || u.octaves > (uint32_t)kMaxOct) return PSC_ERR_UNSUPPORTED;
  const dim3 grid((v.width + kTileW - 1) / kTileW, (v.height + kTileH - 1) / kTileH);
  if (g.wide)
    k_grid_layer_grad<true><<<grid, kThreads, 0, s>>>(u, v, g, out);
  else
    k_grid_layer_grad<false><<<grid, kThreads, 0, s>>>(u, v, g, out);
  return cudaGetLastError() == cudaSuccess ? PSC_OK : PSC_ERR_CUDA;
}

}  // namespace psc
