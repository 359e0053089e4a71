// Voxel-grid form of the cloud march and its adjoint.
//
// Density comes from a trilinearly interpolated FP32 voxel grid (cell
// centres, zero outside) instead of the procedural Schneider density; the
// rest is the reference march loop (cloud_march.wgsl:808-1000): the 6-tap
// light march toward the sun (:543-578), Beer-powder and the Hillaire
// octaves (:888-927), the sun transmittance and sky-view ambient LUTs,
// approx-Mie or dual-lobe HG phase, lightning, and the energy-conserving
// step integral.  For differentiability every step contributes (no density
// gate) and the step integral is (1 - e^-x)/x without the 1e-6 floor; no
// aerial perspective is applied.
//
// A sample whose grid value is 0 adds nothing to L and leaves T as it is, so
// the forward march takes its light taps and LUT lookups only where the grid
// is not empty (see `every` in grid_pixel for grids with infinities or NaN).
//
// Adjoint: one thread per ray runs the forward march, evaluates its pixel's
// loss term (I - target)^2 / N with I = L + background * T, then walks the
// steps backwards, carrying the adjoint of the transmittance.  The
// transmittance before a step is exp(-sigma_t * k * prefix), prefix the sum of
// grid value x step over the steps before it: the forward march sums them in
// FP64 and the reverse sweep takes each step's value off again, each held to
// what makes a step opaque (`cap`) so that no value is lost beside a larger one
// (2^-53 of 256 such steps is 1e-11 of optical depth; 1171 us without it, 1173
// with: the bound comes from the host, found per ray it spilled and took 1.4 %
// more).  Neither checkpoints nor a recomputed segment are needed and the L1 has
// no shared memory to make room for (checkpoints and segment buffers in 25.6 KB
// of shared memory per CTA: 1886 us, without: 1668 us; each KB per CTA more cost
// about 20 us).  d loss / d density at the primary sample and d loss / d optical
// depth toward the sun are scattered into the gradient with vector atomic adds
// over the trilinear weights of the primary sample and of the six light taps,
// one 16-byte add per y row (as 8-byte pairs, four per tap, the scatter took 270
// us of 1668; now 90 of 1362).  Loss and d loss / d density_scale are reduced per
// CTA and added in double.
#include <cuda_runtime.h>
#include <stdint.h>

#include "grid_common.cuh"

namespace psc {
namespace {

constexpr int kTileW = 16;
constexpr int kTileH = 8;
constexpr int kThreads = 128;
// The adjoint's CTAs per SM: 512^2 rays, 96 steps, 256x64x256 cells take
// 1362 us at 5 (96 registers) and 1417 us at 6 (80 registers, 112 bytes
// spilled).
constexpr int kAdjointCtas = 5;
// Adds val x the trilinear weights into the gradient quads: one 16-byte
// vector atomic add per y row.  Entries outside the grid collect weight that
// the fold passes over.
template <bool WIDE>
__device__ __forceinline__ void grid_scatter(const GridDev& g, const Cell<WIDE>& c, float val) {
  if (val == 0.0f) return;
  const float z1 = c.wz * val, z0 = (1.0f - c.wz) * val;
  const float x1 = c.wx, x0 = 1.0f - c.wx;
  const float4 q = make_float4(x0 * z0, x0 * z1, x1 * z0, x1 * z1);
  const float wy[2] = {1.0f - c.wy, c.wy};
#pragma unroll
  for (int dy = 0; dy < 2; ++dy)
    if (wy[dy] != 0.0f && (!WIDE || (dy ? c.hi : c.lo)))
      atomicAdd(g.grads + (c.i + (decltype(c.i))(dy ? g.plane : 0)),
                make_float4(wy[dy] * q.x, wy[dy] * q.y, wy[dy] * q.z, wy[dy] * q.w));
}

template <bool WIDE>
__device__ __forceinline__ float light_sum(const MarchUniforms& u, const GridDev& g, const LightGeo& lg, const Sample& p) {
  float s = 0.0f;
  if (lg.poly) {
    // the tap index as a float, in groups of three
    const float n = (float)u.light_steps;
    float j = 0.5f;
#pragma unroll 1
    for (; j + 2.0f < n; j += 3.0f) {
      float v[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) v[k] = grid_fetch<WIDE>(g, grid_cell<WIDE>(g, light_pos(lg, (j + (float)k) * lg.delta)));
      s = ((s + v[0]) + v[1]) + v[2];
    }
#pragma unroll 1
    for (; j < n; j += 1.0f) s += grid_fetch<WIDE>(g, grid_cell<WIDE>(g, light_pos(lg, j * lg.delta)));
  } else {
#pragma unroll 1
    for (uint32_t j = 0; j < u.light_steps; ++j)
      s += grid_fetch<WIDE>(g, grid_cell<WIDE>(g, light_pos_far(u, g, lg, p, ((float)j + 0.5f) * lg.delta)));
  }
  return s * lg.delta;
}

// d loss / d (light sum) of every tap into the gradient.
template <bool WIDE>
__device__ __forceinline__ void light_scatter(const MarchUniforms& u, const GridDev& g, const LightGeo& lg,
                                              const Sample& p, float val) {
#pragma unroll 1
  for (uint32_t j = 0; j < u.light_steps; ++j) {
    const float t = ((float)j + 0.5f) * lg.delta;
    const GridPos q = lg.poly ? light_pos(lg, t) : light_pos_far(u, g, lg, p, t);
    if (grid_touches(g, q)) grid_scatter<WIDE>(g, grid_cell<WIDE>(g, q), val);
  }
}

// (1 - e^-x) / x with e = e^-x.
__device__ __forceinline__ float phi_of(float x, float e) {
  return fabsf(x) < 0.03f ? fmaf(x, fmaf(x, fmaf(x, -1.0f / 24.0f, 1.0f / 6.0f), -0.5f), 1.0f)
                          : __fdividef(1.0f - e, x);
}

// Per-position lighting of one sample: sun factor per channel (illuminance x
// sun transmittance), octave coefficients (a^n x forward gain x phase_n) and
// the ambient + lightning term.
struct Light {
  float sun[3], amb[3], cf[kMaxOct];
};

__device__ __forceinline__ void lighting(const MarchUniforms& u, const LayerConst& L, const float* coef,
                                         bool cb, float cos_theta, float fwd_gain, const Sample& p, Light& l) {
  const float h = clamp01((p.alt - L.base_m) * L.inv_thickness);
  if (cb) {
    const float mt = smoothstepf(0.60f, 0.85f, h);
    const PhaseConst pc = phase_consts_from_d(mixf(L.droplet_um, 50.0f, mt), u.droplet_bias);
#pragma unroll
    for (int n = 0; n < kMaxOct; ++n)
      l.cf[n] = (n < (int)u.octaves) ? u.apow[n] * fwd_gain * phase_with(u, cos_theta, u.cpow[n], pc) : 0.0f;
  } else {
#pragma unroll
    for (int n = 0; n < kMaxOct; ++n) l.cf[n] = coef[n];
  }
  float3 ts, sky;
  lut_lookups(u, p.alt, p.ux, p.uy, p.uz, ts, sky);
  l.sun[0] = u.sun_illum[0] * ts.x;
  l.sun[1] = u.sun_illum[1] * ts.y;
  l.sun[2] = u.sun_illum[2] * ts.z;
  const float ag = mixf(0.3f, 1.0f, h) * u.ambient;
  float lr = 0.0f, lg = 0.0f, lb = 0.0f;
  if (u.lightning_radius > 0.0f) {
    const float ddx = p.x - u.lightning_origin_x, ddz = p.z - u.lightning_origin_z;
    const float fo = clamp01(1.0f - sqrtf(ddx * ddx + ddz * ddz) / u.lightning_radius);
    const float wgt = fo * fo * (3.0f - 2.0f * fo);
    lr = u.lightning_rgb[0] * wgt;
    lg = u.lightning_rgb[1] * wgt;
    lb = u.lightning_rgb[2] * wgt;
  }
  l.amb[0] = fmaf(sky.x, ag, lr);
  l.amb[1] = fmaf(sky.y, ag, lg);
  l.amb[2] = fmaf(sky.z, ag, lb);
}

// In-scatter source X(od) = sun(od) * energy(od) + ambient for channel c,
// and (DERIV) its derivative in the light optical depth.
template <bool DERIV>
__device__ __forceinline__ float source(const MarchUniforms& u, const Light& l, float st, int c, float od,
                                        float* dX) {
  float S = 0.0f, dS = 0.0f, B = 1.0f;
#pragma unroll
  for (int n = 0; n < kMaxOct; ++n) {
    if (n < (int)u.octaves) {
      const float e = __expf(-st * od * u.bpow[n]);
      if (n == 0) B = e;
      S = fmaf(l.cf[n], e, S);
      if (DERIV) dS = fmaf(-l.cf[n] * st * u.bpow[n], e, dS);
    }
  }
  S *= l.sun[c];
  const float P = 1.0f - B * B;  // 1 - exp(-2 * sigma_t * od)
  const float ps = u.powder;
  const float E = fmaf(ps, 2.0f * B * P - B, B);
  if (DERIV) {
    dS *= l.sun[c];
    const float dB = -st * B, dP = 2.0f * st * B * B;
    const float dE = fmaf(ps, 2.0f * (dB * P + B * dP) - dB, dB);
    *dX = fmaf(dS, E, S * dE);
  }
  return fmaf(S, E, l.amb[c]);
}

template <bool ADJ, bool WIDE>
__device__ __forceinline__ void grid_pixel(const MarchUniforms& u, const ViewDev& v, const GridDev& g,
                                           uint32_t px, uint32_t py, float& loss_out, float& dk_out) {
  RaySetup rs;
  setup_ray(u, v, px, py, rs);
  const LayerConst& L = u.layers[0];
  const float dx = rs.dir[0], dy = rs.dir[1], dz = rs.dir[2];
  const float cx = u.cam[0], cy = u.cam[1], cz = u.cam[2];
  const float ray_r0 = rs.r0, ray_cv = rs.cos_view, ray_h0 = rs.h0;
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
  const bool cb = L.cloud_type == 7u && u.phase_mode == PSC_PHASE_APPROX_MIE;
  float coef[kMaxOct];
  {
    const PhaseConst pc{L.g_hg, L.g_d, L.alpha, L.w_d, L.ice};
#pragma unroll
    for (int n = 0; n < kMaxOct; ++n) {
      float ph = 0.0f;
      if (n < (int)u.octaves) {
        ph = u.phase_mode == PSC_PHASE_DUAL_LOBE_HG
                 ? mixf(hg_phase(cos_theta, u.hg_f * u.cpow[n]), hg_phase(cos_theta, u.hg_b * u.cpow[n]), u.hg_w)
                 : (cb ? 0.0f : phase_with(u, cos_theta, u.cpow[n], pc));
      }
      coef[n] = u.apow[n] * fwd_gain * ph;
    }
  }
  const float st[3] = {L.sigma_t[0], L.sigma_t[1], L.sigma_t[2]};
  const float ss[3] = {u.sigma_s[0], u.sigma_s[1], u.sigma_s[2]};

  float Lc[3] = {0.0f, 0.0f, 0.0f}, T[3] = {1.0f, 1.0f, 1.0f};
  const float t0 = rs.t0[0], t1 = rs.t1[0];
  const bool hit = (rs.hit_mask & 1u) && t1 > t0;
  const float step = hit ? __fdividef(t1 - t0, (float)u.cloud_steps) : 0.0f;
  uint32_t n_exec = 0;
  double pre = 0.0;  // adjoint: sum of grid value x step of the executed steps
  auto summed = [&](float gv) { return (double)fminf(fmaxf(gv * step, -g.cap), g.cap); };
  // an infinity or NaN somewhere in the grid reaches L through the light sum
  // of an empty sample (0 x inf), so such a grid has every sample lit
  const bool every = __ldg(g.nonfinite) != 0u;

  auto position = [&](uint32_t s) {
    Sample p;
    const float t = fmaf((float)s + jitter, step, t0);
    p.x = fmaf(dx, t, cx);
    p.y = fmaf(dy, t, cy);
    p.z = fmaf(dz, t, cz);
    p.alt = alt_from(u, p.x, p.y, p.z, ray_r0, ray_cv, ray_h0, t);
    const float inv_r = __frcp_rn(u.planet_r + p.alt);
    p.ux = p.x * inv_r;
    p.uy = (p.y + u.planet_r) * inv_r;
    p.uz = p.z * inv_r;
    return p;
  };

  if (hit) {
    // The grid values of kAhead steps are fetched together, so that an empty
    // stretch waits for one fetch latency per group: forward 512^2 view 295 us
    // one by one, 258 / 261 / 238 / 248 us in groups of 2 / 4 / 6 / 8; adjoint
    // 1362 us one by one, 1320 / 1332 / 1345 us in groups of 2 / 4 / 6.
    constexpr uint32_t kAhead = ADJ ? 2u : 6u;
    n_exec = u.cloud_steps;
    for (uint32_t s0 = 0; s0 < u.cloud_steps; s0 += kAhead) {
      float gvs[kAhead];
      bool any = every;
#pragma unroll
      for (uint32_t k = 0; k < kAhead; ++k) {
        const Sample p = position(s0 + k);
        const float gv = grid_fetch<WIDE>(g, grid_cell<WIDE>(g, grid_pos(g, p.x, p.alt, p.z)));
        gvs[k] = s0 + k < u.cloud_steps ? gv : 0.0f;
        any = any || gvs[k] != 0.0f;
      }
      if (!any) continue;
      bool done = false;
#pragma unroll 1
      for (uint32_t k = 0; k < kAhead; ++k) {
        const uint32_t s = s0 + k;
        float gv = gvs[0];
#pragma unroll
        for (uint32_t j = 1; j < kAhead; ++j) gv = k == j ? gvs[j] : gv;
        if (s >= u.cloud_steps || (gv == 0.0f && !every)) continue;
        const Sample p = position(s);
        const GridPos gp = grid_pos(g, p.x, p.alt, p.z);
        if constexpr (ADJ) pre += summed(gv);
        const LightGeo lg = light_geo(u, g, L, gp, p);
        const float gl = light_sum<WIDE>(u, g, lg, p);
        const float rho = g.k * gv, od = g.k * gl;
        Light l;
        lighting(u, L, coef, cb, cos_theta, fwd_gain, p, l);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float X = source<false>(u, l, st[c], c, od, nullptr);
          const float x = rho * st[c] * step;
          const float e = __expf(-x);
          Lc[c] = fmaf(T[c], rho * ss[c] * X * step * phi_of(x, e), Lc[c]);
          T[c] *= e;
        }
        if (fmaxf(T[0], fmaxf(T[1], T[2])) < g.exit_t) {
          n_exec = s + 1u;
          done = true;
          break;
        }
      }
      if (done) break;
    }
  }

  const size_t idx = (size_t)py * v.width + px;
  const float4 lo = make_float4(Lc[0], Lc[1], Lc[2], 1.0f);
  const float4 to = make_float4(T[0], T[1], T[2], 1.0f);
  if (v.out_l) v.out_l[idx] = lo;
  if (v.out_t) v.out_t[idx] = to;
  if constexpr (!ADJ) {
    if (u.composite && v.hdr) {
      const float4 d = v.hdr[idx];
      v.hdr[idx] = make_float4(fmaf(d.x, to.x, lo.x), fmaf(d.y, to.y, lo.y), fmaf(d.z, to.z, lo.z),
                               fmaf(d.w, to.w, lo.w));
    }
  } else {

  // ---- loss term and reverse sweep ----
  const float4 bgp = __ldg(g.bg + idx), tg = __ldg(g.target + idx);
  const float bgc[3] = {bgp.x, bgp.y, bgp.z}, tgc[3] = {tg.x, tg.y, tg.z};
  float gI[3], lam[3], loss = 0.0f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float d = fmaf(bgc[c], T[c], Lc[c]) - tgc[c];
    loss = fmaf(d * d, g.inv_n, loss);
    gI[c] = 2.0f * d * g.inv_n;
    lam[c] = gI[c] * bgc[c];
  }
  loss_out = loss;
  float dk = 0.0f;
  if (n_exec > 0) {
    float bT[3] = {T[0], T[1], T[2]};  // transmittance before the step
    for (uint32_t s = n_exec; s-- > 0u;) {
      const Sample p = position(s);
      const GridPos gp = grid_pos(g, p.x, p.alt, p.z);
      const Cell<WIDE> cell = grid_cell<WIDE>(g, gp);
      // outside the grid: no gradient, and lam passes unchanged
      const bool in = grid_touches(g, gp);
      if (!in && !every) continue;
      const float gv = grid_fetch<WIDE>(g, cell);
      if (gv != 0.0f || every) {
        pre -= summed(gv);
        const float p_od = g.k * (float)pre;  // optical depth per unit sigma_t before the step
#pragma unroll
        for (int c = 0; c < 3; ++c) bT[c] = __expf(-st[c] * p_od);
      }
      const LightGeo lg = light_geo(u, g, L, gp, p);
      const float gl = light_sum<WIDE>(u, g, lg, p);
      const float rho = g.k * gv, od = g.k * gl;
      Light l;
      lighting(u, L, coef, cb, cos_theta, fwd_gain, p, l);
      float drho = 0.0f, dod = 0.0f;
      float s_lit = 0.0f;
#pragma unroll
      for (int n = 0; n < kMaxOct; ++n) s_lit += l.cf[n];
      if (gv == 0.0f && !every) {
        // rho = 0: e = 1, the step adds nothing to L and lam stays; only
        // the derivative in rho is left
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          // nothing toward the sun either: every exponential is 1
          const float X = od == 0.0f ? fmaf(s_lit * l.sun[c], 1.0f - u.powder, l.amb[c])
                                     : source<false>(u, l, st[c], c, od, nullptr);
          drho = fmaf(gI[c] * bT[c], ss[c] * X * step, drho);
          drho = fmaf(lam[c] * bT[c], -st[c] * step, drho);
        }
        grid_scatter<WIDE>(g, cell, g.k * drho);
        continue;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        float dX;
        const float X = source<true>(u, l, st[c], c, od, &dX);
        const float x = rho * st[c] * step;
        const float e = __expf(-x), ph = phi_of(x, e);
        const float s_int = rho * ss[c] * X * step * ph;
        const float gT = gI[c] * bT[c];
        drho = fmaf(gT, ss[c] * X * step * e, drho);
        drho = fmaf(lam[c] * bT[c], -st[c] * step * e, drho);
        dod = fmaf(gT * rho * ss[c] * step * ph, dX, dod);
        lam[c] = fmaf(lam[c], e, gI[c] * s_int);
      }
      if (in) grid_scatter<WIDE>(g, cell, g.k * drho);
      const float vl = g.k * lg.delta * dod;
      if (vl != 0.0f) light_scatter<WIDE>(u, g, lg, p, vl);
      dk = fmaf(gv, drho, fmaf(gl, dod, dk));
    }
  }
  dk_out = dk;
  }
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// MINB: CTAs per SM the register allocation is bounded for (0: unbounded).
//
// Both forms are bound by instructions and by fetch latency (the grid and its
// gradient stay in L2).  512^2 rays, 96 + 6 steps, 256x64x256 cells at 13 %
// fill: lighting only the samples the grid is not empty at took the forward
// march from 1204 to 338 us (983 M to 181 M warp instructions) and one light
// march per sample instead of two the adjoint from 3759 to 2211 us (2366 M to
// 1557 M); zero-padded arrays without bounds tests, FP32x2 blends and cubic
// tap heights took them to 295 and 1886 us, and the steps named above to 238
// and 1320 us (801 M).
template <bool ADJ, int MINB, bool WIDE>
__global__ void __launch_bounds__(kThreads, MINB) k_grid_march(const __grid_constant__ MarchUniforms u,
                                                               const __grid_constant__ ViewDev v,
                                                               const __grid_constant__ GridDev g) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t px = blockIdx.x * kTileW + (warp & 1u) * 8u + (lane & 7u);
  const uint32_t py = blockIdx.y * kTileH + (warp >> 1) * 4u + (lane >> 3);
  float loss = 0.0f, dk = 0.0f;
  if (px < v.width && py < v.height) grid_pixel<ADJ, WIDE>(u, v, g, px, py, loss, dk);
  if (!ADJ) return;
  __shared__ double s_red[2][kThreads / 32];
  const double ls = warp_sum((double)loss), ks = warp_sum((double)dk);
  if (lane == 0) {
    s_red[0][warp] = ls;
    s_red[1][warp] = ks;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
      a += s_red[0][w];
      b += s_red[1][w];
    }
    atomicAdd(g.loss, a);
    atomicAdd(g.grad_scale, b * (double)g.inv_sigma_bar);
  }
}

// One warp per (yi, zi) row of quads, so no index is divided per quad.  Sets
// *nonfinite when a value is an infinity or NaN.
// Bounded by its writes; 8 blocks per SM (32 registers), as many as are launched,
// keep it one wave: at 34 registers a grid_512 call takes 1 to 3 us more of 240.
__global__ void __launch_bounds__(256, 8) k_grid_quads(const __grid_constant__ GridDev g, float4* __restrict__ q,
                                                    uint32_t* __restrict__ nonfinite) {
  const uint32_t lane = threadIdx.x & 31u, pad = g.pad, sx = g.row, sz = g.nz + 2u * pad - 1u;
  const uint64_t rows = (uint64_t)(g.ny + 2u * g.pad_y) * sz, warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  bool bad = false;
  for (uint64_t row = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < rows; row += warps) {
    const uint32_t yi = (uint32_t)(row / sz), zi = (uint32_t)(row - (uint64_t)yi * sz);
    const uint32_t y = yi - g.pad_y, z = zi - pad, z1 = z + 1u;  // outside: at or above the count (mod 2^32)
    const bool in = y < g.ny, lo = in && z < g.nz, hi = in && z1 < g.nz;
    const float* const a = g.values + ((size_t)(in ? y : 0u) * g.nz + (lo ? z : 0u)) * g.nx;
    const float* const b = g.values + ((size_t)(in ? y : 0u) * g.nz + (hi ? z1 : 0u)) * g.nx;
    float4* const out = q + (size_t)row * sx;
    for (uint32_t xi = lane; xi < sx; xi += 32u) {
      const uint32_t x = xi - pad, x1 = x + 1u;
      const bool l = x < g.nx, r = x1 < g.nx;
      const float4 t = make_float4(lo && l ? __ldg(a + x) : 0.0f, hi && l ? __ldg(b + x) : 0.0f,
                                   lo && r ? __ldg(a + x1) : 0.0f, hi && r ? __ldg(b + x1) : 0.0f);
      bad = bad || !isfinite(t.w);  // every cell is some quad's upper right corner
      out[xi] = t;
    }
  }
  if (bad) *nonfinite = 1u;
}

// grad += the four quad entries of each cell, one warp per (y, z) row.
__global__ void __launch_bounds__(256) k_grid_fold(const __grid_constant__ GridDev g) {
  const uint32_t lane = threadIdx.x & 31u, warps = gridDim.x * (blockDim.x >> 5), rows = g.ny * g.nz;
  for (uint32_t r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += warps) {
    const uint32_t y = r / g.nz, z = r - y * g.nz;
    // quads whose lower z is z, from the one whose upper x is 0
    const float4* const up = g.grads + (size_t)(y + g.pad_y) * g.plane + (size_t)(z + g.pad) * g.row + (g.pad - 1u);
    const float4* const dn = up - g.row;
    float* const out = g.grad + (size_t)r * g.nx;
    for (uint32_t x = lane; x < g.nx; x += 32u)
      out[x] += (__ldg(up + x + 1u).x + __ldg(up + x).z) + (__ldg(dn + x + 1u).y + __ldg(dn + x).w);
  }
}

}  // namespace

int launch_grid_quads(const GridDev& g, float4* quads, uint32_t* nonfinite, cudaStream_t s) {
  if (cudaMemsetAsync(nonfinite, 0, sizeof(uint32_t), s) != cudaSuccess) return PSC_ERR_CUDA;
  k_grid_quads<<<148u * 8u, 256, 0, s>>>(g, quads, nonfinite);
  return cudaGetLastError() == cudaSuccess ? PSC_OK : PSC_ERR_CUDA;
}

int launch_grid_fold(const GridDev& g, cudaStream_t s) {
  k_grid_fold<<<148u * 8u, 256, 0, s>>>(g);
  return cudaGetLastError() == cudaSuccess ? PSC_OK : PSC_ERR_CUDA;
}

int launch_grid_march(const MarchUniforms& u, const ViewDev& v, const GridDev& g, bool adjoint,
                      cudaStream_t s) {
  if (!g.quads || (adjoint && !g.grads)) return PSC_ERR_INVALID_ARGUMENT;
  if (u.octaves == 0 || u.octaves > (uint32_t)kMaxOct) return PSC_ERR_UNSUPPORTED;
  const dim3 grid((v.width + kTileW - 1) / kTileW, (v.height + kTileH - 1) / kTileH);
  const bool wide = g.wide;
  if (adjoint && wide)
    k_grid_march<true, kAdjointCtas, true><<<grid, kThreads, 0, s>>>(u, v, g);
  else if (adjoint)
    k_grid_march<true, kAdjointCtas, false><<<grid, kThreads, 0, s>>>(u, v, g);
  else if (wide)
    k_grid_march<false, 0, true><<<grid, kThreads, 0, s>>>(u, v, g);
  else
    k_grid_march<false, 0, false><<<grid, kThreads, 0, s>>>(u, v, g);
  return cudaGetLastError() == cudaSuccess ? PSC_OK : PSC_ERR_CUDA;
}

}  // namespace psc
