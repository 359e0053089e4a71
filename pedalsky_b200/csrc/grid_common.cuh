// The voxel grid as the march kernels read it (grid_march.cu,
// grid_layer_grad.cu): cell coordinates, the padded corner quads
// (GridDev::quads), their trilinear fetch and the light path through them.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "march_fast_body.cuh"

namespace psc {
namespace {

// Grid coordinates (cells, cell centres at whole numbers) of a point.
struct GridPos {
  float x, y, z;
};

__device__ __forceinline__ GridPos grid_pos(const GridDev& g, float x, float alt, float z) {
  return {fmaf(x - g.min_x, g.inv_cell_x, -0.5f), fmaf(alt - g.base, g.inv_cell_y, -0.5f),
          fmaf(z - g.min_z, g.inv_cell_z, -0.5f)};
}

// The eight corners around a point: the index of its quad in the stored
// arrays (GridDev::quads, grads) and the weights of the upper corners.  Each
// coordinate is held to [-2, n].  The narrow arrays hold two layers of zeros
// before the first cell of every axis and two behind the last, so a point
// outside reads zeros without a bounds test; in the wide ones (GridDev::wide)
// a row of corners is read where the grid has it.
template <bool WIDE>
struct Cell {
  std::conditional_t<WIDE, size_t, uint32_t> i;  // quad of the lower y row; the upper is g.plane further on
  float wx, wy, wz;
  bool lo, hi;  // WIDE: the array holds the lower, the upper y row
};

template <bool WIDE>
__device__ __forceinline__ Cell<WIDE> grid_cell(const GridDev& g, const GridPos& p) {
  const float x = fminf(fmaxf(p.x, -2.0f), g.fnx), y = fminf(fmaxf(p.y, -2.0f), g.fny),
              z = fminf(fmaxf(p.z, -2.0f), g.fnz);
  Cell<WIDE> c;
  if constexpr (WIDE) {
    const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    const int64_t ix = (int64_t)fx, iy = (int64_t)fy, iz = (int64_t)fz;
    const bool in = (uint64_t)(ix + 1) <= g.nx && (uint64_t)(iz + 1) <= g.nz;
    c.lo = in && (uint64_t)iy < g.ny;
    c.hi = in && (uint64_t)(iy + 1) < g.ny;
    c.i = (size_t)iy * g.plane + (size_t)(iz + 1) * g.row + (size_t)(ix + 1);
    c.wx = x - fx;
    c.wy = y - fy;
    c.wz = z - fz;
  } else {
    // floor_bits counts from 0x4B400000; g.origin takes that and the two
    // layers before the first cell off all three axes at once (mod 2^32)
    const FloorBits fx = floor_bits(x), fy = floor_bits(y), fz = floor_bits(z);
    c.lo = c.hi = true;
    c.i = fy.i * (uint32_t)g.plane + fz.i * g.row + (fx.i - g.origin);
    c.wx = x - fx.f;
    c.wy = y - fy.f;
    c.wz = z - fz.f;
  }
  return c;
}

// The cell's quads at its lower and upper y.
struct Rows {
  float4 a, b;
};
template <bool WIDE>
__device__ __forceinline__ Rows grid_rows(const GridDev& g, const Cell<WIDE>& c) {
  const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  return {!WIDE || c.lo ? __ldg(g.quads + c.i) : none,
          !WIDE || c.hi ? __ldg(g.quads + (c.i + (decltype(c.i))g.plane)) : none};
}

// Whether a point has a corner inside the grid.  One without has grid value
// 0 whatever the grid holds, so its value has no gradient either.
__device__ __forceinline__ bool grid_touches(const GridDev& g, const GridPos& p) {
  return p.x >= -1.0f && p.x < g.fnx && p.y >= -1.0f && p.y < g.fny && p.z >= -1.0f && p.z < g.fnz;
}

// Trilinear fetch: the four (x, z) corners of a y row come as one 16-byte
// quad, blended as two z lanes (FP32x2); a corner outside adds 0.
template <bool WIDE>
__device__ __forceinline__ float grid_fetch(const GridDev& g, const Cell<WIDE>& c) {
  const float wx0 = 1.0f - c.wx, wy0 = 1.0f - c.wy;
  const float2 x0 = make_float2(wx0, wx0), x1 = make_float2(c.wx, c.wx), wz = make_float2(1.0f - c.wz, c.wz);
  const auto [a, b] = grid_rows<WIDE>(g, c);
  const float2 ha = fma2(x1, make_float2(a.z, a.w), mul2(x0, make_float2(a.x, a.y)));
  const float2 hb = fma2(x1, make_float2(b.z, b.w), mul2(x0, make_float2(b.x, b.y)));
  const float2 v = fma2(mul2(make_float2(c.wy, c.wy), wz), hb, mul2(mul2(make_float2(wy0, wy0), wz), ha));
  return v.x + v.y;
}

// A point of the march: position, altitude and local up.
struct Sample {
  float x, y, z, alt, ux, uy, uz;
};

// Light march of one sample (cloud_march.wgsl:543-578) in grid coordinates:
// x and z are affine along the sun ray, and for light paths up to 20 km the
// altitude is the cubic of march_fast_body.cuh's LightRay (truncation below
// 1e-4 m; with its rounding off by 2.1e-4 m rms, 1.0e-3 at most, over paths of
// all lengths, the geometry's form by 2.2e-4 and 1.25e-3); longer ones take the
// altitude of each tap from the geometry.
struct LightGeo {
  float x, z, kx, kz;    // x + kx t, z + kz t
  float c0, c1, c2, c3;  // y = c0 + t (c1 + t (c2 + t c3))
  float delta;           // metres per tap
  bool poly;
};

__device__ __forceinline__ LightGeo light_geo(const MarchUniforms& u, const GridDev& g, const LayerConst& L,
                                              const GridPos& p, const Sample& q) {
  LightGeo lg;
  const float r0 = u.planet_r + q.alt;
  const float cv = fmaf(q.ux, u.sun[0], fmaf(q.uy, u.sun[1], q.uz * u.sun[2]));
  const float dist = fmaxf((L.top_m - q.alt) * u.inv_cos_sun, 1.0f);
  lg.delta = __fdividef(dist, (float)u.light_steps);
  lg.poly = dist <= 20000.0f;
  const float s2 = fmaf(-cv, cv, 1.0f) * __fdividef(0.5f, r0);
  lg.x = p.x;
  lg.z = p.z;
  lg.kx = u.sun[0] * g.inv_cell_x;
  lg.kz = u.sun[2] * g.inv_cell_z;
  lg.c0 = p.y;
  lg.c1 = cv * g.inv_cell_y;
  lg.c2 = s2 * g.inv_cell_y;
  lg.c3 = -cv * __fdividef(s2, r0) * g.inv_cell_y;
  return lg;
}

__device__ __forceinline__ GridPos light_pos(const LightGeo& lg, float t) {
  return {fmaf(lg.kx, t, lg.x), fmaf(t, fmaf(t, fmaf(t, lg.c3, lg.c2), lg.c1), lg.c0), fmaf(lg.kz, t, lg.z)};
}
// The tap of a path over 20 km.
__device__ __forceinline__ GridPos light_pos_far(const MarchUniforms& u, const GridDev& g, const LightGeo& lg,
                                                 const Sample& p, float t) {
  const float qx = fmaf(u.sun[0], t, p.x), qy = fmaf(u.sun[1], t, p.y), qz = fmaf(u.sun[2], t, p.z);
  const float cv = fmaf(p.ux, u.sun[0], fmaf(p.uy, u.sun[1], p.uz * u.sun[2]));
  const float alt = alt_from(u, qx, qy, qz, u.planet_r + p.alt, cv, p.alt, t);
  return {fmaf(lg.kx, t, lg.x), fmaf(alt - g.base, g.inv_cell_y, -0.5f), fmaf(lg.kz, t, lg.z)};
}

}  // namespace
}  // namespace psc
