// Noise-volume bakes on the device: base shape 128^3 RGBA8, detail 32^3
// RGBA8, curl 128^2 RG8 (shaders/clouds/noise_base.comp.wgsl,
// noise_detail.comp.wgsl, noise_curl.comp.wgsl), and the conversion of the
// RGBA8 volumes into the march's storage forms.
//
// This file is compiled with -fmad=false: every FP32 operation rounds on its
// own, in the order written, so the output is byte-identical to a CPU bake
// that evaluates the same expressions in IEEE binary32 (division and sqrt are
// IEEE-rounded by default).  WGSL built-ins are spelled out the same way:
// length(v) = sqrt((x*x + y*y) + z*z), normalize(v) = v / length(v),
// mix(a, b, t) = a*(1-t) + b*t, dot = (a.x*b.x + a.y*b.y) + a.z*b.z.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "psc_internal.h"

namespace psc {
namespace {

__device__ __forceinline__ uint32_t hash3(uint32_t x, uint32_t y, uint32_t z) {
  uint32_t h = x * 0x27d4eb2du + y * 0x165667b1u + z * 0x9e3779b9u;
  h = (h ^ (h >> 15)) * 0x2c1b3c6du;
  h = (h ^ (h >> 12)) * 0x297a2d39u;
  return h ^ (h >> 15);
}
__device__ __forceinline__ float unit16(uint32_t h) { return (float)(h & 0xffffu) / 65535.0f; }
__device__ __forceinline__ uint32_t wrapc(int32_t c, int32_t f) {
  return (uint32_t)(((c % f) + f) % f);
}
__device__ __forceinline__ float sq3(float x, float y, float z) {
  const float xx = x * x, yy = y * y, zz = z * z;
  return (xx + yy) + zz;
}
__device__ __forceinline__ float len3(float x, float y, float z) { return sqrtf(sq3(x, y, z)); }
__device__ __forceinline__ float mixw(float a, float b, float t) { return a * (1.0f - t) + b * t; }
__device__ __forceinline__ float fade(float t) {
  return ((t * t) * t) * (t * (t * 6.0f - 15.0f) + 10.0f);
}
__device__ __forceinline__ uint8_t to_unorm8(float v) {
  return (uint8_t)rintf(fminf(fmaxf(v, 0.0f), 1.0f) * 255.0f);
}

// Worley cell noise, 27 neighbours, tileable at `freq` (noise_base:45-70),
// evaluated per texel (the detail volume).  The least distance is the root of
// the least square: the IEEE square root is monotonic.
__device__ float worley(float px, float py, float pz, uint32_t freq, bool detail_offset) {
  const float fq = (float)freq;
  const float sx = px * fq, sy = py * fq, sz = pz * fq;
  const float flx = floorf(sx), fly = floorf(sy), flz = floorf(sz);
  const int32_t cx = (int32_t)flx, cy = (int32_t)fly, cz = (int32_t)flz;
  const float fx = sx - flx, fy = sy - fly, fz = sz - flz;
  const int32_t f = (int32_t)freq;
  float min_sq = 1.0f;
  for (int32_t dz = -1; dz <= 1; ++dz)
    for (int32_t dy = -1; dy <= 1; ++dy)
      for (int32_t dx = -1; dx <= 1; ++dx) {
        uint32_t wx = wrapc(cx + dx, f), wy = wrapc(cy + dy, f), wz = wrapc(cz + dz, f);
        if (detail_offset) {  // noise_detail.comp.wgsl:49
          wx += 73u;
          wy += 19u;
          wz += 41u;
        }
        const float jx = unit16(hash3(wx, wy, wz));
        const float jy = unit16(hash3(wx + 1u, wy, wz));
        const float jz = unit16(hash3(wx, wy + 1u, wz));
        min_sq = fminf(min_sq, sq3(((float)dx + jx) - fx, ((float)dy + jy) - fy, ((float)dz + jz) - fz));
      }
  return fminf(fmaxf(1.0f - sqrtf(min_sq), 0.0f), 1.0f);
}
__device__ __forceinline__ float fbm3(float a, float b, float c) { return (a * 0.625f + b * 0.25f) + c * 0.125f; }

// The base volume's noises read their cells from tables: per frequency the
// jitter of every cell (Worley) and the unit gradient of every corner
// (Perlin), the hashes, divisions and square roots evaluated once per cell
// instead of 27 or 8 times per texel.  The tables repeat one cell past either
// side, so a neighbour needs no wrap.
// Table t: Worley 0..7 (2, 4, 8, 16, 32, 14, 28, 56 cells), Perlin 8..10 (4, 8, 16).
__host__ __device__ constexpr uint32_t table_freq(int t) { return t < 5 ? 2u << t : (t < 8 ? 14u << (t - 5) : 4u << (t - 8)); }
__host__ __device__ constexpr uint32_t table_at(int t) {  // its first cell
  uint32_t n = 0;
  for (int i = 0; i < t; ++i) n += (table_freq(i) + 2u) * (table_freq(i) + 2u) * (table_freq(i) + 2u);
  return n;
}
constexpr uint32_t kTableCells = table_at(11);

__global__ void __launch_bounds__(256) k_noise_cells(float4* __restrict__ cells) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kTableCells) return;
  float4* const out = cells + i;
  uint32_t f = 0, first = 0;
  bool perlin = false;
#pragma unroll
  for (int t = 0; t < 11; ++t)
    if (i >= table_at(t)) {
      first = table_at(t);
      f = table_freq(t);
      perlin = t >= 8;
    }
  i -= first;
  const uint32_t n = f + 2u, x = i % n, y = (i / n) % n, z = i / (n * n);
  const uint32_t wx = wrapc((int32_t)x - 1, (int32_t)f), wy = wrapc((int32_t)y - 1, (int32_t)f),
                 wz = wrapc((int32_t)z - 1, (int32_t)f);
  const float jx = unit16(hash3(wx, wy, wz)), jy = unit16(hash3(wx + 1u, wy, wz)), jz = unit16(hash3(wx, wy + 1u, wz));
  if (!perlin) {
    *out = make_float4(jx, jy, jz, 0.0f);
    return;
  }
  const float vx = jx * 2.0f - 1.0f, vy = jy * 2.0f - 1.0f, vz = jz * 2.0f - 1.0f;
  const float l = len3(vx, vy, vz);
  *out = make_float4(vx / l, vy / l, vz / l, 0.0f);
}

// Cell of a texel coordinate in a table: index of the cell itself, fractions.
struct CellAt {
  const float4* c;
  float fx, fy, fz;
};
template <uint32_t F>
__device__ __forceinline__ CellAt cell_at(const float4* table, float px, float py, float pz) {
  const float sx = px * (float)F, sy = py * (float)F, sz = pz * (float)F;
  const float flx = floorf(sx), fly = floorf(sy), flz = floorf(sz);
  constexpr uint32_t n = F + 2u;
  return {table + (((uint32_t)(int32_t)flz + 1u) * n + (uint32_t)(int32_t)fly + 1u) * n + (uint32_t)(int32_t)flx + 1u,
          sx - flx, sy - fly, sz - flz};
}
template <int T>
__device__ __forceinline__ float worley_cells(const float4* __restrict__ cells, float px, float py, float pz) {
  constexpr uint32_t F = table_freq(T), n = F + 2u;
  const CellAt c = cell_at<F>(cells + table_at(T), px, py, pz);
  float min_sq = 1.0f;
#pragma unroll 1
  for (int32_t dz = -1; dz <= 1; ++dz)
#pragma unroll
    for (int32_t dy = -1; dy <= 1; ++dy)
#pragma unroll
      for (int32_t dx = -1; dx <= 1; ++dx) {
        const float4 j = __ldg(c.c + (dz * (int32_t)(n * n) + dy * (int32_t)n + dx));
        min_sq = fminf(min_sq, sq3(((float)dx + j.x) - c.fx, ((float)dy + j.y) - c.fy, ((float)dz + j.z) - c.fz));
      }
  return fminf(fmaxf(1.0f - sqrtf(min_sq), 0.0f), 1.0f);
}

template <int T>
__device__ __forceinline__ float perlin_cells(const float4* __restrict__ cells, float px, float py, float pz) {  // noise_base:92-115
  constexpr uint32_t F = table_freq(8 + T), n = F + 2u;
  const CellAt c = cell_at<F>(cells + table_at(8 + T), px, py, pz);
  const float ux = fade(c.fx), uy = fade(c.fy), uz = fade(c.fz);
  float dots[8];
#pragma unroll
  for (int iz = 0; iz < 2; ++iz)
#pragma unroll
    for (int iy = 0; iy < 2; ++iy)
#pragma unroll
      for (int ix = 0; ix < 2; ++ix) {
        const float4 g = __ldg(c.c + (iz * (int)(n * n) + iy * (int)n + ix));
        const float ddx = c.fx - (float)ix, ddy = c.fy - (float)iy, ddz = c.fz - (float)iz;
        dots[ix + iy * 2 + iz * 4] = (g.x * ddx + g.y * ddy) + g.z * ddz;
      }
  const float x00 = mixw(dots[0], dots[1], ux), x10 = mixw(dots[2], dots[3], ux);
  const float x01 = mixw(dots[4], dots[5], ux), x11 = mixw(dots[6], dots[7], ux);
  const float y0 = mixw(x00, x10, uy), y1 = mixw(x01, x11, uy);
  return mixw(y0, y1, uz) * 0.5f + 0.5f;
}

// One texel per thread, a warp along x (its lanes share most cells).  Of the
// twelve Worley octaves of the four channels eight differ.  3.13 ms with the
// cells hashed per texel, 0.27 ms from the tables (their own kernel 6 us).
__global__ void __launch_bounds__(128) k_bake_base(const float4* __restrict__ cells, uint8_t* __restrict__ out) {
  const uint32_t x = threadIdx.x, y = blockIdx.x, z = blockIdx.y;  // noise_base.comp.wgsl:124-139
  const float px = ((float)x + 0.5f) / 128.0f, py = ((float)y + 0.5f) / 128.0f, pz = ((float)z + 0.5f) / 128.0f;
  const float p1 = perlin_cells<0>(cells, px, py, pz), p2 = perlin_cells<1>(cells, px, py, pz),
              p3 = perlin_cells<2>(cells, px, py, pz);
  const float perlin = (p1 * 0.5f + p2 * 0.25f) + p3 * 0.125f;
  const float w2 = worley_cells<0>(cells, px, py, pz), w4 = worley_cells<1>(cells, px, py, pz);
  const float w8 = worley_cells<2>(cells, px, py, pz), w16 = worley_cells<3>(cells, px, py, pz);
  const float w32 = worley_cells<4>(cells, px, py, pz), w14 = worley_cells<5>(cells, px, py, pz);
  const float w28 = worley_cells<6>(cells, px, py, pz), w56 = worley_cells<7>(cells, px, py, pz);
  const float a = fbm3(w4, w8, w16) - 1.0f;
  const float pw = fminf(fmaxf(0.0f + ((perlin - a) * (1.0f - 0.0f)) / fmaxf(1.0f - a, 1e-5f), 0.0f), 1.0f);
  uchar4 t;
  t.x = to_unorm8(pw);
  t.y = to_unorm8(fbm3(w2, w4, w8));
  t.z = to_unorm8(fbm3(w8, w16, w32));
  t.w = to_unorm8(fbm3(w14, w28, w56));
  reinterpret_cast<uchar4*>(out)[(z * 128u + y) * 128u + x] = t;
}

__global__ void k_bake_detail(uint8_t* __restrict__ out) {  // noise_detail.comp.wgsl:62-72
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
  const uint32_t z = blockIdx.z * blockDim.z + threadIdx.z;
  if (x >= 32u || y >= 32u || z >= 32u) return;
  const float px = ((float)x + 0.5f) / 32.0f, py = ((float)y + 0.5f) / 32.0f,
              pz = ((float)z + 0.5f) / 32.0f;
  float w[6];  // frequencies 2, 4, .. 64: of the nine octaves of the channels six differ
#pragma unroll 1
  for (uint32_t k = 0; k < 6u; ++k) w[k] = worley(px, py, pz, 2u << k, true);
  uchar4 t;
  t.x = to_unorm8(fbm3(w[0], w[1], w[2]));
  t.y = to_unorm8(fbm3(w[2], w[3], w[4]));
  t.z = to_unorm8(fbm3(w[3], w[4], w[5]));
  t.w = 0;
  reinterpret_cast<uchar4*>(out)[(z * 32u + y) * 32u + x] = t;
}

__device__ __forceinline__ uint32_t hash2(uint32_t x, uint32_t y) {
  uint32_t h = x * 0x27d4eb2du + y * 0x165667b1u;
  h = (h ^ (h >> 15)) * 0x2c1b3c6du;
  h = (h ^ (h >> 12)) * 0x297a2d39u;
  return h ^ (h >> 15);
}

__device__ float perlin2(float px, float py, uint32_t freq) {  // noise_curl.comp.wgsl:36-56
  const float fq = (float)freq;
  const float sx = px * fq, sy = py * fq;
  const float flx = floorf(sx), fly = floorf(sy);
  const int32_t cx = (int32_t)flx, cy = (int32_t)fly;
  const float fx = sx - flx, fy = sy - fly;
  const float ux = fade(fx), uy = fade(fy);
  const int32_t f = (int32_t)freq;
  float d[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int ox = k & 1, oy = k >> 1;
    const uint32_t wx = wrapc(cx + ox, f), wy = wrapc(cy + oy, f);
    const float rx = (float)(hash2(wx, wy) & 0xffffu) / 65535.0f * 2.0f - 1.0f;
    const float ry = (float)(hash2(wx + 1u, wy) & 0xffffu) / 65535.0f * 2.0f - 1.0f;
    const float l = sqrtf(rx * rx + ry * ry);
    d[k] = (rx / l) * (fx - (float)ox) + (ry / l) * (fy - (float)oy);
  }
  const float x0 = mixw(d[0], d[1], ux), x1 = mixw(d[2], d[3], ux);
  return mixw(x0, x1, uy);
}

__device__ __forceinline__ float potential(float x, float y) {
  return perlin2(x, y, 4u) + 0.5f * perlin2(x, y, 8u);
}

__global__ void k_bake_curl(uint8_t* __restrict__ out) {  // noise_curl.comp.wgsl:62-74
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= 128u || y >= 128u) return;
  const float px = ((float)x + 0.5f) / 128.0f, py = ((float)y + 0.5f) / 128.0f;
  const float eps = 1.0f / 128.0f;
  const float dpdx = (potential(px + eps, py + 0.0f) - potential(px - eps, py - 0.0f)) / (2.0f * eps);
  const float dpdy = (potential(px + 0.0f, py + eps) - potential(px - 0.0f, py - eps)) / (2.0f * eps);
  const float cx = dpdy, cy = -dpdx;
  out[(y * 128u + x) * 2u + 0u] = to_unorm8(fminf(fmaxf(cx * 0.5f + 0.5f, 0.0f), 1.0f));
  out[(y * 128u + x) * 2u + 1u] = to_unorm8(fminf(fmaxf(cy * 0.5f + 0.5f, 0.0f), 1.0f));
}

// RGBA8 texels -> storage form.  F16/BF16 hold the byte value itself
// (integers 0..255 are exact in both); FP8 e4m3 holds v/255 * fp8_scale.
__global__ void k_convert(const uint32_t* __restrict__ src, void* __restrict__ dst, uint32_t n,
                          int storage, float fp8_scale) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t w = src[i];
  const float c[4] = {(float)(w & 0xffu), (float)((w >> 8) & 0xffu), (float)((w >> 16) & 0xffu),
                      (float)(w >> 24)};
  if (storage == PSC_STORAGE_F32) {
    reinterpret_cast<float4*>(dst)[i] =
        make_float4(c[0] / 255.0f, c[1] / 255.0f, c[2] / 255.0f, c[3] / 255.0f);
  } else if (storage == PSC_STORAGE_F16) {
    __half2 a = __floats2half2_rn(c[0], c[1]), b = __floats2half2_rn(c[2], c[3]);
    uint2 o;
    o.x = *reinterpret_cast<uint32_t*>(&a);
    o.y = *reinterpret_cast<uint32_t*>(&b);
    reinterpret_cast<uint2*>(dst)[i] = o;
  } else if (storage == PSC_STORAGE_BF16) {
    __nv_bfloat162 a = __floats2bfloat162_rn(c[0], c[1]), b = __floats2bfloat162_rn(c[2], c[3]);
    uint2 o;
    o.x = *reinterpret_cast<uint32_t*>(&a);
    o.y = *reinterpret_cast<uint32_t*>(&b);
    reinterpret_cast<uint2*>(dst)[i] = o;
  } else if (storage == PSC_STORAGE_FP8) {
    uint32_t o = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const __nv_fp8_e4m3 q(c[k] / 255.0f * fp8_scale);
      o |= (uint32_t)(*reinterpret_cast<const uint8_t*>(&q)) << (8 * k);
    }
    reinterpret_cast<uint32_t*>(dst)[i] = o;
  } else {
    reinterpret_cast<uint32_t*>(dst)[i] = w;
  }
}

// Channel-folded FP16 forms of the noise volumes, read by the FAST schedule.
// The march uses the base volume only through R and the low-frequency fbm
// 0.625 G + 0.25 B + 0.125 A, and the detail volume only through
// 0.625 R + 0.25 G + 0.125 B (cloud_march.wgsl:463-470, 512-515).  Filtering
// is linear, so filtering the folded channel equals folding the filtered
// channels.  On bytes the folds are integers: base (R, 5G + 2B + A) and
// detail 5R + 2G + B, at most 2040, which FP16 holds exactly; the kernels
// rescale by 1/255 and 1/2040 after filtering.
//   fold: one texel per entry (source of the texture arrays);
//   quad: the 2x2 footprint (x, x+1) x (y, y+1) of slab z, repeat-wrapped,
//         per entry, so an exact trilinear tap is one load per slab.
__device__ __forceinline__ uint32_t fold_base_texel(uint32_t w) {
  const uint32_t r = w & 0xffu, g = (w >> 8) & 0xffu, b = (w >> 16) & 0xffu, a = w >> 24;
  const __half2 h = __floats2half2_rn((float)r, (float)(5u * g + 2u * b + a));
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t fold_detail_texel(uint32_t w) {
  const uint32_t r = w & 0xffu, g = (w >> 8) & 0xffu, b = (w >> 16) & 0xffu;
  return __half_as_ushort(__float2half_rn((float)(5u * r + 2u * g + b)));
}

template <uint32_t N>
__global__ void k_fold_base(const uint32_t* __restrict__ src, uint32_t* __restrict__ fold,
                            uint4* __restrict__ quad) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N * N * N) return;
  const uint32_t x = i % N, y = (i / N) % N, z = i / (N * N);
  const uint32_t x1 = (x + 1u) & (N - 1u), y1 = (y + 1u) & (N - 1u);
  const uint32_t row0 = (z * N + y) * N, row1 = (z * N + y1) * N;
  fold[i] = fold_base_texel(src[i]);
  quad[i] = make_uint4(fold_base_texel(src[row0 + x]), fold_base_texel(src[row0 + x1]),
                       fold_base_texel(src[row1 + x]), fold_base_texel(src[row1 + x1]));
}

template <uint32_t N>
__global__ void k_fold_detail(const uint32_t* __restrict__ src, uint16_t* __restrict__ fold,
                              uint2* __restrict__ quad) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N * N * N) return;
  const uint32_t x = i % N, y = (i / N) % N, z = i / (N * N);
  const uint32_t x1 = (x + 1u) & (N - 1u), y1 = (y + 1u) & (N - 1u);
  const uint32_t row0 = (z * N + y) * N, row1 = (z * N + y1) * N;
  fold[i] = (uint16_t)fold_detail_texel(src[i]);
  quad[i] = make_uint2(fold_detail_texel(src[row0 + x]) | (fold_detail_texel(src[row0 + x1]) << 16),
                       fold_detail_texel(src[row1 + x]) | (fold_detail_texel(src[row1 + x1]) << 16));
}

// RGBA8 volume (n^3, n a power of two) as the 2x2 (x, y) footprint of slab z
// per entry, repeat-wrapped: a trilinear tap is two 16-byte loads instead of
// eight 4-byte ones (the exact FAST march of an 853x479 view, two layers, 192
// steps: 3.12 -> 2.41 ms).
__global__ void k_quads_u8(const uint32_t* __restrict__ src, uint4* __restrict__ quad, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * n * n) return;
  const uint32_t x = i & (n - 1u), y = (i / n) & (n - 1u), slab = i - (y * n + x);
  const uint32_t x1 = (x + 1u) & (n - 1u), y1 = (y + 1u) & (n - 1u);
  const uint32_t* const s = src + slab;
  quad[i] = make_uint4(s[y * n + x], s[y * n + x1], s[y1 * n + x], s[y1 * n + x1]);
}

// Curl tile (128^2 RG8) as 2x2 quads of (R, G) half pairs, repeat-wrapped:
// a bilinear curl tap is one 16-byte load.  Bytes are exact in FP16.
__global__ void k_curl_quads(const uint16_t* __restrict__ src, uint4* __restrict__ quad) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 128u * 128u) return;
  const uint32_t x = i & 127u, y = i >> 7, x1 = (x + 1u) & 127u, y1 = (y + 1u) & 127u;
  auto pair = [&](uint32_t xx, uint32_t yy) {
    const uint32_t t = src[yy * 128u + xx];
    const __half2 h = __floats2half2_rn((float)(t & 0xffu), (float)(t >> 8));
    return *reinterpret_cast<const uint32_t*>(&h);
  };
  quad[i] = make_uint4(pair(x, y), pair(x1, y), pair(x, y1), pair(x1, y1));
}

}  // namespace

int launch_curl_quads(const uint8_t* curl, uint4* quad, cudaStream_t s) {
  k_curl_quads<<<128u * 128u / 256u, 256, 0, s>>>(reinterpret_cast<const uint16_t*>(curl), quad);
  return cudaGetLastError() == cudaSuccess ? PSC_OK : PSC_ERR_CUDA;
}

int launch_quads_u8(const uint8_t* src, uint4* quad, uint32_t n, cudaStream_t s) {
  k_quads_u8<<<(n * n * n + 255u) / 256u, 256, 0, s>>>(reinterpret_cast<const uint32_t*>(src), quad, n);
  return cudaGetLastError() == cudaSuccess ? PSC_OK : PSC_ERR_CUDA;
}

int launch_fold_storage(const uint8_t* base_u8, const uint8_t* detail_u8, uint32_t* base_fold,
                        uint4* base_quad, uint16_t* detail_fold, uint2* detail_quad, cudaStream_t s) {
  k_fold_base<128><<<128u * 128u * 128u / 256u, 256, 0, s>>>(
      reinterpret_cast<const uint32_t*>(base_u8), base_fold, base_quad);
  k_fold_detail<32><<<32u * 32u * 32u / 256u, 256, 0, s>>>(
      reinterpret_cast<const uint32_t*>(detail_u8), detail_fold, detail_quad);
  return cudaGetLastError() == cudaSuccess ? PSC_OK : PSC_ERR_CUDA;
}

size_t noise_cells_bytes() { return kTableCells * sizeof(float4); }

int launch_noise_bakes(float4* cells, uint8_t* base, uint8_t* detail, uint8_t* curl, cudaStream_t s) {
  k_noise_cells<<<(kTableCells + 255u) / 256u, 256, 0, s>>>(cells);
  k_bake_base<<<dim3(128, 128), 128, 0, s>>>(cells, base);
  k_bake_detail<<<dim3(8, 8, 8), dim3(4, 4, 4), 0, s>>>(detail);
  k_bake_curl<<<dim3(16, 16), dim3(8, 8), 0, s>>>(curl);
  return cudaGetLastError() == cudaSuccess ? PSC_OK : PSC_ERR_CUDA;
}

int launch_convert_storage(const uint8_t* src, void* dst, uint32_t n_texels, int storage,
                           float fp8_scale, cudaStream_t s) {
  k_convert<<<(n_texels + 255) / 256, 256, 0, s>>>(reinterpret_cast<const uint32_t*>(src), dst,
                                                    n_texels, storage, fp8_scale);
  return cudaGetLastError() == cudaSuccess ? PSC_OK : PSC_ERR_CUDA;
}

}  // namespace psc
