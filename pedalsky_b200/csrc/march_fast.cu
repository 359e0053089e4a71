// Single-view FAST march kernel: one thread per ray, CTA tile 16x8 pixels,
// warps as 8x4 pixel tiles, 8 CTAs per SM for the lean form (64 registers:
// more resident warps hide more fetch latency than the few spilled values
// cost), 7 for the others (72 registers: their extra paths spill more) and 5 for
// launches of few CTAs of the Cumulonimbus form.
// One 4K frame under a Cumulonimbus layer, 256 + 8 steps: 9.21 ms in the full
// form, 8.83 in the Cumulonimbus form (8.98 at 8 CTAs per SM, 9.14 at 6), 8.58
// with its profile's plateau tested first.  The per-ray
// body is march_fast_body.cuh.
#include <cuda_runtime.h>
#include <stdint.h>

#include "march_fast_body.cuh"

namespace psc {
namespace {

constexpr int kTileW = 16;
constexpr int kTileH = 8;
constexpr int kThreads = 128;

// The form a march over this uniform block takes: lean without Cumulonimbus
// layers, a cloud-type grid, Kahan sums, cone sampling and lightning; with
// Cumulonimbus as the only one of them its own; full otherwise.  Launches whose
// CTAs are all resident at 7 per SM gain nothing from that many and take the
// Cumulonimbus form compiled for 5 (92 registers, no spills, no plateau branch):
// there one ray's chain of latencies is the time.  256 + 8 steps, form of 7 /
// of 5 per SM: 96x54 560 / 501 us, 240x135 (255 CTAs) 505 / 457, 400x225 (725)
// 520 / 481, 480x270 (1020) 549 / 519; beyond, 560x315 (1400) 576 / 535, 640x360
// (1800) 602 / 654.
constexpr uint32_t kFewCtas = 148 * 7;
int kernel_form(const MarchUniforms& u, const dim3& grid) {
  if (!needs_full_paths(&u, 1)) return kFormLean;
  if (u.type_grid || u.kahan || u.cone || u.lightning_radius > 0.0f) return kFormFull;
  return grid.x * grid.y <= kFewCtas ? kFormCumulonimbusFew : kFormCumulonimbus;
}

// Shared memory per CTA: the entry/exit distances of each of the view's
// layers and kAuxWords more words, per thread (dynamic, sized at launch).
template <int ST, int FILT, int FORM, int LB>
__global__ void __launch_bounds__(kThreads, FORM == kFormLean ? 8 : FORM == kFormCumulonimbusFew ? 5 : 7)
    k_march_fast(const __grid_constant__ MarchUniforms u, const __grid_constant__ ViewDev v) {
  extern __shared__ float s_dyn[];
  const uint32_t nl = u.layer_count;
  float* const s_t0 = s_dyn;
  float* const s_t1 = s_dyn + nl * kThreads;
  float* const s_aux = s_dyn + 2u * nl * kThreads;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t px = blockIdx.x * kTileW + (warp & 1u) * 8u + (lane & 7u);
  const uint32_t py = blockIdx.y * kTileH + (warp >> 1) * 4u + (lane >> 3);
  if (px >= v.width || py >= v.height) return;
  march_pixel_fast<ST, FILT, FORM, false, LB>(u, v, px, py, s_t0, s_t1, s_aux, kThreads, threadIdx.x);
}

// The instrumented build of the same kernel (psc_count_fetches): every
// thread counts the fetches its ray issues, and each warp adds its sums to
// `out` (kTallyKinds 64-bit counters).  Not a timed kernel.
template <int ST, int FILT, int FORM>
__global__ void __launch_bounds__(kThreads) k_march_fast_tally(const __grid_constant__ MarchUniforms u,
                                                               const __grid_constant__ ViewDev v,
                                                               unsigned long long* out) {
  extern __shared__ float s_dyn[];
  const uint32_t nl = u.layer_count;
  float* const s_t0 = s_dyn;
  float* const s_t1 = s_dyn + nl * kThreads;
  float* const s_aux = s_dyn + 2u * nl * kThreads;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t px = blockIdx.x * kTileW + (warp & 1u) * 8u + (lane & 7u);
  const uint32_t py = blockIdx.y * kTileH + (warp >> 1) * 4u + (lane >> 3);
  uint32_t tc[kTallyKinds];
#pragma unroll
  for (uint32_t k = 0; k < kTallyKinds; ++k) tc[k] = 0u;
  if (px < v.width && py < v.height)
    march_pixel_fast<ST, FILT, FORM, true>(u, v, px, py, s_t0, s_t1, s_aux, kThreads, threadIdx.x, tc);
#pragma unroll
  for (uint32_t k = 0; k < kTallyKinds; ++k) {
    const uint32_t sum = __reduce_add_sync(0xffffffffu, tc[k]);
    if (lane == 0 && sum) atomicAdd(out + k, (unsigned long long)sum);
  }
}

template <int ST, int FILT>
cudaError_t launch_fast_tally(const MarchUniforms& u, const ViewDev& v, unsigned long long* out,
                              cudaStream_t s) {
  const dim3 grid((v.width + kTileW - 1) / kTileW, (v.height + kTileH - 1) / kTileH);
  const size_t smem = (2u * u.layer_count + kAuxWords) * kThreads * sizeof(float);
  switch (kernel_form(u, grid)) {
    case kFormLean: k_march_fast_tally<ST, FILT, kFormLean><<<grid, kThreads, smem, s>>>(u, v, out); break;
    case kFormCumulonimbusFew:  // the same fetches
    case kFormCumulonimbus: k_march_fast_tally<ST, FILT, kFormCumulonimbus><<<grid, kThreads, smem, s>>>(u, v, out); break;
    default: k_march_fast_tally<ST, FILT, kFormFull><<<grid, kThreads, smem, s>>>(u, v, out);
  }
  return cudaGetLastError();
}

template <int ST, int FILT, int LB = 0>
cudaError_t launch_fast(const MarchUniforms& u, const ViewDev& v, cudaStream_t s) {
  const dim3 grid((v.width + kTileW - 1) / kTileW, (v.height + kTileH - 1) / kTileH);
  const size_t smem = (2u * u.layer_count + kAuxWords) * kThreads * sizeof(float);
  switch (kernel_form(u, grid)) {
    case kFormLean: k_march_fast<ST, FILT, kFormLean, LB><<<grid, kThreads, smem, s>>>(u, v); break;
    case kFormCumulonimbusFew:
      k_march_fast<ST, FILT, kFormCumulonimbusFew, LB><<<grid, kThreads, smem, s>>>(u, v);
      break;
    case kFormCumulonimbus: k_march_fast<ST, FILT, kFormCumulonimbus, LB><<<grid, kThreads, smem, s>>>(u, v); break;
    default: k_march_fast<ST, FILT, kFormFull, LB><<<grid, kThreads, smem, s>>>(u, v);
  }
  return cudaGetLastError();
}

}  // namespace

int launch_march_fast_tally(const MarchUniforms& u, const ViewDev& v, const PscMarchOptions& o,
                            unsigned long long* counts, cudaStream_t s) {
  if (u.octaves > (uint32_t)kMaxOct || u.octaves == 0) return PSC_ERR_UNSUPPORTED;
  cudaError_t e;
  if (o.storage == PSC_STORAGE_F16 && o.filter == PSC_FILTER_HYBRID)
    e = launch_fast_tally<PSC_STORAGE_F16, PSC_FILTER_HYBRID>(u, v, counts, s);
  else if (o.storage == PSC_STORAGE_F16 && o.filter == PSC_FILTER_EXACT)
    e = launch_fast_tally<PSC_STORAGE_F16, PSC_FILTER_EXACT>(u, v, counts, s);
  else if (o.storage == PSC_STORAGE_U8 && o.filter == PSC_FILTER_HYBRID)
    e = launch_fast_tally<PSC_STORAGE_U8, PSC_FILTER_HYBRID>(u, v, counts, s);
  else if (o.storage == PSC_STORAGE_U8 && o.filter == PSC_FILTER_EXACT)
    e = u.far_texels ? launch_fast_tally<kStorageU8Far, PSC_FILTER_EXACT>(u, v, counts, s)
                     : launch_fast_tally<PSC_STORAGE_U8, PSC_FILTER_EXACT>(u, v, counts, s);
  else
    return PSC_ERR_UNSUPPORTED;
  return e == cudaSuccess ? PSC_OK : PSC_ERR_CUDA;
}

int launch_march_fast(const MarchUniforms& u, const ViewDev& v, const PscMarchOptions& o,
                      cudaStream_t s) {
  if (u.octaves > (uint32_t)kMaxOct || u.octaves == 0) return PSC_ERR_UNSUPPORTED;
  cudaError_t e = cudaErrorInvalidValue;
  if (o.filter == PSC_FILTER_TEXTURE) {
    if (o.storage == PSC_STORAGE_U8) e = launch_fast<PSC_STORAGE_U8, PSC_FILTER_TEXTURE>(u, v, s);
    else if (o.storage == PSC_STORAGE_F16) e = launch_fast<PSC_STORAGE_F16, PSC_FILTER_TEXTURE>(u, v, s);
    else return PSC_ERR_UNSUPPORTED;
  } else if (o.filter == PSC_FILTER_HYBRID) {
    // the light-march fetch batch is chosen for the F16 hybrid form only
    if (o.storage == PSC_STORAGE_U8) e = launch_fast<PSC_STORAGE_U8, PSC_FILTER_HYBRID>(u, v, s);
    else if (o.storage == PSC_STORAGE_F16 && o.light_batch == 2)
      e = launch_fast<PSC_STORAGE_F16, PSC_FILTER_HYBRID, 2>(u, v, s);
    else if (o.storage == PSC_STORAGE_F16 && o.light_batch == 3)
      e = launch_fast<PSC_STORAGE_F16, PSC_FILTER_HYBRID, 3>(u, v, s);
    else if (o.storage == PSC_STORAGE_F16) e = launch_fast<PSC_STORAGE_F16, PSC_FILTER_HYBRID>(u, v, s);
    else return PSC_ERR_UNSUPPORTED;
  } else {
    switch (o.storage) {
      case PSC_STORAGE_U8:
        e = u.far_texels ? launch_fast<kStorageU8Far, PSC_FILTER_EXACT>(u, v, s)
                         : launch_fast<PSC_STORAGE_U8, PSC_FILTER_EXACT>(u, v, s);
        break;
      case PSC_STORAGE_F32: e = launch_fast<PSC_STORAGE_F32, PSC_FILTER_EXACT>(u, v, s); break;
      case PSC_STORAGE_F16: e = launch_fast<PSC_STORAGE_F16, PSC_FILTER_EXACT>(u, v, s); break;
      case PSC_STORAGE_BF16: e = launch_fast<PSC_STORAGE_BF16, PSC_FILTER_EXACT>(u, v, s); break;
      case PSC_STORAGE_FP8: e = launch_fast<PSC_STORAGE_FP8, PSC_FILTER_EXACT>(u, v, s); break;
      default: return PSC_ERR_INVALID_ARGUMENT;
    }
  }
  return e == cudaSuccess ? PSC_OK : PSC_ERR_CUDA;
}

}  // namespace psc
