// Counts where the divisions and roots of march_common.cuh differ from CUDA's
// IEEE ones (tests/test_gpu_near_division.py).
#include <cuda_runtime.h>
#include <stdint.h>

#include "march_common.cuh"

using namespace psc;

namespace {

enum What { kReciprocal, kRoot, kQuotient, kByKnown, kEstimate };

__device__ uint32_t mixed(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return (uint32_t)((z ^ (z >> 31)) >> 16);
}
__device__ float between(uint32_t r, float lo, float hi) { return lo + (hi - lo) * ((float)r * 0x1p-32f); }

// Reciprocals and roots: the n floats from x0's bits on.  Quotients: n pairs
// of operands over the two ranges.
__global__ void k_count(int what, float x0, float x1, float y0, float y1, uint64_t n, unsigned long long* off) {
  unsigned long long bad = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    if (what == kReciprocal || what == kRoot) {
      const float x = __uint_as_float(__float_as_uint(x0) + (uint32_t)i);
      bad += what == kReciprocal ? rcp_near(x) != __frcp_rn(x) : sqrt_near(x) != __fsqrt_rn(x);
      continue;
    }
    const float x = between(mixed(2 * i + 1), x0, x1), y = between(mixed(2 * i + 0x9e3779b97f4a7c15ull), y0, y1);
    const float q = __fdiv_rn(x, y);
    bad += (what == kQuotient ? div_near(x, y) : what == kByKnown ? div_by(x, y, __frcp_rn(y)) : __fmul_rn(x, __frcp_rn(y))) != q;
  }
  if (bad) atomicAdd(off, bad);
}

}  // namespace

extern "C" int count_off(int what, float x0, float x1, float y0, float y1, uint64_t n, uint64_t* off) {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, sizeof(*d)) != cudaSuccess) return 1;
  cudaMemset(d, 0, sizeof(*d));
  k_count<<<148 * 8, 256>>>(what, x0, x1, y0, y1, n, d);
  const bool ok = cudaGetLastError() == cudaSuccess && cudaMemcpy(off, d, sizeof(*d), cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(d);
  return ok ? 0 : 2;
}
