// probe_sort.cuh -- the spatial probe order of a bake of up to kCountMax probes.
#pragma once

#include "vlb_device.cuh"
#include "vlb_internal.h"

namespace vlbk {

__device__ __forceinline__ uint32_t expand_bits10(uint32_t v) {
  v &= 0x3ffu;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

// Probe order for n <= kCountMax probes in one CTA: a counting sort on the
// top 12 bits of the 24-bit Morton code (16^3 cells inside the bounds) with
// shared-memory histogram, scan and atomic cursors -- a handful of barriers
// instead of the radix sort's dozens.  The order inside a cell follows the
// atomics; the bake's results never depend on the probe order (each ray's
// walk and each probe's sums are independent of its packet), only its speed.
constexpr uint32_t kCountMax = 16384;
constexpr int kCountBins = 4096;

struct ProbeSortShared {
  uint32_t bin[kCountBins], wsum[32];
};

// All T threads (a power of two up to 1024) of a CTA.
template <int T>
__device__ __forceinline__ void probe_sort_count(const float* __restrict__ probes, uint32_t n, float lox, float loy,
                                                 float loz, float sx, float sy, float sz,
                                                 uint32_t* __restrict__ order, ProbeSortShared& sh) {
  constexpr int B = kCountBins / T;  // bins per thread
  uint32_t* bin = sh.bin;
  uint32_t* wsum = sh.wsum;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto cell = [&](uint32_t i) -> uint32_t {
    auto q = [](float c, float lo, float s) -> uint32_t {
      const float v = (c - lo) * s;
      if (!(v > 0.f)) return 0u;
      return min(__float2uint_rz(v), 255u);
    };
    const uint32_t x = q(probes[3 * size_t(i)], lox, sx), y = q(probes[3 * size_t(i) + 1], loy, sy),
                   z = q(probes[3 * size_t(i) + 2], loz, sz);
    return ((expand_bits10(x) << 2) | (expand_bits10(y) << 1) | expand_bits10(z)) >> 12;
  };
  for (uint32_t b = tid; b < kCountBins; b += T) bin[b] = 0;
  __syncthreads();
  for (uint32_t i = tid; i < n; i += T) atomicAdd(&bin[cell(i)], 1u);
  __syncthreads();
  // exclusive scan: B bins per thread, warp shuffles, then the warp totals
  uint32_t v[B], t = 0;
#pragma unroll
  for (int k = 0; k < B; ++k) { v[k] = bin[B * tid + k]; t += v[k]; }
  uint32_t incl = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= uint32_t(o)) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < T / 32 ? wsum[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= uint32_t(o)) wi += y;
    }
    if (lane < T / 32) wsum[lane] = wi - w;
  }
  __syncthreads();
  uint32_t run = wsum[warp] + incl - t;
#pragma unroll
  for (int k = 0; k < B; ++k) { bin[B * tid + k] = run; run += v[k]; }
  __syncthreads();
  for (uint32_t i = tid; i < n; i += T) order[atomicAdd(&bin[cell(i)], 1u)] = i;
}

}  // namespace vlbk
