// k_setup.cu -- what a bake prepares before its walks: the probe order, the
// probe frontiers (front.cuh) and the sun map (sun_map.cuh).
//
// One launch does all three for a single bake: they do not depend on each other,
// each is bound by latency, and a small bake is a few launches long (4096 probes
// x 256 directions: 186 us with a launch each, 170 with one).  CTA 0 sorts the probes (bakes of more than
// kCountMax sort them before, launch_probe_order), the next draw the map, the
// rest expand the frontiers, a warp per probe.  Batches launch the frontiers
// and the maps of all jobs.
#include <algorithm>

#include "front.cuh"
#include "probe_sort.cuh"
#include "sun_map.cuh"

namespace vlbk {
namespace {

constexpr int kSetupThreads = 256, kSetupWarps = kSetupThreads / 32;
static_assert(kSetupThreads == kMapThreads, "one CTA draws one slice of a map's triangle group");

union SetupShared {
  MapShared map;
  ProbeSortShared sort;
};

__global__ void __launch_bounds__(kSetupThreads) k_bake_setup(const SetupArgs a) {
  extern __shared__ __align__(16) unsigned char setup_smem[];
  SetupShared& sh = *reinterpret_cast<SetupShared*>(setup_smem);
  uint32_t cta = blockIdx.x;
  if (a.order) {
    if (cta == 0) {
      if (threadIdx.x == 0) *a.zero_word = 0;  // the trace's work counter
      probe_sort_count<kSetupThreads>(a.front.probes, a.front.nprobes, a.lo[0], a.lo[1], a.lo[2], a.s[0], a.s[1],
                                      a.s[2], a.order, sh.sort);
      return;
    }
    --cta;
  }
  if (cta < a.map_ctas) {
    map_draw(a.map, a.tris, a.front.ntris, cta / a.map_slices, int(cta % a.map_slices), int(a.map_slices), sh.map);
    return;
  }
  const uint32_t warp = threadIdx.x >> 5, p = (cta - a.map_ctas) * kSetupWarps + warp;
  if (p < a.front.nprobes)
    front_probe(a.front, p, *reinterpret_cast<FrontShared*>(setup_smem + warp * front_shared_bytes(a.front.cap)));
}

__global__ void __launch_bounds__(kSetupWarps * 32)
    k_probe_front_batch(const BakeJobDev* __restrict__ jobs, uint32_t njobs, uint32_t total, uint32_t cap) {
  extern __shared__ __align__(16) unsigned char setup_smem[];
  const uint32_t warp = threadIdx.x >> 5, w = blockIdx.x * kSetupWarps + warp;
  if (w >= total) return;
  uint32_t lo = 0, hi = njobs - 1;  // the last job that begins at or before w
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (__ldg(&jobs[mid].front_begin) <= w) lo = mid; else hi = mid - 1;
  }
  const BakeJobDev& j = jobs[lo];
  const uint32_t p = w - j.front_begin;
  if (!j.front || p >= j.nprobes) return;
  const FrontArgs a{j.nodes, j.ntris, j.probes, j.nprobes, j.front_scale, j.front_cap, const_cast<float4*>(j.front),
                    const_cast<uint32_t*>(j.front_n), j.err};
  front_probe(a, p, *reinterpret_cast<FrontShared*>(setup_smem + warp * front_shared_bytes(cap)));
}

__global__ void __launch_bounds__(kMapThreads) k_sun_map_batch(const BakeJobDev* __restrict__ jobs, uint32_t njobs) {
  __shared__ MapShared sh;
  uint32_t lo = 0, hi = njobs - 1;  // the last job that begins at or before this CTA
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (__ldg(&jobs[mid].map_begin) <= blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const BakeJobDev& j = jobs[lo];
  const uint32_t c = blockIdx.x - j.map_begin;
  if (!j.sun_map.cells || c / j.map_slices * kMapThreads >= j.ntris) return;
  map_draw(j.sun_map, j.tris, j.ntris, c / j.map_slices, int(c % j.map_slices), int(j.map_slices), sh);
}

}  // namespace

void launch_bake_setup(SetupArgs a, const float bounds[6], cudaStream_t s) {
  for (int k = 0; k < 3; ++k) {
    const float e = bounds[3 + k] - bounds[k];
    a.lo[k] = bounds[k];
    a.s[k] = e > 0.f ? 256.0f / e : 0.f;
  }
  if (a.map.cells) {
    cudaMemsetAsync(a.map.cells, 0, size_t(a.map.G) * a.map.G * 8, s);
    a.map_slices = sun_map_slices(a.front.ntris);
    a.map_ctas = sun_map_ctas(a.front.ntris);
  } else {
    a.map_ctas = 0;
  }
  const uint32_t grid =
      (a.order ? 1u : 0u) + a.map_ctas + (a.front.ent ? (a.front.nprobes + kSetupWarps - 1) / kSetupWarps : 0u);
  if (!grid) return;
  // the frontiers' lists take the most; a launch without them keeps its CTAs small
  const size_t smem = std::max(sizeof(SetupShared), a.front.ent ? kSetupWarps * front_shared_bytes(a.front.cap) : 0);
  static std::atomic<uint64_t> opted{0};
  smem_opt_in(k_bake_setup, int(std::max(sizeof(SetupShared), kSetupWarps * front_shared_bytes(kFrontCap))), opted);
  k_bake_setup<<<grid, kSetupThreads, smem, s>>>(a);
}

uint32_t probe_order_in_setup(uint32_t nprobes) { return nprobes <= kCountMax; }

void launch_probe_front_batch(const BakeJobDev* jobs, uint32_t njobs, uint32_t total, uint32_t cap, cudaStream_t s) {
  if (!total) return;
  static std::atomic<uint64_t> opted{0};
  smem_opt_in(k_probe_front_batch, int(kSetupWarps * front_shared_bytes(kFrontCap)), opted);
  k_probe_front_batch<<<(total + kSetupWarps - 1) / kSetupWarps, kSetupThreads, kSetupWarps * front_shared_bytes(cap),
                        s>>>(jobs, njobs, total, cap);
}

// CTAs per group of triangles: about seven CTAs per SM in all.
uint32_t sun_map_slices(uint32_t ntris) {
  const uint32_t groups = (ntris + kMapThreads - 1) / kMapThreads;
  return std::min(64u, std::max(2u, 1024u / std::max(groups, 1u)));
}

void launch_sun_map_batch(const BakeJobDev* jobs, uint32_t njobs, uint32_t ctas, void* cells, size_t bytes,
                          cudaStream_t s) {
  if (!ctas) return;
  cudaMemsetAsync(cells, 0, bytes, s);
  k_sun_map_batch<<<ctas, kMapThreads, 0, s>>>(jobs, njobs);
}

}  // namespace vlbk
