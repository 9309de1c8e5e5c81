// k_scene.cu -- device passes of a scene load around the tree builds
// (src/scene_manager.cpp:214-217, 339-442, 496-506): geometry checks and
// bounds, and the traversal node layout.
//
// Node layout: siblings in one 128-byte line.  A walk that leaves node N goes
// to one of N's two children, and the lanes of a warp that leave N together go
// to either; both children therefore take slots 2k and 2k + 1 of the 64-byte
// nodes, pair k going to the k-th node (by build index) with an inner child.
// The root has slot 0 and slot 1 stays empty: at most 2n - 2 slots.  Building
// it here replaces a download, a host walk and an upload (252 k triangles: 30 us; the
// whole load with a first small bake 10.4 -> 1.62 ms with it and the device builds).
#include "vlb_device.cuh"
#include "vlb_internal.h"

namespace vlbk {
namespace {

__device__ __forceinline__ uint32_t ordered(float f) {
  const uint32_t u = __float_as_uint(f);
  return u ^ (uint32_t(int32_t(u) >> 31) | 0x80000000u);
}

__global__ void k_check_init(SceneCheck* c) {
  c->bad_index = 0xffffffffu;
  c->bad_vertex = 0xffffffffu;
  c->depth = 0;
  c->area = 0.0;
  for (int a = 0; a < 3; ++a) { c->lo[a] = 0xffffffffu; c->hi[a] = 0; }
}

// Vertex bounds (ordered integers) and the first vertex that is not finite.
__global__ void __launch_bounds__(256) k_check_vertices(const float* __restrict__ pos, uint32_t stride, uint32_t nverts,
                                                        SceneCheck* __restrict__ c) {
  uint32_t lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0, 0, 0};
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nverts; v += gridDim.x * blockDim.x)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float x = __ldg(pos + size_t(v) * stride + a);
      if (!isfinite(x)) atomicMin(&c->bad_vertex, v);
      const uint32_t k = ordered(x);
      lo[a] = min(lo[a], k);
      hi[a] = max(hi[a], k);
    }
  // one atomic per CTA and bound
  __shared__ uint32_t s_lo[3], s_hi[3];
  if (threadIdx.x < 3) { s_lo[threadIdx.x] = 0xffffffffu; s_hi[threadIdx.x] = 0; }
  __syncthreads();
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    lo[a] = __reduce_min_sync(0xffffffffu, lo[a]);
    hi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&s_lo[a], lo[a]);
      atomicMax(&s_hi[a], hi[a]);
    }
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    atomicMin(&c->lo[threadIdx.x], s_lo[threadIdx.x]);
    atomicMax(&c->hi[threadIdx.x], s_hi[threadIdx.x]);
  }
}

// out[i] = idx[i], or 0 where it is out of range (the first such i is kept: the
// load fails, but nothing reads outside the vertices).  out may be idx.
__global__ void __launch_bounds__(256) k_check_indices(const uint32_t* idx, uint64_t n, uint32_t nverts, uint32_t* out,
                                                       SceneCheck* __restrict__ c) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t v = idx[i];
    if (v >= nverts) atomicMin(&c->bad_index, uint32_t(i));
    out[i] = v < nverts ? v : 0u;
  }
}

// ---- node layout ---------------------------------------------------------------
constexpr int kPairT = 256, kPairPer = 4, kPairTile = kPairT * kPairPer;

__device__ __forceinline__ bool has_inner(const int32_t* __restrict__ child, uint32_t i) {
  return child[2 * size_t(i)] >= 0 || child[2 * size_t(i) + 1] >= 0;
}

// Nodes with an inner child per tile of kPairTile nodes.
__global__ void __launch_bounds__(kPairT) k_pair_count(const int32_t* __restrict__ child, uint32_t nodes,
                                                       uint32_t* __restrict__ tiles) {
  const uint32_t i0 = blockIdx.x * kPairTile + threadIdx.x * kPairPer;
  uint32_t c = 0;
  for (uint32_t k = 0; k < kPairPer; ++k) c += i0 + k < nodes && has_inner(child, i0 + k);
  c = __reduce_add_sync(0xffffffffu, c);
  __shared__ uint32_t s[kPairT / 32];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kPairT / 32; ++w) t += s[w];
    tiles[blockIdx.x] = t;
  }
}

// Exclusive scan of the tiles in place, one CTA.
__global__ void __launch_bounds__(1024) k_pair_scan(uint32_t* __restrict__ tiles, uint32_t n) {
  __shared__ uint32_t s[1024];
  const uint32_t per = (n + 1023) / 1024, b0 = threadIdx.x * per;
  uint32_t run = 0;
  for (uint32_t k = 0; k < per && b0 + k < n; ++k) run += tiles[b0 + k];
  s[threadIdx.x] = run;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {
    const uint32_t x = threadIdx.x >= unsigned(off) ? s[threadIdx.x - off] : 0;
    __syncthreads();
    s[threadIdx.x] += x;
    __syncthreads();
  }
  uint32_t acc = s[threadIdx.x] - run;
  for (uint32_t k = 0; k < per && b0 + k < n; ++k) {
    const uint32_t x = tiles[b0 + k];
    tiles[b0 + k] = acc;
    acc += x;
  }
}

// slot[inner child] and parent[inner child] of every node; the root's.
__global__ void __launch_bounds__(kPairT) k_pair_slots(const int32_t* __restrict__ child, uint32_t nodes,
                                                       const uint32_t* __restrict__ tiles,
                                                       uint32_t* __restrict__ slot, int32_t* __restrict__ parent) {
  const uint32_t i0 = blockIdx.x * kPairTile + threadIdx.x * kPairPer, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t own = 0;
  for (uint32_t k = 0; k < kPairPer; ++k) own += i0 + k < nodes && has_inner(child, i0 + k);
  uint32_t x = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (int(lane) >= o) x += y;
  }
  __shared__ uint32_t s[kPairT / 32];
  if (lane == 31) s[warp] = x;
  __syncthreads();
  uint32_t rank = tiles[blockIdx.x] + x - own;
  for (uint32_t w = 0; w < warp; ++w) rank += s[w];
  for (uint32_t k = 0; k < kPairPer; ++k) {
    const uint32_t i = i0 + k;
    if (i >= nodes) break;
    if (i == 0) { slot[0] = 0; parent[0] = -1; }
    const int32_t c0 = child[2 * size_t(i)], c1 = child[2 * size_t(i) + 1];
    if (c0 < 0 && c1 < 0) continue;
    uint32_t at = 2 + 2 * rank++;
    if (c0 >= 0) { slot[c0] = at++; parent[c0] = int32_t(i); }
    if (c1 >= 0) { slot[c1] = at; parent[c1] = int32_t(i); }
  }
}

// Boxes widened by (|x| + scene scale) 2^-20 per bound, so that the box tests
// are conservative: a ray in a box's face plane or grazing its edge still
// enters it, and only the triangle test decides.
__device__ __forceinline__ float wlo(float x, float s) { return __fsub_rn(x, __fmul_rn(__fadd_rn(fabsf(x), s), 0x1p-20f)); }
__device__ __forceinline__ float whi(float x, float s) { return __fadd_rn(x, __fmul_rn(__fadd_rn(fabsf(x), s), 0x1p-20f)); }

// Packs node i into its slot; a node with a leaf child climbs to the root and
// keeps the longest way (walks of more than kLaneStack levels are all "deep").
__global__ void k_pair_pack(const int32_t* __restrict__ child, const float* __restrict__ ibox,
                            const float* __restrict__ leaf_box, uint32_t nodes, const uint32_t* __restrict__ slot,
                            const int32_t* __restrict__ parent, float4* __restrict__ out, SceneCheck* __restrict__ c) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t depth = 0;
  if (i < nodes) {
    const float* r = ibox;  // root = node 0
    const float scale = fmaxf(fmaxf(fmaxf(fabsf(r[0]), fabsf(r[1])), fmaxf(fabsf(r[2]), fabsf(r[3]))),
                              fmaxf(fabsf(r[4]), fabsf(r[5])));
    const int32_t c0 = child[2 * size_t(i)], c1 = child[2 * size_t(i) + 1];
    const float* p0 = c0 >= 0 ? ibox + 6 * size_t(c0) : leaf_box + 6 * size_t(~c0);
    const float* p1 = c1 >= 0 ? ibox + 6 * size_t(c1) : leaf_box + 6 * size_t(~c1);
    float b0[6], b1[6];
    for (int a = 0; a < 3; ++a) {
      b0[a] = wlo(p0[a], scale); b0[3 + a] = whi(p0[3 + a], scale);
      b1[a] = wlo(p1[a], scale); b1[3 + a] = whi(p1[3 + a], scale);
    }
    pack_node(out + 4 * size_t(slot[i]), b0, b1, c0 >= 0 ? int32_t(slot[c0]) : c0, c1 >= 0 ? int32_t(slot[c1]) : c1);
    if (c0 < 0 || c1 < 0)
      for (int32_t p = int32_t(i); p >= 0 && depth <= uint32_t(kLaneStack); p = parent[p]) ++depth;
  }
  depth = __reduce_max_sync(0xffffffffu, depth);
  if ((threadIdx.x & 31) == 0) atomicMax(&c->depth, depth);
}

}  // namespace

void launch_scene_check(const float* pos, uint32_t stride_floats, uint32_t nverts, const uint32_t* idx, uint64_t nidx,
                        uint32_t* idx_out, SceneCheck* c, int num_sms, cudaStream_t s) {
  k_check_init<<<1, 1, 0, s>>>(c);
  const uint32_t cap = uint32_t(num_sms) * 2;
  auto grid = [&](uint64_t n) { return uint32_t(n / 256 + 1 < cap ? n / 256 + 1 : cap); };
  if (nverts) k_check_vertices<<<grid(nverts), 256, 0, s>>>(pos, stride_floats, nverts, c);
  if (nidx) k_check_indices<<<grid(nidx), 256, 0, s>>>(idx, nidx, nverts, idx_out, c);
}

size_t pair_scratch_bytes(uint32_t ntris) {
  return (size_t(ntris) * 2 + (size_t(ntris) + kPairTile - 1) / kPairTile) * 4 + 256;
}

int launch_pair_siblings(const int32_t* child, const float* ibox, const float* leaf_box, uint32_t ntris, float4* out,
                         void* scratch, SceneCheck* c, cudaStream_t s) {
  if (ntris < 2) return 0;
  const uint32_t nodes = ntris - 1, tiles = (nodes + kPairTile - 1) / kPairTile;
  uint32_t* slot = static_cast<uint32_t*>(scratch);
  int32_t* parent = reinterpret_cast<int32_t*>(slot + ntris);
  uint32_t* tile = slot + 2 * size_t(ntris);
  k_pair_count<<<tiles, kPairT, 0, s>>>(child, nodes, tile);
  k_pair_scan<<<1, 1024, 0, s>>>(tile, tiles);
  k_pair_slots<<<tiles, kPairT, 0, s>>>(child, nodes, tile, slot, parent);
  k_pair_pack<<<(nodes + 255) / 256, 256, 0, s>>>(child, ibox, leaf_box, nodes, slot, parent, out, c);
  return 4;
}

}  // namespace vlbk
