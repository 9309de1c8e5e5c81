// k_ploc.cu -- the traversal BVH: parallel locally-ordered clustering (PLOC,
// Meister and Bittner 2018, "Parallel Locally-Ordered Clustering for Bounding
// Volume Hierarchy Construction") over the Morton-sorted triangles of the LBVH
// build.  Replaces, like the LBVH, the driver's BLAS/TLAS build
// (src/scene_manager.cpp:339-442); the Karras LBVH stays as the exported,
// bit-exact build, this tree is what the trace kernels walk.
//
// Clusters start as the leaves in Morton order.  Each round:
//   1. every cluster finds its nearest neighbour among the R = 16 clusters on
//      either side, distance = surface area of the union box; ties go to the
//      pair with the smaller (|i - j|, parity of the lower index, lower
//      index) -- a symmetric total order on pairs, so the globally closest
//      pair is always mutual and every round merges at least once, and equal
//      neighbours pair up as (2k, 2k+1) instead of one pair per round;
//   2. mutual nearest neighbours merge into a new internal node (the lower
//      index creates it);
//   3. the surviving clusters are compacted in order (an exclusive scan).
// Internal node ids are handed out from n-2 downwards in creation order, so
// the last merge -- the root -- is node 0.  Every step is deterministic: the
// same triangles give the same tree.
//
// A round is two launches: k_ploc_find (neighbours, flags and their scan inside
// a block) and k_ploc_merge (each block adds up the blocks before it).  The
// cluster count lives on the device, so rounds follow each other without the
// host; once kPlocLast clusters are left, one CTA does all remaining rounds in
// shared memory (k_ploc_last).  58 rounds of 252 k triangles: 1.29 ms of
// kernels and 58 synchronisations before, 0.68 ms and one now.
#include <algorithm>
#include <cmath>

#include "vlb_device.cuh"
#include "vlb_internal.h"

namespace vlbk {

constexpr int kPlocR = 16;
constexpr int kPlocT = 256;
constexpr int kPlocOwn = kPlocT - 2 * kPlocR;  // clusters a block of k_ploc_find owns
constexpr int kPlocLast = 2048;
constexpr uint32_t kPlocScanBlocks = 2048;     // blocks up to which a merge block sums its predecessors itself

struct PlocState {
  uint32_t m;        // clusters
  int32_t next_id;   // next internal node
  uint32_t cur;      // buffer that holds them
  uint32_t round;
  uint32_t stalled;  // 1: max_rounds used up, 2: a round merged nothing
};

__device__ __forceinline__ float union_half_area(const float* a, const float* b) {
  const float dx = fmaxf(a[3], b[3]) - fminf(a[0], b[0]);
  const float dy = fmaxf(a[4], b[4]) - fminf(a[1], b[1]);
  const float dz = fmaxf(a[5], b[5]) - fminf(a[2], b[2]);
  return __fadd_rn(__fadd_rn(__fmul_rn(dx, dy), __fmul_rn(dy, dz)), __fmul_rn(dz, dx));
}

// Cluster i's nearest neighbour among its kPlocR neighbours on either side
// (-1 none); box(j) gives cluster j's box.
template <class F>
__device__ __forceinline__ int ploc_nearest(int i, int m, F box) {
  float bi[6];
  box(i, bi);
  float best = INFINITY;
  int bj = -1;
  for (int o = -kPlocR; o <= kPlocR; ++o) {
    const int j = i + o;
    if (o == 0 || j < 0 || j >= m) continue;
    float b[6];
    box(j, b);
    const float d = union_half_area(bi, b);
    bool take = d < best;
    if (!take && d == best) {  // tie: the pair with the smaller (|i-j|, parity of min, min)
      const int g1 = abs(i - j), g2 = abs(i - bj), lo1 = min(i, j), lo2 = min(i, bj);
      take = g1 < g2 || (g1 == g2 && ((lo1 & 1) < (lo2 & 1) || ((lo1 & 1) == (lo2 & 1) && lo1 < lo2)));
    }
    if (take) { best = d; bj = j; }
  }
  return bj;
}

// Inclusive scan across the warp.
__device__ __forceinline__ uint32_t warp_scan(uint32_t v) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
    if (int(lane) >= o) v += y;
  }
  return v;
}

struct PlocBufs {
  int32_t* cref[2];
  float* cbox[2];
  uint32_t* info;   // per cluster: keep, make, their counts before it in the block, the partner's offset
  uint64_t* sums;   // per block: kept << 32 | made, or the exclusive scan of that
  uint64_t* total;
  int32_t* child;
  float* ibox;
  PlocState* state;  // two slots, by round parity of the launches
};

__device__ __forceinline__ bool ploc_done(const PlocState& st) { return st.m <= kPlocLast || st.stalled; }

// Thread t of block b: cluster b * kPlocOwn - kPlocR + t; the outer kPlocR on
// either side are other blocks' clusters, whose neighbours the owned ones need
// to know whether a pair is mutual.
__global__ void __launch_bounds__(kPlocT) k_ploc_find(const PlocBufs s, int slot, uint32_t max_rounds) {
  const PlocState st = s.state[slot];
  if (ploc_done(st) || st.round > max_rounds) return;
  const int m = int(st.m), base = int(blockIdx.x) * kPlocOwn;
  if (base >= m) return;
  __shared__ float sb[6][kPlocT + 2 * kPlocR];
  __shared__ int16_t snn[kPlocT];
  __shared__ uint32_t swarp[kPlocT / 32];
  const float* cbox = s.cbox[st.cur];
  const int tid = int(threadIdx.x), first = base - 2 * kPlocR;
  for (int t = tid; t < (kPlocT + 2 * kPlocR) * 6; t += kPlocT) {
    const int g = first + t / 6;
    sb[t % 6][t / 6] = g >= 0 && g < m ? cbox[size_t(g) * 6 + t % 6] : 0.f;
  }
  __syncthreads();
  const int i = base - kPlocR + tid;
  int nn = -1;
  if (i >= 0 && i < m)
    nn = ploc_nearest(i, m, [&](int j, float* b) {
#pragma unroll
      for (int k = 0; k < 6; ++k) b[k] = sb[k][j - first];
    });
  snn[tid] = int16_t(nn < 0 ? 0 : nn - i);  // 0: none
  __syncthreads();
  const bool owned = tid >= kPlocR && tid < kPlocR + kPlocOwn && i < m;
  const int off = snn[tid];
  const bool mutual = owned && off != 0 && snn[tid + off] == -off;
  const uint32_t make = mutual && off > 0 ? 1u : 0u, keep = owned && !(mutual && off < 0) ? 1u : 0u;
  const uint32_t v = (keep << 16) | make;
  uint32_t x = warp_scan(v);
  if ((tid & 31) == 31) swarp[tid >> 5] = x;
  __syncthreads();
  x -= v;
  for (int w = 0; w < (tid >> 5); ++w) x += swarp[w];
  // partner offset in bits 18..23 (biased), counts before in 0..7 (made) and 8..15 (kept)
  if (owned)
    s.info[i] = (keep << 17) | (make << 16) | ((x >> 16) << 8) | (x & 255u) | (uint32_t(off + 32) << 18);
  if (tid == kPlocT - 1) {
    const uint32_t t = x + v;
    s.sums[blockIdx.x] = (uint64_t(t >> 16) << 32) | (t & 0xffffu);
  }
}

// One CTA: exclusive scan of the block totals in place, the grand total to
// *total (cluster counts above kPlocScanBlocks blocks only).
__global__ void __launch_bounds__(1024) k_ploc_scan(const PlocBufs s, int slot, uint32_t max_rounds) {
  const PlocState st = s.state[slot];
  const uint32_t nb = (st.m + kPlocOwn - 1) / kPlocOwn;
  if (ploc_done(st) || st.round > max_rounds || nb <= kPlocScanBlocks) return;
  __shared__ uint64_t sh[1024];
  const uint32_t per = (nb + 1023) / 1024, b0 = threadIdx.x * per;
  uint64_t run = 0;
  for (uint32_t k = 0; k < per && b0 + k < nb; ++k) run += s.sums[b0 + k];
  sh[threadIdx.x] = run;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {
    const uint64_t x = threadIdx.x >= unsigned(off) ? sh[threadIdx.x - off] : 0;
    __syncthreads();
    sh[threadIdx.x] += x;
    __syncthreads();
  }
  uint64_t acc = sh[threadIdx.x] - run;
  for (uint32_t k = 0; k < per && b0 + k < nb; ++k) {
    const uint64_t x = s.sums[b0 + k];
    s.sums[b0 + k] = acc;
    acc += x;
  }
  if (threadIdx.x == 1023) *s.total = sh[1023];
}

// Merges the mutual pairs and compacts; the last block writes the next state.
__global__ void __launch_bounds__(kPlocT) k_ploc_merge(const PlocBufs s, int slot, uint32_t max_rounds) {
  const PlocState st = s.state[slot];
  PlocState* nx = s.state + (slot ^ 1);
  if (ploc_done(st) || st.round > max_rounds) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      *nx = st;
      if (!ploc_done(st)) nx->stalled = 1;
    }
    return;
  }
  const uint32_t m = st.m, base = blockIdx.x * kPlocOwn, nb = (m + kPlocOwn - 1) / kPlocOwn;
  if (base >= m) return;
  const int tid = int(threadIdx.x);
  __shared__ uint64_t sred[kPlocT / 32];
  __shared__ uint64_t s_before, s_all;
  if (nb > kPlocScanBlocks) {
    if (tid == 0) { s_before = s.sums[blockIdx.x]; s_all = *s.total; }
  } else {
    uint64_t before = 0, all = 0;
    for (uint32_t k = threadIdx.x; k < nb; k += kPlocT) {
      const uint64_t x = __ldg(s.sums + k);
      if (k < blockIdx.x) before += x;
      all += x;
    }
    // kept and made are both below 2^31 in all: one 64-bit sum each way
    for (int pass = 0; pass < 2; ++pass) {
      uint64_t v = pass ? all : before;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if ((tid & 31) == 0) sred[tid >> 5] = v;
      __syncthreads();
      if (tid == 0) {
        uint64_t t = 0;
        for (int w = 0; w < kPlocT / 32; ++w) t += sred[w];
        (pass ? s_all : s_before) = t;
      }
      __syncthreads();
    }
  }
  __syncthreads();
  if (blockIdx.x == 0 && tid == 0) {
    const uint32_t made = uint32_t(s_all), kept = uint32_t(s_all >> 32);
    *nx = PlocState{kept, st.next_id - int32_t(made), st.cur ^ 1, st.round + 1, 0};
    if (made == 0 || kept + made != m) { nx->m = m; nx->stalled = 2; }
  }
  const uint32_t i = base + threadIdx.x;
  if (tid >= kPlocOwn || i >= m) return;
  const uint32_t f = s.info[i];
  if (!(f >> 17 & 1u)) return;
  const uint32_t dst = uint32_t(s_before >> 32) + (f >> 8 & 255u);
  const float* cbox = s.cbox[st.cur];
  const int32_t* cref = s.cref[st.cur];
  float b[6];
  for (int k = 0; k < 6; ++k) b[k] = cbox[size_t(i) * 6 + k];
  int32_t ref = cref[i];
  if (f >> 16 & 1u) {
    const uint32_t j = uint32_t(int(i) + int(f >> 18 & 63u) - 32);
    const int32_t id = st.next_id - int32_t(uint32_t(s_before) + (f & 255u));
    s.child[2 * size_t(id)] = ref;
    s.child[2 * size_t(id) + 1] = cref[j];
    for (int k = 0; k < 3; ++k) {
      b[k] = fminf(b[k], cbox[size_t(j) * 6 + k]);
      b[3 + k] = fmaxf(b[3 + k], cbox[size_t(j) * 6 + 3 + k]);
    }
    for (int k = 0; k < 6; ++k) s.ibox[size_t(id) * 6 + k] = b[k];
    ref = id;
  }
  s.cref[st.cur ^ 1][dst] = ref;
  for (int k = 0; k < 6; ++k) s.cbox[st.cur ^ 1][size_t(dst) * 6 + k] = b[k];
}

// All remaining rounds of at most kPlocLast clusters, two a thread.
constexpr size_t kPlocLastSmem = size_t(kPlocLast) * (6 * 4 + 4 + 2);
__global__ void __launch_bounds__(kPlocLast / 2) k_ploc_last(const PlocBufs s, int slot, uint32_t max_rounds) {
  extern __shared__ float sm[];
  float* sb = sm;  // [6][kPlocLast]
  int32_t* sr = reinterpret_cast<int32_t*>(sm + 6 * kPlocLast);
  int16_t* snn = reinterpret_cast<int16_t*>(sr + kPlocLast);
  __shared__ uint32_t swarp[2][kPlocLast / 64];
  constexpr int H = kPlocLast / 2;
  PlocState st = s.state[slot];
  if (st.stalled || st.m > kPlocLast) return;
  const int tid = int(threadIdx.x);
  int m = int(st.m);
  for (int i = tid; i < m; i += H) {
    for (int k = 0; k < 6; ++k) sb[k * kPlocLast + i] = s.cbox[st.cur][size_t(i) * 6 + k];
    sr[i] = s.cref[st.cur][i];
  }
  __syncthreads();
  while (m > 1) {
    if (st.round > max_rounds) { st.stalled = 1; break; }
    for (int i = tid; i < m; i += H) {
      const int nn = ploc_nearest(i, m, [&](int j, float* b) {
#pragma unroll
        for (int k = 0; k < 6; ++k) b[k] = sb[k * kPlocLast + j];
      });
      snn[i] = int16_t(nn < 0 ? 0 : nn - i);
    }
    __syncthreads();
    uint32_t v[2], x[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = tid + h * H;
      v[h] = 0;
      if (i < m) {
        const int off = snn[i];
        const bool mutual = off != 0 && snn[i + off] == -off;
        v[h] = (mutual && off < 0 ? 0u : 1u << 16) | (mutual && off > 0 ? 1u : 0u);
      }
      x[h] = warp_scan(v[h]);
      if ((tid & 31) == 31) swarp[h][tid >> 5] = x[h];
    }
    __syncthreads();
    uint32_t total = 0;
    for (int h = 0; h < 2; ++h)
      for (int w = 0; w < H / 32; ++w) {
        const uint32_t t = swarp[h][w];
#pragma unroll
        for (int g = 0; g < 2; ++g)
          if (h < g || (h == g && w < (tid >> 5))) x[g] += t;
        total += t;
      }
    float b[2][6];
    int32_t ref[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = tid + h * H;
      if (!(v[h] >> 16)) continue;
      ref[h] = sr[i];
      for (int k = 0; k < 6; ++k) b[h][k] = sb[k * kPlocLast + i];
      if (v[h] & 1u) {
        const int j = i + snn[i];
        const int32_t id = st.next_id - int32_t((x[h] - v[h]) & 0xffffu);
        s.child[2 * size_t(id)] = ref[h];
        s.child[2 * size_t(id) + 1] = sr[j];
        for (int k = 0; k < 3; ++k) {
          b[h][k] = fminf(b[h][k], sb[k * kPlocLast + j]);
          b[h][3 + k] = fmaxf(b[h][3 + k], sb[(3 + k) * kPlocLast + j]);
        }
        for (int k = 0; k < 6; ++k) s.ibox[size_t(id) * 6 + k] = b[h][k];
        ref[h] = id;
      }
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (!(v[h] >> 16)) continue;
      const int dst = int((x[h] - v[h]) >> 16);
      sr[dst] = ref[h];
      for (int k = 0; k < 6; ++k) sb[k * kPlocLast + dst] = b[h][k];
    }
    const int made = int(total & 0xffffu);
    st.next_id -= made;
    ++st.round;
    m = int(total >> 16);
    if (made == 0) { st.stalled = 2; break; }
    __syncthreads();
  }
  if (tid == 0) {
    st.m = uint32_t(m);
    s.state[0] = st;
    s.state[1] = st;
  }
}

__global__ void k_ploc_init(const float* __restrict__ leaf_box, uint32_t n, const PlocBufs s) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) s.state[0] = PlocState{n, int32_t(n) - 2, 0, 0, 0};
  if (i >= n) return;
  s.cref[0][i] = ~int32_t(i);
  for (int k = 0; k < 6; ++k) s.cbox[0][size_t(i) * 6 + k] = leaf_box[size_t(i) * 6 + k];
}

namespace {
size_t carve(uint32_t n, char* base, PlocBufs* s) {
  size_t off = 0;
  auto take = [&](size_t bytes) { char* p = base ? base + off : nullptr; off += (bytes + 255) & ~size_t(255); return p; };
  for (int k = 0; k < 2; ++k) {
    s->cref[k] = reinterpret_cast<int32_t*>(take(size_t(n) * 4));
    s->cbox[k] = reinterpret_cast<float*>(take(size_t(n) * 24));
  }
  s->info = reinterpret_cast<uint32_t*>(take(size_t(n) * 4));
  s->sums = reinterpret_cast<uint64_t*>(take(size_t(n / kPlocOwn + 2) * 8));
  s->total = reinterpret_cast<uint64_t*>(take(8));
  s->state = reinterpret_cast<PlocState*>(take(2 * sizeof(PlocState)));
  s->child = reinterpret_cast<int32_t*>(take(size_t(2) * n * 4));
  s->ibox = reinterpret_cast<float*>(take(size_t(n) * 24));
  return off;
}
}  // namespace

size_t ploc_scratch_bytes(uint32_t ntris) {
  PlocBufs s;
  return carve(ntris, nullptr, &s);
}

int launch_ploc_build(const float* leaf_box, uint32_t n, const int32_t** child, const float** ibox, void* scratch,
                      cudaStream_t st, int* launches) {
  PlocBufs s;
  carve(n, static_cast<char*>(scratch), &s);
  *child = s.child;
  *ibox = s.ibox;
  if (n < 2) return 0;
  static std::atomic<uint64_t> opted{0};
  smem_opt_in(k_ploc_last, int(kPlocLastSmem), opted);
  uint32_t max_rounds = 64;
  for (uint32_t x = n; x > 1; x >>= 1) max_rounds += 8;
  int L = 0, slot = 0;
  k_ploc_init<<<(n + 255) / 256, 256, 0, st>>>(leaf_box, n, s); ++L;
  uint32_t m = n;
  for (;;) {
    // a round leaves about four fifths of the clusters; rounds past the end do nothing
    const int rounds = m <= kPlocLast ? 0 : int(std::log(double(m) / kPlocLast) / std::log(1.25)) + 3;
    const uint32_t g = (m + kPlocOwn - 1) / kPlocOwn;
    for (int r = 0; r < rounds; ++r) {
      k_ploc_find<<<g, kPlocT, 0, st>>>(s, slot, max_rounds); ++L;
      if (g > kPlocScanBlocks) { k_ploc_scan<<<1, 1024, 0, st>>>(s, slot, max_rounds); ++L; }
      k_ploc_merge<<<g, kPlocT, 0, st>>>(s, slot, max_rounds); ++L;
      slot ^= 1;
    }
    k_ploc_last<<<1, kPlocLast / 2, kPlocLastSmem, st>>>(s, slot, max_rounds); ++L;
    PlocState h{};
    if (cudaMemcpyAsync(&h, s.state + slot, sizeof h, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return -1;
    if (launches) *launches += L;
    L = 0;
    if (h.stalled) return h.stalled == 1 ? 1 : -1;  // 1: degenerate input, the caller keeps the LBVH tree
    if (h.m == 1) return h.next_id == -1 ? 0 : -1;
    m = h.m;
  }
}

}  // namespace vlbk
