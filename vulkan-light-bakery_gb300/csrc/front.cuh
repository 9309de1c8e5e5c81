// front.cuh -- probe frontiers: where the rays of one probe enter the
// traversal tree.
//
// All rays of a probe start at one point, so every one of them enters every
// tree node whose box holds that point; in a scene of overlapping boxes that
// is most of a ray's walk (64^3 grid probes, 4096 boxes: 63 of the 87 nodes a
// primary ray tests).  This kernel walks those nodes once per probe: one warp
// expands the tree breadth first from the root wherever the box holds the
// probe, then, while the list is short, the entries that look largest from
// the probe, and lists the boxes and references where the expansion stopped
// (an antichain that covers every triangle), nearest box first.  A lane walk
// tests its ray against that list -- warp-uniform loads, no divergence -- and
// starts from the entries it hits instead of from the root (lr_front).
//
// The boxes written are the tree's own, relative to the probe and widened by
// 2^-20 of the coordinate scale, so a ray enters every entry whose subtree its
// walk from the root would enter with a triangle to hit: its result keeps its
// bits.
//
// Latency bound: some twenty dependent node loads per warp (16 us for 4096
// probes in 778 triangles; 180 us for 32,768 probes in 49,162, 3 % of that bake).
#pragma once

#include "vlb_device.cuh"
#include "vlb_internal.h"

namespace vlbk {

constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ float axis_gap(float lo, float hi, float o) { return fmaxf(fmaxf(lo - o, o - hi), 0.f); }

struct FrontBox {
  float4 a, b;  // [lx ly hx hy] [lz hz ref dist^2]
};

// Child h of node `nd`.
__device__ __forceinline__ FrontBox front_box(const float4* nd, int h) {
  const float4 xy = __ldg(nd + h), z = __ldg(nd + 2), r = __ldg(nd + 3);
  return FrontBox{xy, h ? make_float4(z.z, z.w, r.y, 0.f) : make_float4(z.x, z.y, r.x, 0.f)};
}

// Entries whose box half area exceeds kFrontLarge times the squared distance
// are expanded too, up to kFrontLook entries: with more, a ray group tests
// more boxes than the shorter walks save (16^3 probes x 256 directions, 778
// triangles: 212 us at 10, 223 us without, 234 us at 1; the 4096-box scene,
// whose lists are long already, 11.3 against 11.2 ms with none).
constexpr float kFrontLarge = 10.f;
constexpr int kFrontLook = 32;
constexpr int kFrontRounds = 8;

// Nodes of a level expanded; the rest become entries (16,384 probes in 170,000 boxes,
// lists of 1024: 16.3 ms with 64, 12.2 with 128, 12.7 with 256; fewer boxes alike).
constexpr int kFrontOpen = 128;

// A warp's shared memory: two levels of open nodes (the references of the
// nodes and where they stand), then `cap` entries.  A child is known by its
// parent's slot and its side; its box is read again when the list is written, so
// that an entry is 12 bytes here, not 32, and three times the warps fit.
struct FrontShared {
  int ref[2][kFrontOpen];
  uint32_t src[2][kFrontOpen];  // 2 * parent + side
};
inline __host__ __device__ size_t front_shared_bytes(uint32_t cap) { return sizeof(FrontShared) + size_t(cap) * 12; }
constexpr uint32_t kFrontWide = 1u << 31;  // in an entry's src: looks large from the probe

struct FrontList {
  uint32_t* src;
  int* ref;
  float* d2;
  __device__ __forceinline__ void put(int i, uint32_t s, int r, float d) const { src[i] = s; ref[i] = r; d2[i] = d; }
};

// One warp: sorts the list by distance, then by ref.  Bitonic merges that all
// ascend (each begins by comparing mirrored entries), so the entries past n, as
// if at infinity, stay where they are.  Counting, n steps an entry, takes 1.8 ms
// for 16,384 lists of up to 1024, sorting 0.76 ms; but a sort's steps depend on one
// another, and lists of 32 lose 4 us by it (64 probes x 64 directions: 74 -> 81 us).
constexpr int kFrontSort = 256;
__device__ __forceinline__ void front_sort(const FrontList& l, int n) {
  const int lane = int(threadIdx.x & 31);
  int size = 32;
  while (size < n) size *= 2;
  auto order = [&](int i, int j) {
    if (j >= n) return;
    const float di = l.d2[i], dj = l.d2[j];
    const int ri = l.ref[i], rj = l.ref[j];
    if (dj < di || (dj == di && rj < ri)) {
      const uint32_t si = l.src[i], sj = l.src[j];
      l.put(i, sj, rj, dj);
      l.put(j, si, ri, di);
    }
  };
  for (int k = 2; k <= size; k *= 2) {
    for (int t = lane; t < size / 2; t += 32) {
      const int in = t & (k / 2 - 1), b = (t - in) * 2;
      order(b + in, b + k - 1 - in);
    }
    __syncwarp();
    for (int h = k / 4; h >= 1; h /= 2) {
      for (int t = lane; t < size / 2; t += 32) {
        const int in = t & (h - 1), b = (t - in) * 2;
        order(b + in, b + in + h);
      }
      __syncwarp();
    }
  }
}

// One warp: probe p's frontier.
__device__ __forceinline__ void front_probe(const FrontArgs& a, uint32_t p, FrontShared& sh) {
  const uint32_t lane = threadIdx.x & 31;
  const int cap = int(a.cap);
  const float ox = a.probes[3 * size_t(p)], oy = a.probes[3 * size_t(p) + 1], oz = a.probes[3 * size_t(p) + 2];
  const unsigned below = (1u << lane) - 1u;
  FrontList done;
  done.src = reinterpret_cast<uint32_t*>(&sh + 1);
  done.ref = reinterpret_cast<int*>(done.src + cap);
  done.d2 = reinterpret_cast<float*>(done.ref + cap);
  // the children of node `ref`: their place (with kFrontWide), reference and squared distance
  auto children = [&](int ref, uint32_t* src, int* cr, float* d2) {
    const float4* nd = a.nodes + 4 * size_t(ref);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const FrontBox c = front_box(nd, h);
      const float gx = axis_gap(c.a.x, c.a.z, ox), gy = axis_gap(c.a.y, c.a.w, oy), gz = axis_gap(c.b.x, c.b.y, oz);
      const float ex = c.a.z - c.a.x, ey = c.a.w - c.a.y, ez = c.b.y - c.b.x;
      cr[h] = __float_as_int(c.b.z);
      d2[h] = gx * gx + gy * gy + gz * gz;
      src[h] = 2u * uint32_t(ref) + uint32_t(h);
      if (cr[h] >= 0 && ex * ey + ey * ez + ez * ex > kFrontLarge * d2[h]) src[h] |= kFrontWide;
    }
  };
  if (lane == 0) { sh.ref[0][0] = 0; sh.src[0][0] = 0; }
  __syncwarp();
  int n_open = 1, n_done = 0;
  for (int level = 0; n_open > 0; ++level) {
    const int cur = level & 1, nxt = cur ^ 1;
    int n_next = 0;
    for (int base = 0; base < n_open; base += 32) {
      const bool have = base + int(lane) < n_open;
      // entries live now; expanding one adds one (the root, without a box of its
      // own, always is: there is room for 32)
      const int room = cap - (n_open - base + n_next + n_done);
      const int ref = have ? sh.ref[cur][base + lane] : 0;
      const uint32_t at = have ? sh.src[cur][base + lane] : 0;
      const bool expand = have && int(lane) < room && VLB_INB(ref, 2 * a.ntris - 2, a.err);
      uint32_t cs[2];
      int cr[2];
      float cd[2];
      bool go[2] = {false, false};  // the child is expanded in turn
      if (expand) {
        children(ref, cs, cr, cd);
#pragma unroll
        for (int h = 0; h < 2; ++h) go[h] = cr[h] >= 0 && cd[h] == 0.f;
      }
      {  // no more than the next level holds
        const unsigned w0 = __ballot_sync(kAll, expand && go[0]), w1 = __ballot_sync(kAll, expand && go[1]);
        go[0] = go[0] && n_next + __popc(w0 & below) < kFrontOpen;
        go[1] = go[1] && n_next + __popc(w0) + __popc(w1 & below) < kFrontOpen;
      }
      const unsigned keep = __ballot_sync(kAll, have && !expand);
      const unsigned g0 = __ballot_sync(kAll, expand && go[0]), g1 = __ballot_sync(kAll, expand && go[1]);
      const unsigned d0 = __ballot_sync(kAll, expand && !go[0]), d1 = __ballot_sync(kAll, expand && !go[1]);
      // a node that stays holds the probe
      if (have && !expand) done.put(n_done + __popc(keep & below), at | kFrontWide, ref, 0.f);
      const int nd = n_done + __popc(keep);
      if (expand) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int g = n_next + (h ? __popc(g0) + __popc(g1 & below) : __popc(g0 & below));
          const int d = nd + (h ? __popc(d0) + __popc(d1 & below) : __popc(d0 & below));
          if (go[h]) { sh.ref[nxt][g] = cr[h]; sh.src[nxt][g] = cs[h] & ~kFrontWide; }
          else done.put(d, cs[h], cr[h], cd[h]);
        }
      }
      n_done = nd + __popc(d0) + __popc(d1);
      n_next += __popc(g0) + __popc(g1);
      __syncwarp();
    }
    n_open = n_next;
  }
  // then the entries that look largest from the probe
  const int look = min(kFrontLook, cap);
  for (int round = 0; round < kFrontRounds; ++round) {
    const int n0 = n_done;
    for (int base = 0; base < n0; base += 32) {
      const bool have = base + int(lane) < n0;
      const uint32_t src = have ? done.src[base + lane] : 0;
      const int ref = have ? done.ref[base + lane] : 0;
      const bool want = (src & kFrontWide) && VLB_INB(ref, 2 * a.ntris - 2, a.err);
      const unsigned wm = __ballot_sync(kAll, want);
      const bool expand = want && n_done + __popc(wm & below) < look;
      const unsigned em = __ballot_sync(kAll, expand);
      if (expand) {
        uint32_t cs[2];
        int cr[2];
        float cd[2];
        children(ref, cs, cr, cd);
        done.put(base + int(lane), cs[0], cr[0], cd[0]);
        done.put(n_done + __popc(em & below), cs[1], cr[1], cd[1]);
      }
      n_done += __popc(em);
      __syncwarp();
    }
    if (n_done == n0) break;
  }
  const float m = (fmaxf(fmaxf(fabsf(ox), fabsf(oy)), fabsf(oz)) + a.scale) * 0x1p-20f;
  // nearest first, equal distances by position: short lists by counting the
  // entries before each, long ones sorted, the position in the references' place
  const bool sorted = n_done > kFrontSort;
  if (sorted) {
    for (int i = int(lane); i < n_done; i += 32) done.ref[i] = i;
    __syncwarp();
    front_sort(done, n_done);
  }
  float4* out = a.ent + size_t(p) * a.cap * 2;
  for (int i = int(lane); i < n_done; i += 32) {
    const uint32_t src = done.src[i] & ~kFrontWide;
    FrontBox e = front_box(a.nodes + 4 * size_t(src >> 1), int(src & 1u));
    e.b.w = done.d2[i];
    int rank = sorted ? i : 0;
    for (int j = 0; !sorted && j < n_done; ++j) {
      const float dj = done.d2[j];
      rank += dj < e.b.w || (dj == e.b.w && j < i);
    }
    // relative to the probe, widened by m
    e.a.x = __fsub_rd(e.a.x, ox) - m; e.a.y = __fsub_rd(e.a.y, oy) - m; e.b.x = __fsub_rd(e.b.x, oz) - m;
    e.a.z = __fsub_ru(e.a.z, ox) + m; e.a.w = __fsub_ru(e.a.w, oy) + m; e.b.y = __fsub_ru(e.b.y, oz) + m;
    out[2 * rank] = e.a;
    out[2 * rank + 1] = e.b;
  }
  if (lane == 0) a.cnt[p] = uint32_t(n_done);
}

}  // namespace vlbk
