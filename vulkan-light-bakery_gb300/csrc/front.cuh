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

// The two children of node `ref` with their squared distances to the probe.
__device__ __forceinline__ void front_children(const FrontArgs& a, int ref, float ox, float oy, float oz,
                                               FrontBox* c) {
  const float4* nd = a.nodes + 4 * size_t(ref);
  const float4 n0 = __ldg(nd), n1 = __ldg(nd + 1), n2 = __ldg(nd + 2), n3 = __ldg(nd + 3);
  c[0].a = n0;
  c[0].b = make_float4(n2.x, n2.y, n3.x, 0.f);
  c[1].a = n1;
  c[1].b = make_float4(n2.z, n2.w, n3.y, 0.f);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float gx = axis_gap(c[h].a.x, c[h].a.z, ox), gy = axis_gap(c[h].a.y, c[h].a.w, oy),
                gz = axis_gap(c[h].b.x, c[h].b.y, oz);
    c[h].b.w = gx * gx + gy * gy + gz * gz;
  }
}

// Entries whose box half area exceeds kFrontLarge times the squared distance
// are expanded too, up to kFrontLook entries: with more, a ray group tests
// more boxes than the shorter walks save (16^3 probes x 256 directions, 778
// triangles: 212 us at 10, 223 us without, 234 us at 1; the 4096-box scene,
// whose lists are long already, 11.3 against 11.2 ms with none).
constexpr float kFrontLarge = 10.f;
constexpr int kFrontLook = 32;
constexpr int kFrontRounds = 8;

constexpr int kFrontOpen = 64;  // nodes of a level expanded; the rest become entries
struct FrontShared {
  FrontBox open[2][kFrontOpen], done[kFrontCap];
};

// One warp: probe p's frontier.
__device__ __forceinline__ void front_probe(const FrontArgs& a, uint32_t p, FrontShared& sh) {
  const uint32_t lane = threadIdx.x & 31;
  const int cap = int(a.cap);
  const float ox = a.probes[3 * size_t(p)], oy = a.probes[3 * size_t(p) + 1], oz = a.probes[3 * size_t(p) + 2];
  const unsigned below = (1u << lane) - 1u;
  FrontBox* done = sh.done;
  if (lane == 0) {
    sh.open[0][0].a = make_float4(0.f, 0.f, 0.f, 0.f);
    sh.open[0][0].b = make_float4(0.f, 0.f, __int_as_float(0), 0.f);
  }
  __syncwarp();
  int n_open = 1, n_done = 0;
  for (int level = 0; n_open > 0; ++level) {
    const FrontBox* open = sh.open[level & 1];
    FrontBox* next = sh.open[(level + 1) & 1];
    int n_next = 0;
    for (int base = 0; base < n_open; base += 32) {
      const bool have = base + int(lane) < n_open;
      // entries live now; expanding one adds one
      const int room = cap - (n_open - base + n_next + n_done);
      FrontBox e{};
      if (have) e = open[base + lane];
      const int ref = have ? __float_as_int(e.b.z) : 0;
      const bool expand = have && int(lane) < room && VLB_INB(ref, 2 * a.ntris - 2, a.err);
      FrontBox c[2];
      bool go[2] = {false, false};  // the child is expanded in turn
      if (expand) {
        front_children(a, ref, ox, oy, oz, c);
#pragma unroll
        for (int h = 0; h < 2; ++h) go[h] = __float_as_int(c[h].b.z) >= 0 && c[h].b.w == 0.f;
      }
      {  // no more than the next level holds
        const unsigned w0 = __ballot_sync(kAll, expand && go[0]), w1 = __ballot_sync(kAll, expand && go[1]);
        go[0] = go[0] && n_next + __popc(w0 & below) < kFrontOpen;
        go[1] = go[1] && n_next + __popc(w0) + __popc(w1 & below) < kFrontOpen;
      }
      const unsigned keep = __ballot_sync(kAll, have && !expand);
      const unsigned g0 = __ballot_sync(kAll, expand && go[0]), g1 = __ballot_sync(kAll, expand && go[1]);
      const unsigned d0 = __ballot_sync(kAll, expand && !go[0]), d1 = __ballot_sync(kAll, expand && !go[1]);
      if (have && !expand) done[n_done + __popc(keep & below)] = e;
      int nd = n_done + __popc(keep);
      if (expand) {
        if (go[0]) next[n_next + __popc(g0 & below)] = c[0];
        else done[nd + __popc(d0 & below)] = c[0];
        if (go[1]) next[n_next + __popc(g0) + __popc(g1 & below)] = c[1];
        else done[nd + __popc(d0) + __popc(d1 & below)] = c[1];
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
      FrontBox e{};
      if (have) e = done[base + lane];
      const float ex = e.a.z - e.a.x, ey = e.a.w - e.a.y, ez = e.b.y - e.b.x;
      const int ref = __float_as_int(e.b.z);
      const bool want = have && ref >= 0 && ex * ey + ey * ez + ez * ex > kFrontLarge * e.b.w &&
                        VLB_INB(ref, 2 * a.ntris - 2, a.err);
      const unsigned wm = __ballot_sync(kAll, want);
      const bool expand = want && n_done + __popc(wm & below) < look;
      const unsigned em = __ballot_sync(kAll, expand);
      if (expand) {
        FrontBox c[2];
        front_children(a, ref, ox, oy, oz, c);
        done[base + lane] = c[0];
        done[n_done + __popc(em & below)] = c[1];
      }
      n_done += __popc(em);
      __syncwarp();
    }
    if (n_done == n0) break;
  }
  const float m = (fmaxf(fmaxf(fabsf(ox), fabsf(oy)), fabsf(oz)) + a.scale) * 0x1p-20f;
  // nearest first (rank by distance, then by position)
  float4* out = a.ent + size_t(p) * a.cap * 2;
  for (int i = int(lane); i < n_done; i += 32) {
    FrontBox e = done[i];
    int rank = 0;
    for (int j = 0; j < n_done; ++j) {
      const float dj = done[j].b.w;
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
