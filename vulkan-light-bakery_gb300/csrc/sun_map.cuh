// sun_map.cuh -- sun maps: shadow rays answered without a walk.
//
// All shadow rays of a bake run toward the sun, so they are parallel: seen
// along the sun direction a ray is one point of a plane plus its origin's
// depth.  A kernel rasterises the scene's triangles onto that plane and
// keeps two depths (along the direction to the sun) per cell:
//   cover  the largest depth below which every ray of the cell is occluded:
//          some triangle covers the whole cell and lies above it everywhere;
//   top    a depth above which no ray of the cell meets anything.
// A shadow ray that starts below its cell's cover is occluded, one that
// starts above top is lit, and only the rest walk the tree.  Both bounds are
// conservative against what a walk would find with its FP32 tests, so every ray
// keeps the answer its walk gives.  Cells are widened by `margin` (2^-17 of the
// scene's coordinate scale, for its rounding).  The triangle test misplaces an edge
// by that rounding times up to |e1| |e2| / |e1 x e2 . direction| (`grow`): a covering
// triangle contains the widened cell with that much room, any triangle reaches that
// far beyond its edges, and its plane's depth beyond them is bounded by grow once
// more.  Of triangles seen nearly edge on (steep: grow 256 and more) the test may
// find anything, but a walk tests them only on rays that meet their box, so they
// reach as far as their box looks from the light, and cover nothing.
//
// A point light outside the scene is the same map seen from the light: u and v
// are divided by the distance along the view axis and the depth is its
// reciprocal, so triangles stay triangles and depth planes planes.  A shadow ray
// there runs parallel to the line from the hit to the light, `bias` beside it,
// and drifts by at most bias (1 / nearest - 1 / farthest) in u and v: cells are
// widened by that too (it does not grow: the ray is where it is).
//
// Thread k of a CTA sets up one triangle; the CTA's triangles' cells are then
// numbered through and shared by all its threads (a binary search finds a
// cell's triangle), so slivers and walls cost what their cells cost.  Several
// CTAs (slices) share a group of triangles row by row: the walls of a room
// fill the map and would otherwise be drawn by a single CTA.  A cell is read
// before its atomic maximum: in deep scenes most triangles lie below one
// already drawn.  Latency bound: 15 us for 778 triangles, 40 us for 164 k small
// ones, 130 us for the 49 k faces of 4096 boxes.
#pragma once

#include "vlb_device.cuh"
#include "vlb_internal.h"

namespace vlbk {

constexpr int kMapThreads = 256;
// Order-preserving map of a float to an unsigned integer; 0 is below every float.
__device__ __forceinline__ uint32_t ordered(float f) {
  const uint32_t u = __float_as_uint(f);
  return u ^ (uint32_t(int32_t(u) >> 31) | 0x80000000u);
}

struct MapTri {
  float ea[3], eb[3], ec[3];  // edge k: ea u + eb v + ec = distance inside it
  float au, av, ac;           // depth = au u + av v + ac
  float dmax, slack, pad;     // pad: how far from its edges a ray may be hit or missed by rounding
  int i0, i1, j0, j1, first;  // cells; the slice's first row
  int covers;
};

__device__ __forceinline__ float dotm(float x, float y, float z, float3 a) {
  return fmaf(z, a.z, fmaf(y, a.y, x * a.x));
}

__device__ __forceinline__ void map_setup(const SunMap& m, const float4 a, const float4 e1, const float4 e2,
                                          MapTri& T) {
  float au, av, ad, bu, bv, bd, cu, cv, cd;  // the first vertex, the edges from it
  const float l1 = e1.x * e1.x + e1.y * e1.y + e1.z * e1.z, l2 = e2.x * e2.x + e2.y * e2.y + e2.z * e2.z;
  float det, facing;  // twice the projected area, signed; |e1 x e2 . direction|
  // the triangle's box (its middle from the light, half its edges): how far it reaches
  const float hx = 0.5f * (fmaxf(0.f, fmaxf(e1.x, e2.x)) - fminf(0.f, fminf(e1.x, e2.x)));
  const float hy = 0.5f * (fmaxf(0.f, fmaxf(e1.y, e2.y)) - fminf(0.f, fminf(e1.y, e2.y)));
  const float hz = 0.5f * (fmaxf(0.f, fmaxf(e1.z, e2.z)) - fminf(0.f, fminf(e1.z, e2.z)));
  const float mx = a.x + fminf(0.f, fminf(e1.x, e2.x)) + hx - m.o.x, my = a.y + fminf(0.f, fminf(e1.y, e2.y)) + hy - m.o.y,
              mz = a.z + fminf(0.f, fminf(e1.z, e2.z)) + hz - m.o.z;
  const float dm = dotm(mx, my, mz, m.s), dh = hx * fabsf(m.s.x) + hy * fabsf(m.s.y) + hz * fabsf(m.s.z);
  auto see = [&](float px, float py, float pz, float& u, float& v, float& d) {
    d = 1.0f / dotm(px, py, pz, m.s);
    u = dotm(px, py, pz, m.u) * d;
    v = dotm(px, py, pz, m.v) * d;
  };
  if (m.point) {
    const float x = a.x - m.o.x, y = a.y - m.o.y, z = a.z - m.o.z;
    see(x, y, z, au, av, ad);
    see(x + e1.x, y + e1.y, z + e1.z, bu, bv, bd);
    see(x + e2.x, y + e2.y, z + e2.z, cu, cv, cd);
    bu -= au; bv -= av; bd -= ad;
    cu -= au; cv -= av; cd -= ad;
    det = bu * cv - bv * cu;
    const float nx = e1.y * e2.z - e1.z * e2.y, ny = e1.z * e2.x - e1.x * e2.z, nz = e1.x * e2.y - e1.y * e2.x;
    // the rays to its farthest vertex graze it most
    auto len2 = [](float px, float py, float pz) { return px * px + py * py + pz * pz; };
    const float far2 = fmaxf(len2(x, y, z), fmaxf(len2(x + e1.x, y + e1.y, z + e1.z), len2(x + e2.x, y + e2.y, z + e2.z)));
    facing = fabsf(nx * x + ny * y + nz * z) * rsqrtf(far2);
  } else {
    au = dotm(a.x, a.y, a.z, m.u); av = dotm(a.x, a.y, a.z, m.v); ad = dotm(a.x, a.y, a.z, m.s);
    bu = dotm(e1.x, e1.y, e1.z, m.u); bv = dotm(e1.x, e1.y, e1.z, m.v); bd = dotm(e1.x, e1.y, e1.z, m.s);
    cu = dotm(e2.x, e2.y, e2.z, m.u); cv = dotm(e2.x, e2.y, e2.z, m.v); cd = dotm(e2.x, e2.y, e2.z, m.s);
    det = bu * cv - bv * cu;
    facing = fabsf(det);
  }
  const float grow = sqrtf(l1) * sqrtf(l2) / facing;
  const bool steep = !(grow < 256.f && fabsf(det) > 0.f);
  T.slack = steep ? INFINITY : m.dmargin * (1.f + grow);
  T.pad = steep ? INFINITY : m.margin + m.round * grow;
  T.covers = !steep;
  T.dmax = (m.point ? 1.0f / (dm - dh) : dm + dh) + m.dmargin;
  if (!steep) T.dmax = fminf(T.dmax, ad + fmaxf(0.f, fmaxf(bd, cd)) + T.slack * (1.f + grow));
  const float inv = steep ? 0.f : 1.f / det;
  T.au = (bd * cv - cd * bv) * inv;
  T.av = (cd * bu - bd * cu) * inv;
  T.ac = ad - T.au * au - T.av * av;
  const float sg = det < 0.f ? -1.f : 1.f;
  const float pu[3] = {au, au + bu, au + cu}, pv[3] = {av, av + bv, av + cv};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int n = k == 2 ? 0 : k + 1;
    const float du = pu[n] - pu[k], dv = pv[n] - pv[k];
    const float rn = steep ? 0.f : sg * rsqrtf(fmaxf(du * du + dv * dv, 1e-30f));
    T.ea[k] = -dv * rn;
    T.eb[k] = du * rn;
    T.ec[k] = -(T.ea[k] * pu[k] + T.eb[k] * pv[k]);
  }
  float u0 = fminf(pu[0], fminf(pu[1], pu[2])), u1 = fmaxf(pu[0], fmaxf(pu[1], pu[2]));
  float v0 = fminf(pv[0], fminf(pv[1], pv[2])), v1 = fmaxf(pv[0], fmaxf(pv[1], pv[2])), reach = T.pad;
  if (steep) {
    reach = m.margin;
    if (m.point) {
      for (int k = 0; k < 8; ++k) {
        float u, v, d;
        see(mx + (k & 1 ? hx : -hx), my + (k & 2 ? hy : -hy), mz + (k & 4 ? hz : -hz), u, v, d);
        u0 = fminf(u0, u); u1 = fmaxf(u1, u);
        v0 = fminf(v0, v); v1 = fmaxf(v1, v);
      }
    } else {
      const float u = dotm(mx, my, mz, m.u), uh = hx * fabsf(m.u.x) + hy * fabsf(m.u.y) + hz * fabsf(m.u.z);
      const float v = dotm(mx, my, mz, m.v), vh = hx * fabsf(m.v.x) + hy * fabsf(m.v.y) + hz * fabsf(m.v.z);
      u0 = u - uh; u1 = u + uh;
      v0 = v - vh; v1 = v + vh;
    }
  }
  const float G1 = float(m.G - 1);
  auto cell = [&](float x, float x0) { return int(fminf(fmaxf((x - x0) * m.inv, 0.f), G1)); };
  T.i0 = cell(u0 - reach, m.u0);
  T.i1 = cell(u1 + reach, m.u0);
  T.j0 = cell(v0 - reach, m.v0);
  T.j1 = cell(v1 + reach, m.v0);
}

__device__ __forceinline__ void map_cell(const SunMap& m, const MapTri& T, int i, int j) {
  const float half = 0.5f * m.cell + m.margin;
  const float cu = fmaf(float(i) + 0.5f, m.cell, m.u0), cv = fmaf(float(j) + 0.5f, m.cell, m.v0);
  bool out = false, in = T.covers != 0;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const float d = fmaf(T.ea[e], cu, fmaf(T.eb[e], cv, T.ec[e]));
    const float r = half * (fabsf(T.ea[e]) + fabsf(T.eb[e]));
    out = out || d + r < -T.pad;
    in = in && d - r > T.pad;
  }
  if (out) return;
  const float zc = fmaf(T.au, cu, fmaf(T.av, cv, T.ac)), zr = half * (fabsf(T.au) + fabsf(T.av));
  const float hi = T.covers ? fminf(T.dmax, zc + zr + T.slack) : T.dmax;
  uint32_t* at = m.cells + 2 * (size_t(j) * m.G + i);
  const uint2 now = __ldcg(reinterpret_cast<const uint2*>(at));
  const uint32_t ht = ordered(hi);
  if (now.y < ht) atomicMax(at + 1, ht);
  if (in) {
    const uint32_t hc = ordered(zc - zr - T.slack);
    if (now.x < hc) atomicMax(at, hc);
  }
}

struct MapShared {
  MapTri st[kMapThreads];
  int end[kMapThreads];  // cells of triangles 0 .. k
  int warp[kMapThreads / 32];
};

// One CTA: slice `slice` of a group of kMapThreads triangles, the rows of each
// that are congruent to it modulo the slice count.
__device__ __forceinline__ void map_draw(const SunMap& m, const float4* __restrict__ tris, uint32_t ntris,
                                         uint32_t group, int slice, int slices, MapShared& sh) {
  const int tid = int(threadIdx.x), lane = tid & 31, warp = tid >> 5;
  const uint32_t t = group * kMapThreads + threadIdx.x;
  int n = 0;
  if (t < ntris) {
    MapTri& T = sh.st[tid];
    map_setup(m, __ldg(tris + 3 * size_t(t)), __ldg(tris + 3 * size_t(t) + 1), __ldg(tris + 3 * size_t(t) + 2), T);
    int off = (slice - T.j0) % slices;
    off += off < 0 ? slices : 0;
    T.first = T.j0 + off;
    n = T.first <= T.j1 ? ((T.j1 - T.first) / slices + 1) * (T.i1 - T.i0 + 1) : 0;
  }
  int end = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= o) end += y;
  }
  if (lane == 31) sh.warp[warp] = end;
  __syncthreads();
  for (int k = 0; k < warp; ++k) end += sh.warp[k];
  sh.end[tid] = end;
  __syncthreads();
  const int total = sh.end[kMapThreads - 1];
#pragma unroll 2
  for (int c = tid; c < total; c += kMapThreads) {
    int k = 0;  // the first triangle whose end exceeds c
#pragma unroll
    for (int step = kMapThreads / 2; step > 0; step >>= 1)
      if (sh.end[k + step - 1] <= c) k += step;
    const MapTri& T = sh.st[k];
    const int at = c - (k ? sh.end[k - 1] : 0), w = T.i1 - T.i0 + 1, r = at / w;
    map_cell(m, T, T.i0 + at - r * w, T.first + r * slices);
  }
}

}  // namespace vlbk
