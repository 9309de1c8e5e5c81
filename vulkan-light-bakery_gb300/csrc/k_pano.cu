// k_pano.cu -- SH projection of panoramas and equirect env maps
// (shaders/skybox_sh.comp:23-42, shaders/sh.comp:23-42), row by row.
//
// On an equirect image every basis function of l <= 3 is a trigonometric
// polynomial of degree <= 3 along a row, times a function of the row.  So a row
// needs only seven sums per channel (five for l <= 2) -- the texels times 1,
// cos, sin of phi, 2 phi and 3 phi -- instead of sixteen, and no basis per texel:
//   k_pano_rows     one warp per row segment: the sums, texels in pairs by packed
//                   FMAs, reduced across the warp; 84 bytes per 1024 texels
//   k_pano_combine  one cluster per map: the rows' sums into coefficients
// The reference adds every texel's 48 products into 48 floats with an
// unsynchronised read-modify-write (skybox_sh.comp:39).  Here the segments and
// the order of every sum are functions of the image size, so a map's
// coefficients are the same alone or in a batch.
//
// Sums of FP32 texels are scaled by a power of two (PanoScale) so that no sum of
// finite ones overflows, although a row is added up before its weight is applied.  A sum
// over a row segment that holds infinities or NaNs says little about the products
// with the basis, so such a segment leaves the signs of those products instead
// (kPanoCode): every coefficient is what adding the products one by one gives.
//
// Texel loads need no alignment beyond their own.  One 2048 x 1024 RGBA8 image
// takes 16.8 us a call, most of it the two launches' latency; with a basis per
// texel, 2048 partials per value added by one thread and the tables made on the
// host it took 256 us.
#include <cooperative_groups.h>

#include "vlb_device.cuh"
#include "vlb_internal.h"

namespace vlbk {
namespace {

constexpr int kPanoWarps = 8;
constexpr uint32_t kPanoSeg = 1024;   // texels of a row segment
constexpr int kPanoSums = 24;         // floats per segment: [channel][8], seven sums and a code
// The code, an integer: 0, or for a channel with texels that are not finite bit k:
// coefficient k gets +inf from one of them, bit 16 + k: -inf (both: NaN).
constexpr int kPanoCode = 7;
constexpr int kPanoThreads = 128;

// A segment's sums are multiplied by `down`, coefficients by `up`, its reciprocal: a
// sum times the largest factor of row_coeffs (5) and the row's weight stays finite.
struct PanoScale {
  float down = 1.f;
  double up = 1.0;
  PanoScale(const SkyboxArgs& a) {
    if (a.fmt != VLB_TEXEL_RGB32F) return;
    double most = 16.0 * (a.w < kPanoSeg ? a.w : kPanoSeg);
    const double weight = 2.0 * 3.1415926538 / a.w * (3.1415926538 / a.h);
    if (weight > 1.0) most *= weight;
    while (up < most) { up *= 2.0; down *= 0.5f; }
  }
};

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(d)
      : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)),
        "l"(*reinterpret_cast<uint64_t*>(&c)));
  return *reinterpret_cast<float2*>(&d);
}

template <int FMT>
__device__ __forceinline__ void load_rgb(const void* __restrict__ texels, size_t i, float* c) {
  if constexpr (FMT == 0) {
    const float* f = static_cast<const float*>(texels) + 3 * i;
    c[0] = __ldg(f); c[1] = __ldg(f + 1); c[2] = __ldg(f + 2);
  } else {
    const uint32_t q = __ldg(static_cast<const uint32_t*>(texels) + i);  // UNORM bytes, scaled at the end
    c[0] = float(q & 255u); c[1] = float((q >> 8) & 255u); c[2] = float((q >> 16) & 255u);
  }
}

// The code of channel c of a segment with texels that are not finite (one warp):
// their products with the weighted basis, as the texel-by-texel kernel forms them.
template <int LMAX>
__device__ __noinline__ uint32_t pano_code(const float* __restrict__ row_texels, const float2* __restrict__ col_tab,
                                           const float4 rw, bool pano, uint32_t x0, uint32_t x1, int c) {
  uint32_t code = 0;
  for (uint32_t x = x0 + (threadIdx.x & 31); x < x1; x += 32) {
    const float t = __ldg(row_texels + 3 * size_t(x) + c);
    if (isfinite(t)) continue;
    const float2 cs = __ldg(col_tab + x);
    const float dx = rw.x * cs.x, dy = rw.x * cs.y, dz = rw.y;
    float Y[16];
    sh_basis<LMAX>(dx, pano ? dz : dy, pano ? dy : dz, Y);
#pragma unroll
    for (int k = 0; k < sh_k<LMAX>(); ++k) {
      const float p = t * (Y[k] * rw.z);
      if (!(p < 0.f)) code |= 1u << k;
      if (!(p > 0.f)) code |= 0x10000u << k;
    }
  }
  return __reduce_or_sync(0xffffffffu, code);
}

// rows: [map][row][segment][kPanoSums].  LMAX 2 leaves the 3 phi sums out.
template <int LMAX, int FMT>
__global__ void __launch_bounds__(kPanoWarps * 32) k_pano_rows(const SkyboxArgs a, float* __restrict__ rows,
                                                               uint32_t nseg, uint32_t units, float down) {
  constexpr int M = LMAX == 3 ? 7 : 5;
  const uint32_t lane = threadIdx.x & 31, u = blockIdx.x * kPanoWarps + (threadIdx.x >> 5);
  if (u >= units) return;
  const uint32_t row = u / nseg, seg = u - row * nseg;  // row: over all maps' rows
  const uint32_t x0 = seg * kPanoSeg, x1 = min(a.w, x0 + kPanoSeg);
  const size_t at = size_t(row) * a.w;
  float2 acc[3][M];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int m = 0; m < M; ++m) acc[c][m] = make_float2(0.f, 0.f);
#pragma unroll 4
  for (uint32_t x = x0 + lane; x < x1; x += 64) {
    const bool two = x + 32 < x1;
    float t0[3], t1[3] = {0.f, 0.f, 0.f};
    load_rgb<FMT>(a.texels, at + x, t0);
    if (two) load_rgb<FMT>(a.texels, at + x + 32, t1);
    const float2 p = __ldg(a.col_tab + x), q = __ldg(a.col_tab + (two ? x + 32 : x));
    const float2 c1 = make_float2(p.x, q.x), s1 = make_float2(p.y, q.y);
    const float2 one = make_float2(1.f, 1.f), zero = make_float2(0.f, 0.f);
    const float2 two_c = fma2(c1, one, c1);
    // times `down`, a power of two: the texels' scale, exact here as on them
    const float d = FMT == 0 ? down : 1.f;
    const float2 f0 = make_float2(d, d), f1 = FMT == 0 ? fma2(c1, f0, zero) : c1, f2 = FMT == 0 ? fma2(s1, f0, zero) : s1;
    const float2 c2 = fma2(two_c, f1, make_float2(-d, -d)), s2 = fma2(two_c, f2, zero);  // cos 2phi = 2 cos^2 - 1, sin 2phi
    float2 f[7] = {f0, f1, f2, c2, s2, zero, zero};
    if constexpr (M == 7) {
      f[5] = fma2(two_c, c2, make_float2(-f1.x, -f1.y));  // cos 3phi = 2 cos phi cos 2phi - cos phi
      f[6] = fma2(two_c, s2, make_float2(-f2.x, -f2.y));
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float2 t = make_float2(t0[c], t1[c]);
#pragma unroll
      for (int m = 0; m < M; ++m) acc[c][m] = fma2(t, f[m], acc[c][m]);
    }
  }
  float v[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = i / 8 < 3 && i % 8 < M ? acc[i / 8 < 3 ? i / 8 : 0][i % 8 < M ? i % 8 : 0].x +
                                                                  acc[i / 8 < 3 ? i / 8 : 0][i % 8 < M ? i % 8 : 0].y
                                                            : 0.f;
  float s = warp_sums<32>(v);
  if constexpr (FMT == 0) {
    const unsigned bad = __ballot_sync(0xffffffffu, lane < kPanoSums && !isfinite(s));
    for (int c = 0; bad && c < 3; ++c) {
      if (!(bad >> (8 * c) & 0xffu)) continue;
      const uint32_t code = pano_code<LMAX>(static_cast<const float*>(a.texels) + 3 * at, a.col_tab,
                                            __ldg(a.row_tab + row % a.h), a.layout == VLB_SKY_PANORAMA, x0, x1, c);
      if (lane == uint32_t(8 * c + kPanoCode)) s = __uint_as_float(code);
    }
  }
  if (lane < kPanoSums) rows[size_t(u) * kPanoSums + lane] = s;
}

// A row's coefficients from its sums f = {1, c1, s1, c2, s2, c3, s3} at (sin
// theta, cos theta), without the basis' constants: the products of
// shaders/sh_common.h:26-116 with the powers of sin phi and cos phi written as
// multiple angles.  PANO: the basis at dir.xzy (skybox_sh.comp:39).
template <int LMAX, bool PANO>
__device__ __forceinline__ void row_coeffs(float s, float c, const float* f, float* o) {
  const float s2 = s * s, c2 = c * c, sc = s * c, s3 = s2 * s, s2c = s2 * c;
  o[0] = f[0];
  if constexpr (!PANO) {
    o[1] = -s * f[2];
    o[2] = c * f[0];
    o[3] = -s * f[1];
    o[4] = 0.5f * s2 * f[4];
    o[5] = -sc * f[2];
    o[6] = (2.f * c2 - s2) * f[0];
    o[7] = -sc * f[1];
    o[8] = s2 * f[3];
    if constexpr (LMAX == 3) {
      o[9] = -s3 * f[6];
      o[10] = 0.5f * s2c * f[4];
      o[11] = -s * (4.f * c2 - s2) * f[2];
      o[12] = c * (2.f * c2 - 3.f * s2) * f[0];
      o[13] = -s * (4.f * c2 - s2) * f[1];
      o[14] = s2c * f[3];
      o[15] = -s3 * f[5];
    }
  } else {
    o[1] = -c * f[0];
    o[2] = s * f[2];
    o[3] = -s * f[1];
    o[4] = sc * f[1];
    o[5] = -sc * f[2];
    o[6] = ((0.5f * s2 - c2) * f[0] - 1.5f * s2 * f[3]);
    o[7] = -0.5f * s2 * f[4];
    o[8] = ((0.5f * s2 - c2) * f[0] + 0.5f * s2 * f[3]);
    if constexpr (LMAX == 3) {
      o[9] = -c * ((1.5f * s2 - c2) * f[0] + 1.5f * s2 * f[3]);
      o[10] = 0.5f * s2c * f[4];
      o[11] = -c * ((1.5f * s2 - c2) * f[0] - 2.5f * s2 * f[3]);
      o[12] = (s * (0.75f * s2 - 3.f * c2) * f[2] - 1.25f * s3 * f[6]);
      o[13] = -(s * (0.25f * s2 - c2) * f[1] - 1.25f * s3 * f[5]);
      o[14] = (s * (0.25f * s2 - c2) * f[2] + 0.25f * s3 * f[6]);
      o[15] = -(s * (0.75f * s2 - 3.f * c2) * f[1] + 0.25f * s3 * f[5]);
    }
  }
}

// The constants of shaders/sh_common.h:26-116 by coefficient.
__constant__ double c_sh[16] = {0.282095, 0.488603, 0.488603, 0.488603, 1.092548, 1.092548, 0.315392, 1.092548,
                                0.546274, 0.590044, 2.890611, 0.457046, 0.373176, 0.457046, 1.445306, 0.590044};

// warp_sums of 16 values v + e, e what rounding took from v: lane l < 16 ends with the
// sum of v[l] and e[l].
__device__ __forceinline__ double warp_sums_kept(float (&v)[16], float (&e)[16]) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (int n = 16; n >= 1; n /= 2) {  // first the lane 16 away, all values; then half of the values less a step
    const bool up = n < 16 && (lane & n);
    const int m = n < 16 ? n : 16;
#pragma unroll
    for (int i = 0; i < m; ++i) {
      const int j = n < 16 ? i + n : i;
      const float sv = up ? v[i] : v[j], se = up ? e[i] : e[j], kv = up ? v[j] : v[i], ke = up ? e[j] : e[i];
      const float ov = __shfl_xor_sync(0xffffffffu, sv, n), oe = __shfl_xor_sync(0xffffffffu, se, n);
      v[i] = __fadd_rn(kv, ov);
      e[i] = __fadd_rn(__fadd_rn(ke, oe), sum_error(kv, ov, v[i]));
    }
  }
  return double(v[0]) + double(e[0]);
}

// One cluster per map: a thread takes every n-th row segment, n its threads.  Segments
// are added as the texel-by-texel kernel's partials are, in more than FP32: threads and
// lanes keep, beside their FP32 sums, what rounding took from the products with the
// row's weight and from the sums; warps and CTAs are added in FP64, in order.  (FP64
// adds across the lanes, at 1/64 of the FP32 rate: 256 maps of 256 x 128 at lmax 3 136
// against 41 us a call.)  The basis' constants and the 1 / 255 of 8-bit texels multiply
// the FP64 sum, so neither is rounded to FP32.  A cluster has the CTAs that its segments
// keep busy (pano_ctas): one CTA per map, with FP32 sums, took 18.9 us for 2048 x 1024
// and 207 us for 8192 x 4096, now 16.8 and 142 us.
template <int LMAX, bool PANO>
__global__ void __launch_bounds__(kPanoThreads)
    k_pano_combine(const SkyboxArgs a, const float* __restrict__ rows, uint32_t nseg, double up,
                   float* __restrict__ out) {
  constexpr int K = sh_k<LMAX>();
  __shared__ double s_warp[kPanoThreads / 32][48], s_sum[48];
  __shared__ uint32_t s_code[3];
  namespace cg = cooperative_groups;
  const auto cluster = cg::this_cluster();
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t ctas = cluster.num_blocks(), map = blockIdx.x / ctas, rank = blockIdx.x % ctas, units = a.h * nseg;
  if (tid < 3) s_code[tid] = 0;
  __syncthreads();
  float sum[3][K], lost[3][K];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int k = 0; k < K; ++k) sum[c][k] = lost[c][k] = 0.f;
  for (uint32_t u = rank * kPanoThreads + tid; u < units; u += ctas * kPanoThreads) {
    const float4 rw = __ldg(a.row_tab + u / nseg);  // sin theta, cos theta, weight
    const float4* r = reinterpret_cast<const float4*>(rows) + (size_t(map) * units + u) * (kPanoSums / 4);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float4 x = __ldg(r + 2 * c), y = __ldg(r + 2 * c + 1);
      const bool sums = __float_as_uint(y.w) == 0;
      if (!sums) atomicOr(&s_code[c], __float_as_uint(y.w));
      float f[7] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z}, o[16];
#pragma unroll
      for (int i = 0; i < 7; ++i) f[i] = sums ? f[i] : 0.f;
      row_coeffs<LMAX, PANO>(rw.x, rw.y, f, o);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const float p = __fmul_rn(rw.z, o[k]), t = __fadd_rn(sum[c][k], p);
        lost[c][k] += __fadd_rn(sum_error(sum[c][k], p, t), __fmaf_rn(rw.z, o[k], -p));
        sum[c][k] = t;
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    float v[16], e[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      v[k] = k < K ? sum[c][k < K ? k : 0] : 0.f;
      e[k] = k < K ? lost[c][k < K ? k : 0] : 0.f;
    }
    const double s = warp_sums_kept(v, e);
    if (lane < 16) s_warp[warp][3 * lane + c] = s;
  }
  __syncthreads();
  if (tid < 3 * K) {
    double s = 0.0;
    for (int w = 0; w < kPanoThreads / 32; ++w) s += s_warp[w][tid];
    s_sum[tid] = s;
  }
  cluster.sync();
  if (rank == 0 && tid < 3 * K) {
    const int k = int(tid) / 3, c = int(tid) - 3 * k;
    double s = 0.0;
    uint32_t code = 0;
    for (uint32_t q = 0; q < ctas; ++q) {
      s += *cluster.map_shared_rank(&s_sum[tid], q);
      code |= *cluster.map_shared_rank(&s_code[c], q);
    }
    s *= a.fmt == VLB_TEXEL_RGBA8 ? c_sh[k] / 255.0 : c_sh[k] * up;
    if (code >> k & 1u) s += INFINITY;
    if (code >> (16 + k) & 1u) s -= INFINITY;
    const int co = a.flags & VLB_SKY_REF_BGRA_SWAP ? 2 - c : c;
    out[(size_t(map) * K + k) * 3 + co] = float(s);
  }
  cluster.sync();  // no CTA leaves while its sums are read
}

// CTAs of a map's cluster: two row segments a thread keep a CTA busy.
uint32_t pano_ctas(uint32_t units) {
  uint32_t n = 1;
  while (n < 8 && n * kPanoThreads * 2 <= units) n *= 2;
  return n;
}

template <int LMAX>
void launch(const SkyboxArgs& a, float* rows, float* out, cudaStream_t s) {
  const uint32_t nseg = (a.w + kPanoSeg - 1) / kPanoSeg, units = a.count * a.h * nseg;
  const uint32_t grid = (units + kPanoWarps - 1) / kPanoWarps;
  const PanoScale scale(a);
  if (a.fmt == VLB_TEXEL_RGB32F)
    k_pano_rows<LMAX, 0><<<grid, kPanoWarps * 32, 0, s>>>(a, rows, nseg, units, scale.down);
  else
    k_pano_rows<LMAX, 1><<<grid, kPanoWarps * 32, 0, s>>>(a, rows, nseg, units, scale.down);
  cudaLaunchAttribute cluster{};
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = pano_ctas(a.h * nseg);
  cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(a.count * cluster.val.clusterDim.x);
  cfg.blockDim = dim3(kPanoThreads);
  cfg.stream = s;
  cfg.attrs = &cluster;
  cfg.numAttrs = 1;
  if (a.layout == VLB_SKY_PANORAMA) cudaLaunchKernelEx(&cfg, k_pano_combine<LMAX, true>, a, rows, nseg, scale.up, out);
  else cudaLaunchKernelEx(&cfg, k_pano_combine<LMAX, false>, a, rows, nseg, scale.up, out);
}

}  // namespace

// Direction tables: per column (cos phi, sin phi), per row (sin theta, cos theta,
// pixel weight) with the reference's PI (shaders/sh_common.h:1, :14-22;
// sh.comp:28-33, skybox_sh.comp:28: phi - PI/2).
__global__ void k_pano_tables(float2* col, float4* row, uint32_t w, uint32_t h, int shift) {
  const double pi = 3.1415926538;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < w) {
    double phi = 2.0 * pi * (double(i) + 0.5) / double(w);
    if (shift) phi -= pi / 2.0;
    col[i] = make_float2(float(cos(phi)), float(sin(phi)));
  }
  if (i < h) {
    const double th = pi * (double(i) + 0.5) / double(h);
    const double area = (2.0 * pi / w) * (pi / h);
    row[i] = make_float4(float(sin(th)), float(cos(th)), float(area * sin(th)), 0.f);
  }
}

void launch_pano_tables(float2* col, float4* row, uint32_t w, uint32_t h, bool shift, cudaStream_t s) {
  const uint32_t n = w > h ? w : h;
  k_pano_tables<<<(n + 63) / 64, 64, 0, s>>>(col, row, w, h, shift ? 1 : 0);
}

size_t pano_rows_bytes(uint32_t w, uint32_t h, uint32_t count) {
  return size_t(count) * h * ((w + kPanoSeg - 1) / kPanoSeg) * kPanoSums * sizeof(float);
}

void launch_pano_sh(const SkyboxArgs& a, float* rows, float* out, cudaStream_t s) {
  if (a.lmax == 2) launch<2>(a, rows, out, s);
  else launch<3>(a, rows, out, s);
}

}  // namespace vlbk
