// Voxel-volume transient renderer: confocal forward, its exact adjoint, the
// reference's transposed operator, the measurement-point gradient, and the
// exhaustive (laser/detector) forward with its adjoint.
//
// Reference: src/render/volume_cuda.cu. The reference forward gathers over
// every (point, bin, voxel column) (:12-66), O(N T X Y). The forward here
// scatters only occupied voxels: a voxel at slice k receives samples whose
// interpolation cell is k-1 or k, i.e. a contiguous run of ~4 bins per
// (voxel, point), found by inverting the sphere/column geometry and then
// re-deciding each bin with the reference's FP32 sample arithmetic. Each CTA
// owns a tile of points and keeps their transient rows in shared memory.
#include <cooperative_groups.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>

#include "capi_common.cuh"
#include "tune.cuh"

namespace totri {
namespace volume {

namespace cg = cooperative_groups;

struct Geo {
  int X, Y, Z;
  float ox, oy, oz, sx, sy, sz;
  float scale, dz;  // Z / sz, sz / Z
  float bw, bo;
  float inv_bw;
  int T;
  int exact;     // 1: every sample takes the exact chain (tuning key "volume.exact")
  int all_bins;  // bin width not positive and finite (or offset not finite): walk every bin
};

// Column / slice centre: origin + ((i + 0.5) * size) / n (volume_cuda.cu:35,38).
__device__ __forceinline__ float centre(float o, float s, int n, int i) {
  return xadd(o, xdiv(xmul(xadd((float)i, 0.5f), s), (float)n));
}

struct Sample {
  bool ok;
  int zi;
  float alpha, f1, f2;  // f1 = (depth / tc^2)^2, f2 = f1^2
};

// The reference's sample at (point w, bin t, column x/y) (volume_cuda.cu:23-57):
// FP32 decisions (depth^2 > 0, floor(z_hat), 0 <= zi, zi + 1 < Z) with one
// rounding per operation; alpha and f2 are values.
__device__ __forceinline__ Sample sample(const Geo& g, float wx, float wy, float wz, int t,
                                         float x, float y) {
  Sample s{false, 0, 0.f, 0.f, 0.f};
  const float tc = xadd(xmul((float)t, g.bw), g.bo);
  const float dx = xsub(wx, x), dy = xsub(wy, y);
  const float d2 = xsub(xsub(xmul(tc, tc), xmul(dx, dx)), xmul(dy, dy));
  if (!(d2 > 0.f)) return s;
  const float depth = xsqrt(d2);
  const float z = xadd(wz, depth);
  const float zh = xsub(xmul(xsub(z, g.oz), g.scale), 0.5f);
  const float fl = floorf(zh);
  if (!(fl >= 0.f && fl + 1.f < (float)g.Z)) return s;
  s.ok = true;
  s.zi = (int)fl;
  s.alpha = zh - fl;
  const float q = __fdividef(depth, tc * tc);  // a value: the hardware reciprocal (2 ulp)
  s.f1 = q * q;
  s.f2 = s.f1 * s.f1;
  return s;
}

// The kernels take a sample's cell from a fast path where it is sure to be the exact
// chain's: with u = 2^-24, the depth from the hardware reciprocal square root (within 6 u
// of the exact root) moves z_hat by at most 8 u scale (depth + |wz| + |z| + |oz|) + 4 u |z_hat|,
// so where its fraction is farther than that margin from 0 and 1 (taken at the largest
// magnitudes of a walk), the fast floor is the exact floor; elsewhere sample() decides.
// alpha and f2 are values (few-ulp differences). "volume.exact" = 1: sample() always.

// First bin whose centre t bw + bo (the sample chain's FP32 arithmetic) is not
// negative; 0 unless the bin offset is negative. Bins before it have negative
// centres, whose samples mirror those of the positive centres (the reference
// walks every bin and squares the centre).
__device__ __forceinline__ int first_nonneg_bin(const Geo& g) {
  if (g.all_bins || !(g.bo < 0.f)) return 0;
  const float tf = ceilf(-g.bo * g.inv_bw);
  if (!(tf < (float)g.T)) return g.T;
  int t = max((int)tf - 2, 0);
  while (t > 0 && xadd(xmul((float)(t - 1), g.bw), g.bo) >= 0.f) --t;
  while (t < g.T && xadd(xmul((float)t, g.bw), g.bo) < 0.f) ++t;
  return t;
}

// Bins whose centre's magnitude lies in [cl, ch] widened by eps bins: [p0, p1]
// with non-negative centres (t >= tz) and [n0, n1] with negative ones (t < tz). A span
// whose last bin is before its first is empty; its first may be any up to INT_MAX.
// Every bin when the bin width is degenerate. A NaN bound gives empty spans.
struct Spans {
  int p0, p1, n0, n1;
};
__device__ __forceinline__ Spans tc_spans(const Geo& g, int tz, float cl, float ch, float eps) {
  Spans s{1, 0, 1, 0};
  if (g.all_bins) {
    s.p0 = 0;
    s.p1 = g.T - 1;
    return s;
  }
  if (!(cl <= ch)) return s;
  s.p0 = max(__float2int_ru((cl - g.bo) * g.inv_bw - eps), tz);
  s.p1 = min(__float2int_rd((ch - g.bo) * g.inv_bw + eps), g.T - 1);
  if (tz > 0) {
    s.n0 = max(__float2int_ru((-ch - g.bo) * g.inv_bw - eps), 0);
    s.n1 = min(__float2int_rd((-cl - g.bo) * g.inv_bw + eps), tz - 1);
  }
  return s;
}

// The same spans with first bins of at most T, for walks that add a lane's offset to
// them before the test for an empty span.
__device__ __forceinline__ Spans within_bins(const Geo& g, Spans s) {
  s.p0 = min(s.p0, g.T);
  s.n0 = min(s.n0, g.T);
  return s;
}

// Centre magnitudes [cl, ch] of the bins whose samples from a point at squared
// horizontal distance rho2 and height wz can land in z in [zlo, zhi); false
// when the whole interval lies below the point.
__device__ __forceinline__ bool tc_bounds(float rho2, float wz, float zlo, float zhi, float& cl,
                                          float& ch) {
  const float dhi = zhi - wz;
  if (!(dhi > 0.f)) return false;
  const float dlo = fmaxf(zlo - wz, 0.f);
  cl = sqrtf(dlo * dlo + rho2);
  ch = sqrtf(dhi * dhi + rho2);
  return true;
}

// The widening, in bins, of a span from tc_bounds whose largest centre
// magnitude is ch: the bound of confocal_adjoint_cells_kernel on the FP32
// rounding of the sample chain against that inverse (64 u of the largest
// magnitudes over the bin width, plus 0.01, at most one bin), with the
// largest |tc| of the walked bins at most ch plus one bin.
__device__ __forceinline__ float span_eps(const Geo& g, float ch, float wz) {
  const float u = 5.9604645e-8f;
  const float dmax = 1.001f * (ch + fabsf(g.bw));
  const float zmax = fabsf(wz) + dmax;
  return fminf(64.f * u * (dmax + fabsf(g.bo) + fabsf(wz) + zmax + fabsf(g.oz) +
                           fabsf(1.f / g.scale)) * g.inv_bw + 0.01f,
               1.f);
}

// Bins whose sample may fall in interpolation cells k-1 or k of a column,
// widened by span_eps (a whole bin each side walked about two more bins per
// (voxel, point) pair of the forward).
__device__ __forceinline__ Spans bin_range(const Geo& g, int tz, float rho2, float wz, int k) {
  float cl, ch;
  if (!tc_bounds(rho2, wz, g.oz + ((float)k - 0.5f) / g.scale,
                 g.oz + ((float)k + 1.5f) / g.scale, cl, ch))
    return Spans{1, 0, 1, 0};
  return tc_spans(g, tz, cl, ch, span_eps(g, ch, wz));
}

struct Points {  // measurement points [3, N] with strides
  const float* p;
  int64_t sc, sn;
  __device__ float at(int c, int i) const { return p[c * sc + i * sn]; }
};

// The occupied voxels of a [X][Y][Z] volume as records (column centre x, y,
// value, cell k): the per-voxel decoding (two divisions of the index, two
// correctly rounded divisions for the centres) is done once here instead of
// once per (voxel, point) pair.
__global__ void compact_kernel(Geo g, const float* __restrict__ vol, int64_t n, float4* recs,
                               uint32_t* count) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool occ = i < n && vol[i] != 0.f;
  const uint32_t m = __ballot_sync(0xffffffffu, occ);
  if (!m) return;
  const int lane = threadIdx.x & 31;
  uint32_t base = 0;
  if (lane == __ffs(m) - 1) base = atomicAdd(count, (uint32_t)__popc(m));
  base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
  if (occ) {
    const uint32_t lin = (uint32_t)i;
    const int k = (int)(lin % g.Z);
    const int yi = (int)((lin / g.Z) % g.Y), xi = (int)(lin / ((uint32_t)g.Z * g.Y));
    recs[base + __popc(m & ((1u << lane) - 1u))] =
        make_float4(centre(g.ox, g.sx, g.X, xi), centre(g.oy, g.sy, g.Y, yi), vol[i],
                    __int_as_float(k));
  }
}

constexpr int kPT = 8;  // points per CTA of grad_mp_wide_kernel

// Table entries of two bins each: (tc^2, tc^2, 1 / tc^4, 1 / tc^4) of bins 2 i
// and 2 i + 1, padded to a multiple of four bins. A sample's f2 = (depth / tc^2)^4 is
// (d2 / tc^4)^2: 1 / tc^8 and d2^2, whose product it is too, leave the FP32 range at tc
// of 4e5 and 1e-5 (a scene of a metre in micrometres, or in light microseconds).
__host__ __device__ constexpr int bin_table(int T) { return 2 * ((T + 3) / 4); }

// One measurement point's constants for the walks over occupied voxels.
struct WalkPoint {
  float wx, wy, wz;
  float ea, eb;  // span_eps as ea ch + eb, at most 1
  float ma, mb;  // the margin of a cell fraction as ma ch + mb
};
__device__ __forceinline__ WalkPoint walk_point(const Geo& g, float wx, float wy, float wz) {
  const float u = 5.9604645e-8f;
  WalkPoint p{wx, wy, wz, 0.f, 0.f, 0.f, 0.f};
  // |tc| <= dmax = 1.001 (ch + 2 |bw|) on the walked bins, |z| <= |wz| + dmax
  const float rest = 2.002f * fabsf(g.bw);
  const float za = fabsf(wz), zo = fabsf(g.oz);
  p.ea = 64.f * u * 2.002f * fabsf(g.inv_bw);
  p.eb = 64.f * u * (2.f * rest + fabsf(g.bo) + 2.f * za + zo + fabsf(1.f / g.scale)) *
             fabsf(g.inv_bw) + 0.01f;
  // 8 u scale (dmax + |wz| + |z| + |oz|) + 4 u |zh| + 1e-7, |zh| <= (|z| + |oz|) scale + 1/2,
  // a thousandth wider for the rounding of these bounds
  const float s = fabsf(g.scale) * 1.001f * u;
  p.ma = s * 20.f * 1.002f;
  p.mb = s * (20.f * rest + 20.f * za + 12.f * zo) + 2.5f * u + 1e-7f;
  return p;
}

// Calls f(t, lower, fr, a, b, depth), f2 = (a b)^2, for every sample of the point in the
// interpolation cells of an occupied voxel (column centre x, y, cell k): lower
// is true for cell k (the voxel is its lower node, weight 1 - fr) and false for
// cell k - 1 (weight fr). The bins come from inverting the column geometry,
// widened by span_eps, two at a time from an even one with paired FP32
// instructions; tab holds (tc^2, tc^2, 1 / tc^4, 1 / tc^4) of each two. The depth
// is the hardware reciprocal square root's with one remainder correction
// (within an ulp of the correctly rounded root), the cell coordinate the
// exact chain's operations on it; where its fraction lies within the margin of a
// cell boundary the sample is decided by sample(). A sample with d2 <= 0 has a
// NaN cell. The even bin before a span holds no sample of the voxel; with
// kSigned (negative bin centres) it may belong to the other span and is
// skipped.
template <bool kSigned, class F>
__device__ __forceinline__ void walk_voxel(const Geo& g, const float4* tab, const WalkPoint& p,
                                           int tz, float x, float y, int k, F f) {
  using u64 = unsigned long long;
  const float dx = xsub(p.wx, x), dy = xsub(p.wy, y);
  const float ddx = xmul(dx, dx), ddy = xmul(dy, dy);
  const float rho2 = ddx + ddy;
  const float dhi = fmaf((float)k + 1.5f, g.dz, g.oz) - p.wz;
  if (!(dhi > 0.f)) return;
  const float dlo = fmaxf(fmaf((float)k - 0.5f, g.dz, g.oz) - p.wz, 0.f);
  const float cl = sqrt_approx(fmaf(dlo, dlo, rho2)), ch = sqrt_approx(fmaf(dhi, dhi, rho2));
  const Spans sp = tc_spans(g, tz, cl, ch, fminf(fmaf(p.ea, ch, p.eb), 1.f));
  const float pm = fmaf(p.ma, ch, p.mb);
  const float lim = g.exact || !(pm < 0.5f) ? 0.f : 0.5f - pm;
  const u64 ndx = f2pack(-ddx, -ddx), ndy = f2pack(-ddy, -ddy);
  const u64 wz = f2pack(p.wz, p.wz), noz = f2pack(-g.oz, -g.oz);
  const u64 scale = f2pack(g.scale, g.scale), half = f2pack(-0.5f, -0.5f);
  const u64 big = f2pack(12582912.f, 12582912.f);  // 1.5 2^23
  // cells k (if it has a node above) and k - 1 (if there is one) as bit patterns
  const int lower = k + 1 < g.Z ? 0x4B400000 + k : -2;
  const int upper = k > 0 ? 0x4B400000 + k - 1 : -2;
#pragma unroll 1
  for (int r = 0; r < (kSigned ? 2 : 1); ++r) {
    const int t0 = r ? sp.n0 : sp.p0, t1 = r ? sp.n1 : sp.p1;
#pragma unroll 1
    for (int t = t0 & ~1; t <= t1; t += 2) {
      const float4 tb = tab[t >> 1];
      const u64 d2 = f2add(f2add(f2pack(tb.x, tb.y), ndx), ndy);
      float d[2], z[2], fr[2], off[2], depth[2], i4[2] = {tb.z, tb.w};
      f2unpack(d2, d[0], d[1]);
      const float r0 = rsqrt_approx(d[0]), r1 = rsqrt_approx(d[1]);
      u64 q = f2mul(d2, f2pack(r0, r1));
      q = f2fma(f2fma(f2mul(q, f2pack(-1.f, -1.f)), q, d2), f2mul(f2pack(r0, r1), f2pack(0.5f, 0.5f)),
                q);
      f2unpack(q, depth[0], depth[1]);
      const u64 zh = f2add(f2mul(f2add(f2add(q, wz), noz), scale), half);
      const u64 fx = f2add_rm(zh, big);
      const u64 fr2 = f2sub(zh, f2sub(fx, big));
      f2unpack(fx, z[0], z[1]);
      f2unpack(fr2, fr[0], fr[1]);
      f2unpack(f2add(fr2, half), off[0], off[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (kSigned && (t + h < t0 || t + h > t1)) continue;
        int cell = __float_as_int(z[h]);
        if (fabsf(off[h]) >= lim) {  // (NaN: no)
          const Sample sm = sample(g, p.wx, p.wy, p.wz, t + h, x, y);
          cell = sm.ok ? 0x4B400000 + sm.zi : -1;
          fr[h] = sm.alpha;
          d[h] = sm.f1;
          i4[h] = 1.f;
        }
        if (cell == lower || cell == upper)
          f(t + h, cell == lower, fr[h], d[h], i4[h], depth[h]);
      }
    }
  }
}

// The bin table of walk_voxel, in shared memory; all threads of the CTA.
__device__ __forceinline__ void fill_bin_table(const Geo& g, float4* tab) {
  for (int i = threadIdx.x; i < bin_table(g.T); i += blockDim.x) {
    float tc2[2], i4[2];
    for (int h = 0; h < 2; ++h) {
      const int t = 2 * i + h;
      const float tc = xadd(xmul((float)t, g.bw), g.bo);
      tc2[h] = xmul(tc, tc);
      const float i2 = __fdividef(1.f, tc2[h]);
      i4[h] = i2 * i2;
      if (t >= g.T) tc2[h] = -INFINITY, i4[h] = 0.f;  // padding: no sample
    }
    tab[i] = make_float4(tc2[0], tc2[1], i4[0], i4[1]);
  }
}

// f(p, t) for the n rows of T bins, t fastest, over the threads of the CTA (without a
// division per element: the forward of 8^3 voxels, 16,384 rows of 4,096 bins, took 0.69 ms
// with one and takes 0.56).
template <class F>
__device__ __forceinline__ void for_rows(int n, int T, F f) {
  if (T <= 0) return;
  int p = threadIdx.x / T, t = threadIdx.x - p * T;
  const int dp = blockDim.x / T, dt = blockDim.x - dp * T;
  while (p < n) {
    f(p, t);
    p += dp;
    t += dt;
    if (t >= T) t -= T, ++p;
  }
}

// Confocal forward: a CTA takes PT points and a slice of the occupied voxels,
// and keeps the points' bins in shared memory ([bin][point]: with 32 points the
// lanes of a warp add to 32 banks). A thread walks one point over every
// (blockDim / PT)-th voxel. With several slices the CTAs add into a zeroed output.
// What bounds it: the compare-and-swap adds (the measurement-point gradient,
// with the same walks and reads in their place, takes two thirds of the time)
// and instruction issue. 128^3 voxels (2%) x 16,384 points x 1,024 bins: 7.35 ->
// 5.4 ms; 41 x 37 x 53 (10%) x 899 points x 500 bins: 0.535 -> 0.11 ms.
template <int PT, bool kSigned>
__global__ void __launch_bounds__(32 * PT > 256 ? 32 * PT : 256) confocal_forward_kernel(
    Geo g, const float4* __restrict__ recs, const uint32_t* __restrict__ count, Points mp, int N,
    float* __restrict__ out) {
  extern __shared__ __align__(16) float hist[];  // [T][PT], then the bin table
  float4* tab = reinterpret_cast<float4*>(hist + (((size_t)PT * g.T + 3) & ~(size_t)3));
  const int i0 = blockIdx.x * PT;
  for (int j = threadIdx.x; j < PT * g.T; j += blockDim.x) hist[j] = 0.f;
  fill_bin_table(g, tab);
  __syncthreads();
  const uint32_t nnz = *count;
  const uint32_t v0 = (uint32_t)((uint64_t)nnz * blockIdx.y / gridDim.y);
  const uint32_t v1 = (uint32_t)((uint64_t)nnz * (blockIdx.y + 1) / gridDim.y);
  const int pl = threadIdx.x % PT;
  const int i = i0 + pl;
  const int tz = kSigned ? first_nonneg_bin(g) : 0;
  if (i < N) {
    const WalkPoint p = walk_point(g, mp.at(0, i), mp.at(1, i), mp.at(2, i));
    float* col = hist + pl;
    for (uint32_t v = v0 + threadIdx.x / PT; v < v1; v += blockDim.x / PT) {
      const float4 rec = __ldg(recs + v);
      walk_voxel<kSigned>(g, tab, p, tz, rec.x, rec.y, __float_as_int(rec.w),
                          [&](int t, bool lower, float fr, float a, float b, float) {
                            const float w = lower ? 1.f - fr : fr, f1 = a * b;
                            atomicAdd(col + t * PT, rec.z * w * (f1 * f1));
                          });
    }
  }
  __syncthreads();
  for_rows(min(PT, N - i0), g.T, [&](int p, int t) {
    float* dst = out + (size_t)(i0 + p) * g.T + t;
    const float h = hist[t * PT + p];
    if (gridDim.y == 1) *dst = h;
    else if (h != 0.f) atomicAdd(dst, h);
  });
}

// d transient / d measurement points (volume_cuda.cu:189-265) with the same
// walks: a thread accumulates one point over its share of the voxels, and the shares
// are reduced in shared memory (then added into a zeroed output when there are
// several slices of the voxels). 41 x 37 x 53 voxels (10%) x 899 points x 500 bins: 0.55
// -> 0.10 ms. transient_grad is read in place, a voxel's few bins of a row, or its rows
// are staged in shared memory (kRows: few points, long rows, see the launcher): with the
// rows staged 1,024 bins took as long (0.92 to 1.02 of the time, by voxels and
// points), 2,048 bins 1.3 to 3 times and 4,096 bins 2 to 7 times as long (16,384 rows for
// the 10 voxels of an 8^3 volume 1.2 against 0.18 ms).
template <int PT, bool kSigned, bool kRows>
__global__ void __launch_bounds__(32 * PT > 256 ? 32 * PT : 256) grad_mp_kernel(
    Geo g, const float4* __restrict__ recs, const uint32_t* __restrict__ count, Points mp, int N,
    const float* __restrict__ tg, float* __restrict__ out, int64_t osc, int64_t osn) {
  extern __shared__ __align__(16) float rows[];  // kRows: [T][PT]; then the bin table
  float4* tab = reinterpret_cast<float4*>(rows + (kRows ? ((size_t)PT * g.T + 3) & ~(size_t)3 : 0));
  __shared__ float sum[PT][3];
  const int i0 = blockIdx.x * PT;
  if (kRows)
    for_rows(PT, g.T, [&](int p, int t) {
      rows[t * PT + p] = i0 + p < N ? __ldg(tg + (size_t)(i0 + p) * g.T + t) : 0.f;
    });
  fill_bin_table(g, tab);
  if (threadIdx.x < PT) sum[threadIdx.x][0] = sum[threadIdx.x][1] = sum[threadIdx.x][2] = 0.f;
  __syncthreads();
  const uint32_t nnz = *count;
  const uint32_t v0 = (uint32_t)((uint64_t)nnz * blockIdx.y / gridDim.y);
  const uint32_t v1 = (uint32_t)((uint64_t)nnz * (blockIdx.y + 1) / gridDim.y);
  const int pl = threadIdx.x % PT;
  const int i = i0 + pl;
  float gx = 0.f, gy = 0.f, gz = 0.f;
  const int tz = kSigned ? first_nonneg_bin(g) : 0;
  if (i < N) {
    const WalkPoint p = walk_point(g, mp.at(0, i), mp.at(1, i), mp.at(2, i));
    const float* row = tg + (size_t)i * g.T;
    for (uint32_t v = v0 + threadIdx.x / PT; v < v1; v += blockDim.x / PT) {
      const float4 rec = __ldg(recs + v);
      // with f2 = (depth / tc^2)^4 and w the interpolation weight, d(w f2) / d depth
      // = w 4 f2 / depth +- scale f2, and d depth / d(wx, wy) = -(wx - x, wy - y) / depth
      // (lengths of the quotient in slices, so that it keeps the range of the result)
      float radial = 0.f, axial = 0.f;
      walk_voxel<kSigned>(g, tab, p, tz, rec.x, rec.y, __float_as_int(rec.w),
                          [&](int t, bool lower, float fr, float a, float b, float depth) {
                            const float w = lower ? 1.f - fr : fr, f1 = a * b;
                            const float y = kRows ? rows[t * PT + pl] : __ldg(row + t);
                            const float df2 = y * (f1 * f1);
                            const float slope = lower ? -g.scale * df2 : g.scale * df2;
                            const float inv = __fdividef(1.f, depth);
                            radial += fmaf(4.f * w * df2, inv, slope) * (inv * g.dz);
                            axial += slope;
                          });
      // (an infinite voxel or point without a sample adds nothing)
      gx -= radial != 0.f ? rec.z * ((p.wx - rec.x) * g.scale) * radial : 0.f;
      gy -= radial != 0.f ? rec.z * ((p.wy - rec.y) * g.scale) * radial : 0.f;
      gz += axial != 0.f ? rec.z * axial : 0.f;
    }
  }
  for (int o = PT; o < 32; o <<= 1) {
    gx += __shfl_xor_sync(0xffffffffu, gx, o);
    gy += __shfl_xor_sync(0xffffffffu, gy, o);
    gz += __shfl_xor_sync(0xffffffffu, gz, o);
  }
  if ((threadIdx.x & 31) < PT) {
    atomicAdd(&sum[pl][0], gx);
    atomicAdd(&sum[pl][1], gy);
    atomicAdd(&sum[pl][2], gz);
  }
  __syncthreads();
  if (threadIdx.x < PT && i0 + (int)threadIdx.x < N) {
    const int ii = i0 + threadIdx.x;
    for (int c = 0; c < 3; ++c) {
      float* dst = out + c * osc + ii * osn;
      if (gridDim.y == 1) *dst = sum[threadIdx.x][c];
      else atomicAdd(dst, sum[threadIdx.x][c]);
    }
  }
}

// grad_mp_kernel for bin tables that do not fit shared memory: every sample by the
// exact chain; one thread accumulates one point's gradient over a share of the voxels,
// reduced across the kPT-strided threads in shared memory.
__global__ void __launch_bounds__(256) grad_mp_wide_kernel(Geo g, const float4* __restrict__ recs,
                                                      const uint32_t* __restrict__ count,
                                                      Points mp, int N,
                                                      const float* __restrict__ tg,
                                                      float* __restrict__ out, int64_t osc,
                                                      int64_t osn) {
  __shared__ float red[256][3];
  const int i0 = blockIdx.x * kPT;
  const uint32_t nnz = *count;
  const int pl = threadIdx.x % kPT;
  const int i = i0 + pl;
  float gx = 0.f, gy = 0.f, gz = 0.f;
  const int tz = first_nonneg_bin(g);
  if (i < N) {
    const float wx = mp.at(0, i), wy = mp.at(1, i), wz = mp.at(2, i);
    const float* trow = tg + (size_t)i * g.T;
    for (uint32_t v = threadIdx.x / kPT; v < nnz; v += blockDim.x / kPT) {
      const float4 rec = __ldg(recs + v);
      const float x = rec.x, y = rec.y, val = rec.z;
      const int k = __float_as_int(rec.w);
      const float rho2 = (wx - x) * (wx - x) + (wy - y) * (wy - y);
      const Spans sp = bin_range(g, tz, rho2, wz, k);
      for (int r = 0; r < 2; ++r) {
        const int t0 = r ? sp.n0 : sp.p0, t1 = r ? sp.n1 : sp.p1;
        for (int t = t0; t <= t1; ++t) {
          const Sample s = sample(g, wx, wy, wz, t, x, y);
          if (!s.ok || (s.zi != k && s.zi != k - 1)) continue;
          const float tc = (float)t * g.bw + g.bo;
          const float depth =
              sqrtf(fmaxf(tc * tc - (wx - x) * (wx - x) - (wy - y) * (wy - y), 0.f));
          const float dzx = -(wx - x) / depth, dzy = -(wy - y) / depth;
          const float tc2 = tc * tc, tc4 = tc2 * tc2;
          const float df2 = 4.f * depth * depth * depth / (tc4 * tc4);
          // this voxel is the lower (zi == k) or upper (zi == k-1) interpolation node
          const bool lower = s.zi == k;
          const float wgt = lower ? 1.f - s.alpha : s.alpha;
          const float sgn = lower ? -1.f : 1.f;
          const float dl = __ldg(trow + t) * val;
          gx += dl * (wgt * df2 * dzx + sgn * g.scale * dzx * s.f2);
          gy += dl * (wgt * df2 * dzy + sgn * g.scale * dzy * s.f2);
          gz += dl * (sgn * g.scale * s.f2);
        }
      }
    }
  }
  red[threadIdx.x][0] = gx;
  red[threadIdx.x][1] = gy;
  red[threadIdx.x][2] = gz;
  __syncthreads();
  if (threadIdx.x < kPT && i0 + threadIdx.x < N) {
    float a = 0.f, b = 0.f, c = 0.f;
    for (int j = threadIdx.x; j < blockDim.x; j += kPT) {
      a += red[j][0];
      b += red[j][1];
      c += red[j][2];
    }
    const int ii = i0 + threadIdx.x;
    out[ii * osn] = a;
    out[osc + ii * osn] = b;
    out[2 * osc + ii * osn] = c;
  }
}

// Bins whose samples can land in any interpolation cell of a column seen from
// a point at squared horizontal distance rho2 and height wz: cells 0 .. Z-2
// hold z in [oz + 0.5/scale, oz + (Z - 0.5)/scale), widened by one cell above
// and one bin each side (bin_range's spans for cells 1 and Z - 1).
__device__ __forceinline__ Spans column_span(const Geo& g, int tz, float rho2, float wz) {
  float cl, ch;
  if (!tc_bounds(rho2, wz, g.oz + 0.5f / g.scale, g.oz + ((float)g.Z + 0.5f) / g.scale, cl, ch))
    return Spans{1, 0, 1, 0};
  return within_bins(g, tc_spans(g, tz, cl, ch, 1.f));
}

// Largest |t bw + bo| over the bins of two spans (0 when both are empty).
__device__ __forceinline__ float span_tc_max(const Geo& g, const Spans& s) {
  float m = 0.f;
  if (s.p0 <= s.p1)
    m = fmaxf(fabsf((float)s.p1 * g.bw + g.bo), fabsf((float)s.p0 * g.bw + g.bo));
  if (s.n0 <= s.n1)
    m = fmaxf(m, fmaxf(fabsf((float)s.n1 * g.bw + g.bo), fabsf((float)s.n0 * g.bw + g.bo)));
  return m;
}

// Exact adjoint of the forward: one CTA per voxel column, a warp per point at a
// time, its lanes over the point's bins (neighbouring lanes' samples fall in
// neighbouring cells and the transient row is read 128 bytes at a time). Each
// warp accumulates into its own copy of the column in shared memory (eight
// copies), summed at the end. The per-point work (the column's bin span, the
// exact squared horizontal offsets of the sample chain, the filtered path's
// margin) is done once per point by one lane for 32 points at a time and
// handed to the warp with shuffles, instead of by all 32 lanes for every point
// (148 ms for that version on 128^3 voxels x 16,384 points x 1,024 bins).
// The margin bounds the fast path's over every bin of the span, so every decision is
// the exact chain's.
__global__ void __launch_bounds__(256) confocal_adjoint_kernel(Geo g, Points mp, int N,
                                                               const float* __restrict__ tr,
                                                               float* __restrict__ vol) {
  extern __shared__ float cols[];  // [8][Z]
  const int c = blockIdx.x;
  const int xi = c / g.Y, yi = c - xi * g.Y;
  for (int z = threadIdx.x; z < 8 * g.Z; z += blockDim.x) cols[z] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* col = cols + warp * g.Z;
  const float x = centre(g.ox, g.sx, g.X, xi), y = centre(g.oy, g.sy, g.Y, yi);
  const float u = 5.9604645e-8f;
  const int tz = first_nonneg_bin(g);
  for (int base = warp * 32; base < N; base += 256) {
    // lane j prepares point base + j
    const int ip = base + lane;
    float wx = 0.f, wy = 0.f, wz = 0.f, ddx = 0.f, ddy = 0.f, marg = 0.f;
    Spans sp{1, 0, 1, 0};
    if (ip < N) {
      wx = mp.at(0, ip);
      wy = mp.at(1, ip);
      wz = mp.at(2, ip);
      const float dx = xsub(wx, x), dy = xsub(wy, y);
      ddx = xmul(dx, dx);
      ddy = xmul(dy, dy);
      sp = column_span(g, tz, dx * dx + dy * dy, wz);
      // the margin 8 u scale (depth + |wz| + |z| + |oz|) + 4 u |zh|
      // + 1e-7 with depth, |z| and |zh| at their largest over the spans' bins
      const float dmax = 1.001f * span_tc_max(g, sp);
      const float zmax = fabsf(wz) + dmax;
      const float zhmax = (zmax + fabsf(g.oz)) * g.scale + 0.5f;
      marg = 8.f * u * g.scale * (dmax + fabsf(wz) + zmax + fabsf(g.oz)) + 4.f * u * zhmax +
             1e-7f;
    }
    const int np = min(32, N - base);
    for (int j = 0; j < np; ++j) {
      const int p0 = __shfl_sync(0xffffffffu, sp.p0, j), p1 = __shfl_sync(0xffffffffu, sp.p1, j);
      const int n0 = __shfl_sync(0xffffffffu, sp.n0, j), n1 = __shfl_sync(0xffffffffu, sp.n1, j);
      if (p0 > p1 && n0 > n1) continue;  // warp-uniform
      const float pwx = __shfl_sync(0xffffffffu, wx, j), pwy = __shfl_sync(0xffffffffu, wy, j);
      const float pwz = __shfl_sync(0xffffffffu, wz, j);
      const float pddx = __shfl_sync(0xffffffffu, ddx, j);
      const float pddy = __shfl_sync(0xffffffffu, ddy, j);
      const float pm = __shfl_sync(0xffffffffu, marg, j);
      const float* row = tr + (size_t)(base + j) * g.T;
      for (int r = 0; r < 2; ++r) {
        const int t0 = r ? n0 : p0, t1 = r ? n1 : p1;
        for (int t = t0 + lane; t <= t1; t += 32) {
          // the fast path with the point's constants
          const float tc = xadd(xmul((float)t, g.bw), g.bo);
          const float d2 = xsub(xsub(xmul(tc, tc), pddx), pddy);
          if (!(d2 > 0.f)) continue;
          Sample sm;
          const float depth = d2 * rsqrtf(d2);
          const float zh = fmaf((pwz + depth) - g.oz, g.scale, -0.5f);
          const float fl = floorf(zh);
          const float fr = zh - fl;
          if (!g.exact && fr > pm && fr < 1.f - pm) {
            if (!(fl >= 0.f && fl + 1.f < (float)g.Z)) continue;
            sm.zi = (int)fl;
            sm.alpha = fr;
            const float q = __fdividef(depth, tc * tc);
            sm.f2 = (q * q) * (q * q);
          } else {
            sm = sample(g, pwx, pwy, pwz, t, x, y);
            if (!sm.ok) continue;
          }
          const float v = __ldg(row + t) * sm.f2;
          atomicAdd(col + sm.zi, (1.f - sm.alpha) * v);
          atomicAdd(col + sm.zi + 1, sm.alpha * v);
        }
      }
    }
  }
  __syncthreads();
  for (int z = threadIdx.x; z < g.Z; z += blockDim.x) {
    float sum = 0.f;
    for (int w = 0; w < 8; ++w) sum += cols[w * g.Z + z];
    vol[(size_t)c * g.Z + z] = sum;
  }
}

// Exact adjoint of the forward without atomics, for columns of at most 32 CPL
// cells: one CTA per voxel column, each warp over a share of the points (all
// 32 lanes on the same point), lane l owning the CPL cells z0 = l CPL ..
// z0 + CPL - 1. A sample whose lower interpolation cell zi is the lane's adds
// (1 - alpha) v to cell zi and alpha v to cell zi + 1; when zi + 1 is the next
// lane's first cell that share goes to a per-lane carry register, added in at
// the end. The samples a lane walks are those of the bins whose centres map to
// its cells: the bin coordinate of each cell boundary from one square root,
// widened by eps bins, a bound on the FP32 rounding of the sample chain
// against that inverse (64 u of the largest magnitudes, over the bin width,
// plus 0.01, at most the one bin of column_span, inside which the per-point
// margin holds). Each sample's decisions are the exact chain's (the fast path
// with the per-point margin, as in confocal_adjoint_kernel), so every kept
// sample is the forward's and each lands in exactly one lane.
template <int CPL>
__global__ void __launch_bounds__(256) confocal_adjoint_cells_kernel(Geo g, Points mp, int N,
                                                                     const float* __restrict__ tr,
                                                                     float* __restrict__ vol) {
  __shared__ float cells[8][CPL][32];  // [warp][cell of the lane][lane]
  __shared__ float carry_in[8][32];
  const int c = blockIdx.x;
  const int xi = c / g.Y, yi = c - xi * g.Y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < CPL; ++k) cells[warp][k][lane] = 0.f;
  const float x = centre(g.ox, g.sx, g.X, xi), y = centre(g.oy, g.sy, g.Y, yi);
  const float u = 5.9604645e-8f;
  const int tz = first_nonneg_bin(g);
  // this lane's lower cells zi in [za, zb): z in [zlo, zhi)
  const int za = lane * CPL, zb = min(za + CPL, g.Z - 1);
  const float zlo = g.oz + ((float)za + 0.5f) / g.scale;
  const float zhi = g.oz + ((float)zb + 0.5f) / g.scale;
  float carry = 0.f;
  for (int base = warp * 32; base < N; base += 256) {
    // lane j prepares point base + j
    const int ip = base + lane;
    float wx = 0.f, wy = 0.f, wz = 0.f, ddx = 0.f, ddy = 0.f, marg = 0.f, eps = 0.f;
    if (ip < N) {
      wx = mp.at(0, ip);
      wy = mp.at(1, ip);
      wz = mp.at(2, ip);
      const float dx = xsub(wx, x), dy = xsub(wy, y);
      ddx = xmul(dx, dx);
      ddy = xmul(dy, dy);
      const Spans sp = column_span(g, tz, dx * dx + dy * dy, wz);
      const float dmax = 1.001f * span_tc_max(g, sp);
      const float zmax = fabsf(wz) + dmax;
      const float zhmax = (zmax + fabsf(g.oz)) * g.scale + 0.5f;
      marg = 8.f * u * g.scale * (dmax + fabsf(wz) + zmax + fabsf(g.oz)) + 4.f * u * zhmax +
             1e-7f;
      eps = fminf(64.f * u * (dmax + fabsf(g.bo) + fabsf(wz) + zmax + fabsf(g.oz) +
                              1.f / g.scale) * g.inv_bw + 0.01f,
                  1.f);
    }
    const int np = min(32, N - base);
    for (int j = 0; j < np; ++j) {
      const float pwx = __shfl_sync(0xffffffffu, wx, j), pwy = __shfl_sync(0xffffffffu, wy, j);
      const float pwz = __shfl_sync(0xffffffffu, wz, j);
      const float pddx = __shfl_sync(0xffffffffu, ddx, j);
      const float pddy = __shfl_sync(0xffffffffu, ddy, j);
      const float pm = __shfl_sync(0xffffffffu, marg, j);
      const float pe = __shfl_sync(0xffffffffu, eps, j);
      Spans sp{1, 0, 1, 0};
      float cl, ch;
      if (za < zb && tc_bounds(pddx + pddy, pwz, zlo, zhi, cl, ch))
        sp = tc_spans(g, tz, cl, ch, pe);
      const float* row = tr + (size_t)(base + j) * g.T;
      for (int r = 0; r < 2; ++r) {
        const int t0 = r ? sp.n0 : sp.p0, t1 = r ? sp.n1 : sp.p1;
        for (int t = t0; t <= t1; ++t) {
          const float tc = xadd(xmul((float)t, g.bw), g.bo);
          const float d2 = xsub(xsub(xmul(tc, tc), pddx), pddy);
          if (!(d2 > 0.f)) continue;
          int zi;
          float alpha, f2;
          const float depth = d2 * rsqrtf(d2);
          const float zh = fmaf((pwz + depth) - g.oz, g.scale, -0.5f);
          const float fl = floorf(zh);
          const float fr = zh - fl;
          if (!g.exact && fr > pm && fr < 1.f - pm) {
            if (!(fl >= (float)za && fl < (float)zb)) continue;
            zi = (int)fl;
            alpha = fr;
            const float q = __fdividef(depth, tc * tc);
            f2 = (q * q) * (q * q);
          } else {
            const Sample sm = sample(g, pwx, pwy, pwz, t, x, y);
            if (!sm.ok || sm.zi < za || sm.zi >= zb) continue;
            zi = sm.zi;
            alpha = sm.alpha;
            f2 = sm.f2;
          }
          const float v = __ldg(row + t) * f2;
          const int k = zi - za;
          cells[warp][k][lane] += (1.f - alpha) * v;
          if (k + 1 < CPL) cells[warp][k + 1][lane] += alpha * v;
          else carry += alpha * v;
        }
      }
    }
  }
  carry_in[warp][lane] = carry;
  __syncthreads();
  for (int z = threadIdx.x; z < g.Z; z += blockDim.x) {
    const int l = z / CPL, k = z - l * CPL;
    float sum = 0.f;
    for (int w = 0; w < 8; ++w) {
      sum += cells[w][k][l];
      if (k == 0 && l > 0) sum += carry_in[w][l - 1];
    }
    vol[(size_t)c * g.Z + z] = sum;
  }
}

// Adds w0 to cell row `u` and w1 to the next one of the lane's column (at
// shared-memory address `col`, rows 128 bytes apart) when u < zn. Predicated
// loads and stores: a select of the row or of zero weights took three more
// instructions.
__device__ __forceinline__ void adj_add(uint32_t col, unsigned u, unsigned zn, float w0,
                                        float w1) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .f32 a, b;\n\t"
      "setp.lt.u32 p, %1, %2;\n\t"
      "@p ld.shared.f32 a, [%0];\n\t"
      "@p ld.shared.f32 b, [%0 + 128];\n\t"
      "add.f32 a, a, %3;\n\t"
      "add.f32 b, b, %4;\n\t"
      "@p st.shared.f32 [%0], a;\n\t"
      "@p st.shared.f32 [%0 + 128], b;\n\t"
      "}"
      :: "r"(col + 128u * u), "r"(u), "r"(zn), "f"(w0), "f"(w1)
      : "memory");
}

// A point as the lane's column sees it.
struct AdjPoint {
  float ndx, ndy;  // minus the squared horizontal offsets (the sample chain's)
  float wx, wy, wz;
  float lim;       // 1/2 - margin of a cell fraction
};

// The bins [t0, t1] of one point for the lanes' columns, four at a time from
// the multiple of four at or below t0, in pairs with paired FP32
// instructions. `val` holds the values of the first 32 bins, one per lane;
// each chunk of 32 passes through the warp's buffer, from where four come by
// one broadcast read (as the table entries of two bins do), and the next chunk
// is read ahead. floor(z_hat) is the addition of 1.5 2^23 rounded down, whose
// low mantissa bits are the cell. A sample with d2 <= 0 has a NaN z_hat, whose
// bits are past every cell. Samples within the rounding margin of a cell
// boundary go through the exact chain. The step may touch up to three bins on
// each side of [t0, t1]: without kCheck (no negative bin centres) those are real
// bins, rejected unless they hold a sample, or table padding (tc^2 = -inf); with
// kCheck they belong to the other walk and are skipped. A sample's cell is the exact
// chain's; its fraction and f2 are values of the paired arithmetic or, near a
// boundary, of the exact chain.
template <bool kCheck>
__device__ __forceinline__ void adj_walk(const Geo& g, const float4* __restrict__ tab,
                                         float4* vbuf, const float* __restrict__ row,
                                         const AdjPoint& p, int t0, int t1, float val, int lane,
                                         uint32_t col, float x, float y, int za, int zn) {
  using u64 = unsigned long long;
  const u64 ndx = f2pack(p.ndx, p.ndx), ndy = f2pack(p.ndy, p.ndy);
  const u64 wzo = f2pack(p.wz - g.oz, p.wz - g.oz), scale = f2pack(g.scale, g.scale);
  const u64 half = f2pack(-0.5f, -0.5f);
  const u64 big = f2pack(12582912.f, 12582912.f);  // 1.5 2^23
  const unsigned bias = 0x4B400000u + (unsigned)za;
  for (int c = t0 & ~3; c <= t1; c += 32) {
    __syncwarp();
    reinterpret_cast<float*>(vbuf)[lane] = val;
    // (v - alpha v is NaN where v overflows: chunks with infinite or huge values go
    // through the exact chain, whose (1 - alpha) v is not)
    const float lim = __any_sync(0xffffffffu, !(fabsf(val) < 1e30f)) ? 0.f : p.lim;
    __syncwarp();
    if (c + 32 <= t1) val = c + 32 + lane < g.T ? __ldg(row + c + 32 + lane) : 0.f;
    const int n = min(32, t1 - c + 1);
#pragma unroll 1
    for (int s = 0; s < n; s += 4) {
      const float4 v4 = vbuf[s >> 2];
      unsigned u[4];
      float w0[4], w1[4], off[4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float4 tb = tab[((c + s) >> 1) + h];
        if (kCheck) {
          const int t = c + s + 2 * h;
          if (t < t0 || t > t1) tb.x = -INFINITY;
          if (t + 1 < t0 || t + 1 > t1) tb.y = -INFINITY;
        }
        const u64 d2 = f2add(f2add(f2pack(tb.x, tb.y), ndx), ndy);
        float da, db, xa, xb;
        f2unpack(d2, da, db);
        const u64 zh = f2fma(f2fma(d2, f2pack(rsqrt_approx(da), rsqrt_approx(db)), wzo), scale,
                             half);
        const u64 fx = f2add_rm(zh, big);
        const u64 fr = f2sub(zh, f2sub(fx, big));
        f2unpack(fx, xa, xb);
        f2unpack(f2add(fr, half), off[2 * h], off[2 * h + 1]);
        const u64 fall = f2mul(d2, f2pack(tb.z, tb.w));
        const u64 v = f2mul(f2mul(fall, fall), h ? f2pack(v4.z, v4.w) : f2pack(v4.x, v4.y));
        const u64 upper = f2mul(fr, v);
        f2unpack(upper, w1[2 * h], w1[2 * h + 1]);
        f2unpack(f2sub(v, upper), w0[2 * h], w0[2 * h + 1]);
        u[2 * h] = __float_as_uint(xa) - bias;
        u[2 * h + 1] = __float_as_uint(xb) - bias;
      }
      // (NaN fractions are passed over)
      if (absmax3(absmax3(0.f, off[0], off[1]), off[2], off[3]) >= lim) {
        unsigned slow = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (fabsf(off[q]) >= lim) slow |= 1u << q, u[q] = 0xffffffffu;
        do {
          const int q = __ffs(slow) - 1;
          slow &= slow - 1;
          const Sample sm = sample(g, p.wx, p.wy, p.wz, c + s + q, x, y);
          const float v = reinterpret_cast<const float*>(vbuf)[s + q] * sm.f2;
          if (sm.ok)
            adj_add(col, (unsigned)(sm.zi - za), (unsigned)zn, (1.f - sm.alpha) * v, sm.alpha * v);
        } while (slow);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) adj_add(col, u[q], (unsigned)zn, w0[q], w1[q]);
    }
  }
}

// The end of confocal_adjoint_columns_kernel in a cluster of point groups: a cell's sum
// over the warps' copies of all groups, in order, so that the result does not depend
// on which group ends first (two slabs share a cell, but two terms added to zero
// commute).
__device__ __forceinline__ void add_cluster_columns(const Geo& g, float* acc, int nw, int rows,
                                                    int tx, int ty, int za, float* vol,
                                                    int accumulate) {
  cg::cluster_group cluster = cg::this_cluster();
  const int peers = (int)cluster.num_blocks();
  cluster.sync();  // every group has its copies
  for (int jj = cluster.block_rank() * blockDim.x + threadIdx.x; jj < rows * 32;
       jj += peers * blockDim.x) {
    const int r = jj >> 5, l = jj & 31, z = za + r;
    const int cy = ty + (l & 7), cx = tx + (l >> 3);
    if (cx >= g.X || cy >= g.Y || z >= g.Z) continue;
    float sum = 0.f;
    for (int c = 0; c < peers; ++c) {
      const float* copies = cluster.map_shared_rank(acc, c);
      for (int w = 0; w < nw; ++w) sum += copies[((size_t)w * rows + r) * 32 + l];
    }
    float* dst = vol + ((size_t)cx * g.Y + cy) * g.Z + z;
    if (accumulate) atomicAdd(dst, sum);
    else *dst = sum;
  }
  cluster.sync();  // no group leaves while another reads its copies
}

// Exact adjoint of the forward with the lanes of a warp over 32 neighbouring
// voxel columns (an 8 x 4 tile: y fastest) and all lanes on one point and one
// bin at a time. The point's transient row is then read once per warp (32 bins
// per coalesced load), and the bin's tc^2 (the sample chain's FP32 value) and
// 1 / tc^4 come from a per-CTA table in shared memory (broadcast reads), so f2 =
// (depth / tc^2)^4 = (d2 / tc^4)^2 needs no second special-function op. A CTA
// takes one slab of the columns' cells (the samples whose cell pair starts
// there; the pair's second cell may be the next slab's first, one extra row),
// and each lane owns its column's cells of the slab in shared memory
// ([cell][lane]: no bank conflicts, no atomics), one copy per warp; the warps
// of a CTA take interleaved runs of 32 points of one point group, and the CTA
// adds its summed columns into the volume (which the launcher zeroes) with one
// atomic per cell when there is more than one group or slab. A point's bins
// are those whose samples can land in the slab: the bins walked are the union
// of the lanes' column spans: every valid sample of a lane lies in its own
// span, and a sample outside it is decided (and rejected) like any other, so
// each (column, point, bin) is counted once. Decisions are the exact chain's
// (the fast path's margin, taken over the largest |tc| of the union).
// What bounds it: instruction issue and the four shared-memory accesses of a
// sample's cell pair, about 25 warp instructions per warp-sample (55 with one
// bin at a time in scalar instructions, the values handed out by shuffles and
// floor and conversion on the special-function units). 128^3 voxels x 16,384
// points x 1,024 bins: 62.8 -> 40.1 ms, at 73% of the shared-memory pipe's wavefronts
// (39.7 with a table of 1 / tc^8, which leaves the FP32 range in other units).
// kSigned: there may be negative bin centres (a negative bin offset), whose bins
// are a second walk of a point. kCluster: the point groups form a cluster
// (add_cluster_columns).
template <bool kSigned, bool kCluster>
__global__ void __launch_bounds__(256, 3) confocal_adjoint_columns_kernel(
    Geo g, Points mp, int N, int points_per_group, int run, const float* __restrict__ tr,
    float* __restrict__ vol, int accumulate, int slab) {
  // slab blockIdx.z: the samples in cells [za, za + zn) (cell pairs (z, z + 1)
  // with z < Z - 1), held in rows 0 .. slab of the column copies (row slab is
  // cell za + slab, the next slab's first)
  const int za = blockIdx.z * slab, zb = min(g.Z, za + slab), zn = min(zb, g.Z - 1) - za;
  const int rows = slab + 1;
  // [warp][rows][32], [warp][32] bin values, the bin table
  extern __shared__ __align__(16) float acc[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float4* vbuf = reinterpret_cast<float4*>(acc + (size_t)nw * rows * 32 + warp * 32);
  float4* tab = reinterpret_cast<float4*>(acc + (size_t)nw * (rows + 1) * 32);
  const int tiles_y = (g.Y + 7) >> 3;
  const int ty = (blockIdx.x % tiles_y) * 8, tx = (blockIdx.x / tiles_y) * 4;
  const int yi = ty + (lane & 7), xi = tx + (lane >> 3);
  const bool live = xi < g.X && yi < g.Y;
  for (int j = threadIdx.x; j < nw * rows * 32; j += blockDim.x) acc[j] = 0.f;
  fill_bin_table(g, tab);
  __syncthreads();
  const uint32_t col = (uint32_t)__cvta_generic_to_shared(acc + (size_t)warp * rows * 32 + lane);
  const float x = centre(g.ox, g.sx, g.X, live ? xi : 0);
  const float y = centre(g.oy, g.sy, g.Y, live ? yi : 0);
  // the columns' rectangle (centres are monotone in the index) and the slab's z
  const float xa = centre(g.ox, g.sx, g.X, tx), xb = centre(g.ox, g.sx, g.X, min(tx + 3, g.X - 1));
  const float ya = centre(g.oy, g.sy, g.Y, ty), yb = centre(g.oy, g.sy, g.Y, min(ty + 7, g.Y - 1));
  const float bx0 = fminf(xa, xb), bx1 = fmaxf(xa, xb), by0 = fminf(ya, yb), by1 = fmaxf(ya, yb);
  const float zlo = g.oz + ((float)za + 0.5f) / g.scale;
  const float zhi = g.oz + ((float)zb + 0.5f) / g.scale;
  const float u = 5.9604645e-8f;
  const int tz = kSigned ? first_nonneg_bin(g) : 0;
  const int i0 = blockIdx.y * points_per_group;
  const int i1 = min(N, i0 + points_per_group);
  for (int base = i0 + warp * run; base < i1; base += nw * run) {
    // lane j loads point base + j
    const int ip = base + lane;
    const int np = min(run, i1 - base);
    float lwx = 0.f, lwy = 0.f, lwz = 0.f;
    if (lane < np) {
      lwx = mp.at(0, ip);
      lwy = mp.at(1, ip);
      lwz = mp.at(2, ip);
    }
    // and bounds its bins over the rectangle of the tile's columns: the nearest
    // and the farthest horizontal distance give the union of the columns' spans
    Spans sp{1, 0, 1, 0};
    float lim = 0.f;
    if (lane < np) {
      const float ex = fmaxf(fmaxf(bx0 - lwx, lwx - bx1), 0.f);
      const float ey = fmaxf(fmaxf(by0 - lwy, lwy - by1), 0.f);
      const float fx = fmaxf(fabsf(lwx - bx0), fabsf(lwx - bx1));
      const float fy = fmaxf(fabsf(lwy - by0), fabsf(lwy - by1));
      float cl, ch, unused;
      if (zn > 0 && zlo <= zhi && tc_bounds(ex * ex + ey * ey, lwz, zlo, zhi, cl, unused) &&
          tc_bounds(fx * fx + fy * fy, lwz, zlo, zhi, unused, ch))
        sp = within_bins(g, tc_spans(g, tz, cl, ch, span_eps(g, ch, lwz)));
      // the margin over the spans' largest |tc|
      const float dmax = 1.001f * span_tc_max(g, sp);
      const float zmax = fabsf(lwz) + dmax;
      const float zhmax = (zmax + fabsf(g.oz)) * g.scale + 0.5f;
      const float pm = 8.f * u * g.scale * (dmax + fabsf(lwz) + zmax + fabsf(g.oz)) +
                       4.f * u * zhmax + 1e-7f;
      lim = g.exact || !(pm < 0.5f) ? 0.f : 0.5f - pm;
    }
    // a point's first 32 values are read while the point before it is walked
    auto first = [&](int j) {
      const int t = (__shfl_sync(0xffffffffu, sp.p0, j) & ~3) + lane;
      return t < g.T ? __ldg(tr + (size_t)(base + j) * g.T + t) : 0.f;
    };
    float next = first(0);
    for (int j = 0; j < np; ++j) {
      const float val = next;
      if (j + 1 < np) next = first(j + 1);
      AdjPoint p;
      p.wx = __shfl_sync(0xffffffffu, lwx, j);
      p.wy = __shfl_sync(0xffffffffu, lwy, j);
      p.wz = __shfl_sync(0xffffffffu, lwz, j);
      p.lim = __shfl_sync(0xffffffffu, lim, j);
      const int p0 = __shfl_sync(0xffffffffu, sp.p0, j);
      const int p1 = __shfl_sync(0xffffffffu, sp.p1, j);
      const float dx = xsub(p.wx, x), dy = xsub(p.wy, y);
      p.ndx = live ? -xmul(dx, dx) : -INFINITY;
      p.ndy = live ? -xmul(dy, dy) : 0.f;
      const float* row = tr + (size_t)(base + j) * g.T;
      if (p0 <= p1)
        adj_walk<kSigned>(g, tab, vbuf, row, p, p0, p1, val, lane, col, x, y, za, zn);
      if (kSigned) {
        const int n0 = __shfl_sync(0xffffffffu, sp.n0, j);
        const int n1 = __shfl_sync(0xffffffffu, sp.n1, j);
        const int t = (n0 & ~3) + lane;
        if (n0 <= n1)
          adj_walk<true>(g, tab, vbuf, row, p, n0, n1, t < g.T ? __ldg(row + t) : 0.f, lane, col,
                         x, y, za, zn);
      }
    }
  }
  if constexpr (kCluster) {
    add_cluster_columns(g, acc, nw, rows, tx, ty, za, vol, accumulate);
    return;
  }
  __syncthreads();
  // cell za + r of column l: the sum over the warps' copies (l fastest: no
  // bank conflicts in the reads)
  for (int jj = threadIdx.x; jj < rows * 32; jj += blockDim.x) {
    const int r = jj >> 5, l = jj & 31, z = za + r;
    const int cy = ty + (l & 7), cx = tx + (l >> 3);
    if (cx >= g.X || cy >= g.Y || z >= g.Z) continue;
    float sum = 0.f;
    for (int w = 0; w < nw; ++w) sum += acc[((size_t)w * rows + r) * 32 + l];
    float* dst = vol + ((size_t)cx * g.Y + cy) * g.Z + z;
    if (accumulate) atomicAdd(dst, sum);
    else *dst = sum;
  }
}

// The reference's transposed operator, per voxel (volume_cuda.cu:96-160).
__global__ void confocal_transposed_kernel(Geo g, Points mp, int N, const float* __restrict__ tr,
                                           float* __restrict__ vol) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= (int64_t)g.X * g.Y * g.Z) return;
  const int zi = (int)(v % g.Z), yi = (int)((v / g.Z) % g.Y), xi = (int)(v / ((int64_t)g.Z * g.Y));
  const float x = centre(g.ox, g.sx, g.X, xi), y = centre(g.oy, g.sy, g.Y, yi);
  const float z = centre(g.oz, g.sz, g.Z, zi);
  const float dz = xdiv(g.sz, (float)g.Z);
  const float zz = zi > 0 ? dz : 0.f;
  float value = 0.f;
  for (int i = 0; i < N; ++i) {
    const float wx = mp.at(0, i), wy = mp.at(1, i), wz = mp.at(2, i);
    const float dp2 = xadd(xmul(xsub(x, wx), xsub(x, wx)), xmul(xsub(y, wy), xsub(y, wy)));
    const float a = xsub(xsub(z, zz), wz), m = xsub(z, wz), e = xsub(xadd(z, dz), wz);
    auto tbin = [&](float q) {
      const float d = xsqrt(xadd(dp2, xmul(q, q)));
      const float cb = ceilf(xdiv(xsub(d, g.bo), g.bw));
      return (int)fminf(fmaxf(cb, 0.f), (float)g.T);
    };
    const int ts = tbin(a), tm = tbin(m), te = tbin(e);
    const float* row = tr + (size_t)i * g.T;
    for (int t = ts; t < te; ++t) {
      const float tc = xadd(xmul((float)t, g.bw), g.bo);
      const float d2 = xsub(xmul(tc, tc), dp2);
      if (!(d2 > 0.f)) continue;
      const float depth = xsqrt(d2);
      const float zh = xsub(xmul(xsub(xadd(wz, depth), g.oz), g.scale), 0.5f);
      const float al = zh - floorf(zh);
      const float w = (t >= tm) ? 1.f - al : al;
      const float q = depth / (tc * tc);
      value += w * ((q * q) * (q * q)) * __ldg(row + t);
    }
  }
  vol[v] = value;
}

}  // namespace volume

namespace {

using volume::Geo;
using volume::Points;

int check_volume_args(const totri_array_t* vol, const totri_array_t* mp, int& X, int& Y, int& Z,
                      int& N, Points& pts) {
  TOTRI_TRY(check_array(vol, "volume", 3, -1));
  if (vol->dtype != TOTRI_FLOAT32)
    return fail(TOTRI_ERR_UNSUPPORTED, "volume renderer: only float32 tensors are supported");
  TOTRI_TRY(check_contiguous(vol, "volume"));
  TOTRI_TRY(check_array(mp, "measurement_points", 2, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(mp, "measurement_points", 0, 3));
  X = (int)vol->shape[0];
  Y = (int)vol->shape[1];
  Z = (int)vol->shape[2];
  N = (int)mp->shape[1];
  pts = Points{static_cast<const float*>(mp->data), mp->strides[0], mp->strides[1]};
  return TOTRI_OK;
}

Geo make_geo(int X, int Y, int Z, const float* o, const float* s, float bw, float bo, int T) {
  Geo g;
  g.X = X;
  g.Y = Y;
  g.Z = Z;
  g.ox = o[0];
  g.oy = o[1];
  g.oz = o[2];
  g.sx = s[0];
  g.sy = s[1];
  g.sz = s[2];
  g.scale = (float)Z / s[2];
  g.dz = s[2] / (float)Z;
  g.bw = bw;
  g.bo = bo;
  g.inv_bw = 1.f / bw;
  g.T = T;
  g.exact = tune::get("volume.exact") == 1;
  g.all_bins = !(bw > 0.f) || !std::isfinite(bw) || !std::isfinite(bo) ||
               !std::isfinite(g.inv_bw);
  return g;
}

// the count (in a 256-byte header), then one record per voxel
size_t occupancy_bytes(int64_t nvox) { return align_up(256 + sizeof(float4) * nvox, 256); }

int compact(const Geo& g, const float* vol, int64_t n, void* ws, size_t ws_bytes, float4** recs,
            uint32_t** count, cudaStream_t stream) {
  const size_t need = occupancy_bytes(n);
  if (!ws || ws_bytes < need)
    return fail(TOTRI_ERR_WORKSPACE,
                "workspace of " + std::to_string(need) + " bytes required, got " +
                    std::to_string(ws_bytes));
  *count = static_cast<uint32_t*>(ws);
  *recs = reinterpret_cast<float4*>(static_cast<char*>(ws) + 256);
  TOTRI_CUDA(cudaMemsetAsync(*count, 0, sizeof(uint32_t), stream));
  TOTRI_KERNEL("volume compact", stream,
               volume::compact_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, stream>>>(
                   g, vol, n, *recs, *count));
  return TOTRI_OK;
}

// Points per CTA, threads, shared memory and slices of the occupied voxels for
// the walks of confocal_forward_kernel (rows: the points' bins are in shared memory) and
// grad_mp_kernel. points 0: the rows of 4 points, or the bin table, do not fit.
struct WalkTile {
  int points, threads, slices;
  size_t smem;
};

WalkTile walk_tile(int64_t N, int T, int64_t voxels, bool rows) {
  const size_t budget = 220 * 1024;
  const auto bytes = [&](int pt) {
    return (rows ? sizeof(float) * (((size_t)pt * T + 3) & ~(size_t)3) : 0) +
           sizeof(float4) * volume::bin_table(T);
  };
  WalkTile w{0, 0, 1, 0};
  // 16 points by 32 threads each where their rows fit ("volume.forward.points"
  // sets it), and up to 8 slices of the voxels while there are fewer than 16
  // waves of CTAs and a thread keeps some voxels ("volume.forward.slices"):
  // 128^3 voxels, 16,384 points, 1,024 bins: 16 points 6.1 ms alone, 5.6 in 2
  // slices, 5.4 in 8; 8 points 6.3 / 5.9 / 5.6 ms, 32 points 7.1 / 6.4 / 6.4 ms.
  // 41 x 37 x 53 x 899 points, 500 bins: 16 points 0.43 ms alone, 0.11 in 8.
  int want = tune::get("volume.forward.points");
  if (want < 4) want = 0;  // (fewer than 4 points: the built-in choice)
  for (const int pt : {32, 16, 8, 4}) {
    if (bytes(pt) > budget || pt > (want > 0 ? want : 16)) continue;
    w.points = pt;
    break;
  }
  if (w.points == 0) return w;
  // Without rows: smaller tiles until 8 slices make a CTA per SM, and until the points'
  // rows fit half of the L1 cache (24^3 voxels, half of them, x 1,024 points: 2,048 bins
  // 0.51 ms with 8 points, 1.11 with 16; 4,096 bins 0.95 with 4, 1.21 with 8, 2.05 with
  // 16). Above, not even 4 rows do, and 16 points are the fastest (64^3 voxels x 2,048
  // points x 5,000 bins 13.2 ms, 21.8 with 4) but for few points (256: 4.3 and 3.1 ms).
  while (!rows && want == 0 && w.points > 4 &&
         (8 * ceil_div(N, w.points) < (int64_t)tune::sm_count() ||
          (T <= (N <= 256 ? 6000 : 4096) && sizeof(float) * w.points * T > 64 * 1024)))
    w.points /= 2;
  w.threads = std::max(256, 32 * w.points);
  w.smem = bytes(w.points);
  const int64_t resident = std::max<int64_t>(
      1, std::min<int64_t>(2048 / w.threads, (int64_t)(budget / (w.smem + 1024))));
  int64_t slices = tune::get("volume.forward.slices");
  if (slices <= 0)
    slices = std::max<int64_t>(
        1, std::min({(int64_t)8, 16 * resident * tune::sm_count() / ceil_div(N, w.points),
                     voxels / (16 * w.threads)}));
  w.slices = (int)std::min<int64_t>(slices, 256);
  return w;
}

// launch(points, signed) with compile-time constants.
template <class F>
int for_walk_tile(int points, const Geo& g, F launch) {
  const auto with = [&](auto pt) {
    return g.bo < 0.f && !g.all_bins ? launch(pt, std::true_type{}) : launch(pt, std::false_type{});
  };
  switch (points) {
    case 32: return with(std::integral_constant<int, 32>{});
    case 16: return with(std::integral_constant<int, 16>{});
    case 8: return with(std::integral_constant<int, 8>{});
    default: return with(std::integral_constant<int, 4>{});
  }
}

}  // namespace
}  // namespace totri

using namespace totri;

extern "C" {

size_t totri_volume_workspace(int64_t num_voxels) {
  return num_voxels > 0 ? occupancy_bytes(num_voxels) : 0;
}

int totri_volume_confocal_forward(const totri_array_t* vol, const totri_array_t* mp,
                                  const totri_array_t* tr, const float origin[3],
                                  const float size[3], float bw, float bo, void* ws,
                                  size_t ws_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  int X, Y, Z, N;
  Points pts;
  TOTRI_TRY(check_volume_args(vol, mp, X, Y, Z, N, pts));
  TOTRI_TRY(check_array(tr, "transient", 2, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(tr, "transient", 0, N));
  TOTRI_TRY(check_contiguous(tr, "transient"));
  const int T = (int)tr->shape[1];
  if (N == 0 || T == 0) return TOTRI_OK;
  if (sizeof(float) * 8 * (size_t)T > 200 * 1024)
    return fail(TOTRI_ERR_UNSUPPORTED, "too many bins for one tile");
  const Geo g = make_geo(X, Y, Z, origin, size, bw, bo, T);
  float4* recs;
  uint32_t* count;
  TOTRI_TRY(compact(g, static_cast<const float*>(vol->data), numel(vol), ws, ws_bytes, &recs,
                    &count, stream));
  float* out = static_cast<float*>(tr->data);
  const WalkTile w = walk_tile(N, T, numel(vol), true);
  if (w.slices > 1)
    TOTRI_CUDA(cudaMemsetAsync(out, 0, sizeof(float) * (size_t)N * T, stream));
  return for_walk_tile(w.points, g, [&](auto pt, auto sign) {
    const auto kernel = volume::confocal_forward_kernel<decltype(pt)::value, decltype(sign)::value>;
    TOTRI_CUDA(tune::ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), w.smem));
    const dim3 grid((unsigned)ceil_div(N, w.points), (unsigned)w.slices);
    TOTRI_KERNEL("volume confocal forward", stream,
                 kernel<<<grid, w.threads, w.smem, stream>>>(g, recs, count, pts, N, out));
    return (int)TOTRI_OK;
  });
}

int totri_volume_confocal_adjoint(const totri_array_t* vol, const totri_array_t* mp,
                                  const totri_array_t* tr, const float origin[3],
                                  const float size[3], float bw, float bo, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  int X, Y, Z, N;
  Points pts;
  TOTRI_TRY(check_volume_args(vol, mp, X, Y, Z, N, pts));
  TOTRI_TRY(check_array(tr, "transient", 2, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(tr, "transient", 0, N));
  TOTRI_TRY(check_contiguous(tr, "transient"));
  const int T = (int)tr->shape[1];
  if (numel(vol) == 0) return TOTRI_OK;
  if (N == 0 || T == 0) {
    TOTRI_CUDA(cudaMemsetAsync(vol->data, 0, sizeof(float) * numel(vol), stream));
    return TOTRI_OK;
  }
  const Geo g = make_geo(X, Y, Z, origin, size, bw, bo, T);
  const unsigned grid = (unsigned)(X * Y);
  const float* trd = static_cast<const float*>(tr->data);
  float* vd = static_cast<float*>(vol->data);
  // "volume.adjoint.mode": 0 (default) lanes over columns, 1 shared-memory
  // atomics, 2 lane-owned cells (columns of up to 256 cells)
  const int mode = tune::get("volume.adjoint.mode");
  // lanes over columns: warps per CTA such that two CTAs' copies of 32
  // columns and the bin table fit an SM's shared memory
  // ("volume.adjoint.warps" overrides); bins beyond 4,096 take the atomic kernel
  const size_t table = sizeof(float4) * volume::bin_table(T);
  // The columns split into slabs of at most 64 cells, a CTA per slab: each
  // warp's column copy is then 65 rows (8.3 KB), and 3 CTAs of 8 warps share
  // an SM (24 warps) instead of 2 of 6 with whole 128-cell columns. 128^3
  // voxels x 16,384 points: 65.8 ms with 2 slabs, 75.4 ms with 1 and 72.5 ms
  // with 4 (each slab walks the union of its lanes' bins, so thinner slabs
  // walk more bins in all). "volume.adjoint.slabs" sets the count.
  int slabs = (int)tune::get("volume.adjoint.slabs");
  if (slabs <= 0) slabs = (int)ceil_div(Z, 64);
  slabs = std::min(slabs, Z);
  const int slab = (int)ceil_div(Z, slabs);
  const size_t per_warp = (size_t)(slab + 2) * 32 * sizeof(float);  // cells and bin values
  int warps = T <= 4096 && table < 113 * 1024 ? (int)((113 * 1024 - table) / per_warp) : 0;
  if (tune::get("volume.adjoint.warps") > 0) warps = tune::get("volume.adjoint.warps");
  warps = std::min(warps, 8);
  if (Z < 2) {  // no interpolation pair: no samples
    TOTRI_CUDA(cudaMemsetAsync(vd, 0, sizeof(float) * numel(vol), stream));
    return TOTRI_OK;
  }
  if (mode == 0 && warps >= 1 && T <= 4096) {
    const size_t smem = (size_t)warps * per_warp + table;
    const int64_t tiles = ceil_div(Y, 8) * ceil_div(X, 4);
    // point groups: about 16 CTAs per SM in all, each with at least a run of
    // points per warp; runs of 32 points, or down to 8 while the CTAs would not
    // fill the SMs' three places twice (41 x 37 x 53 voxels x 899 points: 0.60 -> 0.15 ms)
    const int nslab = (int)ceil_div(Z, slab);
    const int64_t want = std::max<int64_t>(1, (16 * tune::sm_count()) / (tiles * nslab));
    int run = 32;
    while (run > 8 && tiles * nslab * ceil_div(N, (int64_t)run * warps) < 6 * tune::sm_count())
      run /= 2;
    const int groups =
        (int)std::max<int64_t>(1, std::min<int64_t>(want, ceil_div(N, (int64_t)run * warps)));
    const int per = (int)(ceil_div(ceil_div(N, groups), run) * run);
    const int used = (int)ceil_div(N, per);
    // The groups of up to two runs of 32 points per warp (at most 8 groups) form a
    // cluster, which sums them in order: the result repeats bit for bit. Those of more
    // points add in the order in which they end: 64^3 voxels x 1,024 points take 346 us
    // so, 390 us in clusters of 4.
    const int peers = N <= 64 * warps && used <= 8 ? used : 1;
    const int accumulate = used > peers || nslab > 1;
    if (accumulate) TOTRI_CUDA(cudaMemsetAsync(vd, 0, sizeof(float) * numel(vol), stream));
    const dim3 grid3((unsigned)tiles, (unsigned)used, (unsigned)nslab);
    const bool negative = g.bo < 0.f && !g.all_bins;
    const auto kernel =
        peers > 1 ? (negative ? volume::confocal_adjoint_columns_kernel<true, true>
                              : volume::confocal_adjoint_columns_kernel<false, true>)
                  : (negative ? volume::confocal_adjoint_columns_kernel<true, false>
                              : volume::confocal_adjoint_columns_kernel<false, false>);
    TOTRI_CUDA(tune::ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem));
    cudaLaunchAttribute cluster[1];
    cluster[0].id = cudaLaunchAttributeClusterDimension;
    cluster[0].val.clusterDim.x = 1;
    cluster[0].val.clusterDim.y = (unsigned)peers;
    cluster[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid3;
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = cluster;
    cfg.numAttrs = peers > 1 ? 1 : 0;
    cudaError_t le = cudaSuccess;
    TOTRI_KERNEL("volume confocal adjoint", stream,
                 le = cudaLaunchKernelEx(&cfg, kernel, g, pts, N, per, run, trd, vd, accumulate,
                                         slab));
    TOTRI_CUDA(le);
    return TOTRI_OK;
  }
  if (Z <= 256 && mode == 2) {
    if (Z <= 32)
      TOTRI_KERNEL("volume confocal adjoint", stream,
                   volume::confocal_adjoint_cells_kernel<1><<<grid, 256, 0, stream>>>(
                       g, pts, N, trd, vd));
    else if (Z <= 64)
      TOTRI_KERNEL("volume confocal adjoint", stream,
                   volume::confocal_adjoint_cells_kernel<2><<<grid, 256, 0, stream>>>(
                       g, pts, N, trd, vd));
    else if (Z <= 128)
      TOTRI_KERNEL("volume confocal adjoint", stream,
                   volume::confocal_adjoint_cells_kernel<4><<<grid, 256, 0, stream>>>(
                       g, pts, N, trd, vd));
    else
      TOTRI_KERNEL("volume confocal adjoint", stream,
                   volume::confocal_adjoint_cells_kernel<8><<<grid, 256, 0, stream>>>(
                       g, pts, N, trd, vd));
    return TOTRI_OK;
  }
  const size_t smem = sizeof(float) * 8 * (size_t)Z;
  if (smem > 200 * 1024) return fail(TOTRI_ERR_UNSUPPORTED, "volume too deep for one column tile");
  TOTRI_CUDA(tune::ensure_dynamic_smem(
      reinterpret_cast<const void*>(volume::confocal_adjoint_kernel), smem));
  TOTRI_KERNEL("volume confocal adjoint", stream,
               volume::confocal_adjoint_kernel<<<grid, 256, smem, stream>>>(g, pts, N, trd, vd));
  return TOTRI_OK;
}

int totri_volume_confocal_grad_volume(const totri_array_t* vol, const totri_array_t* mp,
                                      const totri_array_t* tr, const float origin[3],
                                      const float size[3], float bw, float bo, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  int X, Y, Z, N;
  Points pts;
  TOTRI_TRY(check_volume_args(vol, mp, X, Y, Z, N, pts));
  TOTRI_TRY(check_array(tr, "transient", 2, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(tr, "transient", 0, N));
  TOTRI_TRY(check_contiguous(tr, "transient"));
  const int T = (int)tr->shape[1];
  const int64_t nv = numel(vol);
  if (nv == 0) return TOTRI_OK;
  const Geo g = make_geo(X, Y, Z, origin, size, bw, bo, T);
  TOTRI_KERNEL("volume confocal transposed", stream,
               volume::confocal_transposed_kernel<<<(unsigned)ceil_div(nv, 128), 128, 0, stream>>>(
                   g, pts, N, static_cast<const float*>(tr->data), static_cast<float*>(vol->data)));
  return TOTRI_OK;
}

int totri_volume_confocal_grad_measurement_points(const totri_array_t* mpg,
                                                  const totri_array_t* vol,
                                                  const totri_array_t* mp,
                                                  const totri_array_t* tg, const float origin[3],
                                                  const float size[3], float bw, float bo,
                                                  void* ws, size_t ws_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  int X, Y, Z, N;
  Points pts;
  TOTRI_TRY(check_volume_args(vol, mp, X, Y, Z, N, pts));
  TOTRI_TRY(check_array(mpg, "measurement_points_grad", 2, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(mpg, "measurement_points_grad", 0, 3));
  TOTRI_TRY(check_dim(mpg, "measurement_points_grad", 1, N));
  TOTRI_TRY(check_array(tg, "transient_grad", 2, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(tg, "transient_grad", 0, N));
  TOTRI_TRY(check_contiguous(tg, "transient_grad"));
  const int T = (int)tg->shape[1];
  if (N == 0) return TOTRI_OK;
  const Geo g = make_geo(X, Y, Z, origin, size, bw, bo, T);
  float4* recs;
  uint32_t* count;
  TOTRI_TRY(compact(g, static_cast<const float*>(vol->data), numel(vol), ws, ws_bytes, &recs,
                    &count, stream));
  float* out = static_cast<float*>(mpg->data);
  const int64_t osc = mpg->strides[0], osn = mpg->strides[1];
  // Rows in shared memory for few and long ones only (us, in place against it, half of
  // 24^3 voxels, and 2% of them): 6,400 bins, 64 points 667/490 and 66/70, 256 points
  // 1,789/923 and 99/115, 1,024 points 4,091/2,607 and 200/279; 9,300 bins, 256 points
  // 2,647/1,306 and 137/151. Half of 64^3 voxels x 6,400 bins, 1,024 points 9.9/16.4 ms.
  WalkTile w{0, 0, 1, 0};
  bool staged = T > 6000 && N <= 256;
  if (staged) w = walk_tile(N, T, numel(vol), true);
  if (w.points == 0) {
    staged = false;
    w = walk_tile(N, T, numel(vol), false);
  }
  if (w.points == 0) {  // the bin table is too long for shared memory
    TOTRI_KERNEL("volume confocal grad points", stream,
                 volume::grad_mp_wide_kernel<<<(unsigned)ceil_div(N, volume::kPT), 256, 0, stream>>>(
                     g, recs, count, pts, N, static_cast<const float*>(tg->data), out, osc, osn));
    return TOTRI_OK;
  }
  if (w.slices > 1 && osn == 1 && osc == N)
    TOTRI_CUDA(cudaMemsetAsync(out, 0, sizeof(float) * 3 * (size_t)N, stream));
  else
    w.slices = 1;  // (the slices add into a zeroed output)
  return for_walk_tile(w.points, g, [&](auto pt, auto sign) {
    constexpr int kPoints = decltype(pt)::value;
    constexpr bool kSigned = decltype(sign)::value;
    const auto kernel = staged ? volume::grad_mp_kernel<kPoints, kSigned, true>
                               : volume::grad_mp_kernel<kPoints, kSigned, false>;
    TOTRI_CUDA(tune::ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), w.smem));
    const dim3 grid((unsigned)ceil_div(N, w.points), (unsigned)w.slices);
    TOTRI_KERNEL("volume confocal grad points", stream,
                 kernel<<<grid, w.threads, w.smem, stream>>>(
                     g, recs, count, pts, N, static_cast<const float*>(tg->data), out, osc, osn));
    return (int)TOTRI_OK;
  });
}

}  // extern "C"
