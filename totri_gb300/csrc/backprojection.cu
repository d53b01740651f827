// Backprojection reconstructions: Velten confocal (and its adjoint), Velten
// exhaustive, Arellano exhaustive.
//
// Reference: src/reconstruct/backprojection_cuda.cu (:153-194 Velten
// confocal, :229-287 Velten exhaustive, :11-115 Arellano). The Velten kernels
// gather per voxel; here a CTA of 256 voxels stages scan points (and their
// wall-to-origin distances) in shared memory in tiles, so each scan point is
// read once per CTA rather than once per voxel. The adjoint owns a tile of
// scan points and keeps their transient columns in shared memory.
#include <algorithm>
#include <climits>
#include <cmath>
#include <string>

#include "capi_common.cuh"
#include "mesh_kernels.cuh"
#include "tune.cuh"

namespace totri {
namespace bp {

struct Grid {
  int D, H, W;
  float sx, sy, sz, ex, ey, ez;
};

// start + (i / (n - 1)) * (end - start) (backprojection_cuda.cu:167-170).
__device__ __forceinline__ float grid_coord(float s, float e, int n, int i) {
  return xadd(s, xmul(xdiv((float)i, (float)(n - 1)), xsub(e, s)));
}

__device__ __forceinline__ fv3 voxel_point(const Grid& g, int x, int y, int z) {
  return mkv(grid_coord(g.sx, g.ex, g.W, x), grid_coord(g.sy, g.ey, g.H, y),
             grid_coord(g.sz, g.ez, g.D, z));
}

// floor((dist - offset) / width + 0.5) (backprojection_cuda.cu:187).
__device__ __forceinline__ int nearest_bin(float dist, float bw, float bo) {
  const float b = floorf(xadd(xdiv(xsub(dist, bo), bw), 0.5f));
  if (!(b == b)) return -1;
  if (b > 2.0e9f) return 2000000000;
  if (b < -2.0e9f) return -2000000000;
  return (int)b;
}

// Velten bins with a filtered fast path. The decision is nearest_bin(od2 + 2
// |q - p|) with one IEEE rounding per operation. The fast path evaluates the
// same expression with fused multiply-adds, the hardware reciprocal square
// root (2 ulp) and a precomputed 1/bw; against the exact chain its bin
// coordinate c = (dist - bo)/bw + 1/2 deviates by at most about
// 14 u (dist + |bo|)/bw + 5 u |c| (u = 2^-24: 3 u from the sum of squares,
// 6.5 u from the root, one rounding per remaining operation). Where c lies
// farther than twice that from an integer both floors are equal and the fast
// bin is returned; otherwise (and for NaN or infinite c) the exact chain runs,
// so the bins are those of the exact chain everywhere.
struct FastBin {
  float inv_bw, nbo, k1, k2;
  float kc, kb;  // box_bins' margin: kc dist + kb
};

inline FastBin make_fast_bin(float bw, float bo) {
  const float u = 5.9604645e-8f;  // 2^-24
  FastBin f;
  f.inv_bw = 1.f / bw;
  f.nbo = -bo * f.inv_bw;
  const bool ok = bw > 0.f && std::isfinite(f.inv_bw) && std::isfinite(f.nbo);
  f.k1 = ok ? 32.f * u * f.inv_bw : INFINITY;
  f.k2 = ok ? 32.f * u * std::fabs(bo) * f.inv_bw + 1e-6f : INFINITY;
  f.kc = ok ? 16.f * u * f.inv_bw : INFINITY;
  f.kb = ok ? 16.f * u * std::fabs(bo) * f.inv_bw + 1e-6f : INFINITY;
  return f;
}

__device__ __forceinline__ int velten_bin(fv3 q, float od2, fv3 p, float bw, float bo,
                                          const FastBin& f) {
  const float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
  const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  const float dist = fmaf(2.f, d2 * rsqrtf(d2), od2);
  const float c = fmaf(dist, f.inv_bw, f.nbo) + 0.5f;
  const float t = floorf(c);
  const float fr = c - t;
  const float m = fmaf(f.k1, dist, f.k2) + 1e-6f * fabsf(c);
  if (fr > m && fr < 1.f - m && fabsf(t) < 1.0e9f) return (int)t;
  return nearest_bin(xadd(od2, xmul(2.f, xlen(xsub3(q, p)))), bw, bo);
}

// velten_bin for two voxels of a column at once with paired FP32 instructions,
// the margin bounded once per box of voxels (box_bins) and the +1/2 of the bin
// coordinate folded away. r2, the squared distance in x and y, is shared by
// the column's voxels. The bin is rounded without the conversion units: v =
// dist / bw - bo / bw plus 1.5 2^23 holds rint(v) in its low mantissa bits for
// |v| < 2^22, and floor(v + 1/2) = rint(v) wherever v + 1/2 is farther than
// the margin from an integer, which is the test |v - rint(v)| < 1/2 - m
// (`half_m`; <= 0 sends every pair to the exact chain). The bins are those of
// the exact chain everywhere.
__device__ __forceinline__ void velten_bin_col2(fv3 q, float od2, fv3 pa, fv3 pb, float r2,
                                                float bw, float bo, float inv_bw, float nbo,
                                                float half_m, int& ta, int& tb) {
  const unsigned long long dz = f2sub(f2pack(q.z, q.z), f2pack(pa.z, pb.z));
  const unsigned long long d2 = f2fma(dz, dz, f2pack(r2, r2));
  float d2a, d2b;
  f2unpack(d2, d2a, d2b);
  const unsigned long long prod = f2mul(d2, f2pack(rsqrt_approx(d2a), rsqrt_approx(d2b)));
  const unsigned long long dist = f2fma(f2pack(2.f, 2.f), prod, f2pack(od2, od2));
  const unsigned long long v = f2fma(dist, f2pack(inv_bw, inv_bw), f2pack(nbo, nbo));
  const unsigned long long big = f2pack(12582912.f, 12582912.f);  // 1.5 2^23
  const unsigned long long x = f2add(v, big);
  const unsigned long long rr = f2sub(v, f2sub(x, big));
  float xa, xb, ra, rb;
  f2unpack(x, xa, xb);
  f2unpack(rr, ra, rb);
  ta = fabsf(ra) < half_m ? __float_as_int(xa) - 0x4B400000
                          : nearest_bin(xadd(od2, xmul(2.f, xlen(xsub3(q, pa)))), bw, bo);
  tb = fabsf(rb) < half_m ? __float_as_int(xb) - 0x4B400000
                          : nearest_bin(xadd(od2, xmul(2.f, xlen(xsub3(q, pb)))), bw, bo);
}

struct Pts3 {  // [B, n, 3] with strides
  const float* p;
  int64_t sb, sn, sc;
  __device__ fv3 at(int b, int i) const {
    const float* q = p + b * sb + i * sn;
    return mkv(q[0], q[sc], q[2 * sc]);
  }
};

// Bin coordinates (+1/2) that a scan point q with origin term od2 can reach in
// a box of voxels, [cmin, cmax] (NaN where they are not defined), and the
// margin of the fast bins there. With u = 2^-24 and dist = 2 s + od2, the exact
// chain's own roundings move the coordinate by at most 5 u 2s + 4 u od2 + 3 u
// |bo| (over bw; plus u/2), the fast paths' by 6.2 u 2s + 3 u od2 + 4 u |bo|
// (root: 2^-22.9 from rsqrt and one product), and the two sums of squares
// differ by at most 6 u, 3 u in the root: 14.2 u (dist + |bo|) / bw in all. The
// margin is 16 u of the largest distance of the box, 2% wider still for the
// rounding of these bounds, plus 1e-6; infinite (every pair takes the exact
// chain) where the bounds are not finite or the bins reach 2^21, the range of
// the rounding by addition. With the previous 32 u dist / bw + 1e-6 |c|, three
// times as wide, a warp left the fast path three times as often.
struct BoxBins {
  float cmin, cmax, margin;
  bool away;  // the box keeps a normal distance from the point
};
__device__ __forceinline__ BoxBins box_bins(fv3 q, float od2, fv3 lo, fv3 hi, float bw, float bo,
                                            const FastBin& fb) {
  const float ex = fmaxf(fmaxf(lo.x - q.x, q.x - hi.x), 0.f);
  const float ey = fmaxf(fmaxf(lo.y - q.y, q.y - hi.y), 0.f);
  const float ez = fmaxf(fmaxf(lo.z - q.z, q.z - hi.z), 0.f);
  const float fx = fmaxf(fabsf(lo.x - q.x), fabsf(hi.x - q.x));
  const float fy = fmaxf(fabsf(lo.y - q.y), fabsf(hi.y - q.y));
  const float fz = fmaxf(fabsf(lo.z - q.z), fabsf(hi.z - q.z));
  const float e2 = ex * ex + ey * ey + ez * ez, f2 = fx * fx + fy * fy + fz * fz;
  BoxBins r;
  r.cmin = (od2 + 2.f * sqrtf(e2) - bo) / bw + 0.5f;
  r.cmax = (od2 + 2.f * sqrtf(f2) - bo) / bw + 0.5f;
  const float dmax = fmaf(2.f, sqrtf(f2), od2);
  const float cabs = fmaxf(fabsf(r.cmin), fabsf(r.cmax));
  r.margin = 1.02f * fmaf(fb.kc, dmax, fb.kb);
  if (!(r.margin == r.margin) || !(cabs < 2097152.f) || !(r.cmin == r.cmin))
    r.margin = INFINITY;
  r.away = e2 > 1e-30f;
  return r;
}

constexpr int kTile = 512;

__global__ void __launch_bounds__(256) velten_confocal_kernel(Grid g, int b, int T, int S,
                                                              Pts3 sp, Pts3 so, int has_origin,
                                                              float bw, float bo, FastBin fb,
                                                              const float* __restrict__ tr,
                                                              float* __restrict__ vol) {
  __shared__ float4 pts[kTile];  // scan point xyz, 2 * |scan - origin|
  const int64_t nv = (int64_t)g.D * g.H * g.W;
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int x = (int)(v % g.W), y = (int)((v / g.W) % g.H), z = (int)(v / ((int64_t)g.W * g.H));
  const fv3 p = voxel_point(g, x, y, z);
  const float* trb = tr + (size_t)b * T * S;
  float value = 0.f;
  for (int s0 = 0; s0 < S; s0 += kTile) {
    __syncthreads();
    for (int j = threadIdx.x; j < kTile && s0 + j < S; j += blockDim.x) {
      const fv3 q = sp.at(b, s0 + j);
      const float od = has_origin ? xlen(xsub3(q, so.at(b, s0 + j))) : 0.f;
      pts[j] = make_float4(q.x, q.y, q.z, xmul(2.f, od));
    }
    __syncthreads();
    if (v < nv) {
      const int cnt = min(kTile, S - s0);
      for (int j = 0; j < cnt; ++j) {
        const float4 q = pts[j];
        const int t = velten_bin(mkv(q.x, q.y, q.z), q.w, p, bw, bo, fb);
        if (t >= 0 && t < T) value += __ldg(trb + (size_t)t * S + s0 + j);
      }
    }
  }
  if (v < nv) vol[(size_t)b * nv + v] = value;
}

// Tiled Velten confocal: one CTA of 256 threads per 8 x 8 x (4 VZ) block of
// voxels, each thread VZ voxels of a column, 4 apart in z, and the scan points
// in tiles of ST. Every point of a tile has a window of kWinFloats / ST rows of
// its transient column in shared memory, which holds every bin that the block
// can reach from it (box_bins, one bin more each side); bins outside [0, T) are
// staged as zeros. So a fast bin needs no range test: its shared-memory address
// is one shift and add away from the rounded coordinate. A window starts at
// the first bin of its group of 8 neighbouring points (whose 8 columns of a row
// are one 32-byte sector) or, when a group's bins overflow it, of its own point.
// Tiles whose windows cannot hold their bins, or with bins that need the exact
// chain throughout, read the transient in place (velten_tile_direct).
// Descriptors of 256 points are prepared at a time, one per thread.
//
// What bounds it: instruction issue (73% of slots with 40 warps per SM). Pairs
// within the margin of a bin boundary (about 1e-3 of them at 5 mm bins) take the
// exact chain, one lane at a time, about a tenth of the instructions. 128^3
// voxels x 16,384 points: 33.4 -> 17.2 ms at 1,024 bins and 61.1 -> 26.3 ms at
// 4,096, against a kernel that tested every pair's margin and window row with
// branches. On the way: registers for 5 CTAs per SM (48), 18.1 ms, for 4, 19.4,
// for 6, 20.5; 8 voxels per thread 18.4 ms; the boundary test per point instead
// of per two points 19.8 ms; staging through registers instead of cp.async
// 18.1 ms. The sum runs over the scan points in the order of
// velten_confocal_kernel, so the two give identical volumes.
constexpr int kBX = 8, kBY = 8, kBZ = 4, kWinFloats = 6176, kBatch = 256;
// rows of a window: an odd count, so neighbouring points' windows start on
// different banks (staging writes one row of 32 points)
__host__ __device__ constexpr int win_rows(int ST) { return (kWinFloats / ST - 1) | 1; }

// One tile of scan points [s0, s0 + cnt) against the thread's voxels, bins by
// velten_bin and read in place.
template <int VZ>
__device__ __noinline__ void velten_tile_direct(int b, int T, int S, Pts3 sp, Pts3 so,
                                                int has_origin, float bw, float bo,
                                                const FastBin& fb, const float* __restrict__ trb,
                                                int s0, int cnt, const fv3* p, float* value) {
  for (int j = 0; j < cnt; ++j) {
    const fv3 q = sp.at(b, s0 + j);
    const float od2 = xmul(2.f, has_origin ? xlen(xsub3(q, so.at(b, s0 + j))) : 0.f);
    for (int v = 0; v < VZ; ++v) {
      const int t = velten_bin(q, od2, p[v], bw, bo, fb);
      if ((unsigned)t < (unsigned)T) value[v] += __ldg(trb + (size_t)t * S + s0 + j);
    }
  }
}

enum : int { kTileSkip = 0, kTileFast = 1, kTileDirect = 2 };

template <int VZ, int ST>
__global__ void __launch_bounds__(256, 5) velten_confocal_tiled_kernel(
    Grid g, int b, int T, int S, Pts3 sp, Pts3 so, int has_origin, float bw, float bo,
    FastBin fb, const float* __restrict__ tr, float* __restrict__ vol) {
  using u64 = unsigned long long;
  constexpr int kRows = win_rows(ST), kTiles = kBatch / ST;
  __shared__ float win[kWinFloats];
  __shared__ float4 pa[kBatch];  // x, y, window address less the bin bias, 1/2 - margin
  __shared__ float4 pb[kBatch];  // z, z, od2 / bw - bo / bw twice
  __shared__ int2 prow[kBatch];  // first staged bin, staged rows
  __shared__ int tile_mode[kTiles], tile_inner[kTiles];
  const int lane = threadIdx.x & 31;
  const int x0 = blockIdx.x * kBX, y0 = blockIdx.y * kBY, z0 = blockIdx.z * kBZ * VZ;
  const int x = x0 + (threadIdx.x & 7), y = y0 + ((threadIdx.x >> 3) & 7);
  const int zt = z0 + (threadIdx.x >> 6);  // voxels zt + kBZ v
  // Voxels past the volume's edge compute on a clamped position (inside the
  // block's box) and are never written.
  const fv3 p0 = voxel_point(g, min(x, g.W - 1), min(y, g.H - 1), 0);
  float npz[VZ];  // negated
#pragma unroll
  for (int v = 0; v < VZ; ++v) npz[v] = -grid_coord(g.sz, g.ez, g.D, min(zt + kBZ * v, g.D - 1));
  const float* trb = tr + (size_t)b * T * S;
  const u64 slope = f2pack(2.f * fb.inv_bw, 2.f * fb.inv_bw);
  const u64 big = f2pack(12582912.f, 12582912.f);  // 1.5 2^23
  u64 value[VZ / 2];
#pragma unroll
  for (int v = 0; v < VZ / 2; ++v) value[v] = 0ull;
  for (int i0 = 0; i0 < S; i0 += kBatch) {
    __syncthreads();  // the previous descriptors are consumed
    {
      const int i = i0 + threadIdx.x;
      const bool live = i < S;
      int lo1 = INT_MAX, hi1 = INT_MIN;
      bool fast = true;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f), c = a;
      if (live) {
        const fv3 q = sp.at(b, i);
        const float od2 = has_origin ? xmul(2.f, xlen(xsub3(q, so.at(b, i)))) : 0.f;
        // the block's box: voxel coordinates are monotone in the index
        const fv3 ca = voxel_point(g, x0, y0, z0);
        const fv3 cb = voxel_point(g, min(x0 + kBX, g.W) - 1, min(y0 + kBY, g.H) - 1,
                                   min(z0 + kBZ * VZ, g.D) - 1);
        const fv3 lo = mkv(fminf(ca.x, cb.x), fminf(ca.y, cb.y), fminf(ca.z, cb.z));
        const fv3 hi = mkv(fmaxf(ca.x, cb.x), fmaxf(ca.y, cb.y), fmaxf(ca.z, cb.z));
        const BoxBins bb = box_bins(q, od2, lo, hi, bw, bo, fb);
        fast = bb.margin < 0.25f && bb.away;  // so |cmin|, |cmax| < 2^21
        lo1 = hi1 = 0;
        if (fast) {
          lo1 = (int)floorf(bb.cmin) - 1;
          hi1 = (int)floorf(bb.cmax) + 1;
        }
        a = make_float4(q.x, q.y, 0.f, 0.5f - bb.margin);
        const float c0 = fmaf(od2, fb.inv_bw, fb.nbo);
        c = make_float4(q.z, q.z, c0, c0);
      }
      int lo8 = lo1, hi8 = hi1;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        lo8 = min(lo8, __shfl_xor_sync(0xffffffffu, lo8, o));
        hi8 = max(hi8, __shfl_xor_sync(0xffffffffu, hi8, o));
      }
      // (a dead point's span is empty, and its difference never formed)
      const int rows1 = hi1 >= lo1 ? hi1 - lo1 + 1 : 0, rows8 = hi8 >= lo8 ? hi8 - lo8 + 1 : 0;
      const unsigned mine = ST == 32 ? 0xffffffffu : ((1u << (ST & 31)) - 1u) << (lane & ~(ST - 1));
      const bool in8 = !(__ballot_sync(0xffffffffu, rows8 > kRows) & mine);
      const bool in1 = !(__ballot_sync(0xffffffffu, rows1 > kRows) & mine);
      const bool all_fast = !(__ballot_sync(0xffffffffu, !fast) & mine);
      const bool some = (__ballot_sync(0xffffffffu, hi1 >= 0 && lo1 < T && live) & mine) != 0;
      const int first = in8 ? lo8 : lo1;
      const int rows = in8 ? rows8 : rows1;
      const bool inner =
          (__ballot_sync(0xffffffffu, !live || first < 0 || first + rows > T) & mine) == 0;
      const uint32_t base = (uint32_t)__cvta_generic_to_shared(win) +
                            4u * (uint32_t)((threadIdx.x & (ST - 1)) * kRows);
      const uint32_t bias = 4u * (0x4B400000u + (uint32_t)first);
      if (live) {
        a.z = __uint_as_float(base - bias);
        pa[threadIdx.x] = a;
        pb[threadIdx.x] = c;
        prow[threadIdx.x] = make_int2(first, rows);
        if (i == S - 1 && !(threadIdx.x & 1)) {
          // the odd last point's companion: the same point and rows in the
          // next window, which is staged as zeros
          a.z = __uint_as_float(base + 4u * kRows - bias);
          pa[threadIdx.x + 1] = a;
          pb[threadIdx.x + 1] = c;
          prow[threadIdx.x + 1] = make_int2(-(1 << 30), rows);
        }
      } else if (i > S || !(threadIdx.x & 1)) {
        prow[threadIdx.x] = make_int2(0, 0);
      }
      if ((threadIdx.x & (ST - 1)) == 0) {
        const int tile = threadIdx.x / ST;
        tile_mode[tile] = !(all_fast && in1) ? kTileDirect : (some ? kTileFast : kTileSkip);
        tile_inner[tile] = inner;
      }
    }
    __syncthreads();
    for (int t0 = 0; t0 < kBatch && i0 + t0 < S; t0 += ST) {
      const int cnt = min(ST, S - i0 - t0);
      const int mode = tile_mode[t0 / ST];
      if (mode == kTileSkip) continue;  // every bin is outside [0, T)
      if (mode == kTileDirect) {
        fv3 p[VZ];
        float val[VZ];
#pragma unroll
        for (int v = 0; v < VZ; v += 2) f2unpack(value[v / 2], val[v], val[v + 1]);
#pragma unroll
        for (int v = 0; v < VZ; ++v) p[v] = mkv(p0.x, p0.y, -npz[v]);
        velten_tile_direct<VZ>(b, T, S, sp, so, has_origin, bw, bo, fb, trb, i0 + t0, cnt, p, val);
#pragma unroll
        for (int v = 0; v < VZ; v += 2) value[v / 2] = f2pack(val[v], val[v + 1]);
        continue;
      }
      __syncthreads();  // the previous tile's windows are consumed
      {
        constexpr int kSub = 32 / ST, kStep = 8 * kSub;  // rows a warp, the CTA takes at once
        const int k = lane & (ST - 1);
        const int2 d = prow[t0 + k];
        const int r0 = (threadIdx.x >> 5) * kSub + lane / ST;
        uint32_t dst = (uint32_t)__cvta_generic_to_shared(win) + 4u * (uint32_t)(k * kRows + r0);
        const float* src = trb + i0 + t0 + k + ((int64_t)d.x + r0) * S;
        const int64_t step = (int64_t)kStep * S;
        if (tile_inner[t0 / ST]) {  // every row is a bin
#pragma unroll 4
          for (int r = r0; r < d.y; r += kStep, dst += 4u * kStep, src += step)
            cp_async4(dst, src, 4);
        } else {
          for (int r = r0; r < d.y; r += kStep, dst += 4u * kStep, src += step) {
            const bool bin = (unsigned)(d.x + r) < (unsigned)T;
            cp_async4(dst, bin ? src : trb, bin ? 4 : 0);
          }
        }
        cp_async_wait_all();
      }
      __syncthreads();
      // two points at a time: one test sends the lanes with a bin near a
      // boundary (in either point) to the exact chain. An odd last point is
      // joined by the dead one after it, whose window holds zeros.
#pragma unroll 1
      for (int j = 0; j < cnt; j += 2) {
        float w[2][VZ], off[2][VZ];
        float far = 0.f, near = 1.f;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const float4 a = pa[t0 + j + m], c = pb[t0 + j + m];
          const float dx = a.x - p0.x, dy = a.y - p0.y;
          const float r2 = fmaf(dx, dx, dy * dy);
          const uint32_t base = __float_as_uint(a.z);
          near = fminf(near, a.w);
#pragma unroll
          for (int v = 0; v < VZ; v += 2) {
            const u64 dz = f2add(f2pack(c.x, c.y), f2pack(npz[v], npz[v + 1]));
            float da, db, xa, xb;
            f2unpack(f2fma(dz, dz, f2pack(r2, r2)), da, db);
            const u64 q =
                f2fma(f2pack(sqrt_approx(da), sqrt_approx(db)), slope, f2pack(c.z, c.w));
            const u64 x = f2add(q, big);
            f2unpack(f2sub(q, f2sub(x, big)), off[m][v], off[m][v + 1]);
            f2unpack(x, xa, xb);
            far = absmax3(far, off[m][v], off[m][v + 1]);
            w[m][v] = lds(base + 4u * __float_as_uint(xa));
            w[m][v + 1] = lds(base + 4u * __float_as_uint(xb));
          }
        }
        if (!(far < near)) {
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            const float4 a = pa[t0 + j + m];
            const fv3 q = mkv(a.x, a.y, pb[t0 + j + m].x);
            const int i = min(i0 + t0 + j + m, S - 1);
            const float od2 = has_origin ? xmul(2.f, xlen(xsub3(q, so.at(b, i)))) : 0.f;
#pragma unroll
            for (int v = 0; v < VZ; ++v) {
              if (fabsf(off[m][v]) < a.w) continue;
              // the exact chain's bin is in the window like every other
              const fv3 e = xsub3(q, mkv(p0.x, p0.y, -npz[v]));
              const float t =
                  floorf(xadd(xdiv(xsub(xadd(od2, xmul(2.f, xlen(e))), bo), bw), 0.5f));
              w[m][v] = lds(__float_as_uint(a.z) + 4u * __float_as_uint(t + 12582912.f));
            }
          }
        }
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int v = 0; v < VZ; v += 2)
            value[v / 2] = f2add(value[v / 2], f2pack(w[m][v], w[m][v + 1]));
      }
    }
  }
  float val[VZ];
#pragma unroll
  for (int v = 0; v < VZ; v += 2) f2unpack(value[v / 2], val[v], val[v + 1]);
#pragma unroll
  for (int v = 0; v < VZ; ++v) {
    const int z = zt + kBZ * v;
    if (x < g.W && y < g.H && z < g.D)
      vol[(size_t)b * g.D * g.H * g.W + ((size_t)z * g.H + y) * g.W + x] = val[v];
  }
}

// Adjoint: transient_grad[t][s] = sum of the voxels whose bin from point s is
// t. A CTA keeps the [T][kTS] histogram of kTS scan points in shared memory
// and walks columns of kAZ voxels (all of them, or the share of its slice
// blockIdx.y when there are too few points to fill the GPU: the slices then
// add into a zeroed output). A thread takes one column and visits the kTS
// points in an order that starts at its lane, so the lanes of a warp work on
// all kTS points at once and only every kTS-th lane can meet another one in a
// histogram column; the column's coordinates, values and squared horizontal
// distance serve kAZ voxels. Bins are velten_bin_col2's, with the margin
// taken once per point over the volume's box. What bounds it: the
// compare-and-swap adds of the histogram (32 warps per SM hide their
// latency) and, next, instruction issue. Before, a thread took one point and
// one voxel at a time, with two 64-bit divisions for the voxel's index and three
// correctly rounded ones for its position per pair, in 8 warps per SM at 4,096
// bins: 96 x 88 x 72 voxels x 4,320 points x 4,096 bins took 60.4 ms
// (now 4.5 ms; 5.7 ms with the margin of the wider bound).
constexpr int kTS = 8, kAZ = 4;
__global__ void __launch_bounds__(1024) velten_adjoint_kernel(Grid g, int b, int T, int S, Pts3 sp,
                                                              Pts3 so, int has_origin, float bw,
                                                              float bo, FastBin fb, int64_t per_slice,
                                                              const float* __restrict__ vol,
                                                              float* __restrict__ tr) {
  extern __shared__ float hist[];  // [T][kTS]
  __shared__ float4 pts[kTS];      // scan point xyz, 2 |scan - origin|
  __shared__ float half_m[kTS];
  const int s0 = blockIdx.x * kTS;
  for (int j = threadIdx.x; j < T * kTS; j += blockDim.x) hist[j] = 0.f;
  if (threadIdx.x < kTS) {
    float4 pt = make_float4(0.f, 0.f, 0.f, 0.f);
    float hm = 0.f;
    if (s0 + (int)threadIdx.x < S) {
      const fv3 q = sp.at(b, s0 + threadIdx.x);
      pt = make_float4(q.x, q.y, q.z,
                       xmul(2.f, has_origin ? xlen(xsub3(q, so.at(b, s0 + threadIdx.x))) : 0.f));
      const fv3 ca = voxel_point(g, 0, 0, 0), cb = voxel_point(g, g.W - 1, g.H - 1, g.D - 1);
      const fv3 lo = mkv(fminf(ca.x, cb.x), fminf(ca.y, cb.y), fminf(ca.z, cb.z));
      const fv3 hi = mkv(fmaxf(ca.x, cb.x), fmaxf(ca.y, cb.y), fmaxf(ca.z, cb.z));
      const BoxBins bb = box_bins(q, pt.w, lo, hi, bw, bo, fb);
      hm = 0.5f - bb.margin;
    }
    pts[threadIdx.x] = pt;
    half_m[threadIdx.x] = hm;
  }
  __syncthreads();
  // columns: x fastest, then y, then the z block
  const int64_t plane = max((int64_t)g.H * g.W, (int64_t)1), step = blockDim.x;
  const int64_t units = (int64_t)((g.D + kAZ - 1) / kAZ) * g.H * g.W;
  const int64_t u1 = min(units, (int64_t)(blockIdx.y + 1) * per_slice);
  // (x, y, zb) of the thread's column, advanced by blockDim.x columns a step
  int64_t u = (int64_t)blockIdx.y * per_slice + threadIdx.x;
  const int W = max(g.W, 1), H = max(g.H, 1);
  int x = (int)(u % W), y = (int)((u / W) % H), zb = (int)(u / plane);
  const int sx = (int)(step % W), sy = (int)((step / W) % H), sz = (int)(step / plane);
  const float* vb = vol + (size_t)b * g.D * g.H * g.W;
  for (; u < u1; u += step) {
    float val[kAZ];
    fv3 p[kAZ];
    bool any = false;
#pragma unroll
    for (int k = 0; k < kAZ; ++k) {
      const int z = zb * kAZ + k;
      val[k] = z < g.D ? __ldg(vb + ((size_t)z * g.H + y) * g.W + x) : 0.f;
      any |= val[k] != 0.f;
    }
    if (any) {
#pragma unroll
      for (int k = 0; k < kAZ; ++k)
        p[k] = mkv(0.f, 0.f, grid_coord(g.sz, g.ez, g.D, min(zb * kAZ + k, g.D - 1)));
      p[0].x = grid_coord(g.sx, g.ex, g.W, x);
      p[0].y = grid_coord(g.sy, g.ey, g.H, y);
#pragma unroll
      for (int k = 1; k < kAZ; ++k) p[k].x = p[0].x, p[k].y = p[0].y;
#pragma unroll 1
      for (int i = 0; i < kTS; ++i) {
        const int sl = (threadIdx.x + i) & (kTS - 1);
        if (s0 + sl >= S) continue;
        const float4 q = pts[sl];
        const float hm = half_m[sl];
        const float dx = q.x - p[0].x, dy = q.y - p[0].y;
        const float r2 = fmaf(dx, dx, dy * dy);
#pragma unroll
        for (int k = 0; k < kAZ; k += 2) {
          int t[2];
          velten_bin_col2(mkv(q.x, q.y, q.z), q.w, p[k], p[k + 1], r2, bw, bo, fb.inv_bw, fb.nbo,
                          hm, t[0], t[1]);
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if ((unsigned)t[h] < (unsigned)T && val[k + h] != 0.f)
              atomicAdd(hist + t[h] * kTS + sl, val[k + h]);
        }
      }
    }
    x += sx;
    if (x >= W) x -= W, ++y;
    y += sy;
    if (y >= H) y -= H, ++zb;
    zb += sz;
  }
  __syncthreads();
  float* out = tr + (size_t)b * T * S;
  for (int j = threadIdx.x; j < T * kTS; j += blockDim.x) {
    const int t = j / kTS, c = j - t * kTS;
    if (s0 + c >= S) continue;
    if (gridDim.y == 1) out[(size_t)t * S + s0 + c] = hist[j];
    else if (hist[j] != 0.f) atomicAdd(out + (size_t)t * S + s0 + c, hist[j]);
  }
}

__global__ void __launch_bounds__(128) velten_exhaustive_kernel(Grid g, int b, int T, int S, int L,
                                                                Pts3 sp, Pts3 lp, Pts3 so, Pts3 lo,
                                                                int has_so, int has_lo, float bw,
                                                                float bo,
                                                                const float* __restrict__ tr,
                                                                float* __restrict__ vol) {
  const int64_t nv = (int64_t)g.D * g.H * g.W;
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  const int x = (int)(v % g.W), y = (int)((v / g.W) % g.H), z = (int)(v / ((int64_t)g.W * g.H));
  const fv3 p = voxel_point(g, x, y, z);
  const float* trb = tr + (size_t)b * T * S * L;
  float value = 0.f;
  for (int s = 0; s < S; ++s) {
    const fv3 q = sp.at(b, s);
    const float sv = xlen(xsub3(q, p));
    const float sod = has_so ? xlen(xsub3(q, so.at(b, s))) : 0.f;
    const float a = xadd(sod, sv);
    for (int l = 0; l < L; ++l) {
      const fv3 r = lp.at(b, l);
      const float lv = xlen(xsub3(r, p));
      const float lod = has_lo ? xlen(xsub3(r, lo.at(b, l))) : 0.f;
      const int t = nearest_bin(xadd(xadd(a, lv), lod), bw, bo);
      if (t >= 0 && t < T) value += __ldg(trb + ((size_t)t * S + s) * L + l);
    }
  }
  vol[(size_t)b * nv + v] = value;
}

// Velten exhaustive over blocks of 8 x 8 x 16 voxels, four of a column per
// thread. A path length is the sum of a scan and a laser distance, so a thread
// keeps its voxels' distances to a group of kLG lasers in shared memory, takes
// the distances to each scan point of its slice once per group, and a triple
// costs two additions, the bin (exactly as nearest_bin rounds it: div_fixed and a
// floor by an addition rounded down, two voxels per paired instruction) and one
// read. Transient element (t, s, l) is tr[((s - s_base) L + l) cstep + t bstep]: in
// bins-last order (kLast, bstep 1) the lanes' bins of a pair lie within a few
// cache lines, in place every bin is another sector. What bounds it: the FP32
// pipe (59%) and waits on the reads through L1, at 66% of issue slots.
// 48^3 voxels x 256 scan points x 64 lasers, 1,024 bins: 7.9 ms (two correctly
// rounded roots and a division per triple, in-place reads) -> 1.24 ms.
constexpr int kLG = 8;
template <bool kLast>
__global__ void __launch_bounds__(256, 4) velten_pairs_kernel(
    Grid g, int b, int T, int S, int L, Pts3 sp, Pts3 lp, Pts3 so, Pts3 lo, int has_so, int has_lo,
    float bw, float bo, float inv_bw, int s_base, int s_end, int per_slice,
    const float* __restrict__ tr, int64_t cstep, int64_t bstep, float* __restrict__ vol, int add) {
  using u64 = unsigned long long;
  __shared__ float4 laser[kLG][256];
  __shared__ float lod[kLG];
  const int nbx = (g.W + 7) >> 3, nby = (g.H + 7) >> 3;
  const int x = (int)(blockIdx.x % nbx) * 8 + (threadIdx.x & 7);
  const int y = (int)(blockIdx.x / nbx % nby) * 8 + ((threadIdx.x >> 3) & 7);
  const int z0 = (int)(blockIdx.x / (nbx * nby)) * 16 + (threadIdx.x >> 6);
  // voxels z0 + 4 v; those past the volume's edge work on a clamped position
  fv3 p[4];
#pragma unroll
  for (int v = 0; v < 4; ++v)
    p[v] = voxel_point(g, min(x, g.W - 1), min(y, g.H - 1), min(z0 + 4 * v, g.D - 1));
  const u64 nbo = f2pack(-bo, -bo), nbw = f2pack(-bw, -bw), inv = f2pack(inv_bw, inv_bw);
  const u64 half = f2pack(0.5f, 0.5f), big = f2pack(12582912.f, 12582912.f);  // 1.5 2^23
  const int s0 = s_base + blockIdx.y * per_slice, s1 = min(s_end, s0 + per_slice);
  u64 acc[2] = {0ull, 0ull};
  for (int l0 = 0; l0 < L; l0 += kLG) {
    const int nl = min(kLG, L - l0);
    __syncthreads();  // the previous group's origin terms are consumed
    if ((int)threadIdx.x < nl)
      lod[threadIdx.x] =
          has_lo ? xlen(xsub3(lp.at(b, l0 + threadIdx.x), lo.at(b, l0 + threadIdx.x))) : 0.f;
#pragma unroll 1
    for (int k = 0; k < nl; ++k) {
      const fv3 q = lp.at(b, l0 + k);
      laser[k][threadIdx.x] = make_float4(xlen(xsub3(q, p[0])), xlen(xsub3(q, p[1])),
                                          xlen(xsub3(q, p[2])), xlen(xsub3(q, p[3])));
    }
    __syncthreads();
    for (int s = s0; s < s1; ++s) {
      const fv3 q = sp.at(b, s);
      const float sod = has_so ? xlen(xsub3(q, so.at(b, s))) : 0.f;
      u64 a[2];
#pragma unroll
      for (int h = 0; h < 2; ++h)
        a[h] = f2pack(xadd(sod, xlen(xsub3(q, p[2 * h]))), xadd(sod, xlen(xsub3(q, p[2 * h + 1]))));
      const float* col = tr + ((int64_t)(s - s_base) * L + l0) * cstep;
      u64 part[2] = {0ull, 0ull};
#pragma unroll 2
      for (int k = 0; k < nl; ++k, col += cstep) {
        const float4 d = laser[k][threadIdx.x];
        const u64 o = f2pack(lod[k], lod[k]);
        const u64 ld[2] = {f2pack(d.x, d.y), f2pack(d.z, d.w)};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const u64 n = f2add(f2add(f2add(a[h], ld[h]), o), nbo);
          u64 c = f2mul(n, inv);  // div_fixed
          c = f2fma(f2fma(c, nbw, n), inv, c);
          c = f2fma(f2fma(c, nbw, n), inv, c);
          float xa, xb;
          f2unpack(f2add_rm(f2add(c, half), big), xa, xb);
          // (a bin outside [0, T), or a NaN, reads nothing)
          const unsigned ta = __float_as_uint(xa) - 0x4B400000u;
          const unsigned tb = __float_as_uint(xb) - 0x4B400000u;
          const float va = ta < (unsigned)T ? __ldg(col + (kLast ? (int64_t)ta : ta * bstep)) : 0.f;
          const float vb = tb < (unsigned)T ? __ldg(col + (kLast ? (int64_t)tb : tb * bstep)) : 0.f;
          part[h] = f2add(part[h], f2pack(va, vb));
        }
      }
      acc[0] = f2add(acc[0], part[0]);
      acc[1] = f2add(acc[1], part[1]);
    }
  }
  float val[4];
  f2unpack(acc[0], val[0], val[1]);
  f2unpack(acc[1], val[2], val[3]);
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    if (x >= g.W || y >= g.H || z0 + 4 * v >= g.D) continue;
    // (a slice's volume is its own)
    float* dst = vol + (((size_t)blockIdx.y * g.D + z0 + 4 * v) * g.H + y) * g.W + x;
    *dst = add ? *dst + val[v] : val[v];
  }
}

struct Pts3T {  // [B, 3, n] with strides
  const float* p;
  int64_t sb, sc, sn;
  __device__ fv3 at(int b, int i) const {
    const float* q = p + b * sb + i * sn;
    return mkv(q[0], q[sc], q[2 * sc]);
  }
};

// Arellano (backprojection_cuda.cu:11-115): per (column, scan, laser), scale
// the ellipsoid of constant path length to a sphere along the scan-laser axis
// and deposit each positive bin where the column's ray meets it. int()
// truncation makes the reference's interpolation weight always 0 (nearest).
__global__ void __launch_bounds__(64) arellano_kernel(Grid g, int b, int T, int S, int L, Pts3T sp,
                                                      Pts3T lp, Pts3T so, Pts3T lo, int has_so,
                                                      int has_lo, float bw, float bo,
                                                      const float* __restrict__ tr,
                                                      float* __restrict__ vol) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int s = blockIdx.y, l = blockIdx.z;
  if (c >= g.H * g.W) return;
  const int xi = c % g.W, yi = c / g.W;
  const float xf = xadd(g.sx, xmul(xdiv((float)xi, (float)(g.W - 1)), xsub(g.ex, g.sx)));
  const float yf = xadd(g.sy, xmul(xdiv((float)yi, (float)(g.H - 1)), xsub(g.ey, g.sy)));
  const fv3 sc = sp.at(b, s), lc = lp.at(b, l);
  const float sd = has_so ? xlen(xsub3(sc, so.at(b, s))) : 0.f;
  const float ld = has_lo ? xlen(xsub3(lc, lo.at(b, l))) : 0.f;
  const fv3 center = mkv(xmul(0.5f, xadd(sc.x, lc.x)), xmul(0.5f, xadd(sc.y, lc.y)),
                         xmul(0.5f, xadd(sc.z, lc.z)));
  fv3 nrm = xsub3(sc, lc);
  const float length = xlen(nrm);
  if (length > 1e-6f) {
    const float inv = xdiv(1.f, length);
    nrm = mkv(xmul(inv, nrm.x), xmul(inv, nrm.y), xmul(inv, nrm.z));
  }
  const fv3 rs = xsub3(mkv(xf, yf, g.sz), center);
  const fv3 re = xsub3(mkv(xf, yf, g.ez), center);
  const float* col = tr + (((size_t)b * T) * S + s) * L + l;
  const size_t st = (size_t)S * L;
  float* vb = vol + (size_t)b * g.D * g.H * g.W + c;
  const size_t vs = (size_t)g.H * g.W;
  for (int t = 0; t < T; ++t) {
    const float value = __ldg(col + t * st);
    if (!(value > 0.f)) continue;
    const float tc = xsub(xsub(xadd(xmul((float)t, bw), bo), sd), ld);
    if (!(tc > length)) continue;
    const float r0 = xdiv(tc, 2.f);
    const float r1 = xsqrt(xsub(xmul(r0, r0), xdiv(xmul(length, length), 4.f)));
    const float scale = xdiv(r1, r0);
    const float ks = xmul(xsub(scale, 1.f), xdot(rs, nrm));
    const float ke = xmul(xsub(scale, 1.f), xdot(re, nrm));
    const fv3 st0 = mkv(xfma(ks, nrm.x, rs.x), xfma(ks, nrm.y, rs.y), xfma(ks, nrm.z, rs.z));
    const fv3 et = mkv(xfma(ke, nrm.x, re.x), xfma(ke, nrm.y, re.y), xfma(ke, nrm.z, re.z));
    fv3 dir = xsub3(et, st0);
    const float rl = xlen(dir);
    const float ir = xdiv(1.f, rl);
    dir = mkv(xmul(ir, dir.x), xmul(ir, dir.y), xmul(ir, dir.z));
    const float v0 = xdot(dir, st0);
    float v1 = xsub(xmul(v0, v0), xsub(xdot(st0, st0), xmul(r1, r1)));
    if (!(v1 > 0.f)) continue;
    v1 = xsqrt(v1);
    float d = xsub(-v0, v1);
    if (d < 0.f) d = xadd(-v0, v1);
    const float bf = xadd(xmul(xdiv(d, rl), (float)g.D), 0.5f);
    if (!(bf > -1.f && bf < (float)g.D)) continue;
    atomicAdd(vb + (size_t)(int)bf * vs, value);
  }
}

}  // namespace bp

namespace {

int check_volume_out(const totri_array_t* vol, bp::Grid& g, const float* start, const float* end,
                     int64_t& B) {
  TOTRI_TRY(check_array(vol, "volume", 4, -1));
  if (vol->dtype != TOTRI_FLOAT32)
    return fail(TOTRI_ERR_UNSUPPORTED, "backprojection: only float32 tensors are supported");
  TOTRI_TRY(check_contiguous(vol, "volume"));
  B = vol->shape[0];
  g = bp::Grid{(int)vol->shape[1], (int)vol->shape[2], (int)vol->shape[3], start[0], start[1],
               start[2], end[0], end[1], end[2]};
  return TOTRI_OK;
}

int check_pts3(const totri_array_t* a, const char* name, int64_t B, int64_t& n, bp::Pts3& p) {
  TOTRI_TRY(check_array(a, name, 3, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(a, name, 0, B));
  TOTRI_TRY(check_dim(a, name, 2, 3));
  n = a->shape[1];
  p = bp::Pts3{static_cast<const float*>(a->data), a->strides[0], a->strides[1], a->strides[2]};
  return TOTRI_OK;
}

int check_pts3t(const totri_array_t* a, const char* name, int64_t B, int64_t& n, bp::Pts3T& p) {
  TOTRI_TRY(check_array(a, name, 3, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(a, name, 0, B));
  TOTRI_TRY(check_dim(a, name, 1, 3));
  n = a->shape[2];
  p = bp::Pts3T{static_cast<const float*>(a->data), a->strides[0], a->strides[1], a->strides[2]};
  return TOTRI_OK;
}

int origin_of(const totri_array_t* o, int64_t n, int has) {
  (void)o;
  (void)n;
  return has;
}

}  // namespace
}  // namespace totri

using namespace totri;

extern "C" {

int totri_backprojection_confocal_velten_forward(const totri_array_t* transient,
                                                 const totri_array_t* scan_points,
                                                 const totri_array_t* scan_origin,
                                                 const totri_array_t* volume, const float start[3],
                                                 const float end[3], float bw, float bo,
                                                 void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  bp::Grid g;
  int64_t B, S, So;
  TOTRI_TRY(check_volume_out(volume, g, start, end, B));
  bp::Pts3 sp, so;
  TOTRI_TRY(check_pts3(scan_points, "scan_points", B, S, sp));
  TOTRI_TRY(check_pts3(scan_origin, "scan_origin", B, So, so));
  if (So != 0 && So != S) return fail(TOTRI_ERR_INVALID_ARGUMENT, "scan_origin size mismatch");
  TOTRI_TRY(check_array(transient, "transient", 3, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(transient, "transient", 0, B));
  TOTRI_TRY(check_dim(transient, "transient", 2, S));
  TOTRI_TRY(check_contiguous(transient, "transient"));
  const int T = (int)transient->shape[1];
  const int64_t nv = (int64_t)g.D * g.H * g.W;
  if (nv == 0 || B == 0) return TOTRI_OK;
  if (S == 0 || T == 0) {  // (an empty transient has no address to stage rows from)
    TOTRI_CUDA(cudaMemsetAsync(volume->data, 0, sizeof(float) * (size_t)(B * nv), stream));
    return TOTRI_OK;
  }
  const bool tiled = tune::get("backprojection.velten.mode") != 1;
  int vz = tune::get("backprojection.velten.vz");
  if (vz <= 0) vz = 4;
  if (vz == 1) vz = 2;  // voxels go in pairs: 1 is taken as 2
  if (vz != 2 && vz != 4)
    return fail(TOTRI_ERR_INVALID_ARGUMENT, "backprojection.velten.vz must be 2 or 4");
  const dim3 grid((unsigned)ceil_div(g.W, bp::kBX), (unsigned)ceil_div(g.H, bp::kBY),
                  (unsigned)ceil_div(g.D, bp::kBZ * vz));
  // Points per tile (32, 16 or 8; "backprojection.velten.points" sets it): the
  // most whose windows are a third larger than a block's bins from one point, at
  // most 2 |block diagonal| / bw + 4 rows, so that the bins of 8 neighbouring
  // points mostly fit too (windows per point read the transient 4 bytes at a
  // time). 230 rows of 385 at 16 points: 26.3 ms against 30.0 ms with 8
  // (128^3 x 16,384 points, 4,096 bins); 385 rows of 385: 4.46 ms against 3.73 ms
  // with 8 (96 x 88 x 72 x 4,320, 4,096 bins); 60 rows of 193 at 32 points:
  // 17.2 ms against 18.2 ms with 16 (128^3 x 16,384, 1,024 bins).
  const auto pitch = [](float a, float e, int n) {
    return n > 1 ? std::fabs((double)e - (double)a) / (n - 1) : 0.0;
  };
  const double ex = (bp::kBX - 1) * pitch(g.sx, g.ex, g.W);
  const double ey = (bp::kBY - 1) * pitch(g.sy, g.ey, g.H);
  const double ez = (bp::kBZ * vz - 1) * pitch(g.sz, g.ez, g.D);
  const double rows = 2.0 * std::sqrt(ex * ex + ey * ey + ez * ez) / std::fabs((double)bw) + 4.0;
  int st = tune::get("backprojection.velten.points");
  if (st != 8 && st != 16 && st != 32)
    st = rows <= 0.75 * bp::win_rows(32) ? 32 : (rows <= 0.75 * bp::win_rows(16) ? 16 : 8);
  const bp::FastBin fb = bp::make_fast_bin(bw, bo);
  const float* trp = static_cast<const float*>(transient->data);
  float* volp = static_cast<float*>(volume->data);
  for (int b = 0; b < (int)B; ++b) {
#define TOTRI_VELTEN_TILED(VZ, ST)                                                 \
  TOTRI_KERNEL("backprojection velten confocal", stream,                          \
               bp::velten_confocal_tiled_kernel<VZ, ST><<<grid, 256, 0, stream>>>( \
                   g, b, T, (int)S, sp, so, So > 0, bw, bo, fb, trp, volp))
    if (!tiled)
      TOTRI_KERNEL("backprojection velten confocal", stream,
                   bp::velten_confocal_kernel<<<(unsigned)ceil_div(nv, 256), 256, 0, stream>>>(
                       g, b, T, (int)S, sp, so, So > 0, bw, bo, fb, trp, volp));
    else if (vz == 4 && st == 32)
      TOTRI_VELTEN_TILED(4, 32);
    else if (vz == 4 && st == 16)
      TOTRI_VELTEN_TILED(4, 16);
    else if (vz == 4)
      TOTRI_VELTEN_TILED(4, 8);
    else if (st == 32)
      TOTRI_VELTEN_TILED(2, 32);
    else if (st == 16)
      TOTRI_VELTEN_TILED(2, 16);
    else
      TOTRI_VELTEN_TILED(2, 8);
#undef TOTRI_VELTEN_TILED
  }
  return TOTRI_OK;
}

int totri_backprojection_confocal_velten_adjoint(const totri_array_t* volume,
                                                 const totri_array_t* scan_points,
                                                 const totri_array_t* scan_origin,
                                                 const totri_array_t* transient,
                                                 const float start[3], const float end[3],
                                                 float bw, float bo, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  bp::Grid g;
  int64_t B, S, So;
  TOTRI_TRY(check_volume_out(volume, g, start, end, B));
  bp::Pts3 sp, so;
  TOTRI_TRY(check_pts3(scan_points, "scan_points", B, S, sp));
  TOTRI_TRY(check_pts3(scan_origin, "scan_origin", B, So, so));
  if (So != 0 && So != S) return fail(TOTRI_ERR_INVALID_ARGUMENT, "scan_origin size mismatch");
  TOTRI_TRY(check_array(transient, "transient", 3, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(transient, "transient", 0, B));
  TOTRI_TRY(check_dim(transient, "transient", 2, S));
  TOTRI_TRY(check_contiguous(transient, "transient"));
  const int T = (int)transient->shape[1];
  if (numel(transient) == 0) return TOTRI_OK;
  const size_t smem = sizeof(float) * (size_t)T * bp::kTS;
  if (smem > 200 * 1024) return fail(TOTRI_ERR_UNSUPPORTED, "too many bins for one tile");
  TOTRI_CUDA(tune::ensure_dynamic_smem(
      reinterpret_cast<const void*>(bp::velten_adjoint_kernel), smem));
  // 1,024 threads once the histogram leaves room for one CTA per SM only, else 512,
  // and not many more than there are columns (8^3 voxels x 16,384 points, 1,024 bins: 96
  // us with 512, 67 with 128; nearly all voxels zero 86 and 63). A second grid dimension slices the voxels until about 8 waves of CTAs
  // are in flight, each slice with at least 16 columns per thread (zeroing and
  // flushing the histogram costs about what 1 or 2 take).
  const int64_t units = (int64_t)ceil_div(g.D, bp::kAZ) * g.H * g.W;
  const int threads = smem > 100 * 1024 ? 1024 : (units <= 128 ? 128 : (units <= 256 ? 256 : 512));
  const int64_t tiles = ceil_div(S, bp::kTS);
  const int64_t resident = (int64_t)tune::sm_count() *
                           std::max<int64_t>(1, std::min<int64_t>(2048 / threads,
                                                                  (220 * 1024) / (smem + 1024)));
  const int64_t slices = std::max<int64_t>(
      1, std::min<int64_t>(ceil_div(8 * resident, tiles), units / (16 * (int64_t)threads)));
  const int64_t per = std::max<int64_t>(1, ceil_div(units, slices));
  const dim3 grid((unsigned)tiles, (unsigned)std::max<int64_t>(1, ceil_div(units, per)));
  if (grid.y > 1)
    TOTRI_CUDA(cudaMemsetAsync(transient->data, 0, sizeof(float) * numel(transient), stream));
  for (int b = 0; b < (int)B; ++b)
    TOTRI_KERNEL("backprojection velten adjoint", stream,
                 bp::velten_adjoint_kernel<<<grid, threads, smem, stream>>>(
                     g, b, T, (int)S, sp, so, So > 0, bw, bo, bp::make_fast_bin(bw, bo), per,
                     static_cast<const float*>(volume->data),
                     static_cast<float*>(transient->data)));
  return TOTRI_OK;
}

// The blocked kernel takes its bins from div_fixed (bin widths within 1e-18 .. 1e18)
// and a rounding by addition (bins below 2^21); anything else goes one voxel per
// thread ("backprojection.velten.pairs" = 1: always).
static bool velten_blocked(int64_t S, int64_t L, int64_t T, float bw) {
  const float abw = std::fabs(bw);
  return abw > 1e-18f && abw < 1e18f && T <= (1 << 21) && S > 0 && L > 0 && T > 0 &&
         tune::get("backprojection.velten.pairs") != 1;
}

// Bins-last copies but where a pair's column has more bins than the volume has voxels
// to read them; slices of the scan points until about 4 waves of CTAs (4 per SM), with
// at least 4 scan points each (a slice repeats the lasers' distances).
static mesh::PairPlan velten_plan(int64_t S, int64_t L, int64_t T, int64_t D, int64_t H, int64_t W,
                                  size_t ws_bytes) {
  const int64_t blocks = ceil_div(W, 8) * ceil_div(H, 8) * ceil_div(D, 16);
  return mesh::pair_plan(S, L, T, D * H * W, blocks, 16 * (int64_t)tune::sm_count(), 4,
                         D * H * W >= T, ws_bytes);
}

size_t totri_backprojection_exhaustive_velten_scratch(int64_t S, int64_t L, int64_t T) {
  // Partial sums of a launch: slices of at most 1,024 voxels per CTA, fewer than
  // 2 x 16 CTAs per SM where there is more than one.
  const size_t partial = S < 8 ? 0 : sizeof(float) * 1024 * 32 * (size_t)tune::sm_count();
  return S > 0 && L > 0 && T > 0 ? mesh::exh_grad_scratch_bytes(S, L, T) + partial : 0;
}

size_t totri_backprojection_exhaustive_velten_workspace(int64_t S, int64_t L, int64_t T, int64_t D,
                                                        int64_t H, int64_t W, float bw) {
  if (D <= 0 || H <= 0 || W <= 0 || !velten_blocked(S, L, T, bw)) return 0;
  return velten_plan(S, L, T, D, H, W, SIZE_MAX).bytes;
}

int totri_backprojection_exhaustive_velten_forward_ws(
    const totri_array_t* transient, const totri_array_t* scan_points,
    const totri_array_t* laser_points, const totri_array_t* scan_origin,
    const totri_array_t* laser_origin, const totri_array_t* volume, const float start[3],
    const float end[3], float bw, float bo, void* ws, size_t ws_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  bp::Grid g;
  int64_t B, S, L, So, Lo;
  TOTRI_TRY(check_volume_out(volume, g, start, end, B));
  bp::Pts3 sp, lp, so, lo;
  TOTRI_TRY(check_pts3(scan_points, "scan_points", B, S, sp));
  TOTRI_TRY(check_pts3(laser_points, "laser_points", B, L, lp));
  TOTRI_TRY(check_pts3(scan_origin, "scan_origin", B, So, so));
  TOTRI_TRY(check_pts3(laser_origin, "laser_origin", B, Lo, lo));
  if ((So != 0 && So != S) || (Lo != 0 && Lo != L))
    return fail(TOTRI_ERR_INVALID_ARGUMENT, "origin size mismatch");
  TOTRI_TRY(check_array(transient, "transient", 4, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(transient, "transient", 0, B));
  TOTRI_TRY(check_dim(transient, "transient", 2, S));
  TOTRI_TRY(check_dim(transient, "transient", 3, L));
  TOTRI_TRY(check_contiguous(transient, "transient"));
  const int64_t T = transient->shape[1];
  const int64_t nv = (int64_t)g.D * g.H * g.W;
  if (nv == 0) return TOTRI_OK;
  const float* trp = static_cast<const float*>(transient->data);
  float* volp = static_cast<float*>(volume->data);
  if (!velten_blocked(S, L, T, bw)) {
    for (int b = 0; b < (int)B; ++b)
      TOTRI_KERNEL("backprojection velten exhaustive", stream,
                   bp::velten_exhaustive_kernel<<<(unsigned)ceil_div(nv, 128), 128, 0, stream>>>(
                       g, b, (int)T, (int)S, (int)L, sp, lp, so, lo, So > 0, Lo > 0, bw, bo, trp,
                       volp));
    return TOTRI_OK;
  }
  const mesh::PairPlan plan = velten_plan(S, L, T, g.D, g.H, g.W, ws ? ws_bytes : 0);
  const int64_t blocks = ceil_div(g.W, 8) * ceil_div(g.H, 8) * ceil_div(g.D, 16);
  const int64_t row = S * L;
  float* copy = static_cast<float*>(ws);
  float* part = reinterpret_cast<float*>(static_cast<char*>(ws) + plan.part_at);
  for (int b = 0; b < (int)B; ++b)
    for (int64_t sa = 0; sa < S; sa += plan.step) {
      const int64_t sb = std::min(S, sa + plan.step);
      const int slices = (int)ceil_div(sb - sa, plan.per);
      const dim3 grid((unsigned)blocks, (unsigned)slices);
      const float* tb = trp + (int64_t)b * T * row;
      float* out = volp + (int64_t)b * nv;
      float* dst = slices > 1 ? part : out;
      const int add = slices == 1 && sa > 0;
      if (plan.chunk > 0) {
        TOTRI_TRY(mesh::launch_bins_last(tb + sa * L, copy, (int)T, (int)T, row, (sb - sa) * L,
                                         stream));
        TOTRI_KERNEL("backprojection velten exhaustive", stream,
                     bp::velten_pairs_kernel<true><<<grid, 256, 0, stream>>>(
                         g, b, (int)T, (int)S, (int)L, sp, lp, so, lo, So > 0, Lo > 0, bw, bo,
                         1.f / bw, (int)sa, (int)sb, plan.per, copy, T, 1, dst, add));
      } else {
        TOTRI_KERNEL("backprojection velten exhaustive", stream,
                     bp::velten_pairs_kernel<false><<<grid, 256, 0, stream>>>(
                         g, b, (int)T, (int)S, (int)L, sp, lp, so, lo, So > 0, Lo > 0, bw, bo,
                         1.f / bw, (int)sa, (int)sb, plan.per, tb, 1, row, dst, add));
      }
      if (slices > 1)
        TOTRI_TRY(mesh::launch_sum_slices(part, slices, nv, out, sa > 0, stream));
    }
  return TOTRI_OK;
}

int totri_backprojection_exhaustive_velten_forward(
    const totri_array_t* transient, const totri_array_t* scan_points,
    const totri_array_t* laser_points, const totri_array_t* scan_origin,
    const totri_array_t* laser_origin, const totri_array_t* volume, const float start[3],
    const float end[3], float bw, float bo, void* stream) {
  return totri_backprojection_exhaustive_velten_forward_ws(
      transient, scan_points, laser_points, scan_origin, laser_origin, volume, start, end, bw, bo,
      nullptr, 0, stream);
}

int totri_backprojection_exhaustive_arellano_forward(
    const totri_array_t* transient, const totri_array_t* scan_points,
    const totri_array_t* laser_points, const totri_array_t* scan_origin,
    const totri_array_t* laser_origin, const totri_array_t* volume, const float start[3],
    const float end[3], float bw, float bo, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  bp::Grid g;
  int64_t B, S, L, So, Lo;
  TOTRI_TRY(check_volume_out(volume, g, start, end, B));
  bp::Pts3T sp, lp, so, lo;
  TOTRI_TRY(check_pts3t(scan_points, "scan_points", B, S, sp));
  TOTRI_TRY(check_pts3t(laser_points, "laser_points", B, L, lp));
  TOTRI_TRY(check_pts3t(scan_origin, "scan_origin", B, So, so));
  TOTRI_TRY(check_pts3t(laser_origin, "laser_origin", B, Lo, lo));
  if ((So != 0 && So != S) || (Lo != 0 && Lo != L))
    return fail(TOTRI_ERR_INVALID_ARGUMENT, "origin size mismatch");
  TOTRI_TRY(check_array(transient, "transient", 4, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(transient, "transient", 0, B));
  TOTRI_TRY(check_dim(transient, "transient", 2, S));
  TOTRI_TRY(check_dim(transient, "transient", 3, L));
  TOTRI_TRY(check_contiguous(transient, "transient"));
  const int T = (int)transient->shape[1];
  if (g.H * g.W == 0 || S == 0 || L == 0) return TOTRI_OK;
  for (int b = 0; b < (int)B; ++b) {
    const dim3 grid((unsigned)ceil_div(g.H * g.W, 64), (unsigned)S, (unsigned)L);
    TOTRI_KERNEL("backprojection arellano", stream,
                 bp::arellano_kernel<<<grid, 64, 0, stream>>>(
                     g, b, T, (int)S, (int)L, sp, lp, so, lo, origin_of(scan_origin, S, So > 0),
                     origin_of(laser_origin, L, Lo > 0), bw, bo,
                     static_cast<const float*>(transient->data),
                     static_cast<float*>(volume->data)));
  }
  return TOTRI_OK;
}

}  // extern "C"
