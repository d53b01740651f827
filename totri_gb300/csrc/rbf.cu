// RBF-to-volume splatting and its gradient.
//
// Reference: src/util/rbf2volume_cuda.cu (:50-93 forward, one thread per voxel
// reading every Gaussian from global memory; :124-201 gradient, one block
// column per Gaussian with a shared-memory tree reduction and an atomic per
// (Gaussian, channel, 64 voxels)). Here both kernels work on bricks of voxels,
// skip the Gaussians that contribute exactly zero to the whole brick (the
// underflow cull below), and use that a Gaussian's weight is a product of one
// factor per axis: the forward gives each thread a column of voxels and reads
// the factors from shared memory; the gradient gives each lane a Gaussian and
// sums over the brick axis by axis.
#include <algorithm>
#include <string>

#include "capi_common.cuh"
#include "tune.cuh"

namespace totri {
namespace rbf {

constexpr int kMaxAttr = 8;
constexpr int kTile = 256;

struct Grid {
  int D, H, W;
  float sx, sy, sz, ex, ey, ez;
};

// Voxel coordinate (rbf2volume_cuda.cu:58-60): midpoint for a single-voxel
// axis, else start + ((end - start) * i) / (n - 1).
__device__ __forceinline__ float coord(float s, float e, int n, int i) {
  return n == 1 ? 0.5f * (s + e) : s + ((e - s) * (float)i) / (float)(n - 1);
}

// 2^x from the hardware approximation (ex2.approx, relative error about
// 2^-22; results below the normal range flush to zero): the Gaussians are
// values, compared with tolerances, and -d2 / (2 sigma^2) folds into one
// multiply by a per-Gaussian constant -log2(e) / (2 sigma^2).
__device__ __forceinline__ float exp2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

constexpr float kLog2e = 1.4426950408889634f;

// -log2(e) / (2 sigma^2) as hi + lo: the remainder of the division by sigma^2,
// itself with its rounding error. hi is the FP32 quotient, which the cull and
// the voxel-by-voxel evaluation use.
struct Exponent {
  float hi, lo;
};
__device__ __forceinline__ Exponent exponent(float sigma) {
  const float kh = 0.72134752f, kl = (float)(0.72134752044448170368 - (double)0.72134752f);
  const float s = __fmul_rn(sigma, sigma), se = __fmaf_rn(sigma, sigma, -s);
  Exponent k;
  k.hi = __fdiv_rn(-kh, s);
  k.lo = __fdividef((__fmaf_rn(-k.hi, s, -kh) - kl) - k.hi * se, s);
  if (!isfinite(k.lo)) k.lo = 0.f;
  return k;
}

__device__ __forceinline__ float warp_sum_f(float x) {
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

struct Rbf {  // [B, N, C] with strides
  const float* p;
  int64_t sb, sn, sc;
  __device__ float at(int b, int i, int c) const { return p[b * sb + i * sn + c * sc]; }
};

// Tile-level cull at the underflow radius. ex2.approx.ftz flushes results
// below 2^-126 to zero, so a Gaussian whose exponent argument d2 * k2 lies
// below -126.5 at every voxel of a brick adds exactly +0 (or -0) there, and
// an accumulator that started at +0 is unchanged by it: skipping it leaves the
// sums bit for bit the same, in the same order. The test uses the squared
// distance from the centre to the brick's coordinate box (voxel coordinates
// are monotone in the index), computed in FP32, against 128 / |k2|, which
// leaves a margin far beyond the few ulps of the voxel-level arithmetic.
// Gaussians with a non-finite value are never culled (0 * inf would not be a
// zero term). The tuning key "rbf.cull" = 1 turns the cull off.
constexpr float kCullArg = 128.f;

// Squared distance from (cx, cy, cz) to the box [lo, hi].
__device__ __forceinline__ float box_dist2(float cx, float cy, float cz, const float lo[3],
                                           const float hi[3]) {
  const float dx = fmaxf(fmaxf(lo[0] - cx, cx - hi[0]), 0.f);
  const float dy = fmaxf(fmaxf(lo[1] - cy, cy - hi[1]), 0.f);
  const float dz = fmaxf(fmaxf(lo[2] - cz, cz - hi[2]), 0.f);
  return dx * dx + dy * dy + dz * dz;
}

// Coordinate box of the voxels [i0, i1] of one axis.
__device__ __forceinline__ void axis_box(float s, float e, int n, int i0, int i1, float& lo,
                                         float& hi) {
  const float a = coord(s, e, n, i0), b = coord(s, e, n, i1);
  lo = fminf(a, b);
  hi = fmaxf(a, b);
}

// Block-wide compaction: this thread's slot among the flagged threads (or -1);
// *total receives their count. All threads of the block call it.
__device__ __forceinline__ int block_slot(bool flag, int* warp_counts, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const unsigned bal = __ballot_sync(0xffffffffu, flag);
  if (lane == 0) warp_counts[warp] = __popc(bal);
  __syncthreads();
  int base = 0, sum = 0;
  for (int w = 0; w < nw; ++w) {
    const int c = warp_counts[w];
    base += w < warp ? c : 0;
    sum += c;
  }
  *total = sum;
  return flag ? base + __popc(bal & ((1u << lane) - 1u)) : -1;
}

// Forward: a CTA per brick of 16 x 16 x VZ voxels (x fastest), one column of VZ
// voxels per thread. A Gaussian with finite values separates: its weight at a
// voxel is the product of one factor per axis, 2^(dx^2 k2) 2^(dy^2 k2) 2^(dz^2 k2),
// so the CTA evaluates 32 + VZ factors per surviving Gaussian into shared
// memory instead of one ex2 and one squared distance per voxel; a voxel then
// costs a multiply, an add and a multiply-add per attribute, in pairs with
// paired FP32 instructions. Products below 2^-126 flush to zero, as the single
// ex2 did, so the cull leaves the sums bit for bit the same. Each factor is
// corrected for the rounding of its argument, which the one ex2 carried whole:
// against FP64, 4,096 Gaussians into 128^3 voxels, rel-L2 3.70e-7 (3.79e-7 with one
// ex2 per voxel). Gaussians
// with a non-finite value or exponent factor are evaluated voxel by voxel.
// Gaussians come in tiles of 256, one per thread, each culled against the
// brick's box; the survivors are added in their original order (the non-finite
// ones of a tile after the others). What bounds it: instruction issue, about
// 2.5 instructions per (Gaussian, voxel). 1.16 -> 0.39 ms at that size.
constexpr int kBX = 16, kBY = 16;

// 2^(d^2 k) of one axis within about an ulp, zero below the normal range. The
// rounded exponent t splits into an integer (added to the result's exponent
// bits) and a fraction, to which the rounding errors of d^2 and of the product
// are added; 2^fraction is its Taylor series to degree 7, (ln 2)^n / n! (next
// term below 2^-27 on [-1/2, 1/2]). (With ex2.approx for the three factors the
// volume was 5% further from FP64 than with one ex2 of the whole exponent.)
__device__ __forceinline__ float axis_factor(float d, Exponent k) {
  const float p = __fmul_rn(d, d), t = __fmul_rn(p, k.hi);
  const float e = __fmaf_rn(p, k.lo, __fmaf_rn(__fmaf_rn(d, d, -p), k.hi, __fmaf_rn(p, k.hi, -t)));
  const float x = t + 12582912.f;  // 1.5 2^23: the low mantissa bits hold rint(t)
  const float f = (t - (x - 12582912.f)) + e;
  float y = 1.5252734e-5f;
  y = fmaf(y, f, 1.5403530e-4f);
  y = fmaf(y, f, 1.3333558e-3f);
  y = fmaf(y, f, 9.6181291e-3f);
  y = fmaf(y, f, 5.5504109e-2f);
  y = fmaf(y, f, 2.4022651e-1f);
  y = fmaf(y, f, 6.9314718e-1f);
  y = fmaf(y, f, 1.f);
  y = __int_as_float(__float_as_int(y) + (__float_as_int(x) << 23));
  return t < -126.f ? 0.f : (t <= 0.f ? y : t);  // (NaN: NaN)
}

// a b in each half, results below the normal range flushed to zero.
__device__ __forceinline__ unsigned long long f2mul_ftz(unsigned long long a,
                                                        unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float mul_ftz(float a, float b) {
  float d;
  asm("mul.rn.ftz.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}

// kA attributes at most.
template <int kA, int VZ>
__global__ void __launch_bounds__(256) forward_kernel(Grid g, int b, Rbf r, int N, int C, int cull,
                                                      float* __restrict__ vol) {
  using u64 = unsigned long long;
  constexpr int kFac = kBX + kBY + VZ;  // factors of one Gaussian: x | y | z
  constexpr int kHalf = 128;            // Gaussians whose factors are held at once
  __shared__ float tile[kTile][5];  // x y z, exponent (hi, lo)
  __shared__ __align__(16) u64 rows[kTile][kA];  // attributes, each twice
  __shared__ __align__(16) float fac[kHalf][kFac];
  __shared__ float axis[kFac];  // the brick's voxel coordinates
  __shared__ int counts[8];
  const int A = C - 4;
  const int64_t nv = (int64_t)g.D * g.H * g.W;
  const int tid = threadIdx.x;
  const int bx = blockIdx.x * kBX, by = blockIdx.y * kBY, bz = blockIdx.z * VZ;
  const int lx = tid & (kBX - 1), ly = tid / kBX;
  if (tid < kBX) axis[tid] = coord(g.sx, g.ex, g.W, bx + tid);
  else if (tid < kBX + kBY) axis[tid] = coord(g.sy, g.ey, g.H, by + tid - kBX);
  else if (tid < kFac) axis[tid] = coord(g.sz, g.ez, g.D, bz + tid - kBX - kBY);
  float lo[3], hi[3];
  axis_box(g.sx, g.ex, g.W, bx, min(bx + kBX, g.W) - 1, lo[0], hi[0]);
  axis_box(g.sy, g.ey, g.H, by, min(by + kBY, g.H) - 1, lo[1], hi[1]);
  axis_box(g.sz, g.ez, g.D, bz, min(bz + VZ, g.D) - 1, lo[2], hi[2]);
  u64 sum[VZ / 2], attr[VZ / 2][kA];
#pragma unroll
  for (int v = 0; v < VZ / 2; ++v) {
    sum[v] = 0ull;
#pragma unroll
    for (int a = 0; a < kA; ++a) attr[v][a] = 0ull;
  }
  for (int i0 = 0; i0 < N; i0 += kTile) {
    __syncthreads();  // the previous tile has been read
    float val[5 + kA];
    bool keep = false, finite = true;
    if (i0 + tid < N) {
#pragma unroll
      for (int c = 0; c < 4 + kA; ++c) {
        const float v = c < C ? r.at(b, i0 + tid, c) : 0.f;
        finite = finite && isfinite(v);
        val[c < 4 ? c : c + 1] = v;
      }
      const Exponent k = exponent(val[3]);
      val[3] = k.hi;
      val[4] = k.lo;
      finite = finite && isfinite(val[3]);
      keep = !cull || !finite ||
             !(box_dist2(val[0], val[1], val[2], lo, hi) * -val[3] > kCullArg);
    }
    int cnt, special = 0;
    int at = block_slot(keep && finite, counts, &cnt);
    if (__syncthreads_or(keep && !finite)) {  // the non-finite ones follow the others
      const int sat = block_slot(keep && !finite, counts, &special);
      if (keep && !finite) at = cnt + sat;
    }
    if (keep) {
#pragma unroll
      for (int c = 0; c < 5; ++c) tile[at][c] = val[c];
#pragma unroll
      for (int a = 0; a < kA; ++a) rows[at][a] = f2pack(val[5 + a], val[5 + a]);
    }
    __syncthreads();
    for (int h0 = 0; h0 < cnt; h0 += kHalf) {
      const int hn = min(kHalf, cnt - h0);
      if (h0 > 0) __syncthreads();  // the previous factors have been read
      for (int j = tid; j < hn * kFac; j += 256) {
        const int i = j / kFac, f = j - i * kFac;
        const float* t = tile[h0 + i];
        fac[i][f] = axis_factor(t[f < kBX ? 0 : (f < kBX + kBY ? 1 : 2)] - axis[f],
                                Exponent{t[3], t[4]});
      }
      __syncthreads();
#pragma unroll 4
      for (int i = 0; i < hn; ++i) {
        const float exy = mul_ftz(fac[i][lx], fac[i][kBX + ly]);
        const u64 e2 = f2pack(exy, exy);
        const float4* ez = reinterpret_cast<const float4*>(&fac[i][kBX + kBY]);
        u64 ra[kA];
        if constexpr (kA == 1) {
          ra[0] = rows[h0 + i][0];
        } else {
#pragma unroll
          for (int a = 0; a < kA; a += 2) {
            const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(&rows[h0 + i][a]);
            ra[a] = q.x;
            ra[a + 1] = q.y;
          }
        }
#pragma unroll
        for (int q = 0; q < VZ / 4; ++q) {
          const float4 z = ez[q];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const u64 w = f2mul_ftz(e2, h ? f2pack(z.z, z.w) : f2pack(z.x, z.y));
            sum[2 * q + h] = f2add(sum[2 * q + h], w);
#pragma unroll
            for (int a = 0; a < kA; ++a)
              attr[2 * q + h][a] = f2fma(w, ra[a], attr[2 * q + h][a]);
          }
        }
      }
    }
    for (int i = cnt; i < cnt + special; ++i) {
      const float dx = tile[i][0] - axis[lx], dy = tile[i][1] - axis[kBX + ly];
#pragma unroll
      for (int v = 0; v < VZ; v += 2) {
        float w[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float dz = tile[i][2] - axis[kBX + kBY + v + h];
          w[h] = exp2_approx(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) * tile[i][3]);
        }
        const u64 w2 = f2pack(w[0], w[1]);
        sum[v / 2] = f2add(sum[v / 2], w2);
#pragma unroll
        for (int a = 0; a < kA; ++a)
          if (a < A)
            attr[v / 2][a] = f2fma(w2, rows[i][a], attr[v / 2][a]);
      }
    }
  }
  const int xi = bx + lx, yi = by + ly;
  if (xi >= g.W || yi >= g.H) return;
  float* out = vol + (size_t)b * (1 + A) * nv;
#pragma unroll
  for (int v = 0; v < VZ; ++v) {
    if (bz + v >= g.D) break;
    const int64_t o = ((int64_t)(bz + v) * g.H + yi) * g.W + xi;
    float p[2];
    f2unpack(sum[v / 2], p[0], p[1]);
    const float s = p[v & 1];
    out[o] = s;
    const float norm = s < 1e-8f ? 1.f : s;
#pragma unroll
    for (int a = 0; a < kA; ++a)
      if (a < A) {
        f2unpack(attr[v / 2][a], p[0], p[1]);
        out[(size_t)(1 + a) * nv + o] = p[v & 1] / norm;
      }
  }
}

// Gradient (rbf2volume_cuda.cu:124-201): a CTA per brick of 8 x 8 x 8 voxels.
// With dl = d loss / d vol[0] + sum_a d loss / d vol[1 + a] (r_a - vol[1 + a]) /
// vol[0] at a voxel (vol[0] < 1e-8 counting as 1) and w the Gaussian's weight,
//   d/d centre = sum w dl (voxel - centre) / sigma^2,
//   d/d sigma  = sum w dl |voxel - centre|^2 / sigma^3,
//   d/d r_a    = sum w d loss / d vol[1 + a] / vol[0].
// The brick's d loss / d vol[0], vol[1 + a] and d loss / d vol[1 + a] / vol[0] are
// staged in shared memory with z fastest. The Gaussians that survive the cull
// (as in the forward) are collected until there are 256, a lane takes one, and
// walks the brick's columns: the weight separates into per-axis factors, so a
// column is four dot products over z with the lane's factors 2^(dz^2 k2) times 1,
// dz and dz^2 (paired FP32, the voxels by broadcast reads), and the sums over y and
// then x fold in the other axes' factors. Nothing is reduced across lanes, and a
// Gaussian issues 4 + A atomics per brick. With fewer than 129 Gaussians left,
// several warps share a batch of 32, split the brick's x and add up before the atomics.
// What bounds it: instruction issue, about 5.5 instructions per (Gaussian, voxel) with
// one attribute. 4,096 Gaussians, 128^3 voxels: 3.15 -> 0.85 ms (1.05 with the voxel
// coordinates taken per Gaussian and row), against a warp per two Gaussians whose lanes
// took the voxels, one ex2 per pair and a shuffle reduction per Gaussian and brick.
constexpr int kGB = 8;  // brick side

// kA attributes at most.
template <int kA>
__global__ void __launch_bounds__(256, 2) grad_kernel(
    Grid g, int b, Rbf r, int N, int C, int cull, const float* __restrict__ vol,
    const float* __restrict__ vgrad, float* __restrict__ rgrad, int64_t gsb, int64_t gsn,
    int64_t gsc) {
  using u64 = unsigned long long;
  constexpr int kVox = kGB * kGB * kGB;
  // [1 + 2 A][column y + 8 x][z]: d loss / d vol[0] | vol[1 + a] | d loss / d vol[1 + a] / vol[0]
  extern __shared__ __align__(16) float sm[];
  __shared__ float yfac[8][kGB][32];  // [warp][y][lane]: the lane's Gaussian's y factor
  __shared__ float share[8][4 + kA][32];  // the warps' sums of a Gaussian
  __shared__ float axis[3 * kGB];  // the brick's voxel coordinates: x | y | z
  __shared__ int list[2 * kTile];
  __shared__ int counts[8];
  const int A = C - 4;
  const int64_t nv = (int64_t)g.D * g.H * g.W;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bx = blockIdx.x * kGB, by = blockIdx.y * kGB, bz = blockIdx.z * kGB;
  const float* vb = vol + (size_t)b * (1 + A) * nv;
  const float* gb = vgrad + (size_t)b * (1 + A) * nv;
  for (int j = tid; j < kVox; j += blockDim.x) {
    const int lx = j & 7, ly = (j >> 3) & 7, lz = j >> 6;
    const int xi = bx + lx, yi = by + ly, zi = bz + lz;
    const bool in = xi < g.W && yi < g.H && zi < g.D;
    const int64_t v = in ? ((int64_t)zi * g.H + yi) * g.W + xi : 0;
    float* e = sm + (lx * kGB + ly) * kGB + lz;
    e[0] = in ? gb[v] : 0.f;
    float v0 = in && A > 0 ? vb[v] : 1.f;
    if (v0 < 1e-8f) v0 = 1.f;
    const float inv = 1.f / v0;
    for (int a = 0; a < A; ++a) {
      e[(1 + a) * kVox] = in ? vb[(size_t)(1 + a) * nv + v] : 0.f;
      e[(1 + A + a) * kVox] = in ? gb[(size_t)(1 + a) * nv + v] * inv : 0.f;
    }
  }
  if (tid < kGB) axis[tid] = coord(g.sx, g.ex, g.W, bx + tid);
  else if (tid < 2 * kGB) axis[tid] = coord(g.sy, g.ey, g.H, by + tid - kGB);
  else if (tid < 3 * kGB) axis[tid] = coord(g.sz, g.ez, g.D, bz + tid - 2 * kGB);
  float lo[3], hi[3];
  axis_box(g.sx, g.ex, g.W, bx, min(bx + 7, g.W - 1), lo[0], hi[0]);
  axis_box(g.sy, g.ey, g.H, by, min(by + 7, g.H - 1), lo[1], hi[1]);
  axis_box(g.sz, g.ez, g.D, bz, min(bz + 7, g.D - 1), lo[2], hi[2]);
  // The Gaussians of list[0, cnt), cnt <= 256; all threads of the CTA.
  auto process = [&](int cnt) {
    const int batches = (cnt + 31) >> 5;
    const int parts = batches <= 1 ? 8 : (batches <= 2 ? 4 : (batches <= 4 ? 2 : 1));
    const int batch = warp / parts, part = warp % parts;
    const bool mine = batch * 32 + lane < cnt;  // (a batch past the last one has none)
    const int i = list[mine ? batch * 32 + lane : 0];
    const float xr = r.at(b, i, 0), yr = r.at(b, i, 1), zr = r.at(b, i, 2);
    const float sigma = r.at(b, i, 3);
    const float is2 = 1.f / (sigma * sigma);
    const Exponent k2 = exponent(sigma);
    u64 ra[kA];
#pragma unroll
    for (int a = 0; a < kA; ++a) {
      const float v = a < A ? r.at(b, i, 4 + a) : 0.f;
      ra[a] = f2pack(v, v);
    }
    // the z factors times 1, dz, dz^2 (voxels past the grid carry zeros)
    u64 z0[4], z1[4], z2[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float f[2], d[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        d[h] = axis[2 * kGB + 2 * q + h] - zr;
        f[h] = axis_factor(d[h], k2);
      }
      z0[q] = f2pack(f[0], f[1]);
      z1[q] = f2mul(z0[q], f2pack(d[0], d[1]));
      z2[q] = f2mul(z1[q], f2pack(d[0], d[1]));
    }
#pragma unroll
    for (int y = 0; y < kGB; ++y)
      yfac[warp][y][lane] = axis_factor(axis[kGB + y] - yr, k2);
    float gx = 0.f, gy = 0.f, gz = 0.f, gs = 0.f, ga[kA];
#pragma unroll
    for (int a = 0; a < kA; ++a) ga[a] = 0.f;
    __syncwarp();
#pragma unroll 1
    for (int x = part * (kGB / parts); x < (part + 1) * (kGB / parts); ++x) {
      if (bx + x >= g.W || batch >= batches) break;
      float u0 = 0.f, uy = 0.f, uz = 0.f, u2 = 0.f, ua[kA];
#pragma unroll
      for (int a = 0; a < kA; ++a) ua[a] = 0.f;
#pragma unroll 2
      for (int y = 0; y < kGB; ++y) {
        const float4* e = reinterpret_cast<const float4*>(sm + (x * kGB + y) * kGB);
        u64 m0 = 0ull, m1 = 0ull, m2 = 0ull, mq[kA];
#pragma unroll
        for (int a = 0; a < kA; ++a) mq[a] = 0ull;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float4 d4 = e[q];
          u64 dl[2] = {f2pack(d4.x, d4.y), f2pack(d4.z, d4.w)};
#pragma unroll
          for (int a = 0; a < kA; ++a) {
            if (a >= A) break;
            const float4 v4 = e[(1 + a) * (kVox / 4) + q], q4 = e[(1 + A + a) * (kVox / 4) + q];
            const u64 va[2] = {f2pack(v4.x, v4.y), f2pack(v4.z, v4.w)};
            const u64 qa[2] = {f2pack(q4.x, q4.y), f2pack(q4.z, q4.w)};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              dl[h] = f2fma(f2sub(ra[a], va[h]), qa[h], dl[h]);
              mq[a] = f2fma(z0[2 * q + h], qa[h], mq[a]);
            }
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            m0 = f2fma(z0[2 * q + h], dl[h], m0);
            m1 = f2fma(z1[2 * q + h], dl[h], m1);
            m2 = f2fma(z2[2 * q + h], dl[h], m2);
          }
        }
        float ha, hb;
        const float dy = axis[kGB + y] - yr;
        const float fy = yfac[warp][y][lane];
        f2unpack(m0, ha, hb);
        const float s0 = fy * (ha + hb);
        u0 += s0;
        uy = fmaf(dy, s0, uy);
        u2 = fmaf(dy * dy, s0, u2);
        f2unpack(m1, ha, hb);
        uz = fmaf(fy, ha + hb, uz);
        f2unpack(m2, ha, hb);
        u2 = fmaf(fy, ha + hb, u2);
#pragma unroll
        for (int a = 0; a < kA; ++a) {
          f2unpack(mq[a], ha, hb);
          ua[a] = fmaf(fy, ha + hb, ua[a]);
        }
      }
      const float dx = axis[x] - xr;
      const float fx = axis_factor(dx, k2);
      const float fd = fx * dx;
      gx = fmaf(fd, u0, gx);
      gs = fmaf(fd * dx, u0, gs);
      gy = fmaf(fx, uy, gy);
      gz = fmaf(fx, uz, gz);
      gs = fmaf(fx, u2, gs);
#pragma unroll
      for (int a = 0; a < kA; ++a) ga[a] = fmaf(fx, ua[a], ga[a]);
    }
    if (parts > 1) {
      // the warps of a batch add up in shared memory: one atomic per brick and sum (all
      // bricks meet in the same few words: 64 Gaussians into 160^3 voxels took 1.53 ms
      // with an atomic per warp)
      share[warp][0][lane] = gx;
      share[warp][1][lane] = gy;
      share[warp][2][lane] = gz;
      share[warp][3][lane] = gs;
#pragma unroll
      for (int a = 0; a < kA; ++a) share[warp][4 + a][lane] = ga[a];
      __syncthreads();
      if (part == 0)
        for (int w = warp + 1; w < warp + parts; ++w) {
          gx += share[w][0][lane];
          gy += share[w][1][lane];
          gz += share[w][2][lane];
          gs += share[w][3][lane];
#pragma unroll
          for (int a = 0; a < kA; ++a) ga[a] += share[w][4 + a][lane];
        }
    }
    if (!mine || part > 0) return;
    float* out = rgrad + b * gsb + i * gsn;
    atomicAdd(out, is2 * gx);
    atomicAdd(out + gsc, is2 * gy);
    atomicAdd(out + 2 * gsc, is2 * gz);
    atomicAdd(out + 3 * gsc, is2 / sigma * gs);
#pragma unroll
    for (int a = 0; a < kA; ++a)
      if (a < A) atomicAdd(out + (4 + a) * gsc, ga[a]);
  };
  // A Gaussian with a non-finite value or exponent factor: the whole CTA over
  // the voxels, one weight per voxel.
  auto process_special = [&](int i) {
    const float xr = r.at(b, i, 0), yr = r.at(b, i, 1), zr = r.at(b, i, 2);
    const float sigma = r.at(b, i, 3);
    const float is2 = 1.f / (sigma * sigma), k2 = -0.5f * kLog2e * is2, is3 = is2 / sigma;
    float s[4 + kA];
#pragma unroll
    for (int c = 0; c < 4 + kA; ++c) s[c] = 0.f;
    for (int j = tid; j < kVox; j += blockDim.x) {
      const int lz = j & 7, ly = (j >> 3) & 7, lx = j >> 6;
      if (bx + lx >= g.W || by + ly >= g.H || bz + lz >= g.D) continue;
      const float ex = coord(g.sx, g.ex, g.W, bx + lx) - xr;
      const float ey = coord(g.sy, g.ey, g.H, by + ly) - yr;
      const float ez = coord(g.sz, g.ez, g.D, bz + lz) - zr;
      const float d2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
      const float w = exp2_approx(d2 * k2), wi = is2 * w;
      float dl = sm[j];
#pragma unroll
      for (int a = 0; a < kA; ++a)
        if (a < A) {
          const float q = sm[(1 + A + a) * kVox + j];
          dl = fmaf(r.at(b, i, 4 + a) - sm[(1 + a) * kVox + j], q, dl);
          s[4 + a] = fmaf(w, q, s[4 + a]);
        }
      s[0] += ex * wi * dl;
      s[1] += ey * wi * dl;
      s[2] += ez * wi * dl;
      s[3] += d2 * is3 * w * dl;
    }
#pragma unroll
    for (int c = 0; c < 4 + kA; ++c) {
      const float t = warp_sum_f(s[c]);
      if (lane == 0 && c < 4 + A) atomicAdd(rgrad + b * gsb + i * gsn + c * gsc, t);
    }
  };
  int have = 0;  // Gaussians in the list
  for (int i0 = 0; i0 < N; i0 += kTile) {
    bool keep = false, finite = true;
    if (i0 + tid < N) {
      const float cx = r.at(b, i0 + tid, 0), cy = r.at(b, i0 + tid, 1);
      const float cz = r.at(b, i0 + tid, 2), sg = r.at(b, i0 + tid, 3);
      const float k2 = -0.5f * kLog2e * (1.f / (sg * sg));
      finite = isfinite(cx) && isfinite(cy) && isfinite(cz) && isfinite(k2);
      keep = !cull || !finite || !(box_dist2(cx, cy, cz, lo, hi) * -k2 > kCullArg);
      for (int a = 0; a < A; ++a) finite = finite && isfinite(r.at(b, i0 + tid, 4 + a));
    }
    __syncthreads();  // the staged voxels are written; the counts have been read
    int cnt;
    const int at = block_slot(keep && finite, counts, &cnt);
    if (keep && finite) list[have + at] = i0 + tid;
    have += cnt;
    if (__syncthreads_or(keep && !finite)) {  // (also: the list is written)
      int n;
      const int sat = block_slot(keep && !finite, counts, &n);
      if (keep && !finite) list[have + sat] = i0 + tid;
      __syncthreads();
      for (int q = 0; q < n; ++q) process_special(list[have + q]);
      __syncthreads();
    }
    if (have >= kTile) {
      process(kTile);
      __syncthreads();
      have -= kTile;
      const int moved = tid < have ? list[kTile + tid] : 0;
      __syncthreads();
      if (tid < have) list[tid] = moved;
      __syncthreads();
    }
  }
  if (have > 0) process(have);
}

}  // namespace rbf

namespace {

int check_rbf(const totri_array_t* r, const totri_array_t* vol, rbf::Grid& g, rbf::Rbf& rr,
              int64_t& B, int64_t& N, int& C, const float* start, const float* end) {
  TOTRI_TRY(check_array(r, "rbf", 3, -1));
  if (r->dtype != TOTRI_FLOAT32)
    return fail(TOTRI_ERR_UNSUPPORTED, "rbf2volume: only float32 tensors are supported");
  B = r->shape[0];
  N = r->shape[1];
  C = (int)r->shape[2];
  if (C < 4 || C > 4 + rbf::kMaxAttr)
    return fail(TOTRI_ERR_INVALID_ARGUMENT, "rbf must be [B, N, 4+A] with A <= 8");
  TOTRI_TRY(check_array(vol, "volume", 5, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(vol, "volume", 0, B));
  TOTRI_TRY(check_dim(vol, "volume", 1, C - 3));
  TOTRI_TRY(check_contiguous(vol, "volume"));
  g = rbf::Grid{(int)vol->shape[2], (int)vol->shape[3], (int)vol->shape[4], start[0], start[1],
                start[2], end[0], end[1], end[2]};
  rr = rbf::Rbf{static_cast<const float*>(r->data), r->strides[0], r->strides[1], r->strides[2]};
  return TOTRI_OK;
}

}  // namespace
}  // namespace totri

using namespace totri;

extern "C" {

int totri_rbf2volume_gaussian_forward(const totri_array_t* r, const totri_array_t* vol,
                                      const float start[3], const float end[3], void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  rbf::Grid g;
  rbf::Rbf rr;
  int64_t B, N;
  int C;
  TOTRI_TRY(check_rbf(r, vol, g, rr, B, N, C, start, end));
  const int64_t nv = (int64_t)g.D * g.H * g.W;
  if (nv == 0 || B == 0) return TOTRI_OK;
  const int cull = tune::get("rbf.cull") != 1;
  // columns of 8 voxels, of 4 with several attributes (their accumulators are
  // registers)
  float* vp = static_cast<float*>(vol->data);
  const int vz = C <= 5 ? 8 : 4;
  const dim3 grid((unsigned)ceil_div(g.W, rbf::kBX), (unsigned)ceil_div(g.H, rbf::kBY),
                  (unsigned)ceil_div(g.D, vz));
  for (int b = 0; b < (int)B; ++b) {
    if (C <= 5)
      TOTRI_KERNEL("rbf2volume forward", stream,
                   rbf::forward_kernel<1, 8><<<grid, 256, 0, stream>>>(g, b, rr, (int)N, C, cull,
                                                                       vp));
    else if (C <= 8)
      TOTRI_KERNEL("rbf2volume forward", stream,
                   rbf::forward_kernel<4, 4><<<grid, 256, 0, stream>>>(g, b, rr, (int)N, C, cull,
                                                                       vp));
    else
      TOTRI_KERNEL("rbf2volume forward", stream,
                   rbf::forward_kernel<rbf::kMaxAttr, 4><<<grid, 256, 0, stream>>>(
                       g, b, rr, (int)N, C, cull, vp));
  }
  return TOTRI_OK;
}

int totri_rbf2volume_gaussian_grad(const totri_array_t* r, const totri_array_t* vol,
                                   const totri_array_t* vgrad, const totri_array_t* rgrad,
                                   const float start[3], const float end[3], void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  rbf::Grid g;
  rbf::Rbf rr;
  int64_t B, N;
  int C;
  TOTRI_TRY(check_rbf(r, vol, g, rr, B, N, C, start, end));
  TOTRI_TRY(check_array(vgrad, "volume_grad", 5, TOTRI_FLOAT32));
  for (int d = 0; d < 5; ++d)
    if (vgrad->shape[d] != vol->shape[d])
      return fail(TOTRI_ERR_INVALID_ARGUMENT, "volume_grad must have the shape of volume");
  TOTRI_TRY(check_contiguous(vgrad, "volume_grad"));
  TOTRI_TRY(check_array(rgrad, "rbf_grad", 3, TOTRI_FLOAT32));
  for (int d = 0; d < 3; ++d)
    if (rgrad->shape[d] != r->shape[d])
      return fail(TOTRI_ERR_INVALID_ARGUMENT, "rbf_grad must have the shape of rbf");
  const int64_t nv = (int64_t)g.D * g.H * g.W;
  if (nv == 0 || N == 0 || B == 0) return TOTRI_OK;
  const int A = C - 4;
  const size_t smem = sizeof(float) * 512 * (1 + 2 * A);
  const int cull = tune::get("rbf.cull") != 1;
  const dim3 grid((unsigned)ceil_div(g.W, rbf::kGB), (unsigned)ceil_div(g.H, rbf::kGB),
                  (unsigned)ceil_div(g.D, rbf::kGB));
  const auto kernel = A <= 1   ? rbf::grad_kernel<1>
                      : A <= 4 ? rbf::grad_kernel<4>
                               : rbf::grad_kernel<rbf::kMaxAttr>;
  TOTRI_CUDA(tune::ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem));
  for (int b = 0; b < (int)B; ++b)
    TOTRI_KERNEL("rbf2volume grad", stream,
                 kernel<<<grid, 256, smem, stream>>>(
                     g, b, rr, (int)N, C, cull, static_cast<const float*>(vol->data),
                     static_cast<const float*>(vgrad->data), static_cast<float*>(rgrad->data),
                     rgrad->strides[0], rgrad->strides[1], rgrad->strides[2]));
  return TOTRI_OK;
}

}  // extern "C"
