// Exhaustive (separate laser and detector points) volume renderer and its
// adjoint with respect to the volume.
//
// Reference: src/render/volume_cuda.cu:298-377 (forward, one thread per
// (voxel column, scan point, laser point) with global atomics) and :415-466
// (gradient: an empty kernel). Here the forward gives each CTA one scan point
// and a tile of laser points, walks the occupied voxels and splats each
// voxel's path-length interval into a shared [T][tile] histogram that is
// flushed with row stores; the adjoint (the forward is linear in the volume)
// gathers per voxel. A voxel's path length is the sum of a scan and a laser
// distance, so each distance is taken once and serves a whole tile of pairs.
#include <algorithm>
#include <cmath>
#include <string>

#include "capi_common.cuh"
#include "mesh_kernels.cuh"
#include "tune.cuh"

namespace totri {
namespace vexh {

struct Geo {
  int D, H, W, S, L, T;
  float sx, sy, sz, ex, ey, ez, bw, bo;
  float inv_bw;  // 1 / bw for div_fixed; NaN where it does not apply (every pair is exact)
};

struct Pts {  // [B, 3, n] with strides
  const float* p;
  int64_t sb, sc, sn;
  __device__ fv3 at(int b, int i) const {
    const float* q = p + b * sb + i * sn;
    return mkv(q[0], q[sc], q[2 * sc]);
  }
};

struct Interval {
  bool ok;
  int first, last;
  float bf0, bf1, range;
};

// The two ends of a voxel's z extent (volume_cuda.cu:314-330), each value with
// one rounding per operation.
struct Ends {
  fv3 p0, p1;
};
__device__ __forceinline__ Ends voxel_ends(const Geo& g, int xi, int yi, int zi) {
  const float xf = xadd(g.sx, xmul(xdiv(xadd((float)xi, 0.5f), (float)g.W), xsub(g.ex, g.sx)));
  const float yf = xadd(g.sy, xmul(xdiv(xadd((float)yi, 0.5f), (float)g.H), xsub(g.ey, g.sy)));
  const float zf = xadd(g.sz, xmul(xdiv(xadd((float)zi, 0.5f), (float)g.D), xsub(g.ez, g.sz)));
  const float half = xmul(xdiv(0.5f, (float)g.D), xsub(g.ez, g.sz));
  return Ends{mkv(xf, yf, xsub(zf, half)), mkv(xf, yf, xadd(zf, half))};
}

// Path-length interval of a voxel for a pair whose path lengths to its two
// ends are d0 and d1, binned (volume_cuda.cu:331-364); FP32 decisions as in the
// oracle. The quotients come from div_fixed and the floors from an addition
// of 1.5 2^23 rounded down while both bin coordinates lie within 2^21, from
// the correctly rounded division and floorf otherwise (NaN and infinities too):
// the same values either way.
template <bool kForward>
__device__ __forceinline__ Interval interval(const Geo& g, float d0, float d1) {
  Interval r{false, 0, 0, 0.f, 0.f, 0.f};
  if (d1 < d0) {
    const float t = d0;
    d0 = d1;
    d1 = t;
  }
  float bf0 = div_fixed(xsub(d0, g.bo), g.bw, g.inv_bw);
  float bf1 = div_fixed(xsub(d1, g.bo), g.bw, g.inv_bw);
  int first, last;
  if (bf0 > -2097152.f && bf1 < 2097152.f) {
    first = __float_as_int(__fadd_rd(bf0, 12582912.f)) - 0x4B400000;
    last = __float_as_int(__fadd_rd(bf1, 12582912.f)) - 0x4B400000;
  } else {
    bf0 = xdiv(xsub(d0, g.bo), g.bw);
    bf1 = xdiv(xsub(d1, g.bo), g.bw);
    first = (int)floorf(bf0);
    last = (int)floorf(bf1);
  }
  const float range = xsub(bf1, bf0);
  // With a negative bin width the first bin is the later one: neither test implies that
  // the other bin is inside. (Both at once took the forward 162 us and the tests apart
  // 169 at 32^3 voxels x 1,024 x 4 points, the gradient 2.77 and 2.61 ms at 8^3 x 64 x 64.)
  if (kForward && (last < 0 || first >= g.T)) return r;
  if (first < 0) {
    if (!kForward && last < 0) return r;
    bf0 = 0.f;
    first = 0;
  }
  if (last >= g.T) {
    if (!kForward && first >= g.T) return r;
    bf1 = (float)(g.T - 1);
    last = g.T - 1;
  }
  if (!kForward && g.bw < 0.f && (last < 0 || first >= g.T)) return r;
  r.ok = true;
  r.first = first;
  r.last = last;
  r.bf0 = bf0;
  r.bf1 = bf1;
  r.range = range;
  return r;
}

__global__ void compact_kernel(const float* __restrict__ vol, int64_t n, uint32_t* list,
                               uint32_t* count) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool occ = i < n && vol[i] != 0.f;
  const uint32_t m = __ballot_sync(0xffffffffu, occ);
  if (!m) return;
  const int lane = threadIdx.x & 31;
  uint32_t base = 0;
  if (lane == __ffs(m) - 1) base = atomicAdd(count, (uint32_t)__popc(m));
  base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
  if (occ) list[base + __popc(m & ((1u << lane) - 1u))] = (uint32_t)i;
}

template <int LT>
__global__ void __launch_bounds__(256) forward_kernel(Geo g, int b, const float* __restrict__ vol,
                                                      const uint32_t* __restrict__ list,
                                                      const uint32_t* __restrict__ count, Pts sp,
                                                      Pts lp, float* __restrict__ out) {
  extern __shared__ float hist[];  // [T][LT]
  const int s = blockIdx.x;
  const int l0 = blockIdx.y * LT;
  for (int j = threadIdx.x; j < g.T * LT; j += blockDim.x) hist[j] = 0.f;
  __syncthreads();
  const uint32_t nnz = *count;
  // A thread takes one occupied voxel at a time to the lasers of the tile, in an order
  // that starts at its lane: the lanes of a warp add to different histogram columns.
  // Where the voxels are fewer than the threads, 2, 4 .. LT threads share a voxel's
  // lasers.
  __shared__ float laser[LT][3];
  if (threadIdx.x < LT && l0 + (int)threadIdx.x < g.L) {
    const fv3 q = lp.at(b, l0 + threadIdx.x);
    laser[threadIdx.x][0] = q.x;
    laser[threadIdx.x][1] = q.y;
    laser[threadIdx.x][2] = q.z;
  }
  __syncthreads();
  const fv3 sc = sp.at(b, s);
  const int nl = min(LT, g.L - l0);
  uint32_t share = 1;
  while (share < LT && 2 * share * nnz <= blockDim.x) share *= 2;
  for (uint32_t v = threadIdx.x / share; v < nnz; v += blockDim.x / share) {
    const uint32_t lin = __ldg(list + v);
    const int xi = (int)(lin % g.W), yi = (int)((lin / g.W) % g.H);
    const int zi = (int)(lin / ((uint32_t)g.W * g.H));
    const Ends e = voxel_ends(g, xi, yi, zi);
    const float occ = __ldg(vol + lin);
    const float s0 = xlen(xsub3(sc, e.p0)), s1 = xlen(xsub3(sc, e.p1));
#pragma unroll 1
    for (int i = 0; i < LT; i += share) {
      const int ll = (threadIdx.x + i) & (LT - 1);
      if (ll >= nl) continue;
      const fv3 lc = mkv(laser[ll][0], laser[ll][1], laser[ll][2]);
      const Interval iv = interval<true>(g, xadd(s0, xlen(xsub3(lc, e.p0))),
                                   xadd(s1, xlen(xsub3(lc, e.p1))));
      if (!iv.ok) continue;
      float* col = hist + ll;
      if (iv.first == iv.last) {
        atomicAdd(col + iv.first * LT, occ);
        continue;
      }
      const float fo = occ / iv.range;
      atomicAdd(col + iv.first * LT, (1.f - (iv.bf0 - (float)iv.first)) * fo);
      for (int t = iv.first + 1; t < iv.last; ++t) atomicAdd(col + t * LT, fo);
      atomicAdd(col + iv.last * LT, (iv.bf1 - (float)iv.last) * fo);
    }
  }
  __syncthreads();
  // out[b][t][s][l0 .. l0+LT)
  const size_t base = ((size_t)b * g.T * g.S + s) * g.L + l0;
  for (int j = threadIdx.x; j < g.T * LT; j += blockDim.x) {
    const int t = j / LT, c = j - t * LT;
    if (l0 + c < g.L) out[base + (size_t)t * g.S * g.L + c] = hist[j];
  }
}

// x held within the finite range, sign kept; a NaN gives a finite value.
__device__ __forceinline__ float clamp_finite(float x) {
  float r;
  asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(3.4028235e38f));
  return r;
}

// d loss / d volume: per voxel, the forward weights against transient_grad. A
// CTA takes a block of 8 x 8 x 4 voxels, one per thread, and the scan points of
// its slice; a thread holds the distances of its voxel's ends to kLC lasers in
// registers and walks the scan points, so a pair costs two additions, the
// division by the bin width and its bins. transient_grad element (t, s, l) is
// tg[((s - s_base) L + l) cstep + t bstep]: in bins-last order (bstep 1) the bins that
// the block can reach in a pair are one run of memory, which a warp copies to
// shared memory (cp.async, the next scan point's while this one's are used). A window past kRows bins, or without
// sound bounds, is read in place. 56 x 40 x 48 voxels x 256 scan points x 36
// lasers, 1,024 bins: 21.8 ms (four square roots and eight divisions per pair,
// every bin another sector of the in-place order) -> 3.68 ms,
// at 91% of issue slots: about 50 instructions per pair and 5 per bin.
constexpr int kLC = 8, kRows = 256;

// A pair's weighted bins, read in place.
__device__ __noinline__ float pair_direct(Geo g, float d0, float d1, const float* __restrict__ col,
                                          int64_t bstep) {
  const Interval iv = interval<false>(g, d0, d1);
  if (!iv.ok) return 0.f;
  if (iv.first == iv.last) return __ldg(col + iv.first * bstep);
  float sum = (1.f - (iv.bf0 - (float)iv.first)) * __ldg(col + iv.first * bstep);
  for (int t = iv.first + 1; t < iv.last; ++t) sum += __ldg(col + t * bstep);
  sum += (iv.bf1 - (float)iv.last) * __ldg(col + iv.last * bstep);
  return sum / iv.range;
}

// window_far: the farthest path whose bins have sound bounds. With u = 2^-24 the exact
// chain's lengths and the bounds' each lie within 8 u far of the true ones, and the
// offset adds u |bo| to either difference: a window's extra bin each side holds them
// while 16 u (far + |bo|) is below half a bin width. (At a bin width of 2e-8, a path of
// 2.26 less an offset of 2.26 missed one bin in 2,000 by more.)
__global__ void __launch_bounds__(256, 4) adjoint_kernel(Geo g, int b, Pts sp, Pts lp, int s_base,
                                                         int s_end, int per_slice,
                                                         const float* __restrict__ tg,
                                                         int64_t cstep, int64_t bstep,
                                                         float* __restrict__ vg, int add,
                                                         float window_far) {
  using u64 = unsigned long long;
  __shared__ float win[2][kLC][kRows];
  __shared__ float2 laser[kLC][256];  // distances of the thread's voxel ends to the lasers
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;  // warp w stages laser l0 + w
  const int nbx = (g.W + 7) >> 3, nby = (g.H + 7) >> 3;
  const int x0 = (blockIdx.x % nbx) * 8, y0 = (blockIdx.x / nbx) % nby * 8;
  const int z0 = blockIdx.x / (nbx * nby) * 4;
  const int xi = x0 + (threadIdx.x & 7), yi = y0 + ((threadIdx.x >> 3) & 7);
  const int zi = z0 + (threadIdx.x >> 6);
  // threads past the volume's edge work on a clamped voxel and write nothing
  const Ends e = voxel_ends(g, min(xi, g.W - 1), min(yi, g.H - 1), min(zi, g.D - 1));
  float box[6];  // of the block: voxel positions are monotone in the index
  {
    const Ends a = voxel_ends(g, x0, y0, z0);
    const Ends c = voxel_ends(g, min(x0 + 8, g.W) - 1, min(y0 + 8, g.H) - 1,
                              min(z0 + 4, g.D) - 1);
    box[0] = fminf(a.p0.x, c.p0.x), box[3] = fmaxf(a.p0.x, c.p0.x);
    box[1] = fminf(a.p0.y, c.p0.y), box[4] = fmaxf(a.p0.y, c.p0.y);
    box[2] = fminf(fminf(a.p0.z, a.p1.z), fminf(c.p0.z, c.p1.z));
    box[5] = fmaxf(fmaxf(a.p0.z, a.p1.z), fmaxf(c.p0.z, c.p1.z));
  }
  // nearest and farthest distance from q to the box (NaN for a NaN point)
  auto reach = [&](fv3 q, float& near, float& far) {
    const float ex = fmaxf(fmaxf(box[0] - q.x, q.x - box[3]), 0.f);
    const float ey = fmaxf(fmaxf(box[1] - q.y, q.y - box[4]), 0.f);
    const float ez = fmaxf(fmaxf(box[2] - q.z, q.z - box[5]), 0.f);
    const float fx = fmaxf(fabsf(q.x - box[0]), fabsf(q.x - box[3]));
    const float fy = fmaxf(fabsf(q.y - box[1]), fabsf(q.y - box[4]));
    const float fz = fmaxf(fabsf(q.z - box[2]), fabsf(q.z - box[5]));
    near = sqrtf(ex * ex + ey * ey + ez * ez);
    far = sqrtf(fx * fx + fy * fy + fz * fz);
  };
  const int s0 = s_base + blockIdx.y * per_slice, s1 = min(s_end, s0 + per_slice);
  const u64 nbo = f2pack(-g.bo, -g.bo), nbw = f2pack(-g.bw, -g.bw);
  const u64 inv = f2pack(g.inv_bw, g.inv_bw), big = f2pack(12582912.f, 12582912.f);
  const float bins = (float)min(g.T, 2097152);
  float acc = 0.f;
  for (int l0 = 0; l0 < g.L; l0 += kLC) {
    const int nl = min(kLC, g.L - l0);
#pragma unroll 1
    for (int k = 0; k < nl; ++k) {
      const fv3 lc = lp.at(b, l0 + k);
      laser[k][threadIdx.x] = make_float2(xlen(xsub3(lc, e.p0)), xlen(xsub3(lc, e.p1)));
    }
    float lnear, lfar;  // lane k: laser l0 + k
    reach(lp.at(b, min(l0 + (lane & (kLC - 1)), g.L - 1)), lnear, lfar);
    float snear = 0.f, sfar = 0.f;  // lane j: scan point s0 + 32 i + j
    // Stages the windows of scan point s; lane k receives laser l0 + k's first
    // bin and bins (none: read in place).
    auto stage = [&](int s, int buf) {
      if (((s - s0) & 31) == 0) reach(sp.at(b, min(s + lane, s_end - 1)), snear, sfar);
      const float near = __shfl_sync(0xffffffffu, snear, (s - s0) & 31) + lnear;
      const float far = __shfl_sync(0xffffffffu, sfar, (s - s0) & 31) + lfar;
      const float c0 = (near - g.bo) / g.bw, c1 = (far - g.bo) / g.bw;
      int2 w = make_int2(0, 0);
      if (far < window_far && c0 > -262144.f && c1 < 262144.f) {  // (NaN: no window)
        w.x = max((int)floorf(c0) - 1, 0);
        w.y = min((int)floorf(c1) + 1, g.T - 1) - w.x + 1;
        if (w.y > kRows || w.y < 0) w.y = 0;
      }
      const int first = __shfl_sync(0xffffffffu, w.x, warp);
      const int rows = __shfl_sync(0xffffffffu, w.y, warp);
      if (l0 + warp < g.L) {
        const float* src =
            tg + ((int64_t)(s - s_base) * g.L + l0 + warp) * cstep + (first + lane) * bstep;
        uint32_t dst = (uint32_t)__cvta_generic_to_shared(&win[buf][warp][lane]);
        for (int r = lane; r < rows; r += 32, dst += 128, src += 32 * bstep)
          cp_async4(dst, src, 4);
      }
      return w;
    };
    __syncthreads();  // the previous lasers' windows are consumed
    int2 next = stage(s0, 0);
    for (int s = s0; s < s1; ++s) {
      const int2 w = next;
      const int buf = (s - s0) & 1;
      cp_async_wait_all();
      __syncthreads();  // this point's windows are there, the other buffer's are consumed
      if (s + 1 < s1) next = stage(s + 1, buf ^ 1);
      const fv3 sc = sp.at(b, s);
      const u64 d = f2pack(xlen(xsub3(sc, e.p0)), xlen(xsub3(sc, e.p1)));
      float part = 0.f;
#pragma unroll 1
      for (int k = 0; k < nl; ++k) {
        // interval() for bins inside [0, T): the ends' quotients in pairs
        const float2 e2 = laser[k][threadIdx.x];
        float da, db;
        f2unpack(f2add(d, f2pack(e2.x, e2.y)), da, db);
        const u64 a = f2add(f2pack(min_nan(da, db), max_nan(da, db)), nbo);
        u64 q = f2mul(a, inv);
        q = f2fma(f2fma(q, nbw, a), inv, q);
        q = f2fma(f2fma(q, nbw, a), inv, q);
        const u64 x = f2add_rm(q, big);
        float q0, q1, x0, x1, f0, f1;
        f2unpack(q, q0, q1);
        f2unpack(x, x0, x1);
        f2unpack(f2sub(q, f2sub(x, big)), f0, f1);  // the ends' bin fractions
        const int lo = __shfl_sync(0xffffffffu, w.x, k);
        const int rows = __shfl_sync(0xffffffffu, w.y, k);
        if (rows > 0 && q0 >= 0.f && q1 < bins) {  // (NaN: no)
          const int n = __float_as_int(x1) - __float_as_int(x0);
          const uint32_t c = (uint32_t)__cvta_generic_to_shared(&win[buf][k][0]) +
                             4u * (__float_as_uint(x0) - 0x4B400000u - (uint32_t)lo);
          const float c0 = lds(c);
          float sum = (1.f - f0) * c0 + f1 * lds(c + 4u * n);
#pragma unroll 1
          for (int i = 1; i < n; i += 4) {
            const uint32_t ci = c + 4u * i;
            const float v0 = lds(ci), v1 = i + 1 < n ? lds(ci + 4u) : 0.f;
            const float v2 = i + 2 < n ? lds(ci + 8u) : 0.f, v3 = i + 3 < n ? lds(ci + 12u) : 0.f;
            sum += (v0 + v1) + (v2 + v3);
          }
          // sum / range: the hardware reciprocal and one remainder correction (a finite
          // one: an infinite quotient stays)
          const float range = q1 - q0, r = __fdividef(1.f, range), y = sum * r;
          part += n == 0 ? c0 : fmaf(clamp_finite(fmaf(-y, range, sum)), r, y);
        } else {
          part += pair_direct(g, da, db, tg + ((int64_t)(s - s_base) * g.L + l0 + k) * cstep,
                              bstep);
        }
      }
      acc += part;
    }
  }
  if (xi >= g.W || yi >= g.H || zi >= g.D) return;
  // (a slice's volume is its own)
  float* dst = vg + (((size_t)blockIdx.y * g.D + zi) * g.H + yi) * g.W + xi;
  *dst = add ? *dst + acc : acc;
}

}  // namespace vexh

namespace {

int check_pts(const totri_array_t* a, const char* name, int64_t B, int64_t& n, vexh::Pts& p) {
  TOTRI_TRY(check_array(a, name, 3, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(a, name, 0, B));
  TOTRI_TRY(check_dim(a, name, 1, 3));
  n = a->shape[2];
  p = vexh::Pts{static_cast<const float*>(a->data), a->strides[0], a->strides[1], a->strides[2]};
  return TOTRI_OK;
}

vexh::Geo make_geo(const totri_array_t* vol, int64_t S, int64_t L, int64_t T, const float* start,
                   const float* end, float bw, float bo) {
  vexh::Geo g{(int)vol->shape[1], (int)vol->shape[2], (int)vol->shape[3], (int)S, (int)L, (int)T,
              start[0], start[1], start[2], end[0], end[1], end[2], bw, bo, 1.f / bw};
  const float a = std::fabs(bw);
  if (!(a > 1e-18f && a < 1e18f)) g.inv_bw = NAN;  // div_fixed's range
  return g;
}

template <int LT>
int launch_fwd(const vexh::Geo& g, int b, const float* vol, const uint32_t* list,
               const uint32_t* count, const vexh::Pts& sp, const vexh::Pts& lp, float* out,
               cudaStream_t stream) {
  const size_t smem = sizeof(float) * (size_t)g.T * LT;
  TOTRI_CUDA(tune::ensure_dynamic_smem(
      reinterpret_cast<const void*>(vexh::forward_kernel<LT>), smem));
  const dim3 grid((unsigned)g.S, (unsigned)ceil_div(g.L, LT));
  TOTRI_KERNEL("volume exhaustive forward", stream,
               vexh::forward_kernel<LT><<<grid, 256, smem, stream>>>(g, b, vol, list, count, sp,
                                                                     lp, out));
  return TOTRI_OK;
}

}  // namespace
}  // namespace totri

using namespace totri;

extern "C" {

int totri_volume_exhaustive_forward(const totri_array_t* vol, const totri_array_t* scan_points,
                                    const totri_array_t* laser_points,
                                    const totri_array_t* scan_origin,
                                    const totri_array_t* laser_origin,
                                    const totri_array_t* transient, const float start[3],
                                    const float end[3], float bw, float bo, void* ws,
                                    size_t ws_bytes, void* stream_) {
  (void)scan_origin;  // unused by the reference kernel (volume_cuda.cu:312-313)
  (void)laser_origin;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  TOTRI_TRY(check_array(vol, "volume", 4, -1));
  if (vol->dtype != TOTRI_FLOAT32)
    return fail(TOTRI_ERR_UNSUPPORTED, "volume renderer: only float32 tensors are supported");
  TOTRI_TRY(check_contiguous(vol, "volume"));
  const int64_t B = vol->shape[0];
  int64_t S, L;
  vexh::Pts sp, lp;
  TOTRI_TRY(check_pts(scan_points, "scan_points", B, S, sp));
  TOTRI_TRY(check_pts(laser_points, "laser_points", B, L, lp));
  TOTRI_TRY(check_array(transient, "transient", 4, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(transient, "transient", 0, B));
  TOTRI_TRY(check_dim(transient, "transient", 2, S));
  TOTRI_TRY(check_dim(transient, "transient", 3, L));
  TOTRI_TRY(check_contiguous(transient, "transient"));
  const vexh::Geo g = make_geo(vol, S, L, transient->shape[1], start, end, bw, bo);
  if (numel(transient) == 0) return TOTRI_OK;
  const int64_t nv = (int64_t)g.D * g.H * g.W;
  const size_t need = align_up(sizeof(uint32_t) * (nv + 64), 256);
  if (!ws || ws_bytes < need)
    return fail(TOTRI_ERR_WORKSPACE, "workspace of " + std::to_string(need) + " bytes required");
  uint32_t* count = static_cast<uint32_t*>(ws);
  uint32_t* list = count + 64;
  for (int b = 0; b < (int)B; ++b) {
    const float* vb = static_cast<const float*>(vol->data) + (size_t)b * nv;
    TOTRI_CUDA(cudaMemsetAsync(count, 0, sizeof(uint32_t), stream));
    TOTRI_KERNEL("volume compact", stream,
                 vexh::compact_kernel<<<(unsigned)ceil_div(nv, 256), 256, 0, stream>>>(
                     vb, nv, list, count));
    float* out = static_cast<float*>(transient->data);
    const size_t budget = 200 * 1024;
    const int64_t fill = 2 * (int64_t)tune::sm_count();  // CTAs, two per SM
    const int want = tune::get("volume.exhaustive.lt");
    if (want == 1 || want == 8 || want == 32) {
      if ((size_t)g.T * want * 4 > budget)
        return fail(TOTRI_ERR_INVALID_ARGUMENT, "tuned laser tile too large for the bin count");
      if (want == 32) TOTRI_TRY(launch_fwd<32>(g, b, vb, list, count, sp, lp, out, stream));
      else if (want == 8) TOTRI_TRY(launch_fwd<8>(g, b, vb, list, count, sp, lp, out, stream));
      else TOTRI_TRY(launch_fwd<1>(g, b, vb, list, count, sp, lp, out, stream));
    } else if (want != 0) {
      return fail(TOTRI_ERR_INVALID_ARGUMENT, "laser tile must be 1, 8 or 32");
    } else if ((size_t)g.T * 32 * 4 <= 40 * 1024 && L >= 32 && S * ceil_div(L, 32) >= fill)
      // 32 lasers (a column per lane) where several CTAs fit an SM and there are CTAs
      // for two per SM: 4 x 64 x 64 voxels x 100 x 100 points, 300 bins, 0.35 ms (5% of the
      // voxels) and 4.7 ms (all), with 8 lasers 0.44 and 7.2; 32^3 x 64 x 64, 256 bins: 0.31
      // and 0.15 ms.
      TOTRI_TRY(launch_fwd<32>(g, b, vb, list, count, sp, lp, out, stream));
    else if ((size_t)g.T * 8 * 4 <= budget && L >= 6 && S * ceil_div(L, 8) >= fill)
      // 8 lasers: several CTAs per SM up to 1,600 bins or so, and whole 32-byte
      // sectors of the output (36 lasers, 1,024 bins, 256 scan points x 2,150
      // voxels: 0.27 ms; 1 laser 0.35 ms; 32 lasers, one CTA per SM and a second tile
      // of 4 lasers: 1.06 ms). Fewer CTAs or lasers: 1 laser (64^3 x 16 x 16 0.15 against
      // 0.49 ms, 96^3 x 9 x 9 0.35 against 1.04; 32^3 x 1,024 x 4, 5: 0.15, 0.18 against 0.20).
      TOTRI_TRY(launch_fwd<8>(g, b, vb, list, count, sp, lp, out, stream));
    else if ((size_t)g.T * 4 <= budget)
      TOTRI_TRY(launch_fwd<1>(g, b, vb, list, count, sp, lp, out, stream));
    else
      return fail(TOTRI_ERR_UNSUPPORTED, "too many bins for one tile");
  }
  return TOTRI_OK;
}

// Bins-last copies (one read and write of transient_grad, where a pair's reads in place
// are a sector per voxel and bin); slices of the scan points until about 8 waves of
// CTAs (4 per SM), with at least 8 scan points each (a slice repeats the lasers'
// distances).
static mesh::PairPlan grad_plan(int64_t S, int64_t L, int64_t T, int64_t D, int64_t H, int64_t W,
                                size_t ws_bytes) {
  const int64_t blocks = ceil_div(W, 8) * ceil_div(H, 8) * ceil_div(D, 4);
  return mesh::pair_plan(S, L, T, D * H * W, blocks, 32 * (int64_t)tune::sm_count(), 8, true,
                         ws_bytes);
}

size_t totri_volume_exhaustive_grad_scratch(int64_t S, int64_t L, int64_t T) {
  // Partial sums of a launch: slices of at most 256 voxels per CTA, fewer than 2 x 32
  // CTAs per SM where there is more than one.
  const size_t partial = S < 16 ? 0 : sizeof(float) * 256 * 64 * (size_t)tune::sm_count();
  return S > 0 && L > 0 && T > 0 ? mesh::exh_grad_scratch_bytes(S, L, T) + partial : 0;
}

size_t totri_volume_exhaustive_grad_workspace(int64_t S, int64_t L, int64_t T, int64_t D, int64_t H,
                                              int64_t W) {
  if (S <= 0 || L <= 0 || T <= 0 || D <= 0 || H <= 0 || W <= 0) return 0;
  return grad_plan(S, L, T, D, H, W, SIZE_MAX).bytes;
}

int totri_volume_exhaustive_grad_volume_ws(const totri_array_t* tg,
                                           const totri_array_t* scan_points,
                                           const totri_array_t* laser_points,
                                           const totri_array_t* scan_origin,
                                           const totri_array_t* laser_origin,
                                           const totri_array_t* vg, const float start[3],
                                           const float end[3], float bw, float bo, void* ws,
                                           size_t ws_bytes, void* stream_) {
  (void)scan_origin;
  (void)laser_origin;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  TOTRI_TRY(check_array(vg, "volume_grad", 4, TOTRI_FLOAT32));
  TOTRI_TRY(check_contiguous(vg, "volume_grad"));
  const int64_t B = vg->shape[0];
  int64_t S, L;
  vexh::Pts sp, lp;
  TOTRI_TRY(check_pts(scan_points, "scan_points", B, S, sp));
  TOTRI_TRY(check_pts(laser_points, "laser_points", B, L, lp));
  TOTRI_TRY(check_array(tg, "transient_grad", 4, TOTRI_FLOAT32));
  TOTRI_TRY(check_dim(tg, "transient_grad", 0, B));
  TOTRI_TRY(check_dim(tg, "transient_grad", 2, S));
  TOTRI_TRY(check_dim(tg, "transient_grad", 3, L));
  TOTRI_TRY(check_contiguous(tg, "transient_grad"));
  const int64_t T = tg->shape[1];
  const vexh::Geo g = make_geo(vg, S, L, T, start, end, bw, bo);
  const int64_t n = numel(vg);
  if (n == 0) return TOTRI_OK;
  float* out = static_cast<float*>(vg->data);
  if (S == 0 || L == 0 || T == 0) {
    TOTRI_CUDA(cudaMemsetAsync(out, 0, sizeof(float) * n, stream));
    return TOTRI_OK;
  }
  const mesh::PairPlan plan = grad_plan(S, L, T, g.D, g.H, g.W, ws ? ws_bytes : 0);
  const float window_far = std::fma(524288.f, bw, -std::fabs(bo));
  const int64_t blocks = ceil_div(g.W, 8) * ceil_div(g.H, 8) * ceil_div(g.D, 4);
  const int64_t row = S * L, nv = (int64_t)g.D * g.H * g.W;
  float* copy = static_cast<float*>(ws);
  float* part = reinterpret_cast<float*>(static_cast<char*>(ws) + plan.part_at);
  for (int b = 0; b < (int)B; ++b) {
    const float* tb = static_cast<const float*>(tg->data) + (int64_t)b * T * row;
    for (int64_t sa = 0; sa < S; sa += plan.step) {
      const int64_t sb = std::min(S, sa + plan.step);
      const int slices = (int)ceil_div(sb - sa, plan.per);
      const dim3 grid((unsigned)blocks, (unsigned)slices);
      float* sum = out + b * nv;
      float* dst = slices > 1 ? part : sum;
      const int add = slices == 1 && sa > 0;
      if (plan.chunk > 0) {
        TOTRI_TRY(mesh::launch_bins_last(tb + sa * L, copy, (int)T, (int)T, row, (sb - sa) * L,
                                         stream));
        TOTRI_KERNEL("volume exhaustive adjoint", stream,
                     vexh::adjoint_kernel<<<grid, 256, 0, stream>>>(
                         g, b, sp, lp, (int)sa, (int)sb, plan.per, copy, T, 1, dst, add,
                         window_far));
      } else {
        TOTRI_KERNEL("volume exhaustive adjoint", stream,
                     vexh::adjoint_kernel<<<grid, 256, 0, stream>>>(
                         g, b, sp, lp, (int)sa, (int)sb, plan.per, tb, 1, row, dst, add,
                         window_far));
      }
      if (slices > 1) TOTRI_TRY(mesh::launch_sum_slices(part, slices, nv, sum, sa > 0, stream));
    }
  }
  return TOTRI_OK;
}

int totri_volume_exhaustive_grad_volume(const totri_array_t* tg,
                                        const totri_array_t* scan_points,
                                        const totri_array_t* laser_points,
                                        const totri_array_t* scan_origin,
                                        const totri_array_t* laser_origin,
                                        const totri_array_t* vg, const float start[3],
                                        const float end[3], float bw, float bo, void* stream) {
  return totri_volume_exhaustive_grad_volume_ws(tg, scan_points, laser_points, scan_origin,
                                                laser_origin, vg, start, end, bw, bo, nullptr, 0,
                                                stream);
}

}  // extern "C"
