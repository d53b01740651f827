// Exhaustive (separate laser and detector points) mesh transient rendering:
// forward splat and vertex / albedo gradient.
//
// Reference: src/render/program/mesh_exhaustive_forward_optix.cu:18-169 and
// mesh_exhaustive_grad_verts_optix.cu:18-248: one OptiX thread per (face,
// scan, laser) triple tracing two visibility rays, global atomics into
// transient[b][bin][s][l]. Here visibility is separable: face f is visible
// from scan point s and from laser point l independently, so the two masks
// are computed once (S + L rows of the shared mask buffer) and each triple is
// their AND. The forward gives each CTA one scan point and a tile of laser
// points with a [T][tile] shared histogram flushed as rows of the [T][S][L]
// output; the gradient gives each CTA 32 faces and a slice of scan points and
// walks every (s, l) pair of the slice.
#include <cooperative_groups.h>

#include <algorithm>

#include "capi_common.cuh"
#include "mesh.cuh"
#include "mesh_kernels.cuh"
#include "tune.cuh"

namespace cg = cooperative_groups;

namespace totri {
namespace mesh {

struct ExhPair {
  fv3 v[3];
  int perm[3];
  float d[3];   // scan + laser path length (sort key)
  float ds[3];  // vertex - scan distance
  float dl[3];  // vertex - laser distance
  float c[3];
  int bin[3];
};

__device__ __forceinline__ void exh_sort(ExhPair& q) {
  auto sw = [&](int i, int j) {
    float t = q.d[i]; q.d[i] = q.d[j]; q.d[j] = t;
    t = q.ds[i]; q.ds[i] = q.ds[j]; q.ds[j] = t;
    t = q.dl[i]; q.dl[i] = q.dl[j]; q.dl[j] = t;
    fv3 tv = q.v[i]; q.v[i] = q.v[j]; q.v[j] = tv;
    int tp = q.perm[i]; q.perm[i] = q.perm[j]; q.perm[j] = tp;
  };
  if (q.d[0] > q.d[1]) sw(0, 1);
  if (q.d[1] > q.d[2]) sw(1, 2);
  if (q.d[0] > q.d[1]) sw(0, 1);
}

// FP32 decisions exactly as the oracle takes them (exhaustive_geom).
__device__ __forceinline__ void exh_pair(float4 s0, float4 s1, float4 s2, fv3 sp, fv3 lp, float od,
                                         float bw, float bo, ExhPair& q) {
  q.v[0] = mkv(s0.x, s0.y, s0.z);
  q.v[1] = mkv(s1.x, s1.y, s1.z);
  q.v[2] = mkv(s2.x, s2.y, s2.z);
  for (int k = 0; k < 3; ++k) {
    q.perm[k] = k;
    q.ds[k] = xlen(xsub3(q.v[k], sp));
    q.dl[k] = xlen(xsub3(q.v[k], lp));
    q.d[k] = xadd(q.ds[k], q.dl[k]);
  }
  exh_sort(q);
  for (int k = 0; k < 3; ++k) {
    q.c[k] = xdiv(xsub(xadd(q.d[k], od), bo), bw);
    q.bin[k] = bin_of(q.c[k]);
  }
}

// exh_pair with a filtered fast path (FastBins). The six lengths come from
// the hardware reciprocal square root and the bin coordinates from a fused
// multiply-add with a precomputed 1/bw. Against the exact chain each path
// length d = |v - s| + |v - l| deviates by at most 8 u d (u = 2^-24), so when
// the three fast lengths are separated by more than 16 u max(d) the exact
// sort gives the same order, and a bin coordinate farther than
// 32 u (d + od + |bo|)/bw + 8 u |c| from an integer truncates to the exact
// bin. Only then are the fast values kept (they differ from the exact ones
// by a few ulps, which the value tolerances absorb); otherwise, and for
// NaN or huge coordinates, the exact exh_pair runs. Bins and vertex order
// are therefore always those of the exact chain.
__device__ __forceinline__ void exh_pair_filtered(float4 s0, float4 s1, float4 s2, fv3 sp,
                                                  fv3 lp, float od, float bw, float bo,
                                                  const FastBins& fb, ExhPair& q) {
  q.v[0] = mkv(s0.x, s0.y, s0.z);
  q.v[1] = mkv(s1.x, s1.y, s1.z);
  q.v[2] = mkv(s2.x, s2.y, s2.z);
  for (int k = 0; k < 3; ++k) {
    q.perm[k] = k;
    q.ds[k] = len_fast(q.v[k] - sp);
    q.dl[k] = len_fast(q.v[k] - lp);
    q.d[k] = q.ds[k] + q.dl[k];
  }
  exh_sort(q);
  const float u = 5.9604645e-8f;
  bool ok = q.d[1] - q.d[0] > 16.f * u * q.d[2] && q.d[2] - q.d[1] > 16.f * u * q.d[2];
  for (int k = 0; k < 3; ++k) {
    const float c = fmaf(q.d[k] + od, fb.inv_bw, fb.nbo);
    const float m = fmaf(fb.kc, q.d[k] + od, fb.kb) + 8.f * u * fabsf(c);
    ok = ok && fabsf(c - rintf(c)) > m && fabsf(c) < 1.0e9f;
    q.c[k] = c;
    q.bin[k] = __float2int_rz(c);
  }
  if (!ok) exh_pair(s0, s1, s2, sp, lp, od, bw, bo, q);
}

// AlphaExhaustive (mesh_common.h:505-531), wall normals (0,0,1).
__device__ __forceinline__ float alpha_exhaustive(const ExhPair& q, fv3 c, fv3 sp, fv3 lp,
                                                  float rho) {
  const fv3 n = cross(q.v[1] - q.v[0], q.v[2] - q.v[0]);
  const fv3 rs = c - sp, rl = c - lp;
  if (!(rs.z > 0.f) || !(rl.z > 0.f)) return 0.f;
  const float rss = dot(rs, rs), rll = dot(rl, rl);
  return vdiv(100.f * rho * rs.z * rl.z * fabsf(dot(n, rs)) * fabsf(dot(n, rl)) *
                  rsqrtf(dot(n, n)),
              (rss * rss) * (rll * rll));
}

__device__ __forceinline__ float origin_term(const Origins& o, int b, int s, int l, fv3 sp,
                                             fv3 lp) {
  float od = 0.f;
  if (o.has_so) od = xlen(xsub3(sp, mkv(o.so.at(b, s, 0), o.so.at(b, s, 1), o.so.at(b, s, 2))));
  if (o.has_lo)
    od = xadd(od, xlen(xsub3(lp, mkv(o.lo.at(b, l, 0), o.lo.at(b, l, 1), o.lo.at(b, l, 2)))));
  return od;
}

// One CTA per (scan point, tile of LT lasers): the tile's [T][LT] histogram in
// shared memory, flushed once. With CL > 1 the CTAs of a cluster of CL
// neighbouring tiles (CL LT = 8 lasers) each flush every CL-th bin row for the
// whole cluster, reading the other tiles' histograms through distributed
// shared memory, so every row piece is one full 32-byte sector: a 4-laser
// tile's own 16-byte pieces make the memory read, merge and write back each
// sector (8.75 GB of DRAM traffic for a 2 GB transient).
template <int LT, int kOcc = 1, int CL = 1>
__global__ void __launch_bounds__(256, kOcc) exh_splat_kernel(Scene sc, View3f sp, View3f lp, Origins org,
                                                        int S, int L, float* __restrict__ out,
                                                        int T, float bw, float bo, FastBins fb) {
  extern __shared__ float hist[];  // [T][LT]
  const int b = blockIdx.z;
  const int s = blockIdx.x;
  const int l0 = blockIdx.y * LT;
  for (int i = threadIdx.x; i < T * LT; i += blockDim.x) hist[i] = 0.f;
  __syncthreads();
  const int n = sc.meta[b].n;
  const int ll = threadIdx.x % LT;
  const int l = l0 + ll;
  if (l < L) {
    const fv3 p = mkv(sp.at(b, s, 0), sp.at(b, s, 1), sp.at(b, s, 2));
    const fv3 q = mkv(lp.at(b, l, 0), lp.at(b, l, 1), lp.at(b, l, 2));
    const float od = origin_term(org, b, s, l, p, q);
    const uint32_t* ms = sc.mask + ((size_t)b * sc.P + s) * sc.nch;
    const uint32_t* ml = sc.mask + ((size_t)b * sc.P + S + l) * sc.nch;
    const float4* shade = sc.shade + (size_t)b * sc.F * 4;
    Hist<LT> h{hist, ll, T};
    for (int k = threadIdx.x / LT; k < n; k += blockDim.x / LT) {
      const uint32_t bit = 1u << (k & 31);
      if (!(__ldg(ms + (k >> 5)) & bit) || !(__ldg(ml + (k >> 5)) & bit)) continue;
      const float4 s0r = __ldg(shade + 4 * k), s1r = __ldg(shade + 4 * k + 1);
      const float4 s2r = __ldg(shade + 4 * k + 2), s3r = __ldg(shade + 4 * k + 3);
      ExhPair e;
      exh_pair_filtered(s0r, s1r, s2r, p, q, od, bw, bo, fb, e);
      const float alpha = alpha_exhaustive(e, mkv(s3r.x, s3r.y, s3r.z), p, q, s0r.w);
      if (!(alpha > 0.f)) continue;
      splat_tent(h, e.c, e.bin, alpha);
    }
  }
  __syncthreads();
  if (CL == 1) {
    // rows out[b][t][s][l0 .. l0+LT)
    float* ob = out + (((size_t)b * T) * S + s) * L + l0;
    for (int i = threadIdx.x; i < T * LT; i += blockDim.x) {
      const int t = i / LT, c = i - t * LT;
      if (l0 + c < L) ob[(size_t)t * S * L + c] = hist[i];
    }
  } else {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();  // every tile of the cluster has its histogram
    const int rank = (int)cluster.block_rank();
    const int L0 = l0 - rank * LT;  // the cluster's first laser
    float* ob = out + (((size_t)b * T) * S + s) * L + L0;
    const int rows = (T - rank + CL - 1) / CL;
    for (int i = threadIdx.x; i < rows * CL * LT; i += blockDim.x) {
      const int t = rank + CL * (i / (CL * LT)), j = i % (CL * LT);
      const int src = j / LT, c = j - src * LT;
      const float* rh = cluster.map_shared_rank(hist, src);
      if (L0 + j < L) ob[(size_t)t * S * L + j] = rh[t * LT + c];
    }
    cluster.sync();  // no tile leaves while another still reads its histogram
  }
}

// Forward with the visible triples compacted first (tuning option). Visibility is separable,
// so for the CTA's scan point s and each of its LT lasers the visible faces of
// a 32-face chunk are one AND of two mask words. Each warp walks its chunks,
// appends the visible (face, laser) pairs to a per-warp queue in shared memory
// and evaluates them 32 at a time, one per lane: every lane does useful work
// instead of most lanes waiting on mask tests that fail.
constexpr int kExhQueue = 64;

template <int LT>
__global__ void __launch_bounds__(256) exh_splat_compact_kernel(Scene sc, View3f sp, View3f lp,
                                                                Origins org, int S, int L,
                                                                float* __restrict__ out, int T,
                                                                float bw, float bo, FastBins fb) {
  extern __shared__ float hist[];  // [T][LT]
  __shared__ float lpt[LT][4];     // laser point, laser-origin term
  __shared__ int queue[8][kExhQueue];
  const int b = blockIdx.z;
  const int s = blockIdx.x;
  const int l0 = blockIdx.y * LT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < T * LT; i += blockDim.x) hist[i] = 0.f;
  const fv3 p = mkv(sp.at(b, s, 0), sp.at(b, s, 1), sp.at(b, s, 2));
  if (threadIdx.x < LT && l0 + (int)threadIdx.x < L) {
    const int l = l0 + threadIdx.x;
    const fv3 q = mkv(lp.at(b, l, 0), lp.at(b, l, 1), lp.at(b, l, 2));
    lpt[threadIdx.x][0] = q.x;
    lpt[threadIdx.x][1] = q.y;
    lpt[threadIdx.x][2] = q.z;
    lpt[threadIdx.x][3] = origin_term(org, b, s, l, p, q);
  }
  __syncthreads();
  const int n = sc.meta[b].n;
  const int nchu = (n + 31) >> 5;
  const uint32_t* ms = sc.mask + ((size_t)b * sc.P + s) * sc.nch;
  const uint32_t* ml = sc.mask + ((size_t)b * sc.P + S) * sc.nch;
  const float4* shade = sc.shade + (size_t)b * sc.F * 4;
  const int lts = min(LT, L - l0);
  const uint32_t below = (1u << lane) - 1u;
  int* qw = queue[warp];
  int cnt = 0;  // warp-uniform
  auto run = [&](int e) {
    const int k = e >> 5, l = e & 31;
    const float4 s0r = __ldg(shade + 4 * k), s1r = __ldg(shade + 4 * k + 1);
    const float4 s2r = __ldg(shade + 4 * k + 2), s3r = __ldg(shade + 4 * k + 3);
    const fv3 q = mkv(lpt[l][0], lpt[l][1], lpt[l][2]);
    ExhPair ep;
    exh_pair_filtered(s0r, s1r, s2r, p, q, lpt[l][3], bw, bo, fb, ep);
    const float alpha = alpha_exhaustive(ep, mkv(s3r.x, s3r.y, s3r.z), p, q, s0r.w);
    if (!(alpha > 0.f)) return;
    const Hist<LT> h{hist, l, T};
    splat_tent(h, ep.c, ep.bin, alpha);
  };
  for (int ch = warp; ch < nchu; ch += 8) {
    const uint32_t msw = __ldg(ms + ch);
    if (msw == 0u) continue;
    const uint32_t lw =
        lane < lts ? (__ldg(ml + (size_t)(l0 + lane) * sc.nch + ch) & msw) : 0u;
    for (int l = 0; l < lts; ++l) {
      const uint32_t bits = __shfl_sync(0xffffffffu, lw, l);
      if (bits == 0u) continue;
      if ((bits >> lane) & 1u) qw[cnt + __popc(bits & below)] = ((ch * 32 + lane) << 5) | l;
      cnt += __popc(bits);
      if (cnt >= 32) {
        __syncwarp();
        const int e = qw[lane];
        __syncwarp();
        if (lane < cnt - 32) qw[lane] = qw[32 + lane];
        cnt -= 32;
        __syncwarp();
        run(e);
      }
    }
  }
  __syncwarp();
  if (lane < cnt) run(qw[lane]);
  __syncthreads();
  // rows out[b][t][s][l0 .. l0+LT)
  float* ob = out + (((size_t)b * T) * S + s) * L + l0;
  for (int i = threadIdx.x; i < T * LT; i += blockDim.x) {
    const int t = i / LT, c = i - t * LT;
    if (l0 + c < L) ob[(size_t)t * S * L + c] = hist[i];
  }
}

// The origin terms |s - o_s| + |l - o_l| as a double-float (zero without origins).
__device__ __forceinline__ DFloat origin_term_df(const Origins& o, int b, int s, int l, fv3 sp,
                                                 fv3 lp) {
  DFloat od{0.f, 0.f};
  if (o.has_so) od = len_df(sp, mkv(o.so.at(b, s, 0), o.so.at(b, s, 1), o.so.at(b, s, 2)));
  if (o.has_lo)
    od = df_add(od, len_df(lp, mkv(o.lo.at(b, l, 0), o.lo.at(b, l, 1), o.lo.at(b, l, 2))));
  return od;
}

// The tent corners of a triple relative to its first bin, from double-float
// path lengths |v_k - s| + |v_k - l| + od (bin_offset).
__device__ __forceinline__ void exh_corners(const ExhPair& q, fv3 sp, fv3 lp, DFloat od, float bw,
                                            float inv_bw, float bo, float x[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const DFloat d = df_add(df_add(len_df(q.v[k], sp), len_df(q.v[k], lp)), od);
    x[k] = bin_offset(d, bo, bw, inv_bw, q.bin[0]);
  }
}

// Gradient of one visible triple w.r.t. the sorted vertices and the albedo
// (mesh_exhaustive_grad_verts_optix.cu:336-412, AlphaExhaustiveGradVerts
// mesh_common.h:549-630), with the tent corners x taken relative to bin[0]
// (exh_corners).
__device__ __forceinline__ bool triple_grad(const ExhPair& q, const float x[3], fv3 c, fv3 sp,
                                            fv3 lp, float rho, float bw,
                                            const float* __restrict__ col, int64_t stride, int T,
                                            fv3 dv[3], float& dmat) {
  const float alpha = alpha_exhaustive(q, c, sp, lp, rho);
  if (!(alpha > 0.f)) return false;
  if (q.bin[0] >= T || q.bin[2] < 0) return false;
  const fv3 e1 = q.v[1] - q.v[0], e2 = q.v[2] - q.v[0];
  const fv3 n = cross(e1, e2);
  const fv3 rs = c - sp, rl = c - lp;
  const float kn = vdiv(-1.f, dot(n, n));
  const float krs = vdiv(-4.f, 3.f * dot(rs, rs)), krl = vdiv(-4.f, 3.f * dot(rl, rl));
  const float kw = vdiv(1.f, 3.f * rs.z) + vdiv(1.f, 3.f * rl.z);
  const float knrs = vdiv(1.f, dot(n, rs)), knrl = vdiv(1.f, dot(n, rl));
  const fv3 w = kn * n + knrs * rs + knrl * rl;
  const fv3 g1 = cross(e2, w), g2 = cross(w, e1);
  const fv3 common = krs * rs + krl * rl + ((knrs + knrl) * (1.f / 3.f)) * n + mkv(0.f, 0.f, kw);
  const fv3 da0 = alpha * (common - g1 - g2);
  const fv3 da1 = alpha * (common + g1);
  const fv3 da2 = alpha * (common + g2);
  const float dadm = vdiv(alpha, rho);
  if (q.bin[0] == q.bin[2]) {
    const float g = __ldg(col + (size_t)q.bin[0] * stride);
    dv[0] = g * da0;
    dv[1] = g * da1;
    dv[2] = g * da2;
    dmat = g * dadm;
    return true;
  }
  TentGrad tgr;
  tent_grad(col, stride, T, x, q.bin, tgr);
  const float span = x[2] - x[0];
  const float kk = vdiv(-2.f, bw * span * span);
  fv3 dc[3];
  for (int k = 0; k < 3; ++k)
    dc[k] = vdiv(1.f, bw * q.dl[k]) * (q.v[k] - lp) + vdiv(1.f, bw * q.ds[k]) * (q.v[k] - sp);
  const fv3 dyc0 = kk * (vdiv(-1.f, q.dl[0]) * (q.v[0] - lp) + vdiv(-1.f, q.ds[0]) * (q.v[0] - sp));
  const fv3 dyc2 = kk * (vdiv(1.f, q.dl[2]) * (q.v[2] - lp) + vdiv(1.f, q.ds[2]) * (q.v[2] - sp));
  dv[0] = tgr.part0 * da0 + alpha * (tgr.ayc * dyc0 + tgr.a0 * dc[0]);
  dv[1] = tgr.part0 * da1 + alpha * (tgr.a1 * dc[1]);
  dv[2] = tgr.part0 * da2 + alpha * (tgr.ayc * dyc2 + tgr.a2 * dc[2]);
  dmat = dadm * tgr.part0;
  return true;
}

__global__ void __launch_bounds__(256) exh_grad_kernel(Scene sc, View3f sp, View3f lp, Origins org,
                                                       int S, int L,
                                                       const float* __restrict__ tgrad, int T,
                                                       float bw, float bo, FastBins fb, GradOut out) {
  extern __shared__ uint32_t mcol[];  // [S + L] mask words of this 32-face chunk
  const int b = blockIdx.y;
  const int ch = blockIdx.x;
  const int n = sc.meta[b].n;
  if (ch * 32 >= n) return;
  // scan-point slice [s0, s1) of this CTA (gridDim.z slices); all laser rows
  const int s0 = (int)((int64_t)S * blockIdx.z / gridDim.z);
  const int s1 = (int)((int64_t)S * (blockIdx.z + 1) / gridDim.z);
  for (int i = threadIdx.x; i < S + L; i += blockDim.x)
    if (i >= S || (i >= s0 && i < s1)) mcol[i] = sc.mask[((size_t)b * sc.P + i) * sc.nch + ch];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const float* tgb = tgrad + (size_t)b * T * S * L;
  const int64_t stride = (int64_t)S * L;
  const float4* shade = sc.shade + (size_t)b * sc.F * 4;
  for (int j = warp; j < 32; j += nw) {
    const int k = ch * 32 + j;
    if (k >= n) break;
    const float4 s0r = __ldg(shade + 4 * k), s1r = __ldg(shade + 4 * k + 1);
    const float4 s2r = __ldg(shade + 4 * k + 2), s3r = __ldg(shade + 4 * k + 3);
    const fv3 c = mkv(s3r.x, s3r.y, s3r.z);
    fv3 acc[3] = {mkv(0.f, 0.f, 0.f), mkv(0.f, 0.f, 0.f), mkv(0.f, 0.f, 0.f)};
    float accm = 0.f;
    for (int s = s0; s < s1; ++s) {
      if (!((mcol[s] >> j) & 1u)) continue;
      const fv3 p = mkv(sp.at(b, s, 0), sp.at(b, s, 1), sp.at(b, s, 2));
      for (int l = lane; l < L; l += 32) {
        if (!((mcol[S + l] >> j) & 1u)) continue;
        const fv3 q = mkv(lp.at(b, l, 0), lp.at(b, l, 1), lp.at(b, l, 2));
        ExhPair e;
        exh_pair_filtered(s0r, s1r, s2r, p, q, origin_term(org, b, s, l, p, q), bw, bo, fb,
                          e);
        if (e.bin[0] >= T || e.bin[2] < 0) continue;
        float x[3];
        exh_corners(e, p, q, origin_term_df(org, b, s, l, p, q), bw, fb.inv_bw, bo, x);
        fv3 dv[3];
        float dm;
        if (!triple_grad(e, x, c, p, q, s0r.w, bw, tgb + (size_t)s * L + l, stride, T, dv, dm))
          continue;
        add_permuted(acc, dv, e.perm);
        accm += dm;
      }
    }
    scatter_face_grad(out, b, s1r, s2r, s3r, acc, accm, sc.status);
  }
}

// Gradient with the visible (scan point, laser) pairs of each face compacted:
// the CTA holds its 32 faces' scan-mask words for a slice of scan points and,
// per face, the set of lasers that see it (transposed from the laser rows by
// warp ballots). A warp walks one face at a time, queues its visible
// (s, l) pairs and evaluates them 32 at a time, one per lane; the face's
// gradient stays in registers and is reduced and scattered once per CTA.
__global__ void __launch_bounds__(256) exh_grad_compact_kernel(
    Scene sc, View3f sp, View3f lp, Origins org, int S, int L, const float* __restrict__ tgrad,
    int T, float bw, float bo, FastBins fb, GradOut out) {
  extern __shared__ uint32_t words[];  // [slice] scan words | [32][LW] laser sets
  __shared__ int qs[8][kExhQueue], ql[8][kExhQueue];
  const int b = blockIdx.y;
  const int ch = blockIdx.x;
  const int n = sc.meta[b].n;
  if (ch * 32 >= n) return;
  const int s0 = (int)((int64_t)S * blockIdx.z / gridDim.z);
  const int s1 = (int)((int64_t)S * (blockIdx.z + 1) / gridDim.z);
  const int ns = s1 - s0;
  const int LW = (L + 31) >> 5;
  uint32_t* mcs = words;
  uint32_t* lvis = words + ns;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t* mrow = sc.mask + (size_t)b * sc.P * sc.nch + ch;
  for (int i = threadIdx.x; i < ns; i += blockDim.x) mcs[i] = mrow[(size_t)(s0 + i) * sc.nch];
  for (int wl = warp; wl < LW; wl += 8) {
    const int l = wl * 32 + lane;
    const uint32_t m = l < L ? mrow[(size_t)(S + l) * sc.nch] : 0u;
    for (int j = 0; j < 32; ++j) {
      const uint32_t bal = __ballot_sync(0xffffffffu, (m >> j) & 1u);
      if (lane == 0) lvis[j * LW + wl] = bal;
    }
  }
  __syncthreads();
  const float* tgb = tgrad + (size_t)b * T * S * L;
  const int64_t stride = (int64_t)S * L;
  const float4* shade = sc.shade + (size_t)b * sc.F * 4;
  const uint32_t below = (1u << lane) - 1u;
  for (int j = warp; j < 32; j += 8) {
    const int k = ch * 32 + j;
    if (k >= n) break;
    const float4 s0r = __ldg(shade + 4 * k), s1r = __ldg(shade + 4 * k + 1);
    const float4 s2r = __ldg(shade + 4 * k + 2), s3r = __ldg(shade + 4 * k + 3);
    const fv3 c = mkv(s3r.x, s3r.y, s3r.z);
    fv3 acc[3] = {mkv(0.f, 0.f, 0.f), mkv(0.f, 0.f, 0.f), mkv(0.f, 0.f, 0.f)};
    float accm = 0.f;
    auto run = [&](int s, int l) {
      const fv3 p = mkv(sp.at(b, s, 0), sp.at(b, s, 1), sp.at(b, s, 2));
      const fv3 q = mkv(lp.at(b, l, 0), lp.at(b, l, 1), lp.at(b, l, 2));
      ExhPair e;
      exh_pair_filtered(s0r, s1r, s2r, p, q, origin_term(org, b, s, l, p, q), bw, bo, fb,
                          e);
      if (e.bin[0] >= T || e.bin[2] < 0) return;
      float x[3];
      exh_corners(e, p, q, origin_term_df(org, b, s, l, p, q), bw, fb.inv_bw, bo, x);
      fv3 dv[3];
      float dm;
      if (!triple_grad(e, x, c, p, q, s0r.w, bw, tgb + (size_t)s * L + l, stride, T, dv, dm))
        return;
      add_permuted(acc, dv, e.perm);
      accm += dm;
    };
    const uint32_t* lv = lvis + j * LW;
    int cnt = 0;  // warp-uniform
    for (int si = 0; si < ns; ++si) {
      if (!((mcs[si] >> j) & 1u)) continue;
      for (int wl = 0; wl < LW; ++wl) {
        const uint32_t bits = lv[wl];
        if (bits == 0u) continue;
        if ((bits >> lane) & 1u) {
          const int at = cnt + __popc(bits & below);
          qs[warp][at] = s0 + si;
          ql[warp][at] = wl * 32 + lane;
        }
        cnt += __popc(bits);
        if (cnt >= 32) {
          __syncwarp();
          const int es = qs[warp][lane], el = ql[warp][lane];
          __syncwarp();
          if (lane < cnt - 32) {
            qs[warp][lane] = qs[warp][32 + lane];
            ql[warp][lane] = ql[warp][32 + lane];
          }
          cnt -= 32;
          __syncwarp();
          run(es, el);
        }
      }
    }
    __syncwarp();
    if (lane < cnt) run(qs[warp][lane], ql[warp][lane]);
    __syncwarp();
    scatter_face_grad(out, b, s1r, s2r, s3r, acc, accm, sc.status);
  }
}

// Gradient that uses the separability of the triple terms. For one face,
// everything that depends on the scan point s alone or the laser point l alone
// is computed once per point into a shared-memory record:
//   - the exact FP32 lengths |v_m - p| that decide the vertex order and bins
//     (the same chain as exh_pair) and their double-float low parts;
//   - the origin term |p - o_p| (exact FP32 and low part);
//   - the point's alpha factor A_p = max(0, r.z) |n.r| / |r|^4 (r = c - p),
//     with alpha = 100 rho |n|^-1 A_s A_l (AlphaExhaustive, mesh_common.h:505-531);
//   - its parts of d log(alpha) / d v_m: cm = -4/3 r/|r|^2 + n/(3 n.r) +
//     (0, 0, 1/(3 r.z)), the same for every vertex, and wv = r/(n.r), which
//     enters through the normal's Jacobian (AlphaExhaustiveGradVerts,
//     mesh_common.h:549-630);
//   - the unit vectors u_m = (v_m - p)/|v_m - p| that make up d c_k / d v.
// A triple then only needs its two factors P = alpha area-weighted gradient and Q_m
// = alpha times the tent's weight of vertex m: the vertex gradients are linear in
// the two records, sum P (cm_s + cm_l), sum P (wv_s + wv_l) and sum Q_m (u_s + u_l),
// the alpha gradient being taken in the face's own vertex order (the formula is
// the same in any order). A lane therefore keeps one point's record while its warp
// walks the other points: it adds the other point's part triple by triple, 16
// multiply-adds, and its own part once at the end, times the sums of P and Q; the
// normal's Jacobian is applied to the face's sum. The lanes stand for the scan or
// the laser points, whichever fill 32 better. A CTA takes its faces one at a time
// over a slice of at most kFaceSlice scan points and the lasers in chunks of
// kFaceSlice. The decisions (vertex order, bins) are those of exh_pair.
// 20,000 faces x 400 x 144 points, 2,048 bins: 8.2 ms (71% of the issue slots, the
// ALU pipe 70% busy with selects and compares) against 11.9 ms when each of
// a pair's 48 record fields was read per triple, the tent's three parts were walked
// apart and bins were read one by one; 768 faces x 143 x 35 points: 76 against 458
// us, of which one face per CTA instead of 8 gave 368 (96 CTAs before).
constexpr int kFaceSlice = 256;
constexpr int kFacesPerCta = 1;
// Most bytes of one bins-last copy of transient_grad (a range of scan points
// of one batch item; launch_exhaustive_grad).
constexpr size_t kGradChunkBytes = size_t(2) << 30;
constexpr int kRec = 28;  // floats per point record (fields below; 28 keeps 16-byte reads of
                          // 8 neighbouring records on distinct banks)
enum : int {
  kRecD = 0,     // [3] exact FP32 lengths
  kRecA = 3,     // alpha factor
  kRecDlo = 4,   // [3] the lengths' low parts
  kRecOdlo = 7,  // the origin term's low part
  kRecCm = 8,    // [3]
  kRecWv = 11,   // [3]
  kRecU = 14,    // [9] unit vectors u_m
  kRecOd = 23,   // origin term, FP32
  kRecAt = 24,   // the point's index (int)
};

// Fills the record of point p (origin o if has_o) for the face (v, c, n);
// rec[f] is field f.
__device__ __forceinline__ void exh_point_record(const fv3 v[3], fv3 c, fv3 n, fv3 p, bool has_o,
                                                 fv3 o, float* rec) {
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const float d = xlen(xsub3(v[m], p));
    const DFloat df = len_df(v[m], p);
    rec[kRecD + m] = d;
    rec[kRecDlo + m] = (df.hi - d) + df.lo;
    const float inv = vdiv(1.f, d);
    const fv3 u = inv * (v[m] - p);
    rec[kRecU + 3 * m] = u.x;
    rec[kRecU + 3 * m + 1] = u.y;
    rec[kRecU + 3 * m + 2] = u.z;
  }
  float od = 0.f, odlo = 0.f;
  if (has_o) {
    od = xlen(xsub3(p, o));
    const DFloat df = len_df(p, o);
    odlo = (df.hi - od) + df.lo;
  }
  rec[kRecOd] = od;
  rec[kRecOdlo] = odlo;
  const fv3 r = c - p;
  const float rr = dot(r, r), nr = dot(n, r);
  const bool front = r.z > 0.f;
  rec[kRecA] = front ? vdiv(r.z * fabsf(nr), rr * rr) : 0.f;
  const float kr = vdiv(-4.f, 3.f * rr), knr = vdiv(1.f, nr), kw = vdiv(1.f, 3.f * r.z);
  const fv3 cm = kr * r + (knr * (1.f / 3.f)) * n + mkv(0.f, 0.f, front ? kw : 0.f);
  rec[kRecCm] = cm.x;
  rec[kRecCm + 1] = cm.y;
  rec[kRecCm + 2] = cm.z;
  rec[kRecWv] = knr * r.x;
  rec[kRecWv + 1] = knr * r.y;
  rec[kRecWv + 2] = knr * r.z;
}

// Block-wide compaction: returns this thread's slot among the threads whose
// flag is set (or -1) and leaves their count in *total. All 256 threads call it.
__device__ __forceinline__ int block_slot(bool flag, int* warp_counts, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned bal = __ballot_sync(0xffffffffu, flag);
  if (lane == 0) warp_counts[warp] = __popc(bal);
  __syncthreads();
  int base = 0, sum = 0;
  for (int w = 0; w < 8; ++w) {
    const int c = warp_counts[w];
    base += w < warp ? c : 0;
    sum += c;
  }
  *total = sum;
  return flag ? base + __popc(bal & ((1u << lane) - 1u)) : -1;
}

// kForward: the bin width is positive.
template <int kOcc, bool kLast, bool kForward>
__global__ void __launch_bounds__(256, kOcc) exh_grad_face_kernel(
    Scene sc, View3f sp, View3f lp, Origins org, int S, int L, const float* __restrict__ tgrad,
    int T, float bw, float bo, int fixed, GradOut out, int faces_per_cta, int lchunk, int sslice,
    int b0, int s_base, int s_end, int64_t bstride, int64_t cstep, int64_t bstep) {
  // Batch item b0 + blockIdx.y, scan points [s_base, s_end); transient_grad
  // element (t, s, l) of item b is tgrad[(b - b0) bstride + ((s - s_base) L +
  // l) cstep + t bstep]: the caller's [B, T, S, L] tensor (b0 = s_base = 0,
  // bstride = T S L, cstep = 1, bstep = S L) or one item's bins-last copy of
  // a range of scan points (cstep = T, bstep = 1).
  extern __shared__ float4 recs4[];  // scan-point then laser-point records
  float* srec = reinterpret_cast<float*>(recs4);
  float* lrec = srec + kRec * kFaceSlice;
  __shared__ int counts[2][8];
  __shared__ float red[8][16], tot[16];
  const int b = b0 + blockIdx.y;
  const int n = sc.meta[b].n;
  const int nlc = (L + lchunk - 1) / lchunk;
  const int s0 = s_base + (blockIdx.z / nlc) * sslice;
  const int ns_all = min(sslice, s_end - s0);
  const int la = (blockIdx.z % nlc) * lchunk, lb = min(L, la + lchunk);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* tgb = tgrad + (int64_t)(b - b0) * bstride;
  const float4* shade = sc.shade + (size_t)b * sc.F * 4;
  const uint32_t* mrows = sc.mask + (size_t)b * sc.P * sc.nch;
  const float inv_bw = __frcp_rn(bw);
  const bool plain = !org.has_so && !org.has_lo && bo == 0.f;  // nothing added to a path
  for (int fi = 0; fi < faces_per_cta; ++fi) {
    const int k = blockIdx.x * faces_per_cta + fi;
    if (k >= n) break;  // CTA-uniform
    const float4 s0r = __ldg(shade + 4 * k), s1r = __ldg(shade + 4 * k + 1);
    const float4 s2r = __ldg(shade + 4 * k + 2), s3r = __ldg(shade + 4 * k + 3);
    const fv3 v[3] = {mkv(s0r.x, s0r.y, s0r.z), mkv(s1r.x, s1r.y, s1r.z), mkv(s2r.x, s2r.y, s2r.z)};
    const fv3 c = mkv(s3r.x, s3r.y, s3r.z);
    const fv3 nrm = cross(v[1] - v[0], v[2] - v[0]);
    const float nn = dot(nrm, nrm);
    const float kf = xdiv(100.f * s0r.w, xsqrt(nn));
    const int ch = k >> 5;
    const uint32_t bit = 1u << (k & 31);
    // the face's scan-point records over this slice
    int ns;
    {
      const int s = s0 + tid;
      const bool vis = tid < ns_all && (mrows[(size_t)s * sc.nch + ch] & bit);
      const int at = block_slot(vis, counts[0], &ns);
      if (vis) {
        const fv3 p = mkv(sp.at(b, s, 0), sp.at(b, s, 1), sp.at(b, s, 2));
        const fv3 o = org.has_so ? mkv(org.so.at(b, s, 0), org.so.at(b, s, 1), org.so.at(b, s, 2))
                                 : mkv(0.f, 0.f, 0.f);
        exh_point_record(v, c, nrm, p, org.has_so, o, srec + at * kRec);
        srec[at * kRec + kRecAt] = __int_as_float(s - s_base);
      }
    }
    // pairs of sum P cm [3], sum P wv [3], sum Q_m u_m [9], sum P
    unsigned long long acc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] = 0ull;
    for (int l0 = la; l0 < lb && ns > 0; l0 += kFaceSlice) {
      int nl;
      {
        const int l = l0 + tid;
        const bool vis = l < lb && tid < kFaceSlice &&
                         (mrows[(size_t)(S + l) * sc.nch + ch] & bit);
        const int at = block_slot(vis, counts[1], &nl);
        if (vis) {
          const fv3 p = mkv(lp.at(b, l, 0), lp.at(b, l, 1), lp.at(b, l, 2));
          const fv3 o = org.has_lo ? mkv(org.lo.at(b, l, 0), org.lo.at(b, l, 1), org.lo.at(b, l, 2))
                                   : mkv(0.f, 0.f, 0.f);
          exh_point_record(v, c, nrm, p, org.has_lo, o, lrec + at * kRec);
          lrec[at * kRec + kRecAt] = __int_as_float(l);
        }
      }
      __syncthreads();
      // The lanes take the points that fill the last warp row better; laser points
      // unless that is a third worse where their bins lie side by side.
      const int gs = (ns + 31) >> 5, gl = (nl + 31) >> 5;
      const bool over_s = kLast ? ns * gl >= nl * gs : 3 * ns * gl > 4 * nl * gs;
      const float* mine = over_s ? srec : lrec;
      const float* other = over_s ? lrec : srec;
      const int nm = over_s ? ns : nl, no = over_s ? nl : ns, gm = over_s ? gs : gl;
      const int64_t mstep = (over_s ? (int64_t)L : 1) * cstep;
      const int64_t ostep = (over_s ? 1 : (int64_t)L) * cstep;
      // rows (32 points of one side, one point of the other), split over the warps
      int r = (int)((int64_t)warp * gm * no / 8);
      const int r_end = (int)((int64_t)(warp + 1) * gm * no / 8);
      while (r < r_end) {
        const int grp = r / no;
        int j = r - grp * no;
        const int j_end = min(no, j + r_end - r);
        r += j_end - j;
        const int i = grp * 32 + lane;
        const float* rm = mine + min(i, nm - 1) * kRec;
        const float4 m0 = *reinterpret_cast<const float4*>(rm);      // D, A
        const float4 m1 = *reinterpret_cast<const float4*>(rm + 4);  // Dlo, odlo
        const float mod = rm[kRecOd];
        const float am = i < nm ? m0.w * kf : 0.f;
        const float* colm = tgb + __float_as_int(rm[kRecAt]) * mstep;
        float gP = 0.f, gQ0 = 0.f, gQ1 = 0.f, gQ2 = 0.f;
        bool used = false;
        for (; j < j_end; ++j) {
          const float* ro = other + j * kRec;
          const float4 o0 = *reinterpret_cast<const float4*>(ro);
          const float alpha = am * o0.w;
          if (!(alpha > 0.f)) continue;
          const float4 o1 = *reinterpret_cast<const float4*>(ro + 4);
          // path lengths: hi is the FP32 chain's sum, lo what it rounds off
          DFloat e0 = two_sum(m0.x, o0.x), e1 = two_sum(m0.y, o0.y), e2 = two_sum(m0.z, o0.z);
          e0.lo += m1.x + o1.x;
          e1.lo += m1.y + o1.y;
          e2.lo += m1.z + o1.z;
          // the vertex order of exh_sort (stable compare-swaps on the path length)
          const PathOrder order = sort_paths(e0, e1, e2);
          if (!plain) {
            const float ood = ro[kRecOd];
            const DFloat od = df_add(DFloat{mod, m1.w}, DFloat{ood, o1.w});
            e0 = path_offset(e0, od, bo);
            e1 = path_offset(e1, od, bo);
            e2 = path_offset(e2, od, bo);
          }
          const float* col = colm + __float_as_int(ro[kRecAt]) * ostep;
          float4 w;  // area, weights of the vertices
          if (!pair_weights<kLast, kForward>(col, bstep, T, e0, e1, e2, bw, inv_bw, fixed, order, w))
            continue;
          const float P = alpha * w.x, Q0 = alpha * w.y, Q1 = alpha * w.z, Q2 = alpha * w.w;
          used = true;
          gP += P;
          gQ0 += Q0;
          gQ1 += Q1;
          gQ2 += Q2;
          const ulonglong2 o2 = *reinterpret_cast<const ulonglong2*>(ro + 8);   // cm, wv
          const ulonglong2 o3 = *reinterpret_cast<const ulonglong2*>(ro + 12);  // wv, u
          const ulonglong2 o4 = *reinterpret_cast<const ulonglong2*>(ro + 16);
          const ulonglong2 o5 = *reinterpret_cast<const ulonglong2*>(ro + 20);  // u, od
          const unsigned long long PP = f2pack(P, P), Q00 = f2pack(Q0, Q0), Q11 = f2pack(Q1, Q1);
          const unsigned long long Q22 = f2pack(Q2, Q2);
          acc[0] = f2fma(PP, o2.x, acc[0]);
          acc[1] = f2fma(PP, o2.y, acc[1]);
          acc[2] = f2fma(PP, o3.x, acc[2]);
          acc[3] = f2fma(Q00, o3.y, acc[3]);
          acc[4] = f2fma(f2pack(Q0, Q1), o4.x, acc[4]);
          acc[5] = f2fma(Q11, o4.y, acc[5]);
          acc[6] = f2fma(Q22, o5.x, acc[6]);
          float u8, ood;
          f2unpack(o5.y, u8, ood);
          acc[7] = f2fma(f2pack(Q2, P), f2pack(u8, 1.f), acc[7]);
        }
        if (used) {  // this lane's own point
          const unsigned long long PP = f2pack(gP, gP);
          const ulonglong2* q = reinterpret_cast<const ulonglong2*>(rm + 8);
          acc[0] = f2fma(PP, q[0].x, acc[0]);
          acc[1] = f2fma(PP, q[0].y, acc[1]);
          acc[2] = f2fma(PP, q[1].x, acc[2]);
          acc[3] = f2fma(f2pack(gQ0, gQ0), q[1].y, acc[3]);
          acc[4] = f2fma(f2pack(gQ0, gQ1), q[2].x, acc[4]);
          acc[5] = f2fma(f2pack(gQ1, gQ1), q[2].y, acc[5]);
          acc[6] = f2fma(f2pack(gQ2, gQ2), q[3].x, acc[6]);
          acc[7] = f2fma(f2pack(gQ2, 0.f), f2pack(rm[kRecU + 8], 0.f), acc[7]);
        }
      }
      __syncthreads();  // records are rewritten for the next laser chunk / face
    }
    if (ns > 0) {  // CTA-uniform
      // the face's sums, then one thread per vertex component
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        float x, y;
        f2unpack(acc[q], x, y);
        x = warp_sum(x);
        y = warp_sum(y);
        if (lane == 0) {
          red[warp][2 * q] = x;
          red[warp][2 * q + 1] = y;
        }
      }
      __syncthreads();
      if (tid < 16) {
        float t = 0.f;
        for (int w = 0; w < 8; ++w) t += red[w][tid];
        tot[tid] = t;
      }
      __syncthreads();
      const int vi[3] = {__float_as_int(s1r.w), __float_as_int(s2r.w), __float_as_int(s3r.w)};
      if (tid < 9) {
        const int m = tid / 3, a = tid - 3 * m;
        // d alpha: w = sum P (wf + wv), wf = -n / |n|^2, through the normal's Jacobian
        // (a face without a pair adds zeros, whatever its normal and albedo; 1 / |n|^2 is
        // first multiplied by n: with the sum it leaves the FP32 range in small units)
        fv3 w = mkv(tot[3], tot[4], tot[5]);
        if (tot[15] != 0.f) w = tot[15] * (vdiv(-1.f, nn) * nrm) + w;
        const fv3 g1 = cross(v[2] - v[0], w), g2 = cross(w, v[1] - v[0]);
        const fv3 g = m == 0 ? -(g1 + g2) : (m == 1 ? g1 : g2);
        const float t = tot[a] + (a == 0 ? g.x : (a == 1 ? g.y : g.z)) + tot[6 + tid];
        if (vi[m] < 0 || vi[m] >= out.V) {
          atomicOr(sc.status, kStatusFaceIndexRange);
        } else if (out.vg) {
          atomicAdd(out.vg + b * out.vsb + vi[m] * out.vsv + a * out.vsc, t);
        }
      } else if (tid == 9 && out.mg) {
        const float t = tot[15] != 0.f ? xdiv(tot[15], s0r.w) : 0.f;
        for (int m = 0; m < 3; ++m)
          if (vi[m] >= 0 && vi[m] < out.V)
            atomicAdd(out.mg + b * out.msb + vi[m] * out.msv, (1.f / 3.f) * t);
      }
    }
    // the face's counts, records and sums have been read (a face that no scan point
    // sees has come here past one barrier only)
    __syncthreads();
  }
}

// The bins [w0, w1) of one output column in shared memory: bin b at h[(b - w0) CT].
template <int CT>
struct Window {
  float* h;
  int w0, w1;
  __device__ __forceinline__ int lo() const { return w0; }
  __device__ __forceinline__ int hi() const { return w1; }
  __device__ __forceinline__ bool in(int b) const { return b >= w0 && b < w1; }
  __device__ __forceinline__ void add(int b, float v) const { atomicAdd(h + (b - w0) * CT, v); }
};

// splat_tent with one sum per bin: the rising and the falling side over the
// bin's interval, relative to the tent's feet. Coordinates truncate toward zero:
// bin 0 reaches back to a corner in (-1, 0), and where the first foot is in a bin
// below 0 the sides are cut at 0, each if its peak is (splat_segment's terms).
template <int CT>
__device__ __forceinline__ void splat_tent_columns(const Window<CT>& w, float c0, float c1,
                                                   float c2, float alpha) {
  // (a NaN coordinate: a path length of NaN, in bin -1e9 as in bin_of's
  // -2147483647 on no transient)
  const int b0 = __float2int_rz(fminf(fmaxf(c0, -1.0e9f), 1.0e9f));
  const int b2 = __float2int_rz(fminf(fmaxf(c2, -1.0e9f), 1.0e9f));
  if (b0 >= w.w1 || b2 < w.w0) return;
  if (b0 == b2) {
    w.add(b0, alpha);
    return;
  }
  const float d1 = c1 - c0, d2 = c2 - c1, span = c2 - c0;
  // half slopes; a side narrower than 1e-12 bin has no area to speak of
  const float hs1 = d1 > 1e-12f ? vdiv(alpha, span * d1) : 0.f;
  const float hs2 = d2 > 1e-12f ? vdiv(-alpha, span * d2) : 0.f;
  const int first = max(b0, w.w0), last = min(b2, w.w1 - 1);
  const float e0 = (float)first;
  // the bin's lower edge from the feet, clamped to the sides
  const bool in1 = c1 > -1.f;  // the peak's bin is not below 0
  unsigned long long from =
      first > b0 && (b0 >= 0 || first > 0)
          ? f2pack(fminf(e0 - c0, d1), fminf(fmaxf(c2 - e0, 0.f), d2))
          : f2pack(b0 >= 0 ? 0.f : (in1 ? e0 - c0 : d1), in1 ? d2 : c2 - e0);
  const unsigned long long feet = f2pack(-c0, c2);
  unsigned long long edge = f2pack(e0, -e0);
  float* at = w.h + (first - w.w0) * CT;
  for (int i = first; i <= last; ++i, at += CT) {
    edge = f2add(edge, f2pack(1.f, -1.f));
    float t, u, up, down;
    f2unpack(f2add(edge, feet), t, u);
    const unsigned long long to = f2pack(fminf(t, d1), fminf(fmaxf(u, 0.f), d2));
    // (the falling side's difference is negative, and so is its half slope)
    f2unpack(f2mul(f2sub(to, from), f2add(to, from)), up, down);
    atomicAdd(at, fmaf(up, hs1, down * hs2));
    from = to;
  }
}

// What a face adds to every pair of one wall point p: the squared distances of its
// vertices and the point's factor of alpha, |n.r| r.z / |r|^4 with r = c - p.
__device__ __forceinline__ float4 splat_record(fv3 v0, fv3 v1, fv3 v2, fv3 c, fv3 n, fv3 p) {
  const fv3 r = c - p;
  const float rr = dot(r, r);
  const float a = r.z > 0.f ? vdiv(r.z * fabsf(dot(n, r)), rr * rr) : 0.f;
  return make_float4(xlen2(v0 - p), xlen2(v1 - p), xlen2(v2 - p), a);
}

// Forward over CT output columns (s, l) per CTA: column = s L + l, the order of the
// output's rows. A lane owns a column (with CT = 8, four lanes do), so the
// adds of a warp never meet in a word; a warp walks its 32-face chunks, prepares
// the faces that some column sees (vertices, centroid, normal, 100 rho / |n|) and,
// for tiles over at most two scan points, those points' records, one face per
// lane, and then takes the faces one by one with all lanes (four by four with CT =
// 8). The columns' bins are a window [w0, w0 + W) of the T, W rows of shared
// memory: where T > W the CTA first bounds each column's path lengths over the
// chunks it sees, and walks the faces again for every further W bins, but for the
// chunks that the window cannot hold.
// Instruction issue bounds it (72% of the slots at 26 warps per SM): of 8.8 ms for
// 20,000 faces x 400 x 144 points and 2,048 bins with 16 warps, the tents took 4.0
// (1.1 of it the compare-and-swap of a float add in shared memory), the laser
// records 1.9, the corners 0.9 and the rest 2.2), as it did the CTA per scan point
// and 4 lasers (10.3 ms), whose lanes met in the same bins and computed both
// points' lengths for every pair. 32 warps over one window of 1,024 bins (one CTA
// per SM) take 7.9 ms, as fewer columns need a second pass. The coordinates are
// exh_pair_filtered's, bit for bit; exact ones from a square root per length and
// a fixed division were 0.5 ms faster, but moved single bins by 1e-3.
constexpr int kColScan = 2;  // scan points with records prepared per face
constexpr int kColStage = 32 * (16 + 4 * kColScan);  // floats per warp
// kConfocal: a column is a scan point, its path twice one length (L = 1, lp unused).
// 20,480 faces x 4,096 points, 1,024 bins: 0.76 ms with blocks of 8 points whose
// lanes met in the same bins, 0.54 ms.
// kWindows: T > W.
template <int CT, int kColWarps, bool kConfocal, bool kWindows>
__global__ void __launch_bounds__(32 * kColWarps, 32 / kColWarps) splat_columns_kernel(
    Scene sc, View3f sp, View3f lp, Origins org, int S, int L, float* __restrict__ out, int T,
    float bw, float bo, FastBins fb, int W) {
  extern __shared__ float4 smem4[];
  __shared__ int range[2][CT];
  __shared__ float spts[kColScan][3];
  constexpr int G = 32 / CT;  // faces taken together
  const int b = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cl = lane & (CT - 1), grp = lane / CT;
  const int64_t C = (int64_t)S * L;
  const int64_t col0 = (int64_t)blockIdx.x * CT;
  const bool ok = col0 + cl < C;
  const int64_t col = ok ? col0 + cl : col0;
  const int s_first = (int)(col0 / L);
  const int s = (int)(col / L), l = (int)(col - (int64_t)s * L);
  // (CTA-uniform)
  const bool tab = !kConfocal && (int)((min(col0 + CT, C) - 1) / L) - s_first < kColScan;
  float4* stage = smem4 + warp * (kColStage / 4);
  float* hist = reinterpret_cast<float*>(smem4 + kColWarps * (kColStage / 4));
  const fv3 p = mkv(sp.at(b, s, 0), sp.at(b, s, 1), sp.at(b, s, 2));
  const fv3 q = kConfocal ? p : mkv(lp.at(b, l, 0), lp.at(b, l, 1), lp.at(b, l, 2));
  float od = origin_term(org, b, s, l, p, q);
  if (kConfocal) od = xmul(2.f, od);
  if (!kConfocal && threadIdx.x < kColScan) {
    const int si = min(s_first + (int)threadIdx.x, S - 1);
    for (int a = 0; a < 3; ++a) spts[threadIdx.x][a] = sp.at(b, si, a);
  }
  if (threadIdx.x < CT) {
    range[0][threadIdx.x] = T;
    range[1][threadIdx.x] = -1;
  }
  const int n = sc.meta[b].n;
  const int nchu = (n + 31) >> 5;
  const uint32_t* ms = sc.mask + ((size_t)b * sc.P + s) * sc.nch;
  const uint32_t* ml = sc.mask + ((size_t)b * sc.P + S + l) * sc.nch;
  const float4* shade = sc.shade + (size_t)b * sc.F * 4;
  auto seen = [&](int ch) {  // the column's faces of a chunk
    const uint32_t m = ok ? (kConfocal ? __ldg(ms + ch) : __ldg(ms + ch) & __ldg(ml + ch)) : 0u;
    return n - ch * 32 >= 32 ? m : m & ((1u << (n - ch * 32)) - 1u);
  };
  // The bins that the column's paths over a chunk can reach, [lo, hi] within [0, T)
  // (all lanes).
  auto reach = [&](int ch, int& lo, int& hi) {
    const int k = min(ch * 32 + lane, n - 1);
    const float4 s0r = __ldg(shade + 4 * k), s1r = __ldg(shade + 4 * k + 1);
    const float4 s2r = __ldg(shade + 4 * k + 2);
    // the chunk's box (a face with a NaN coordinate adds nothing)
    const float bx0 = warp_min_f(fminf(fminf(s0r.x, s1r.x), s2r.x));
    const float by0 = warp_min_f(fminf(fminf(s0r.y, s1r.y), s2r.y));
    const float bz0 = warp_min_f(fminf(fminf(s0r.z, s1r.z), s2r.z));
    const float bx1 = warp_max_f(fmaxf(fmaxf(s0r.x, s1r.x), s2r.x));
    const float by1 = warp_max_f(fmaxf(fmaxf(s0r.y, s1r.y), s2r.y));
    const float bz1 = warp_max_f(fmaxf(fmaxf(s0r.z, s1r.z), s2r.z));
    auto near = [&](fv3 o) {
      const float x = fmaxf(fmaxf(bx0 - o.x, o.x - bx1), 0.f);
      const float y = fmaxf(fmaxf(by0 - o.y, o.y - by1), 0.f);
      const float z = fmaxf(fmaxf(bz0 - o.z, o.z - bz1), 0.f);
      return sqrtf(fmaf(x, x, fmaf(y, y, z * z)));
    };
    auto far = [&](fv3 o) {
      const float x = fmaxf(bx1 - o.x, o.x - bx0), y = fmaxf(by1 - o.y, o.y - by0);
      const float z = fmaxf(bz1 - o.z, o.z - bz0);
      return sqrtf(fmaf(x, x, fmaf(y, y, z * z)));
    };
    // Each length and sum of the exact chain and of this one is within a few
    // roundings of its value: 4e-6 of the terms and two bins cover them.
    const float dn = near(p) + near(q), df = far(p) + far(q);
    const float inv_bw = fb.inv_bw;
    const float m = fmaf(4e-6f * inv_bw, df + od + fabsf(bo), 2.f);
    const float clo = (dn + od - bo) * inv_bw - m, chi = (df + od - bo) * inv_bw + m;
    // (NaN or infinite bounds: the whole range)
    lo = clo > 0.f ? (clo < (float)T ? (int)clo : T) : 0;
    hi = chi < (float)T ? (chi >= 0.f ? (int)chi : -1) : T - 1;
  };
  __syncthreads();
  int w0 = 0, passes = 1;
  if (kWindows) {
    int lo = T, hi = -1;
    for (int ch = warp; ch < nchu; ch += kColWarps) {
      const uint32_t bits = seen(ch);
      if (!__any_sync(0xffffffffu, bits != 0u)) continue;
      int clo, chi;
      reach(ch, clo, chi);
      if (bits == 0u) continue;
      lo = min(lo, clo);
      hi = max(hi, chi);
    }
    atomicMin(&range[0][cl], lo);
    atomicMax(&range[1][cl], hi);
    __syncthreads();
    for (int i = 0; i < CT; ++i) {
      const int bins = range[1][i] - range[0][i] + 1;
      passes = max(passes, (bins + W - 1) / W);
    }
    w0 = range[0][cl];
  }
  for (int pass = 0; pass < passes; ++pass, w0 += W) {
    for (int i = threadIdx.x; i < W * CT; i += blockDim.x) hist[i] = 0.f;
    __syncthreads();
    const Window<CT> win{hist + cl, w0, min(w0 + W, T)};
    for (int ch = warp; ch < nchu; ch += kColWarps) {
      uint32_t bits = seen(ch);
      uint32_t any = __reduce_or_sync(0xffffffffu, bits);
      if (any == 0u) continue;
      if (kWindows && passes > 1) {  // but for columns whose window the chunk cannot reach
        int clo, chi;
        reach(ch, clo, chi);
        if (chi < w0 || clo >= w0 + W) bits = 0u;
        any = __reduce_or_sync(0xffffffffu, bits);
        if (any == 0u) continue;
      }
      __syncwarp();  // the last chunk's stage has been read
      if ((any >> lane) & 1u) {
        const int k = ch * 32 + lane;
        const float4 s0r = __ldg(shade + 4 * k), s1r = __ldg(shade + 4 * k + 1);
        const float4 s2r = __ldg(shade + 4 * k + 2), s3r = __ldg(shade + 4 * k + 3);
        const fv3 v0 = mkv(s0r.x, s0r.y, s0r.z), v1 = mkv(s1r.x, s1r.y, s1r.z);
        const fv3 v2 = mkv(s2r.x, s2r.y, s2r.z), c = mkv(s3r.x, s3r.y, s3r.z);
        const fv3 nn = cross(v1 - v0, v2 - v0);
        stage[lane] = make_float4(v0.x, v0.y, v0.z, v1.x);
        stage[32 + lane] = make_float4(v1.y, v1.z, v2.x, v2.y);
        stage[64 + lane] = make_float4(v2.z, c.x, c.y, c.z);
        stage[96 + lane] = make_float4(nn.x, nn.y, nn.z, 100.f * s0r.w * rsqrtf(dot(nn, nn)));
        if (tab)
#pragma unroll
          for (int i = 0; i < kColScan; ++i)
            stage[128 + 32 * i + lane] =
                splat_record(v0, v1, v2, c, nn, mkv(spts[i][0], spts[i][1], spts[i][2]));
      }
      __syncwarp();
      while (any) {
        uint32_t mine = any;
        if (G > 1) {
#pragma unroll
          for (int i = 1; i < G; ++i) mine = grp >= i ? mine & (mine - 1u) : mine;
        }
        const int j = __ffs(mine) - 1;
#pragma unroll
        for (int i = 0; i < G; ++i) any &= any - 1u;
        if (j < 0 || !((bits >> j) & 1u)) continue;
        const float4 a0 = stage[j], a1 = stage[32 + j], a2 = stage[64 + j], a3 = stage[96 + j];
        const fv3 v0 = mkv(a0.x, a0.y, a0.z), v1 = mkv(a0.w, a1.x, a1.y);
        const fv3 v2 = mkv(a1.z, a1.w, a2.x), c = mkv(a2.y, a2.z, a2.w);
        const fv3 nn = mkv(a3.x, a3.y, a3.z);
        const float4 rl = splat_record(v0, v1, v2, c, nn, q);
        const float4 rs = kConfocal ? rl
                          : tab     ? stage[128 + 32 * (s - s_first) + j]
                                    : splat_record(v0, v1, v2, c, nn, p);
        const float alpha = rs.w * rl.w * a3.w;
        if (!(alpha > 0.f)) continue;
        // exh_pair_filtered's (confocal_pair_filtered's) coordinates and tests, on the
        // sorted lengths alone (the sum of two lengths contracted as there; NaN for a
        // length of zero)
        auto sum = [](float ds2, float dl2) {
          const float dl = dl2 * rsqrt_approx(dl2);
          return kConfocal ? dl : fmaf(ds2, rsqrt_approx(ds2), dl);
        };
        float d[3] = {sum(rs.x, rl.x), sum(rs.y, rl.y), sum(rs.z, rl.z)}, c3[3];
        auto sort = [&]() {
          const float m01 = fminf(d[0], d[1]), x01 = fmaxf(d[0], d[1]), m12 = fminf(x01, d[2]);
          d[2] = fmaxf(x01, d[2]);
          d[0] = fminf(m01, m12);
          d[1] = fmaxf(m01, m12);
        };
        sort();
        const float u = 5.9604645e-8f;
        bool sure = d[1] - d[0] > 16.f * u * d[2] && d[2] - d[1] > 16.f * u * d[2];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float x = kConfocal ? fmaf(2.f, d[k], od) : d[k] + od;
          const float cc = fmaf(x, fb.inv_bw, fb.nbo);
          const float m = fmaf(fb.kc, x, fb.kb) + 8.f * u * fabsf(cc);
          sure = sure && fabsf(cc - rintf(cc)) > m && fabsf(cc) < 1.0e9f;
          c3[k] = cc;
        }
        if (!sure) {
          auto both = [&](fv3 v) {
            const float dl = xlen(xsub3(v, q));
            return kConfocal ? xmul(2.f, dl) : xadd(xlen(xsub3(v, p)), dl);
          };
          d[0] = both(v0);
          d[1] = both(v1);
          d[2] = both(v2);
          sort();
#pragma unroll
          for (int k = 0; k < 3; ++k) c3[k] = xdiv(xsub(xadd(d[k], od), bo), bw);
        }
        splat_tent_columns<CT>(win, c3[0], c3[1], c3[2], alpha);
      }
    }
    __syncthreads();
    // rows out[b][t][col0 .. col0 + CT): a pass writes its window, the first
    // one also what lies before, the last one what lies after
    if (ok) {
      float* ob = out + (size_t)b * T * C + col;
      const int ta = pass == 0 ? 0 : w0, tb = pass == passes - 1 ? T : min(w0 + W, T);
      for (int t = warp * G + grp; t < T; t += kColWarps * G) {
        if (t < ta || t >= tb) continue;
        ob[(size_t)t * C] = win.in(t) ? hist[(t - w0) * CT + cl] : 0.f;
      }
    }
    __syncthreads();
  }
}

template <int CT, int kColWarps, bool kConfocal>
static int launch_columns(const Scene& sc, const View3f& sp, const View3f& lp,
                          const Origins& org, int S, int L, float* out, int T, float bw, float bo,
                          int W, cudaStream_t stream) {
  const FastBins fast = make_fast_bins(
      bw, bo, tune::get(kConfocal ? "mesh.confocal.exact" : "mesh.exhaustive.exact") != 1);
  const size_t smem = sizeof(float) * ((size_t)kColWarps * kColStage + (size_t)W * CT);
  const dim3 grid((unsigned)ceil_div((int64_t)S * L, CT), (unsigned)sc.B);
  auto* kern = T > W ? splat_columns_kernel<CT, kColWarps, kConfocal, true>
                     : splat_columns_kernel<CT, kColWarps, kConfocal, false>;
  TOTRI_CUDA(tune::ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem));
  TOTRI_KERNEL(kConfocal ? "mesh confocal splat" : "mesh exhaustive splat", stream,
               kern<<<grid, 32 * kColWarps, smem, stream>>>(sc, sp, lp, org, S, L, out, T, bw, bo,
                                                            fast, W));
  return TOTRI_OK;
}

template <int LT>
static int launch_exh_splat(const Scene& sc, const View3f& sp, const View3f& lp,
                            const Origins& org, int S, int L, float* out, int T, float bw,
                            float bo, cudaStream_t stream) {
  const FastBins fast = make_fast_bins(bw, bo, tune::get("mesh.exhaustive.exact") != 1);
  const size_t smem = sizeof(float) * (size_t)T * LT;
  const dim3 grid((unsigned)S, (unsigned)ceil_div(L, LT), (unsigned)sc.B);
  // Per-thread mask tests by default: on the 32-mesh batch (2048 bins, 64x64
  // detector x 16x16 laser points) they took 4.4 s against 4.9 s for the
  // compacted variant, which "mesh.exhaustive.splat.mode" = 1 selects.
  if (tune::get("mesh.exhaustive.splat.mode") != 1) {
    // Tiles narrower than a 32-byte sector flush through a cluster of
    // 8 / LT tiles ("mesh.exhaustive.splat.cluster" = 1: each tile alone).
    constexpr int CL = LT < 8 ? 8 / LT : 1;
    if (CL > 1 && tune::get("mesh.exhaustive.splat.cluster") != 1) {
      const bool capped = tune::get("mesh.exhaustive.splat.occupancy") != 1;
      auto* kern = capped ? exh_splat_kernel<LT, 5, CL> : exh_splat_kernel<LT, 1, CL>;
      TOTRI_CUDA(tune::ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem));
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(grid.x, (unsigned)(ceil_div(grid.y, CL) * CL), grid.z);
      cfg.blockDim = dim3(256);
      cfg.dynamicSmemBytes = smem;
      cfg.stream = stream;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 1;
      attr[0].val.clusterDim.y = CL;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      cudaError_t le = cudaSuccess;
      TOTRI_KERNEL("mesh exhaustive splat", stream,
                   le = cudaLaunchKernelEx(&cfg, kern, sc, sp, lp, org, S, L, out, T, bw, bo,
                                           fast));
      TOTRI_CUDA(le);
      return TOTRI_OK;
    }
    // Registers capped for 5 CTAs per SM (48, no spills): 36.5 ms against
    // 38.1 ms uncapped (58 registers; "mesh.exhaustive.splat.occupancy" = 1)
    // on one 20k-face mesh, 32x32 x 16x16 points, 2,048 bins.
    if (tune::get("mesh.exhaustive.splat.occupancy") != 1) {
      TOTRI_CUDA(tune::ensure_dynamic_smem(
          reinterpret_cast<const void*>(exh_splat_kernel<LT, 5>), smem));
      TOTRI_KERNEL("mesh exhaustive splat", stream,
                   (exh_splat_kernel<LT, 5><<<grid, 256, smem, stream>>>(
                       sc, sp, lp, org, S, L, out, T, bw, bo, fast)));
      return TOTRI_OK;
    }
    TOTRI_CUDA(tune::ensure_dynamic_smem(
        reinterpret_cast<const void*>(exh_splat_kernel<LT>), smem));
    TOTRI_KERNEL("mesh exhaustive splat", stream,
                 exh_splat_kernel<LT><<<grid, 256, smem, stream>>>(sc, sp, lp, org, S, L, out, T,
                                                                   bw, bo, fast));
    return TOTRI_OK;
  }
  TOTRI_CUDA(tune::ensure_dynamic_smem(
      reinterpret_cast<const void*>(exh_splat_compact_kernel<LT>), smem));
  TOTRI_KERNEL("mesh exhaustive splat", stream,
               exh_splat_compact_kernel<LT><<<grid, 256, smem, stream>>>(
                   sc, sp, lp, org, S, L, out, T, bw, bo, fast));
  return TOTRI_OK;
}

// The tile's kernel: windows of W bins (0: as many as fit, two CTAs per SM up to 496
// bins of 32 columns, else 32 warps over one window).
template <bool kConfocal>
static int launch_tile(int ct, const Scene& sc, const View3f& sp, const View3f& lp,
                       const Origins& org, int S, int L, float* out, int T, float bw, float bo,
                       int W, cudaStream_t stream) {
  if (W <= 0) W = ct == 32 ? (T <= 496 ? 496 : 1024) : 1984;
  const bool full = W > 496;
  W = std::min(W, T);
  if (ct == 32 && full)
    return launch_columns<32, 32, kConfocal>(sc, sp, lp, org, S, L, out, T, bw, bo, W, stream);
  if (ct == 32)
    return launch_columns<32, 16, kConfocal>(sc, sp, lp, org, S, L, out, T, bw, bo, W, stream);
  if (ct == 8)
    return launch_columns<8, 16, kConfocal>(sc, sp, lp, org, S, L, out, T, bw, bo, W, stream);
  return fail(TOTRI_ERR_INVALID_ARGUMENT, "column tile must be 8 or 32");
}

int launch_confocal_columns(const Scene& sc, const View3f& sp, const View3f& so, int has_origin,
                            int ct, float* transient, int T, int S, float bw, float bo,
                            cudaStream_t stream) {
  return launch_tile<true>(ct, sc, sp, sp, Origins{so, so, has_origin, 0}, S, 1, transient, T, bw,
                           bo, tune::get("mesh.confocal.splat.window"), stream);
}

int launch_exhaustive_splat(const Scene& sc, const View3f& sp, const View3f& lp,
                            const Origins& org, int S, int L, float* out, int T, float bw,
                            float bo, cudaStream_t stream) {
  const size_t budget = 200 * 1024;
  const int want = tune::get("mesh.exhaustive.splat.lt");
  if (want > 0) {
    if ((size_t)T * want * 4 > budget)
      return fail(TOTRI_ERR_INVALID_ARGUMENT, "tuned laser tile too large for the bin count");
    switch (want) {
      case 1: return launch_exh_splat<1>(sc, sp, lp, org, S, L, out, T, bw, bo, stream);
      case 4: return launch_exh_splat<4>(sc, sp, lp, org, S, L, out, T, bw, bo, stream);
      case 8: return launch_exh_splat<8>(sc, sp, lp, org, S, L, out, T, bw, bo, stream);
      case 16: return launch_exh_splat<16>(sc, sp, lp, org, S, L, out, T, bw, bo, stream);
      case 32: return launch_exh_splat<32>(sc, sp, lp, org, S, L, out, T, bw, bo, stream);
      default: return fail(TOTRI_ERR_INVALID_ARGUMENT, "laser tile must be 1, 4, 8, 16 or 32");
    }
  }
  // Columns (splat_columns_kernel) from 1,024 columns on (ms, the tiles below against 8
  // and 32 columns; 400 x 144, 64 x 144, 169 x 36 and 64 x 16 points):
  //   20,000 faces, 1,024 bins  8.30 / 6.85 / 5.86   1.68 / 1.21 / 1.07
  //                             1.39 / 0.94 / 1.18   0.68 / 0.30 / 0.83
  //   20,000 faces, 2,048 bins 10.27 / 9.31 / 7.80   1.88 / 1.66 / 1.44
  //                             1.61 / 1.26 / 1.87   0.52 / 0.41 / 1.32
  //                3,072 bins  13.70 /11.43 / 9.69   2.48 / 2.07 / 1.78
  //                             2.03 / 1.64 / 1.88   0.64 / 0.54 / 0.98
  //                4,096 bins  18.98 /13.38 /14.42   3.34 / 2.43 / 2.63
  //                             2.76 / 1.91 / 2.81   0.73 / 0.63 / 1.45
  //                6,000 bins  31.98 /16.88 /18.02   5.49 / 3.08 / 3.25
  //   5,000 faces, 1,024 bins   2.61 / 2.60 / 2.26   0.54 / 0.47 / 0.44
  //                             0.45 / 0.37 / 0.43   0.23 / 0.13 / 0.34
  //                3,072 bins   5.39 / 5.31 / 4.65   0.99 / 0.97 / 0.91
  //                4,096 bins   7.87 / 6.48 / 6.72   1.40 / 1.19 / 1.31
  //   1,500 faces, 1,024 bins   1.08 / 1.43 / 1.16   0.24 / 0.27 / 0.25
  //                             0.19 / 0.21 / 0.25   0.12 / 0.09 / 0.22
  //                4,096 bins   4.36 / 3.62 / 4.30   0.79 / 0.66 / 0.79
  //   500 faces, 1,024 bins     0.58 / 0.92 / 0.65   0.13 / 0.17 / 0.14
  //                             0.10 / 0.13 / 0.15   0.06 / 0.05 / 0.12
  //                3,072 bins   1.97 / 2.23 / 2.81   0.37 / 0.41 / 0.55
  //                4,096 bins   3.12 / 2.83 / 3.62   0.56 / 0.51 / 0.69
  // These are spheres, whose paths span 0.6 m of 5.12; a mesh that spans more than a
  // window needs more passes over its faces, each over the chunks that its window
  // reaches (20,000 faces that span 3 m, 400 x 144 points: 10.21 / 10.15 / 9.46 at 2,048
  // bins, 14.2 / 12.9 / 13.4 at 3,072, 20.5 / 16.5 / 17.0 at 4,096; 5,000 faces 4.18 / 4.94
  // / 4.95, 6.2 / 6.7 / 7.7 and 9.4 / 8.8 / 10.4). Hence above 2,048 bins only meshes of
  // 12,288 faces, and from 4,096 bins on, where the tiles are one or two lasers wide,
  // 8 columns from 1,500 faces. Small meshes spend the time on the rows, not on the
  // faces: they take 8 columns only where the tiles leave SMs idle (up to 16 columns
  // per SM and 1,024 bins, or 48 with two faces per bin: 0.16 against 0.15 ms for 1,500
  // faces, 512 bins, 169 x 36 points). A window of 496 bins leaves room for two CTAs per
  // SM.
  // "mesh.exhaustive.splat.columns" = 1 turns the kernel off, 8 and 32 select a
  // tile, ".window" its bins.
  const int cols = tune::get("mesh.exhaustive.splat.columns");
  // Its sides and windows run forwards in time: the tiles take negative bin widths.
  if (cols != 1 && bw > 0.f && tune::get("mesh.exhaustive.splat.mode") != 1 &&
      (size_t)T * 4 <= budget) {
    const int64_t all = (int64_t)S * L * sc.B;
    const int sms = tune::sm_count();
    const bool many = sc.F >= (T <= 2048 ? 4096 : 12288);
    const bool few = all <= 16 * sms && T <= 1024;
    const bool middling = all <= 48 * sms && sc.F >= 2 * T;
    const bool rows = T >= 4096 && sc.F >= 1500;
    const int ct = cols > 1 ? cols
                   : all < 1024 || !(many || few || middling || rows) ? 0
                   : many && !rows && all >= 48 * sms                 ? 32
                                                                      : 8;
    const int W = tune::get("mesh.exhaustive.splat.window");
    if (ct != 0) return launch_tile<false>(ct, sc, sp, lp, org, S, L, out, T, bw, bo, W, stream);
  }
  // Built-in choice: the widest laser tile whose histogram stays within 40 KB,
  // so several CTAs share an SM (2048 bins x 64x64 x 16x16, 32 meshes: 4.4 s
  // with 4 lasers per tile, 12.7 s with 16, whose 128 KB tile leaves one CTA
  // per SM).
  const size_t kTileBytes = 40 * 1024;
  if ((size_t)T * 16 * 4 <= kTileBytes && L >= 16)
    return launch_exh_splat<16>(sc, sp, lp, org, S, L, out, T, bw, bo, stream);
  if ((size_t)T * 8 * 4 <= kTileBytes && L >= 8)
    return launch_exh_splat<8>(sc, sp, lp, org, S, L, out, T, bw, bo, stream);
  if ((size_t)T * 4 * 4 <= budget && L >= 4)
    return launch_exh_splat<4>(sc, sp, lp, org, S, L, out, T, bw, bo, stream);
  if ((size_t)T * 4 <= budget)
    return launch_exh_splat<1>(sc, sp, lp, org, S, L, out, T, bw, bo, stream);
  return fail(TOTRI_ERR_UNSUPPORTED, "number of bins too large for the shared-memory tile");
}

// out[c Tp + t] = in[t row + c] for c < n, t < T: a [T][n] block of rows of
// length `row` into bins-last order (rows of Tp >= T), through 32 x 32 tiles in shared memory
// (coalesced reads and writes).
__global__ void __launch_bounds__(256) bins_last_kernel(const float* __restrict__ in,
                                                        float* __restrict__ out, int T, int Tp,
                                                        int64_t row, int64_t n) {
  __shared__ float tile[32][33];
  const int64_t c0 = (int64_t)blockIdx.x * 32;
  const int t0 = blockIdx.y * 32;
  const float* src = in;
  float* dst = out;
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int t = t0 + r;
    const int64_t c = c0 + threadIdx.x;
    tile[r][threadIdx.x] = (t < T && c < n) ? src[(int64_t)t * row + c] : 0.f;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int64_t c = c0 + r;
    const int t = t0 + threadIdx.x;
    if (t < T && c < n) dst[c * Tp + t] = tile[threadIdx.x][r];
  }
}

int launch_bins_last(const float* in, float* out, int T, int Tp, int64_t row, int64_t n,
                     cudaStream_t stream) {
  constexpr int kBins = 65535 * 32;  // a grid has 65,535 rows of tiles
  for (int64_t t0 = 0; t0 < T; t0 += kBins) {
    const int bins = (int)std::min<int64_t>(T - t0, kBins);
    TOTRI_KERNEL("mesh grad layout", stream,
                 bins_last_kernel<<<dim3((unsigned)ceil_div(n, 32), (unsigned)ceil_div(bins, 32)),
                                    dim3(32, 8), 0, stream>>>(in + t0 * row, out + t0, bins, Tp,
                                                              row, n));
  }
  return TOTRI_OK;
}

int64_t exh_grad_chunk_points(int64_t S, int64_t L, int64_t T) {
  if (S <= 0 || L <= 0 || T <= 0) return 0;
  int64_t c = (int64_t)(kGradChunkBytes / ((size_t)L * (size_t)T * sizeof(float)));
  if (c <= 0) return 0;
  if (c >= S) return S;
  return c >= kFaceSlice ? c / kFaceSlice * kFaceSlice : c;
}

size_t exh_grad_scratch_bytes(int64_t S, int64_t L, int64_t T) {
  const int64_t c = exh_grad_chunk_points(S, L, T);
  return c > 0 ? align_up((size_t)c * (size_t)L * (size_t)T * sizeof(float), 256) : 0;
}

PairPlan pair_plan(int64_t S, int64_t L, int64_t T, int64_t voxels, int64_t blocks, int64_t ctas,
                   int64_t least, bool copies, size_t ws_bytes) {
  PairPlan p{};
  p.chunk = copies ? exh_grad_chunk_points(S, L, T) : 0;
  size_t copy = (size_t)p.chunk * (size_t)L * (size_t)T * sizeof(float);
  if (copy > ws_bytes) p.chunk = 0, copy = 0;
  p.part_at = align_up(copy, 256);
  p.step = p.chunk > 0 ? p.chunk : S;
  const int64_t volume = voxels * (int64_t)sizeof(float);
  const int64_t room = ws_bytes > p.part_at && volume > 0
                           ? (int64_t)((ws_bytes - p.part_at) / (size_t)volume) : 0;
  const int64_t slices = std::max<int64_t>(
      1, std::min({ceil_div(ctas, blocks), p.step / least, room}));
  p.per = (int)ceil_div(p.step, slices);
  p.slices = (int)ceil_div(p.step, p.per);
  p.bytes = p.slices > 1 ? p.part_at + (size_t)(p.slices * volume) : copy;
  return p;
}

__global__ void __launch_bounds__(256) sum_slices_kernel(const float* __restrict__ part, int slices,
                                                         int64_t n, float* __restrict__ out,
                                                         int add) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float sum = add ? out[i] : 0.f;
  for (int s = 0; s < slices; ++s) sum += __ldg(part + s * n + i);
  out[i] = sum;
}

int launch_sum_slices(const float* part, int slices, int64_t n, float* out, bool add,
                      cudaStream_t stream) {
  TOTRI_KERNEL("sum of slices", stream,
               sum_slices_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, stream>>>(
                   part, slices, n, out, add));
  return TOTRI_OK;
}

// The mesh gradient's copies have rows of a multiple of 4 bins.
static int64_t padded_bins(int64_t T) { return (T + 3) & ~(int64_t)3; }
size_t mesh_grad_scratch_bytes(int64_t S, int64_t L, int64_t T) {
  return exh_grad_scratch_bytes(S, L, padded_bins(T));
}

int launch_exhaustive_grad(const Scene& sc, const View3f& sp, const View3f& lp,
                           const Origins& org, int S, int L, const float* tgrad, int T, float bw,
                           float bo, const GradOut& out, void* scratch, size_t scratch_bytes,
                           cudaStream_t stream) {
  const FastBins fast = make_fast_bins(bw, bo, tune::get("mesh.exhaustive.exact") != 1);
  // At most 512 scan points per CTA: a warp walks one face over its slice and
  // then the next face over the same slice, re-reading the same transient_grad
  // rows (slice x L x the chunk's bins), which then stay in L2 (one 20k-face
  // mesh, 1024 x 256 wall points: 92 ms with 512-point slices, 139 ms with
  // 2048).
  constexpr int kMaxSlice = 512;
  const int split =
      tune::grad_split("mesh.exhaustive.grad.split", (int64_t)sc.nch * sc.B, S, kMaxSlice);
  const int64_t slice = ceil_div(S, split);
  // Separable point records (exh_grad_face_kernel) by default;
  // "mesh.exhaustive.grad.mode" = 1 selects per-lane mask tests and 2 the
  // compacted triples (14.7 s against 17.7 s for per-lane mask tests on the
  // 32-mesh batch).
  const int mode = tune::get("mesh.exhaustive.grad.mode");
  if (mode != 1 && mode != 2) {
    // "mesh.exhaustive.grad.faces": faces per CTA (default 1: within 2% of 2 and 8
    // on 20,000 faces, 1.8 to 5 times faster than 8 on 500 and 1,500);
    // "mesh.exhaustive.grad.occupancy" = 4: registers capped for 4 CTAs per SM
    // (64, with spills) instead of 3 (80); "mesh.exhaustive.grad.sslice" /
    // ".lchunk": scan points / lasers per CTA.
    int fpc = tune::get("mesh.exhaustive.grad.faces");
    if (fpc <= 0) fpc = kFacesPerCta;
    const int fixed = fixed_division(bw, bo);
    const bool occ4 = tune::get("mesh.exhaustive.grad.occupancy") == 4;
    const size_t smem = sizeof(float) * 2 * kRec * kFaceSlice;
    auto launch = [&](const float* tg, int lchunk, int sslice, int b0, int nb, int sa, int sb,
                      int64_t bstride, int64_t cstep, int64_t bstep, bool last) -> int {
      const dim3 grid((unsigned)ceil_div(sc.F, fpc), (unsigned)nb,
                      (unsigned)(ceil_div(sb - sa, sslice) * ceil_div(L, lchunk)));
      auto* kern = last ? (occ4 ? exh_grad_face_kernel<4, true, true>
                                : exh_grad_face_kernel<3, true, true>)
                        : (occ4 ? exh_grad_face_kernel<4, false, true>
                                : exh_grad_face_kernel<3, false, true>);
      if (!(bw > 0.f))
        kern = last ? exh_grad_face_kernel<3, true, false> : exh_grad_face_kernel<3, false, false>;
      TOTRI_CUDA(tune::ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem));
      TOTRI_KERNEL("mesh exhaustive grad", stream,
                   kern<<<grid, 256, smem, stream>>>(sc, sp, lp, org, S, L, tg, T, bw, bo, fixed,
                                                     out, fpc, lchunk, sslice, b0, sa, sb, bstride,
                                                     cstep, bstep));
      return TOTRI_OK;
    };
    int lchunk = tune::get("mesh.exhaustive.grad.lchunk");
    int sslice = tune::get("mesh.exhaustive.grad.sslice");
    // Bins-last copies. A triple reads a few consecutive bins of its (s, l)
    // column; in the caller's [T, S, L] order they lie S L floats apart, one
    // L2 sector each, read one after another. When the workspace holds the
    // scratch (totri_mesh_exhaustive_grad_scratch), each item's transient_grad
    // is copied, one range of scan points at a time, into [s][l][t] order,
    // where those bins share one or two sectors: one 20k-face mesh, 2,048
    // bins, 16x16 laser points: 333 -> 189 ms at 64x64 scan points, 54.2 ->
    // 51.0 ms at 32x32 (copies included), with whole 256 x 256 tiles.
    // "mesh.exhaustive.grad.layout" = 2 reads transient_grad in place;
    // "mesh.exhaustive.grad.chunk" caps the scan points per copy.
    int64_t cpts = exh_grad_chunk_points(S, L, padded_bins(T));
    const int64_t cap = tune::get("mesh.exhaustive.grad.chunk");
    if (cap > 0) cpts = std::min(cpts, cap);
    if (tune::get("mesh.exhaustive.grad.layout") != 2 && cpts > 0 && scratch &&
        scratch_bytes >= (size_t)cpts * L * padded_bins(T) * sizeof(float)) {
      if (lchunk <= 0 || lchunk > kFaceSlice) lchunk = kFaceSlice;
      if (sslice <= 0 || sslice > kFaceSlice) sslice = kFaceSlice;
      sslice = (int)std::min<int64_t>(sslice, cpts);
      float* copy = static_cast<float*>(scratch);
      const int64_t row = (int64_t)S * L, Tp = padded_bins(T);
      for (int b = 0; b < sc.B; ++b)
        for (int64_t sa = 0; sa < S; sa += cpts) {
          const int64_t sb = std::min<int64_t>(S, sa + cpts), n = (sb - sa) * L;
          TOTRI_TRY(launch_bins_last(tgrad + ((int64_t)b * T) * row + sa * L, copy, T, (int)Tp, row, n,
                                     stream));
          TOTRI_TRY(launch(copy, lchunk, sslice, b, 1, (int)sa, (int)sb, 0, Tp, 1, true));
        }
      return TOTRI_OK;
    }
    // In place: each CTA takes `sslice` scan points and `lchunk` lasers,
    // faces varying fastest over the grid, so the CTAs that run together
    // read the transient_grad rows of one (scan slice, laser chunk). When a
    // bin row of transient_grad (S L floats) reaches 2 MB the per-pair cost
    // grows (one 20k-face mesh, 2,048 bins: 0.23 ms per thousand pairs at
    // 64x64 x 8x8 points, 0.36 at 64x64 x 16x16), and 128 scan points by 32
    // lasers per CTA recover part of it (378 -> 331 ms at 64x64 x 16x16; at
    // 32x32 x 16x16 whole 256 x 256 tiles stay faster, 54.8 against 58.5 ms).
    const bool wide_rows = (int64_t)S * L >= (int64_t)1 << 19;
    if (lchunk <= 0 || lchunk > kFaceSlice) lchunk = wide_rows ? 32 : kFaceSlice;
    if (sslice <= 0 || sslice > kFaceSlice) sslice = wide_rows ? 128 : kFaceSlice;
    return launch(tgrad, lchunk, sslice, 0, sc.B, 0, S, (int64_t)T * S * L, 1, (int64_t)S * L,
                  false);
  }
  if (mode == 1) {
    const size_t smem = sizeof(uint32_t) * (size_t)(S + L);
    if (smem > 200 * 1024)
      return fail(TOTRI_ERR_UNSUPPORTED, "too many wall points for one tile");
    TOTRI_CUDA(tune::ensure_dynamic_smem(
        reinterpret_cast<const void*>(exh_grad_kernel), smem));
    const dim3 grid((unsigned)sc.nch, (unsigned)sc.B, (unsigned)split);
    TOTRI_KERNEL("mesh exhaustive grad", stream,
                 exh_grad_kernel<<<grid, 256, smem, stream>>>(sc, sp, lp, org, S, L, tgrad, T,
                                                              bw, bo, fast, out));
    return TOTRI_OK;
  }
  const size_t smem = sizeof(uint32_t) * (size_t)(slice + 32 * ceil_div(L, 32));
  if (smem > 180 * 1024) return fail(TOTRI_ERR_UNSUPPORTED, "too many laser points for one tile");
  TOTRI_CUDA(tune::ensure_dynamic_smem(
      reinterpret_cast<const void*>(exh_grad_compact_kernel), smem));
  // (three CTAs per SM at 80 registers spills and runs 6% slower: 93.5 ms
  // against 87.8 ms on one 20k-face mesh; CTAs of 5 or 6 warps capped at 96
  // registers for 4 or 3 CTAs per SM spill and took 98 and 95 ms against
  // 69 ms for this kernel on that mesh)
  const dim3 grid((unsigned)sc.nch, (unsigned)sc.B, (unsigned)split);
  TOTRI_KERNEL("mesh exhaustive grad", stream,
               exh_grad_compact_kernel<<<grid, 256, smem, stream>>>(
                   sc, sp, lp, org, S, L, tgrad, T, bw, bo, fast, out));
  return TOTRI_OK;
}

}  // namespace mesh
}  // namespace totri
