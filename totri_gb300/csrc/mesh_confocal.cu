// Confocal mesh transient rendering: visibility masks, forward splat and the
// vertex / albedo gradient.
//
// Reference: src/render/program/mesh_confocal_forward_optix.cu:18-129 and
// mesh_confocal_grad_verts_optix.cu:18-190 (one OptiX thread per
// (face, scan point) with global atomics into transient[b][bin][s] and into
// verts_grad). Here:
//  * visibility runs once per (scan point, face) into a bit mask
//    [B][P][ceil(F/32)] (one warp per 32 Morton-ordered faces of a point);
//  * the forward gives each CTA a tile of TS scan points and walks all faces,
//    splatting into a shared-memory histogram [T][TS] with shared atomics, and
//    flushes the tile with coalesced float4 stores (no global atomics, no
//    separate zero fill);
//  * the gradient gives each CTA one 32-face mask word and a slice of the scan
//    points (lanes over s, so transient_grad reads are row-coalesced; slices
//    keep every SM busy when there are few faces), keeps
//    the per-face gradient in registers, reduces it across the warp and issues
//    12 atomics per face instead of 9 + 3M per visible pair.
#include <algorithm>
#include <cmath>

#include "mesh.cuh"
#include "mesh_kernels.cuh"
#include "tune.cuh"

namespace totri {
namespace mesh {

namespace {

// One warp per (wall point, 32 Morton-consecutive faces): the 32 rays share
// their origin and end on a compact patch of the surface, so they walk
// largely the same BVH nodes. kVisRayPostponed lets each lane
// walk alone with its triangle tests postponed until the warp runs them
// together (target_visible_pp; 22.8 ms against 27.0 ms for kVisRay, the plain
// per-lane walk target_visible, on the 20,480-face sphere seen from a 64x64
// wall), kVisPacket walks the 32 rays as one warp packet (packet_visible;
// about twice the node visits there), kVisBrute tests every face; all four
// give the same bits. The patch kernels (one CTA per 32 Morton-consecutive
// wall points and up to 8 chunks of 32 faces) walk per lane after the
// seeded surface walk (kVisPatch, the default), as a packet, over the 4-wide
// tree, or (kVisPatchShaft) gather one candidate list per target with a
// warp-wide walk of the hull of the warp's wall points and the target's hit
// box and test it per lane: 9.7 ms against 8.5 ms for kVisPatch on the
// 20,480-face workload. The lanes of a warp already share the top of their
// walks in SIMT, and near the target a lane's own slab tests prune finer
// than one hull does.
constexpr int kVisBrute = 0;
constexpr int kVisRay = 1;
constexpr int kVisPacket = 2;
constexpr int kVisRayPostponed = 3;
constexpr int kVisPatch = 4;
constexpr int kVisPatchPacket = 5;
constexpr int kVisPatchWide = 6;
constexpr int kVisPatchShaft = 7;
constexpr int kShaftFrontier = 128;
constexpr int kShaftCand = 128;

template <int kMode>
__global__ void __launch_bounds__(256) visibility_kernel(Scene sc, View3f pts, int P, int row0) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t per_b = (int64_t)P * sc.nch;
  if (gw >= per_b * sc.B) return;  // whole warp
  const int b = (int)(gw / per_b);
  const int64_t rem = gw - (int64_t)b * per_b;
  const int p = (int)(rem / sc.nch);
  const int ch = (int)(rem - (int64_t)p * sc.nch);
  const int n = sc.meta[b].n;
  const int k = ch * 32 + lane;
  const fv3 o = mkv(pts.at(b, p, 0), pts.at(b, p, 1), pts.at(b, p, 2));
  bool vis = false;
  if (kMode == kVisPacket) {
    if (ch * 32 < n) {  // warp-uniform
      Target tg{};
      tg.k = k;
      if (k < n) tg = load_target(sc, b, k);
      vis = packet_visible(sc, b, n, k < n, tg, o, sc.status);
    }
  } else if (kMode == kVisRayPostponed) {
    int seed = -1;
    if (k < n) vis = target_visible_pp(sc, b, n, load_target(sc, b, k), o, sc.status, seed,
                                       kSeedOff, 0);
  } else if (k < n) {
    int cache = -1;
    vis = target_visible<kMode == kVisBrute>(sc, b, n, load_target(sc, b, k), o, cache,
                                             sc.status);
  }
  const uint32_t word = __ballot_sync(0xffffffffu, vis);
  if (lane == 0) sc.mask[((size_t)b * sc.P + row0 + p) * sc.nch + ch] = word;
}

// One CTA per (block of 32 wall points in their order, run of `chunks`
// 32-face chunks): each warp takes one face of the run at a time and its 32
// lanes cast the rays from the 32 points, which lie on a compact patch of
// the wall and end on the same centroid, so the lanes walk nearly the same BVH
// nodes (lockstep model on the 20,480-face sphere: 12% fewer warp iterations
// and 8.3 -> 5.7 distinct nodes per iteration against point-major warps;
// measured 15.3 ms against 22.6 ms for point-major warps with the same
// postponed-leaf walk). The eight warps of a CTA work on neighbouring faces
// from the same points, so they share their BVH nodes in L1 (a variant
// without the CTA, one warp per 32 x 32 block, took 23.2 ms).
//
// With the binary walk (kWalk 0) each point keeps a seed in shared memory: the
// last occluder any warp of the CTA found for it. Faces of neighbouring Morton
// positions are close on the surface, and so are the faces that hide them from
// one wall point, so a short surface walk from the seed (surface_walk) settles
// most hidden targets without a BVH walk. A CTA starts from the seeds that
// earlier CTAs of the same points left in global memory (the first quarter of
// the point scratch, -1 after the point sort) and leaves its own there. Seeds
// are read and written without synchronisation, as any face is a valid (if
// slower) start. The bits of every chunk are transposed in shared memory into
// one mask word per point and chunk. This is the default visibility kernel.
constexpr int kMaxPatchChunks = 16;

// The wall-point sets of one launch: blocks of 32 points, set 0 in blocks
// [0, blocks0), set 1 (if any) after them.
struct Walls {
  View3f pts0, pts1;
  int P0, P1, row0, row1;
  unsigned blocks0;
};

// kWalk 0: target_visible_pp, 1: packet_visible, 2: target_visible_pp4, 3: shaft
// search, 4: target_visible_pp's prefix and a 4-wide BVH search
// (bvh_occluded_wide); kOcc: CTAs per SM that the register allocation must allow.
template <int kWalk, int kOcc = 1, int kWarps = 8>
__global__ void __launch_bounds__(32 * kWarps, kOcc) visibility_patch_kernel(Scene sc, Walls walls,
                                                               int chunks,
                                                               int seed_mode, int seed_steps,
                                                               int shaft_cap) {
  __shared__ uint32_t bits[kMaxPatchChunks][32];  // [chunk][face j]: visible from point lane
  __shared__ int seeds[32];
  __shared__ int next_face;
  // per warp: two frontiers and the candidate list of the shaft search
  __shared__ int shaft_buf[kWalk == 3 ? kWarps * (2 * kShaftFrontier + kShaftCand) : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.z;
  const int ch0 = blockIdx.y * chunks;
  // one or two sets of wall points, the blocks of the second after the first's
  const bool second = blockIdx.x >= walls.blocks0;
  const View3f pts = second ? walls.pts1 : walls.pts0;
  const int P = second ? walls.P1 : walls.P0, row0 = second ? walls.row1 : walls.row0;
  uint32_t* scratch = sc.pscratch + 4 * (size_t)sc.B * row0;
  // position in the order
  const int i = (int)(blockIdx.x - (second ? walls.blocks0 : 0u)) * 32 + lane;
  const int n = sc.meta[b].n;
  const bool okp = i < P;
  const uint32_t* order = scratch + 3 * (size_t)sc.B * P + (size_t)b * P;
  int p = okp ? (int)order[i] : 0;
  if (!TOTRI_INDEX_OK((unsigned)p < (unsigned)P, sc.status)) p = 0;
  const fv3 o = okp ? mkv(pts.at(b, p, 0), pts.at(b, p, 1), pts.at(b, p, 2)) : mkv(0.f, 0.f, 0.f);
  volatile int* vseeds = seeds;
  volatile int* gseeds = reinterpret_cast<int*>(scratch) + (size_t)b * P;
  if (threadIdx.x < 32) seeds[lane] = okp ? gseeds[i] : -1;
  if (threadIdx.x == 0) next_face = 0;
  __syncthreads();
  const int nc = min(chunks, sc.nch - ch0);
  // The warp's wall points bound every ray's start (shaft search only).
  float plo[3] = {0.f, 0.f, 0.f}, phi[3] = {0.f, 0.f, 0.f}, pad = 0.f;
  if (kWalk == 3) {
    const float oc[3] = {o.x, o.y, o.z};
    float mag = 0.f;
    for (int a = 0; a < 3; ++a) {
      float lo = okp ? oc[a] : INFINITY, hi = okp ? oc[a] : -INFINITY;
      for (int off = 16; off; off >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, off));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, off));
      }
      plo[a] = lo;
      phi[a] = hi;
      mag = fmaxf(mag, fmaxf(fabsf(lo), fabsf(hi)));
    }
    // the hit-point margin, plus room for the rounding of far wall points
    pad = sc.meta[b].delta + ldexpf(isfinite(mag) ? mag : 0.f, -14);
    for (int a = 0; a < 3; ++a) {
      plo[a] -= pad;
      phi[a] += pad;
    }
  }
  // Faces are handed out one at a time from a shared counter, in Morton
  // order: a hidden face settled by a short surface walk costs a fraction of a
  // visible one, so fixed shares would leave warps idle at the final barrier.
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(&next_face, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= nc * 32) break;
    const int c = t >> 5, j = t & 31;
    const int k = (ch0 + c) * 32 + j;
    bool vis = false;
    if (k < n) {  // warp-uniform
      const Target tg = load_target(sc, b, k);
      if (kWalk == 1) {
        vis = packet_visible(sc, b, n, okp, tg, o, sc.status);
      } else if (kWalk == 2) {
        vis = okp && target_visible_pp4(sc, b, n, tg, o, sc.status);
      } else if (kWalk == 3) {
        int seed = okp ? vseeds[lane] : -1;
        const int s0 = seed;
        fv3 dir = mkv(0.f, 0.f, 0.f);
        float tmax = 0.f, tf = 0.f;
        int need = 0;
        if (okp)
          need = query_prefix(sc, b, n, tg, o, seed, seed_mode, seed_steps, dir, tmax, tf, vis);
        if (__any_sync(0xffffffffu, need)) {
          // every ray ends at its accepted hit on the target, which tri_hit
          // keeps inside the target's hit box (not near the centroid: for a
          // grazing target t is ill-conditioned along the ray)
          const float clo[3] = {tg.a2.y - pad, tg.a2.z - pad, tg.a2.w - pad};
          const float chi[3] = {tg.a3.x + pad, tg.a3.y + pad, tg.a3.z + pad};
          const Shaft h = make_shaft(plo, phi, clo, chi);
          int* wb = shaft_buf + warp * (2 * kShaftFrontier + kShaftCand);
          int* cand = wb + 2 * kShaftFrontier;
          const int ncand = shaft_candidates<kShaftFrontier, kShaftCand>(
              sc, b, n, tg.k, h, wb, wb + kShaftFrontier, cand, lane, shaft_cap);
          if (need) {
            bool occ = false;
            if (ncand >= 0) {
              for (int j = 0; j < ncand; ++j) {
                const int kk = cand[j];
                if ((unsigned)kk >= (unsigned)n) {
                  atomicOr(sc.status, kStatusTraversalCap);
                  continue;
                }
                const float4* q = tri_at(sc, b, kk);
                const float4 q0 = __ldg(q), q1 = __ldg(q + 1), q2 = __ldg(q + 2),
                             q3 = __ldg(q + 3);
                float tq;
                if (tri_hit(q0, q1, q2, q3, o, dir, tmax, tq) &&
                    (tq < tf || (tq == tf && __float_as_int(q3.w) < tg.f))) {
                  occ = true;
                  seed = kk;
                  break;
                }
              }
            } else {
              occ = bvh_occluded(sc, b, n, tg.k, tg.f, o, dir, tmax, tf, sc.status, seed);
            }
            vis = !occ;
          }
        }
        if (okp && seed != s0) vseeds[lane] = seed;
      } else if (kWalk == 4) {
        if (okp) {
          const int s0 = vseeds[lane];
          int seed = s0;
          fv3 dir;
          float tmax, tf;
          if (query_prefix(sc, b, n, tg, o, seed, seed_mode, seed_steps, dir, tmax, tf, vis))
            vis = !bvh_occluded_wide(sc, b, n, tg.k, tg.f, o, dir, tmax, tf, sc.status, seed);
          if (seed != s0) vseeds[lane] = seed;
        }
      } else if (okp) {
        const int s0 = vseeds[lane];
        int seed = s0;
        vis = target_visible_pp(sc, b, n, tg, o, sc.status, seed, seed_mode, seed_steps);
        if (seed != s0) vseeds[lane] = seed;
      }
    }
    const uint32_t w = __ballot_sync(0xffffffffu, vis);
    if (lane == 0) bits[c][j] = w;
  }
  __syncthreads();
  if (threadIdx.x < 32 && okp && (kWalk == 0 || kWalk == 3 || kWalk == 4)) gseeds[i] = seeds[lane];
  for (int c = warp; c < nc; c += kWarps) {
    if (!okp) continue;
    uint32_t word = 0u;
#pragma unroll
    for (int j = 0; j < 32; ++j) word |= ((bits[c][j] >> lane) & 1u) << j;
    sc.mask[((size_t)b * sc.P + row0 + p) * sc.nch + ch0 + c] = word;
  }
}

// visibility_patch_kernel<0> with the BVH searches compacted. After a face's
// prefix (the target's own hit and, for faces seen from behind, the surface
// walk) only some lanes are still undecided: most hidden targets are settled
// by the walk, so a face seen from behind typically leaves a few rays, and
// the warp used to run their BVH walks with the other lanes idle. Here each
// undecided ray goes into its warp's queue in shared memory (its direction,
// limits and target), and the warp walks the BVH only for full batches of 32
// queued rays, one per lane, drawn from the faces it has taken so far (and the
// last partial batch at the end). A face's mask word is written when its
// prefix ends, with the queued rays counted visible, and a walk that finds an
// occluder clears its bit. The decisions per ray are those of
// target_visible_pp (same prefix, same search), so the masks are unchanged.
constexpr int kVisQueue = 64;  // entries per warp: < 32 left over + 32 added

template <int kOcc>
__global__ void __launch_bounds__(256, kOcc) visibility_queue_kernel(Scene sc, View3f pts, int P,
                                                                    int row0, int chunks,
                                                                    int seed_mode,
                                                                    int seed_steps) {
  __shared__ uint32_t bits[kMaxPatchChunks][32];
  __shared__ int seeds[32];
  __shared__ int next_face;
  __shared__ float opts[3][32];  // the block's wall points (ray origins)
  // per warp: (dir.xyz, tf) and (tmax, target k << 5 | point lane, face index, -)
  __shared__ float4 queue[8][kVisQueue][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.z;
  const int ch0 = blockIdx.y * chunks;
  const int i = blockIdx.x * 32 + lane;  // position in the order
  const int n = sc.meta[b].n;
  const bool okp = i < P;
  const uint32_t* order = sc.pscratch + 3 * (size_t)sc.B * P + (size_t)b * P;
  int p = okp ? (int)order[i] : 0;
  if (!TOTRI_INDEX_OK((unsigned)p < (unsigned)P, sc.status)) p = 0;
  const fv3 o = okp ? mkv(pts.at(b, p, 0), pts.at(b, p, 1), pts.at(b, p, 2)) : mkv(0.f, 0.f, 0.f);
  volatile int* vseeds = seeds;
  volatile int* gseeds = reinterpret_cast<int*>(sc.pscratch) + (size_t)b * P;
  if (threadIdx.x < 32) {
    seeds[lane] = okp ? gseeds[i] : -1;
    opts[0][lane] = o.x;
    opts[1][lane] = o.y;
    opts[2][lane] = o.z;
  }
  if (threadIdx.x == 0) next_face = 0;
  __syncthreads();
  const int nc = min(chunks, sc.nch - ch0);
  const uint32_t below = (1u << lane) - 1u;
  float4(*q)[2] = queue[warp];
  int cnt = 0;  // queued rays (warp-uniform)
  // Walks queue entries [0, m), entry `lane` on lane `lane`.
  auto walk = [&](int m) {
    if (lane < m) {
      const float4 a = q[lane][0], e = q[lane][1];
      const int code = __float_as_int(e.y);
      const int k = code >> 5, pl = code & 31;
      const fv3 oo = mkv(opts[0][pl], opts[1][pl], opts[2][pl]);
      int seed = -1;
      if (bvh_occluded(sc, b, n, k, __float_as_int(e.z), oo, mkv(a.x, a.y, a.z), e.x, a.w,
                       sc.status, seed)) {
        const int t = k - ch0 * 32;
        atomicAnd(&bits[t >> 5][t & 31], ~(1u << pl));
        vseeds[pl] = seed;
      }
    }
  };
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(&next_face, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= nc * 32) break;
    const int c = t >> 5, j = t & 31;
    const int k = (ch0 + c) * 32 + j;
    if (k >= n) {  // warp-uniform
      if (lane == 0) bits[c][j] = 0u;
      continue;
    }
    bool vis = false;
    int need = 0;
    const Target tg = load_target(sc, b, k);
    fv3 dir = mkv(0.f, 0.f, 0.f);
    float tmax = 0.f, tf = 0.f;
    if (okp) {
      const int s0 = vseeds[lane];
      int seed = s0;
      need = query_prefix(sc, b, n, tg, o, seed, seed_mode, seed_steps, dir, tmax, tf, vis);
      if (seed != s0) vseeds[lane] = seed;
    }
    const uint32_t nm = __ballot_sync(0xffffffffu, need);
    const uint32_t w = __ballot_sync(0xffffffffu, vis || need);
    if (lane == 0) bits[c][j] = w;
    if (need) {
      const int at = cnt + __popc(nm & below);
      q[at][0] = make_float4(dir.x, dir.y, dir.z, tf);
      q[at][1] = make_float4(tmax, __int_as_float((k << 5) | lane), __int_as_float(tg.f), 0.f);
    }
    cnt += __popc(nm);
    if (cnt >= 32) {
      __syncwarp();
      walk(32);
      __syncwarp();
      if (lane < cnt - 32) {
        q[lane][0] = q[32 + lane][0];
        q[lane][1] = q[32 + lane][1];
      }
      cnt -= 32;
      __syncwarp();
    }
  }
  __syncwarp();
  walk(cnt);
  __syncthreads();
  if (threadIdx.x < 32 && okp) gseeds[i] = seeds[lane];
  for (int c = warp; c < nc; c += 8) {
    if (!okp) continue;
    uint32_t word = 0u;
#pragma unroll
    for (int j = 0; j < 32; ++j) word |= ((bits[c][j] >> lane) & 1u) << j;
    sc.mask[((size_t)b * sc.P + row0 + p) * sc.nch + ch0 + c] = word;
  }
}

constexpr int kListWarps = 4, kListFaces = 8, kListFrontier = 256, kListCand = 512;

// Visibility over dense wall grids, in two kernels.
//
// visibility_walk_kernel decides the targets seen from behind as
// visibility_patch_kernel does (surface walk from the last occluder, then the
// BVH) and leaves the bits of front-facing targets set. A warp takes one block
// of 32 wall points (one per lane) and a run of consecutive 32-face chunks from a
// global queue, and keeps each point's last occluder in a register: a target's
// neighbour in Morton order was decided just before by the same warp, so the
// walks start closer than from seeds shared by eight warps on eight faces (3.5
// -> 2.5 ms on the 20,480-face workload; runs of 2, 4 and 8 chunks 2.4, 2.5 and 2.5
// ms there, but 3.1, 3.3, 3.7 and 5.2 ms for 1 to 8 chunks on a 12,288-face box).
//
// visibility_list_kernel then decides the front-facing targets without BVH
// walks. A warp takes 32 wall points and kListFaces consecutive faces and
// collects every face whose box meets the hull of the wall points and those
// faces' hit boxes (shaft_candidates, about 100 of them). For each target the
// lanes test that list, 32 boxes at a time, against the hull of the wall points
// and the rays' own accepted hits on the target: an accepted occluder has t
// in [0, tf], so its hit point lies on a segment from a wall point to such a
// hit. That hull ends in a point for all but grazing targets, so a few
// neighbours remain (8 on the 20,480-face workload, 18 on the box), and they get
// the exact triangle test, all lanes on one face. When the list overflows, the
// target's own hull is walked for its candidates; when those overflow too, or
// fewer than two rays need it, the lanes search the BVH. Every accepted hit's
// box is in the list and passes the second hull (both are padded beyond the
// rounding, as make_shaft describes), so the bits are those of brute force.
// What bounds them: instruction issue. Both together: 7.9 -> 4.6 ms on the
// 20,480-face workload (4,096 points), 17.0 -> 7.5 ms on the box (6,767 points).
// Lists for 4, 16 and 32 faces at a time took 2.4, 2.4 and 3.5 ms against 2.2 ms
// on the 20,480-face workload, 4.9, 7.6 and 11.4 against 5.5 ms on the box.
template <int kOcc>
__global__ void __launch_bounds__(32 * kListWarps, kOcc) visibility_walk_kernel(
    Scene sc, View3f pts, int P, int row0, uint32_t* next_unit, int parts, int seed_mode,
    int seed_steps) {
  const int lane = threadIdx.x & 31;
  const int patches = (P + 31) >> 5;
  const unsigned units = (unsigned)patches * sc.nch * sc.B * parts;
  const int run = 32 / parts;
  for (;;) {
    unsigned unit = 0;
    if (lane == 0) unit = atomicAdd(next_unit, 1u);
    unit = __shfl_sync(0xffffffffu, unit, 0);
    if (unit >= units) break;
    const int j0 = (int)(unit % parts) * run, up = unit / parts;
    const int ch = up % sc.nch, pb = up / sc.nch;
    const int b = pb / patches, i = (pb - b * patches) * 32 + lane;
    const int n = sc.meta[b].n;
    const bool okp = i < P;
    const uint32_t* order = sc.pscratch + 3 * (size_t)sc.B * P + (size_t)b * P;
    int p = okp ? (int)order[i] : 0;
    if (!TOTRI_INDEX_OK((unsigned)p < (unsigned)P, sc.status)) p = 0;
    const fv3 o = okp ? mkv(pts.at(b, p, 0), pts.at(b, p, 1), pts.at(b, p, 2)) : mkv(0.f, 0.f, 0.f);
    volatile int* gseeds = reinterpret_cast<int*>(sc.pscratch) + (size_t)b * P;
    int seed = okp ? gseeds[i] : -1;
    const int s0 = seed;
    uint32_t word = 0u;
    for (int j = j0; j < j0 + run && ch * 32 + j < n; ++j) {  // warp-uniform
      const Target tg = load_target(sc, b, ch * 32 + j);
      bool vis = false;
      if (okp) {
        fv3 dir;
        float tmax, tf;
        const fv3 nrm = cross(mkv(tg.a0.w, tg.a1.x, tg.a1.y), mkv(tg.a1.z, tg.a1.w, tg.a2.x));
        if (n > 1 && !(dot(nrm, tg.c - o) > 0.f))
          vis = true;  // left to visibility_list_kernel
        else if (query_prefix(sc, b, n, tg, o, seed, seed_mode, seed_steps, dir, tmax, tf, vis))
          vis = !bvh_occluded_wide(sc, b, n, tg.k, tg.f, o, dir, tmax, tf, sc.status, seed);
      }
      __syncwarp();
      word |= (uint32_t)vis << j;
    }
    uint32_t* mw = sc.mask + ((size_t)b * sc.P + row0 + p) * sc.nch + ch;
    if (okp && parts == 1) *mw = word;
    // (a run of 8 faces is a byte of the word)
    if (okp && parts == 4) reinterpret_cast<uint8_t*>(mw)[j0 >> 3] = (uint8_t)(word >> j0);
    if (okp && seed != s0) gseeds[i] = seed;
  }
}

template <int kOcc>
__global__ void __launch_bounds__(32 * kListWarps, kOcc) visibility_list_kernel(
    Scene sc, View3f pts, int P, int row0, uint32_t* next_unit, int list_cap) {
  __shared__ int buf[kListWarps][2 * kListFrontier + kListCand];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int* fr0 = buf[warp];
  int* cand = fr0 + 2 * kListFrontier;
  const int patches = (P + 31) >> 5, per_chunk = 32 / kListFaces;
  const unsigned units = (unsigned)patches * sc.nch * per_chunk * sc.B;
  for (;;) {
    unsigned unit = 0;
    if (lane == 0) unit = atomicAdd(next_unit, 1u);
    unit = __shfl_sync(0xffffffffu, unit, 0);
    if (unit >= units) break;
    const int part = unit % per_chunk;
    const unsigned r = unit / per_chunk;
    const int ch = r % sc.nch, pb = r / sc.nch;
    const int b = pb / patches, i = (pb - b * patches) * 32 + lane;
    const int n = sc.meta[b].n;
    const int k0 = ch * 32 + part * kListFaces;
    if (k0 >= n || n == 1) continue;
    const bool okp = i < P;
    const uint32_t* order = sc.pscratch + 3 * (size_t)sc.B * P + (size_t)b * P;
    int p = okp ? (int)order[i] : 0;
    if (!TOTRI_INDEX_OK((unsigned)p < (unsigned)P, sc.status)) p = 0;
    uint32_t* mrow = sc.mask + ((size_t)b * sc.P + row0 + p) * sc.nch + ch;
    const uint32_t open0 = okp ? (*mrow >> (part * kListFaces)) & ((1u << kListFaces) - 1u) : 0u;
    const uint32_t faces = __reduce_or_sync(0xffffffffu, open0);
    if (faces == 0u) continue;
    const fv3 o = okp ? mkv(pts.at(b, p, 0), pts.at(b, p, 1), pts.at(b, p, 2)) : mkv(0.f, 0.f, 0.f);
    float plo[3], phi[3], pad = 0.f;  // the wall points' padded box
    {
      const float oc[3] = {o.x, o.y, o.z};
      float mag = 0.f;
      for (int a = 0; a < 3; ++a) {
        plo[a] = warp_min_f(okp ? oc[a] : INFINITY);
        phi[a] = warp_max_f(okp ? oc[a] : -INFINITY);
        mag = fmaxf(mag, fmaxf(fabsf(plo[a]), fabsf(phi[a])));
      }
      pad = sc.meta[b].delta + ldexpf(isfinite(mag) ? mag : 0.f, -14);
      for (int a = 0; a < 3; ++a) {
        plo[a] -= pad;
        phi[a] += pad;
      }
    }
    uint32_t hidden = 0u;
    int ncand = -2;  // -2: not collected yet, -1: overflow
    for (uint32_t m = faces; m; m &= m - 1) {
      const int j = __ffs(m) - 1, k = k0 + j;
      const Target tg = load_target(sc, b, k);
      const bool open = (open0 >> j) & 1u;
      // the prefix's ray and own hit
      const fv3 D = xsub3(tg.c, o);
      const float dist = xlen(D);
      const fv3 dir = mkv(xdiv(D.x, dist), xdiv(D.y, dist), xdiv(D.z, dist));
      const float tmax = xadd(xmul(dist, 1.01f), 1e-3f);
      float tf = 0.f;
      const bool need =
          open && dist >= 1e-6f && tri_hit(tg.a0, tg.a1, tg.a2, tg.a3, o, dir, tmax, tf);
      const fv3 nrm = cross(mkv(tg.a0.w, tg.a1.x, tg.a1.y), mkv(tg.a1.z, tg.a1.w, tg.a2.x));
      const bool front = need && !(dot(nrm, dir) > 0.f);
      bool occ = false;
      bool search = need;
      if (__popc(__ballot_sync(0xffffffffu, front)) >= 2) {
        if (ncand == -2) {
          // the hull of the wall points and the open faces' hit boxes
          float4 t2 = make_float4(0.f, INFINITY, INFINITY, INFINITY);
          float4 t3 = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
          if (lane < kListFaces && ((faces >> lane) & 1u)) {
            const float4* q = tri_at(sc, b, k0 + lane);
            t2 = __ldg(q + 2);
            t3 = __ldg(q + 3);
          }
          const float clo[3] = {warp_min_f(t2.y) - pad, warp_min_f(t2.z) - pad,
                                warp_min_f(t2.w) - pad};
          const float chi[3] = {warp_max_f(t3.x) + pad, warp_max_f(t3.y) + pad,
                                warp_max_f(t3.z) + pad};
          ncand = shaft_candidates<kListFrontier, kListCand>(
              sc, b, n, -1, make_shaft(plo, phi, clo, chi), fr0, fr0 + kListFrontier, cand, lane,
              list_cap);
        }
        {
          // the hull of the wall points and the rays' hits on the target
          const float hx = fmaf(tf, dir.x, o.x), hy = fmaf(tf, dir.y, o.y);
          const float hz = fmaf(tf, dir.z, o.z);
          const float clo[3] = {warp_min_f(need ? hx : INFINITY) - pad,
                                warp_min_f(need ? hy : INFINITY) - pad,
                                warp_min_f(need ? hz : INFINITY) - pad};
          const float chi[3] = {warp_max_f(need ? hx : -INFINITY) + pad,
                                warp_max_f(need ? hy : -INFINITY) + pad,
                                warp_max_f(need ? hz : -INFINITY) + pad};
          const Shaft h = make_shaft(plo, phi, clo, chi);
          int count = ncand;
          if (ncand == -1)
            count = shaft_candidates<kListFrontier, kListCand>(sc, b, n, k, h, fr0,
                                                               fr0 + kListFrontier, cand, lane,
                                                               list_cap);
          for (int base = 0; base < count; base += 32) {
            const int kk = base + lane < count ? cand[base + lane] : k;
            bool in = false;
            if ((unsigned)kk >= (unsigned)n) {
              atomicOr(sc.status, kStatusTraversalCap);
            } else if (kk != k) {
              const float4* q = tri_at(sc, b, kk);
              const float4 t2 = __ldg(q + 2), t3 = __ldg(q + 3);
              in = shaft_box(h, t2.y, t2.z, t2.w, t3.x, t3.y, t3.z);
            }
            uint32_t mm = __ballot_sync(0xffffffffu, in);
            while (mm) {
              const int g = __shfl_sync(0xffffffffu, kk, __ffs(mm) - 1);
              mm &= mm - 1;
              if (search && !occ) {
                const float4* q = tri_at(sc, b, g);
                const float4 q0 = __ldg(q), q1 = __ldg(q + 1), q2 = __ldg(q + 2),
                             q3 = __ldg(q + 3);
                float tq;
                if (tri_hit(q0, q1, q2, q3, o, dir, tmax, tq) &&
                    (tq < tf || (tq == tf && __float_as_int(q3.w) < tg.f)))
                  occ = true;
              }
            }
          }
          if (count >= 0) search = false;
        }
      }
      if (search) {
        int seed = -1;
        occ = bvh_occluded_wide(sc, b, n, tg.k, tg.f, o, dir, tmax, tf, sc.status, seed);
      }
      __syncwarp();
      hidden |= (uint32_t)(occ || (open && !need)) << j;
    }
    if (okp && hidden) atomicAnd(mrow, ~(hidden << (part * kListFaces)));
  }
}

// Per-pair confocal geometry: FP32 decisions exactly as the oracle takes them.
struct ConfocalPair {
  fv3 v[3];
  int perm[3];
  float d[3];
  float c[3];
  int bin[3];
};

__device__ __forceinline__ void confocal_pair(const float4 s0, const float4 s1, const float4 s2,
                                              fv3 sp, float od, float bw, float bo,
                                              ConfocalPair& q) {
  q.v[0] = mkv(s0.x, s0.y, s0.z);
  q.v[1] = mkv(s1.x, s1.y, s1.z);
  q.v[2] = mkv(s2.x, s2.y, s2.z);
  for (int k = 0; k < 3; ++k) {
    q.perm[k] = k;
    q.d[k] = xlen(xsub3(q.v[k], sp));
  }
  sort3(q);
  for (int k = 0; k < 3; ++k) {
    q.c[k] = xdiv(xsub(xadd(xmul(2.f, q.d[k]), od), bo), bw);
    q.bin[k] = bin_of(q.c[k]);
  }
}

// confocal_pair with a filtered fast path (FastBins): lengths from the
// hardware reciprocal square root, bin coordinates from one fused
// multiply-add. Each fast length is within 8 u d of the exact chain's
// (u = 2^-24), so three lengths separated by more than 16 u max(d) sort as the
// exact ones do, and a bin coordinate farther than
// 32 u (2d + od + |bo|)/bw + 8 u |c| + 1e-6 from an integer truncates to the
// exact bin. Only then are the fast values kept; otherwise (ties, NaN, huge
// coordinates) the exact confocal_pair runs. Bins and vertex order are always
// those of the exact chain; values differ from it by a few ulps. Used by the
// forward splat only: the gradient's FP32 cancellation amplifies those ulps
// (2.8e-4 rel-L2 on the 20,480-face vertex gradient), so the gradient keeps
// the exact chain.
__device__ __forceinline__ void confocal_pair_filtered(const float4 s0, const float4 s1,
                                                       const float4 s2, fv3 sp, float od,
                                                       float bw, float bo, const FastBins& fb,
                                                       ConfocalPair& q) {
  q.v[0] = mkv(s0.x, s0.y, s0.z);
  q.v[1] = mkv(s1.x, s1.y, s1.z);
  q.v[2] = mkv(s2.x, s2.y, s2.z);
  for (int k = 0; k < 3; ++k) {
    q.perm[k] = k;
    q.d[k] = len_fast(q.v[k] - sp);
  }
  sort3(q);
  const float u = 5.9604645e-8f;
  bool ok = q.d[1] - q.d[0] > 16.f * u * q.d[2] && q.d[2] - q.d[1] > 16.f * u * q.d[2];
  for (int k = 0; k < 3; ++k) {
    const float x = fmaf(2.f, q.d[k], od);
    const float c = fmaf(x, fb.inv_bw, fb.nbo);
    const float m = fmaf(fb.kc, x, fb.kb) + 8.f * u * fabsf(c);
    ok = ok && fabsf(c - rintf(c)) > m && fabsf(c) < 1.0e9f;
    q.c[k] = c;
    q.bin[k] = __float2int_rz(c);
  }
  if (!ok) confocal_pair(s0, s1, s2, sp, od, bw, bo, q);
}

// alpha of AlphaConfocal (mesh_common.h:394-413):
// 100 rho (n_w.r)^2 (n.r)^2 / (|n| |r|^8), n_w = (0,0,1), r = c - s.
__device__ __forceinline__ float alpha_confocal(const ConfocalPair& q, fv3 c, fv3 sp,
                                                float rho) {
  const fv3 n = cross(q.v[1] - q.v[0], q.v[2] - q.v[0]);
  const fv3 r = c - sp;
  if (!(r.z > 0.f)) return 0.f;
  const float nr = dot(n, r), rr = dot(r, r), nn = dot(n, n);
  const float rr2 = rr * rr;
  return vdiv(100.f * rho * (r.z * r.z) * (nr * nr) * rsqrtf(nn), rr2 * rr2);
}

template <int TS>
__global__ void __launch_bounds__(256) splat_kernel(Scene sc, View3f sp, View3f so, int has_origin,
                                                    float* __restrict__ transient, int T, int S,
                                                    float bw, float bo, FastBins fb) {
  extern __shared__ float hist[];  // [T][TS]
  const int b = blockIdx.y;
  const int s0 = blockIdx.x * TS;
  for (int i = threadIdx.x; i < T * TS; i += blockDim.x) hist[i] = 0.f;
  __syncthreads();
  const int n = sc.meta[b].n;
  const int sl = threadIdx.x % TS;
  const int s = s0 + sl;
  if (s < S) {
    const fv3 p = mkv(sp.at(b, s, 0), sp.at(b, s, 1), sp.at(b, s, 2));
    float od = 0.f;
    if (has_origin) od = xmul(2.f, xlen(xsub3(p, mkv(so.at(b, s, 0), so.at(b, s, 1), so.at(b, s, 2)))));
    const uint32_t* mrow = sc.mask + ((size_t)b * sc.P + s) * sc.nch;
    const float4* shade = sc.shade + (size_t)b * sc.F * 4;
    Hist<TS> h{hist, sl, T};
    for (int k = threadIdx.x / TS; k < n; k += blockDim.x / TS) {
      if (!((__ldg(mrow + (k >> 5)) >> (k & 31)) & 1u)) continue;
      const float4 s0r = __ldg(shade + 4 * k), s1r = __ldg(shade + 4 * k + 1);
      const float4 s2r = __ldg(shade + 4 * k + 2), s3r = __ldg(shade + 4 * k + 3);
      ConfocalPair q;
      confocal_pair_filtered(s0r, s1r, s2r, p, od, bw, bo, fb, q);
      const float alpha = alpha_confocal(q, mkv(s3r.x, s3r.y, s3r.z), p, s0r.w);
      if (!(alpha > 0.f)) continue;
      splat_tent(h, q.c, q.bin, alpha);
    }
  }
  __syncthreads();
  flush_tile<TS>(hist, transient + (size_t)b * T * S, T, S, s0);
}

// splat_kernel with the visible pairs compacted first: each warp walks
// 32-face chunks (lane = face), gathers each face's visibility over the TS
// scan points of the tile, queues the visible (face, point) pairs in shared
// memory and evaluates them 32 at a time, one per lane, instead of leaving the
// lanes of occluded pairs idle. A face hands out its points starting at a
// lane-dependent offset, so the 32 pairs of a batch fall on different
// histogram columns and their shared atomics seldom collide.
template <int TS>
__global__ void __launch_bounds__(256, 2) splat_compact_kernel(Scene sc, View3f sp, View3f so,
                                                            int has_origin,
                                                            float* __restrict__ transient, int T,
                                                            int S, float bw, float bo,
                                                            FastBins fb) {
  extern __shared__ float hist[];  // [T][TS]
  __shared__ float pts[TS][4];     // scan point, 2 |scan - origin|
  __shared__ int queue[8][64];
  const int b = blockIdx.y;
  const int s0 = blockIdx.x * TS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < T * TS; i += blockDim.x) hist[i] = 0.f;
  if (threadIdx.x < TS && s0 + (int)threadIdx.x < S) {
    const int s = s0 + threadIdx.x;
    const fv3 p = mkv(sp.at(b, s, 0), sp.at(b, s, 1), sp.at(b, s, 2));
    pts[threadIdx.x][0] = p.x;
    pts[threadIdx.x][1] = p.y;
    pts[threadIdx.x][2] = p.z;
    pts[threadIdx.x][3] =
        has_origin ? xmul(2.f, xlen(xsub3(p, mkv(so.at(b, s, 0), so.at(b, s, 1), so.at(b, s, 2)))))
                   : 0.f;
  }
  __syncthreads();
  const int n = sc.meta[b].n;
  const int nchu = (n + 31) >> 5;
  const int ts = min(TS, S - s0);
  const uint32_t* m0 = sc.mask + ((size_t)b * sc.P + s0) * sc.nch;
  const float4* shade = sc.shade + (size_t)b * sc.F * 4;
  const uint32_t below = (1u << lane) - 1u;
  int* qw = queue[warp];
  int cnt = 0;  // warp-uniform
  auto run = [&](int e) {
    const int k = e >> 4, sl = e & 15;
    const float4 s0r = __ldg(shade + 4 * k), s1r = __ldg(shade + 4 * k + 1);
    const float4 s2r = __ldg(shade + 4 * k + 2), s3r = __ldg(shade + 4 * k + 3);
    const fv3 p = mkv(pts[sl][0], pts[sl][1], pts[sl][2]);
    ConfocalPair q;
    confocal_pair_filtered(s0r, s1r, s2r, p, pts[sl][3], bw, bo, fb, q);
    const float alpha = alpha_confocal(q, mkv(s3r.x, s3r.y, s3r.z), p, s0r.w);
    if (!(alpha > 0.f)) return;
    const Hist<TS> h{hist, sl, T};
    splat_tent(h, q.c, q.bin, alpha);
  };
  const int rot = lane & (TS - 1);
  for (int ch = warp; ch < nchu; ch += 8) {
    const uint32_t w = lane < ts ? __ldg(m0 + (size_t)lane * sc.nch + ch) : 0u;
    // vm: this lane's face, bit sl = visible from scan point s0 + sl; faces
    // at or past n never count, whatever the mask words hold there.
    uint32_t vm = 0u;
    for (int sl = 0; sl < ts; ++sl) vm |= ((__shfl_sync(0xffffffffu, w, sl) >> lane) & 1u) << sl;
    if (ch * 32 + lane >= n) vm = 0u;
    while (__any_sync(0xffffffffu, vm != 0u)) {
      const bool has = vm != 0u;
      int sl = 0;
      if (has) {  // next visible point, counting from this lane's offset
        const uint32_t r = ((vm >> rot) | (vm << ((TS - rot) & 31))) & ((1u << TS) - 1u);
        sl = (__ffs(r) - 1 + rot) & (TS - 1);
        vm &= ~(1u << sl);
      }
      const uint32_t take = __ballot_sync(0xffffffffu, has);
      if (has) qw[cnt + __popc(take & below)] = ((ch * 32 + lane) << 4) | sl;
      cnt += __popc(take);  // below 64: at most 31 queued before, 32 added
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
  flush_tile<TS>(hist, transient + (size_t)b * T * S, T, S, s0);
}

// The gradient of a face over its visible scan points, following
// mesh_confocal_grad_verts_optix.cu:248-314 and AlphaConfocalGradVerts
// (mesh_common.h:429-463), as sums that are linear in the pair's two factors: P =
// alpha times the gradient over the tent's area, and Q_m = alpha times the tent's
// weight of vertex m (pair_weights). With r = c - p,
//   d log(alpha) / d v_k = J_n^T (kn n + knr r) + kr r + (knr/3) n + kw n_w
// and d path / d v_m = 2 u_m, u_m the unit vector from the point, so a pair adds
// P kr r, P knr r, P knr, P kw, P and 2 Q_m u_m; the normal and its Jacobian follow
// once per face.
struct FaceSums {
  unsigned long long a[9];  // pairs: kr r and knr r (x y, z x, y z), (knr, kw), (P, u0 x), ...
};

// |v - p| as the FP32 chain's length and its low part (len_df's sums, with the
// Newton step taken from the chain's square root).
__device__ __forceinline__ DFloat len_exact(fv3 v, fv3 p, float& inv) {
  const DFloat dx = two_sum(v.x, -p.x), dy = two_sum(v.y, -p.y), dz = two_sum(v.z, -p.z);
  const float d = xlen(mkv(dx.hi, dy.hi, dz.hi));
  const float hx = __fmul_rn(dx.hi, dx.hi), hy = __fmul_rn(dy.hi, dy.hi);
  const float hz = __fmul_rn(dz.hi, dz.hi);
  const float lx = __fmaf_rn(dx.hi, dx.hi, -hx), ly = __fmaf_rn(dy.hi, dy.hi, -hy);
  const float lz = __fmaf_rn(dz.hi, dz.hi, -hz);
  const DFloat s1 = two_sum(hx, hy);
  const DFloat s2 = two_sum(s1.hi, hz);
  const float lo = (s1.lo + s2.lo) + (lx + ly + lz) +
                   2.f * (dx.hi * dx.lo + dy.hi * dy.lo + dz.hi * dz.lo);
  inv = vdiv(1.f, d);
  return DFloat{d, d > 0.f ? (__fmaf_rn(-d, d, s2.hi) + lo) * (0.5f * inv) : 0.f};
}

// Instruction issue bounds it (75% of the slots). 20,480 faces x 4,096 points, 1,024
// bins: 1.44 ms when each pair built the vertices' gradients, took every length
// twice (chain and double-float) and walked the tent's three parts apart (1,200
// instructions per 32 visible pairs), 1.03 ms now; 320 faces x 1,024 points: 46 and
// 37 us. Two CTAs per SM (no spills) against 1.05 ms and 40 us with three.
// kForward: the bin width is positive.
template <bool kForward>
__global__ void __launch_bounds__(256, 2) grad_kernel(Scene sc, View3f sp, View3f so, int has_origin,
                                                   const float* __restrict__ tgrad, int T, int S,
                                                   float bw, float bo, int fixed, GradOut out) {
  extern __shared__ uint32_t mcol[];  // [slice] mask words of this 32-face chunk
  __shared__ int gq[8][64];           // per-warp queue of visible scan points
  const int b = blockIdx.y;
  const int ch = blockIdx.x;
  const int n = sc.meta[b].n;
  if (ch * 32 >= n) return;
  // scan-point slice [s0, s1) of this CTA (gridDim.z slices)
  const int s0 = (int)((int64_t)S * blockIdx.z / gridDim.z);
  const int s1 = (int)((int64_t)S * (blockIdx.z + 1) / gridDim.z);
  for (int s = s0 + threadIdx.x; s < s1; s += blockDim.x)
    mcol[s - s0] = sc.mask[((size_t)b * sc.P + s) * sc.nch + ch];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const float* tgb = tgrad + (size_t)b * T * S;
  const float4* shade = sc.shade + (size_t)b * sc.F * 4;
  const float inv_bw = __frcp_rn(bw);
  const bool plain = !has_origin && bo == 0.f;  // nothing added to a path
  for (int j = warp; j < 32; j += nw) {
    const int k = ch * 32 + j;
    if (k >= n) break;
    const float4 s0r = __ldg(shade + 4 * k), s1r = __ldg(shade + 4 * k + 1);
    const float4 s2r = __ldg(shade + 4 * k + 2), s3r = __ldg(shade + 4 * k + 3);
    const fv3 c = mkv(s3r.x, s3r.y, s3r.z);
    const fv3 v0 = mkv(s0r.x, s0r.y, s0r.z), v1 = mkv(s1r.x, s1r.y, s1r.z);
    const fv3 v2 = mkv(s2r.x, s2r.y, s2r.z);
    const fv3 e1 = v1 - v0, e2 = v2 - v0;
    const fv3 nrm = cross(e1, e2);
    const float nn = dot(nrm, nrm);
    const float kf = xdiv(100.f * s0r.w, xsqrt(nn));
    FaceSums sums;
    bool used = false;
#pragma unroll
    for (int i = 0; i < 9; ++i) sums.a[i] = 0ull;
    auto run = [&](int s) {
      const fv3 p = mkv(sp.at(b, s, 0), sp.at(b, s, 1), sp.at(b, s, 2));
      const fv3 r = c - p;
      if (!(r.z > 0.f)) return;
      const float nr = dot(nrm, r), rr = dot(r, r);
      // (the square of r.z nr / |r|^4: |r|^8 leaves the FP32 range in small units)
      const float fall = vdiv(r.z * nr, rr * rr), alpha = kf * fall * fall;
      if (!(alpha > 0.f)) return;
      float i0, i1, i2;  // 1 / |v_m - p|
      auto path = [&](fv3 v, float& inv) {
        const DFloat d = len_exact(v, p, inv);
        return DFloat{2.f * d.hi, 2.f * d.lo};
      };
      DFloat d0 = path(v0, i0), d1 = path(v1, i1), d2 = path(v2, i2);
      const PathOrder order = sort_paths(d0, d1, d2);
      if (!plain) {
        DFloat od{0.f, 0.f};
        if (has_origin) {
          const fv3 o = mkv(so.at(b, s, 0), so.at(b, s, 1), so.at(b, s, 2));
          float unused;
          const DFloat d = len_exact(p, o, unused);
          od = DFloat{2.f * d.hi, 2.f * d.lo};
        }
        d0 = path_offset(d0, od, bo);
        d1 = path_offset(d1, od, bo);
        d2 = path_offset(d2, od, bo);
      }
      float4 w;
      if (!pair_weights<false, kForward>(tgb + s, S, T, d0, d1, d2, bw, inv_bw, fixed, order, w)) return;
      const float P = alpha * w.x, knr = vdiv(2.f, nr), kw = vdiv(2.f, 3.f * r.z);
      const float pr = P * vdiv(-8.f, 3.f * rr), pn = P * knr;
      const float q0 = 2.f * alpha * w.y * i0, q1 = 2.f * alpha * w.z * i1;
      const float q2 = 2.f * alpha * w.w * i2;
      const fv3 r0 = v0 - p, r1 = v1 - p, r2 = v2 - p;
      used = true;
      sums.a[0] = f2fma(f2pack(pr, pr), f2pack(r.x, r.y), sums.a[0]);
      sums.a[1] = f2fma(f2pack(pr, pn), f2pack(r.z, r.x), sums.a[1]);
      sums.a[2] = f2fma(f2pack(pn, pn), f2pack(r.y, r.z), sums.a[2]);
      sums.a[3] = f2fma(f2pack(P, P), f2pack(knr, kw), sums.a[3]);
      sums.a[4] = f2fma(f2pack(P, q0), f2pack(1.f, r0.x), sums.a[4]);
      sums.a[5] = f2fma(f2pack(q0, q0), f2pack(r0.y, r0.z), sums.a[5]);
      sums.a[6] = f2fma(f2pack(q1, q1), f2pack(r1.x, r1.y), sums.a[6]);
      sums.a[7] = f2fma(f2pack(q1, q2), f2pack(r1.z, r2.x), sums.a[7]);
      sums.a[8] = f2fma(f2pack(q2, q2), f2pack(r2.y, r2.z), sums.a[8]);
    };
    // visible scan points are queued and evaluated 32 at a time, one per lane
    int* qw = gq[warp];
    int cnt = 0;  // warp-uniform
    for (int base = s0; base < s1; base += 32) {
      const int s = base + lane;
      const bool v = s < s1 && ((mcol[s - s0] >> j) & 1u);
      const uint32_t bits = __ballot_sync(0xffffffffu, v);
      if (v) qw[cnt + __popc(bits & ((1u << lane) - 1u))] = s;
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
    __syncwarp();
    if (lane < cnt) run(qw[lane]);
    __syncwarp();
    float t[18];
#pragma unroll
    for (int i = 0; i < 9; ++i) f2unpack(sums.a[i], t[2 * i], t[2 * i + 1]);
    const float sP = t[8];
    // (a lane without a pair leaves zeros: the face's normal may be anything)
    fv3 acc[3] = {mkv(0.f, 0.f, 0.f), mkv(0.f, 0.f, 0.f), mkv(0.f, 0.f, 0.f)};
    float accm = 0.f;
    if (used) {
      // (1 / |n|^2 is first multiplied by n: with the sum it leaves the FP32 range in
      // small units)
      const fv3 jw = sP * (vdiv(-1.f, nn) * nrm) + mkv(t[3], t[4], t[5]);
      const fv3 g1 = cross(e2, jw), g2 = cross(jw, e1);
      const fv3 common = mkv(t[0], t[1], t[2]) + (t[6] * (1.f / 3.f)) * nrm + mkv(0.f, 0.f, t[7]);
      acc[0] = common - g1 - g2 + mkv(t[9], t[10], t[11]);
      acc[1] = common + g1 + mkv(t[12], t[13], t[14]);
      acc[2] = common + g2 + mkv(t[15], t[16], t[17]);
      accm = xdiv(sP, s0r.w);
    }
    scatter_face_grad(out, b, s1r, s2r, s3r, acc, accm, sc.status);
  }
}

// Re-indexes mask bits from Morton order (bit k) to input face order (bit f).
__global__ void mask_unsort_kernel(Scene sc, int P, uint32_t* out) {
  const int b = blockIdx.y;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int n = sc.meta[b].n;
  if (i >= (int64_t)P * n) return;
  const int p = (int)(i / n), k = (int)(i - (int64_t)p * n);
  const uint32_t w = sc.mask[((size_t)b * sc.P + p) * sc.nch + (k >> 5)];
  if (!((w >> (k & 31)) & 1u)) return;
  const int f = __float_as_int(tri_at(sc, b, k)[3].w);
  if (!TOTRI_INDEX_OK((unsigned)f < (unsigned)sc.F, sc.status)) return;
  atomicOr(out + ((size_t)b * P + p) * sc.nch + (f >> 5), 1u << (f & 31));
}

}  // namespace

int launch_mask_unsort(const Scene& sc, int P, uint32_t* out, cudaStream_t stream) {
  TOTRI_CUDA(cudaMemsetAsync(out, 0, sizeof(uint32_t) * (size_t)sc.B * P * sc.nch, stream));
  const dim3 grid((unsigned)ceil_div((int64_t)P * sc.F, 256), (unsigned)sc.B);
  TOTRI_KERNEL("mesh mask unsort", stream, mask_unsort_kernel<<<grid, 256, 0, stream>>>(sc, P, out));
  return TOTRI_OK;
}

// Dense wall grids (blocks of 32 points narrow enough for the hulls) with
// enough (block, chunk) units to feed the queues: from 1,024 points and 5,000 units
// on the two kernels took 0.50-0.99x of the patch kernel's time on spheres, boxes
// and displaced icospheres of 1,280 to 20,480 faces at 1,024 to 10,201 points (us:
// 20,480 faces, 4,096 points 4,540 against 7,966; 8,000, 3,136 points 1,736 against
// 2,444, a box 2,751 against 5,842; 1,280, 4,096 points 324 against 361). Below,
// 1.0-1.3x, and 1.1-1.4x at 576 points (20,000 faces 2,333 against 2,067).
// "mesh.visibility.list": 1 always, 2 never; ".list.cap" lowers the list's capacity.
static bool list_rule(const Scene& sc, int P, const VisKeys& keys) {
  const int64_t units = ceil_div(P, 32) * sc.nch * sc.B;
  return keys.mode == 0 && keys.wide != 2 && keys.queue != 1 && keys.occupancy == 0 &&
         (keys.list == 1 || (keys.list == 0 && P >= 1024 && units >= 5000)) &&
         units < ((int64_t)1 << 29);
}

VisKeys visibility_keys(bool brute) {
  return VisKeys{brute,
                 tune::get("mesh.visibility.mode"),
                 tune::get("mesh.visibility.queue"),
                 tune::get("mesh.visibility.list"),
                 tune::get("mesh.visibility.wide"),
                 tune::get("mesh.visibility.occupancy")};
}

bool VisKeys::ordered() const {
  return !brute && mode != kVisRay && mode != kVisPacket && mode != kVisRayPostponed;
}

static int launch_visibility_sets(const Scene& sc0, const WallSet* sets, int nsets,
                                  const VisKeys& keys, cudaStream_t stream) {
  // (the kernels over one set find its scratch at sc.pscratch)
  const View3f& pts = sets[0].pts;
  const int row0 = sets[0].row0;
  const int P = sets[0].P;
  Scene sc = sc0;
  sc.pscratch += 4 * (size_t)sc.B * row0;
  const int P2 = nsets > 1 ? sets[1].P : 0;
  const Walls walls{pts, nsets > 1 ? sets[1].pts : pts, P, P2, row0, nsets > 1 ? sets[1].row0 : 0,
                    (unsigned)ceil_div(P, 32)};
  const int64_t units = (int64_t)sc.B * P * sc.nch;
  if (units == 0) return TOTRI_OK;
  const unsigned blocks = (unsigned)ceil_div(units * 32, 256);
  if (keys.brute) {
    TOTRI_KERNEL("mesh visibility brute", stream,
                 visibility_kernel<kVisBrute><<<blocks, 256, 0, stream>>>(sc, pts, P, row0));
  } else if (keys.mode == kVisRay) {
    TOTRI_KERNEL("mesh visibility", stream,
                 visibility_kernel<kVisRay><<<blocks, 256, 0, stream>>>(sc, pts, P, row0));
  } else if (keys.mode == kVisPacket) {
    TOTRI_KERNEL("mesh visibility", stream,
                 visibility_kernel<kVisPacket><<<blocks, 256, 0, stream>>>(sc, pts, P, row0));
  } else if (keys.mode == kVisRayPostponed) {
    TOTRI_KERNEL("mesh visibility", stream,
                 visibility_kernel<kVisRayPostponed><<<blocks, 256, 0, stream>>>(sc, pts, P,
                                                                                  row0));
  } else {
    // Chunks per CTA: up to 8 while the grid keeps 32 CTAs per SM (20,480 faces x
    // 4,096 points: 9.15 ms at 8, 9.3 at 4, 9.6 at 2, 10.4 at 1, 10.5 at 16; 20,000
    // faces x 400 and 144 points: 3.2 ms at the 6 and 2 that 8 CTAs per SM gave,
    // 2.7 ms at 1).
    const int64_t patches = ceil_div(P, 32) + ceil_div(P2, 32);
    int chunks = tune::get("mesh.visibility.chunks");
    if (chunks <= 0)
      chunks = (int)std::max<int64_t>(
          1, std::min<int64_t>(8, patches * sc.nch * sc.B / (32 * tune::sm_count())));
    if (chunks > kMaxPatchChunks)
      return fail(TOTRI_ERR_INVALID_ARGUMENT, "at most 16 face chunks per visibility block");
    const int seed_mode = tune::get("mesh.visibility.seed");
    if (seed_mode < kSeedBack || seed_mode > kSeedFront)
      return fail(TOTRI_ERR_INVALID_ARGUMENT, "visibility seed mode must be 0..3");
    int seed_steps = tune::get("mesh.visibility.seed.steps");
    if (seed_steps <= 0) seed_steps = 48;
    // candidate capacity of the shaft search (tests lower it to force the
    // per-lane search)
    int shaft_cap = tune::get("mesh.visibility.shaft.cap");
    if (shaft_cap <= 0 || shaft_cap > kShaftCand) shaft_cap = kShaftCand;
    const dim3 grid((unsigned)patches, (unsigned)ceil_div(sc.nch, chunks),
                    (unsigned)sc.B);
    const int64_t cta_count = (int64_t)grid.x * grid.y * grid.z;
    if (keys.mode == kVisPatchPacket)
      TOTRI_KERNEL("mesh visibility", stream,
                   visibility_patch_kernel<1><<<grid, 256, 0, stream>>>(
                       sc0, walls, chunks, kSeedOff, 0, 0));
    else if (keys.mode == kVisPatchWide)
      TOTRI_KERNEL("mesh visibility", stream,
                   visibility_patch_kernel<2><<<grid, 256, 0, stream>>>(
                       sc0, walls, chunks, kSeedOff, 0, 0));
    else if (keys.mode == kVisPatchShaft)
      TOTRI_KERNEL("mesh visibility", stream,
                   visibility_patch_kernel<3><<<grid, 256, 0, stream>>>(
                       sc0, walls, chunks, seed_mode, seed_steps, shaft_cap));
    else if (nsets == 1 && list_rule(sc, P, keys)) {
      int cap = tune::get("mesh.visibility.list.cap");
      if (cap <= 0 || cap > kListCand) cap = kListCand;
      // the queues' counters: the second quarter of the point scratch is free
      // once the points are sorted (it holds at least one word)
      uint32_t* next = sc.pscratch + (size_t)sc.B * P;
      const unsigned ctas = 8u * (unsigned)tune::sm_count();
      // Walks in runs of 8 faces where whole chunks are few for 4,864 warps (5,000
      // faces, 2,304 points: 0.84 against 0.98 of the patch kernel's time), of 32 else
      // (a run's faces seed each other: 20,480 faces, 4,096 points 2.5 against 3.7 ms).
      int parts = tune::get("mesh.visibility.list.parts");
      if (parts != 1 && parts != 4) parts = ceil_div(P, 32) * sc.nch * sc.B < 24576 ? 4 : 1;
      TOTRI_CUDA(cudaMemsetAsync(next, 0, sizeof(uint32_t), stream));
      TOTRI_KERNEL("mesh visibility", stream,
                   visibility_walk_kernel<8><<<ctas, 32 * kListWarps, 0, stream>>>(
                       sc, pts, P, row0, next, parts, seed_mode, seed_steps));
      TOTRI_CUDA(cudaMemsetAsync(next, 0, sizeof(uint32_t), stream));
      TOTRI_KERNEL("mesh visibility list", stream,
                   visibility_list_kernel<8><<<ctas, 32 * kListWarps, 0, stream>>>(
                       sc, pts, P, row0, next, cap));
    }
    // The default: the surface-walk prefix, then the 4-wide BVH search
    // (bvh_occluded_wide) with registers for 4 CTAs per SM (60, no spills):
    // 8.81 ms against 9.19 ms for the binary search at 5 CTAs per SM (48
    // registers, spilling) and 9.26 ms for the 4-wide search capped at 5, per
    // mesh_visibility call on the differentiable workload (build included).
    // "mesh.visibility.wide" = 2 selects the binary search.
    else if (keys.wide != 2 && keys.queue != 1) {
      if (keys.occupancy == 5)
        TOTRI_KERNEL("mesh visibility", stream,
                     visibility_patch_kernel<4, 5><<<grid, 256, 0, stream>>>(
                         sc0, walls, chunks, seed_mode, seed_steps, 0));
      // Grids that fill less than a wave: more warps per CTA, fewer faces in a row
      // per warp (768 faces x 143 and 35 points: 275 us with 8 warps, 190 with 16,
      // 152 with 32; 320 faces x 1,024 points: 77, 65 and 74 us).
      else if (cta_count <= tune::sm_count())
        TOTRI_KERNEL("mesh visibility", stream,
                     visibility_patch_kernel<4, 1, 32><<<grid, 1024, 0, stream>>>(
                         sc0, walls, chunks, seed_mode, seed_steps, 0));
      else if (cta_count <= 4 * tune::sm_count())
        TOTRI_KERNEL("mesh visibility", stream,
                     visibility_patch_kernel<4, 2, 16><<<grid, 512, 0, stream>>>(
                         sc0, walls, chunks, seed_mode, seed_steps, 0));
      else
        TOTRI_KERNEL("mesh visibility", stream,
                     visibility_patch_kernel<4, 4><<<grid, 256, 0, stream>>>(
                         sc0, walls, chunks, seed_mode, seed_steps, 0));
    }
    // The queued BVH searches (visibility_queue_kernel) when
    // "mesh.visibility.queue" = 1; queue entries pack the target's Morton
    // position in 26 bits.
    else if (keys.queue == 1 && sc.F < (1 << 26)) {
      if (keys.occupancy == 4)
        TOTRI_KERNEL("mesh visibility", stream,
                     visibility_queue_kernel<4><<<grid, 256, 0, stream>>>(
                         sc, pts, P, row0, chunks, seed_mode, seed_steps));
      else
        TOTRI_KERNEL("mesh visibility", stream,
                     visibility_queue_kernel<5><<<grid, 256, 0, stream>>>(
                         sc, pts, P, row0, chunks, seed_mode, seed_steps));
    }
    // Registers capped for 5 CTAs per SM (48 a thread, 28 bytes of spills):
    // 8.84 ms against 9.33 ms uncapped (60 registers, 4 CTAs) and 9.03 ms at
    // 6 CTAs (40 registers) inside the differentiable 20,480-face step.
    else if (keys.occupancy == 1)
      TOTRI_KERNEL("mesh visibility", stream,
                   visibility_patch_kernel<0, 1><<<grid, 256, 0, stream>>>(
                       sc0, walls, chunks, seed_mode, seed_steps, 0));
    else if (keys.occupancy == 4)
      TOTRI_KERNEL("mesh visibility", stream,
                   visibility_patch_kernel<0, 4><<<grid, 256, 0, stream>>>(
                       sc0, walls, chunks, seed_mode, seed_steps, 0));
    else if (keys.occupancy == 6)
      TOTRI_KERNEL("mesh visibility", stream,
                   visibility_patch_kernel<0, 6><<<grid, 256, 0, stream>>>(
                       sc0, walls, chunks, seed_mode, seed_steps, 0));
    else
      TOTRI_KERNEL("mesh visibility", stream,
                   visibility_patch_kernel<0, 5><<<grid, 256, 0, stream>>>(
                       sc0, walls, chunks, seed_mode, seed_steps, 0));
  }
  return TOTRI_OK;
}

int launch_visibility(const Scene& sc, const WallSet* sets, int nsets, const VisKeys& keys,
                      bool order, cudaStream_t stream) {
  if (order && keys.ordered()) {
    const int st = launch_point_order(sc, sets, nsets, stream);
    if (st != TOTRI_OK) return st;
  }
  // Two sets go in one launch of visibility_patch_kernel where that is the
  // kernel for both (no key selects another one, neither set takes the lists).
  const bool one = nsets == 2 && !keys.brute && keys.mode == 0 && keys.queue != 1 &&
                   sets[0].P > 0 && sets[1].P > 0 && !list_rule(sc, sets[0].P, keys) &&
                   !list_rule(sc, sets[1].P, keys);
  if (one) return launch_visibility_sets(sc, sets, 2, keys, stream);
  for (int j = 0; j < nsets; ++j) {
    const int st = launch_visibility_sets(sc, sets + j, 1, keys, stream);
    if (st != TOTRI_OK) return st;
  }
  return TOTRI_OK;
}

template <int TS>
static int launch_splat_ts(const Scene& sc, const View3f& sp, const View3f& so, int has_origin,
                           float* transient, int T, int S, float bw, float bo,
                           cudaStream_t stream) {
  const size_t smem = sizeof(float) * (size_t)T * TS;
  const dim3 grid((unsigned)ceil_div(S, TS), (unsigned)sc.B);
  if (tune::get("mesh.confocal.splat.mode") == 1) {
    TOTRI_CUDA(tune::ensure_dynamic_smem(
        reinterpret_cast<const void*>(splat_compact_kernel<TS>), smem));
    TOTRI_KERNEL("mesh confocal splat", stream,
                 splat_compact_kernel<TS><<<grid, 256, smem, stream>>>(
                     sc, sp, so, has_origin, transient, T, S, bw, bo,
                     make_fast_bins(bw, bo, tune::get("mesh.confocal.exact") != 1)));
    return TOTRI_OK;
  }
  TOTRI_CUDA(tune::ensure_dynamic_smem(
      reinterpret_cast<const void*>(splat_kernel<TS>), smem));
  TOTRI_KERNEL("mesh confocal splat", stream,
               splat_kernel<TS><<<grid, 256, smem, stream>>>(
                   sc, sp, so, has_origin, transient, T, S, bw, bo,
                   make_fast_bins(bw, bo, tune::get("mesh.confocal.exact") != 1)));
  return TOTRI_OK;
}

int launch_confocal_splat(const Scene& sc, const View3f& sp, const View3f& so, int has_origin,
                          float* transient, int T, int S, float bw, float bo,
                          cudaStream_t stream) {
  const size_t budget = 200 * 1024;
  const int want = tune::get("mesh.confocal.splat.ts");
  if (want > 0) {
    if ((size_t)T * want * 4 > budget)
      return fail(TOTRI_ERR_INVALID_ARGUMENT, "tuned scan tile too large for the bin count");
    switch (want) {
      case 1: return launch_splat_ts<1>(sc, sp, so, has_origin, transient, T, S, bw, bo, stream);
      case 2: return launch_splat_ts<2>(sc, sp, so, has_origin, transient, T, S, bw, bo, stream);
      case 4: return launch_splat_ts<4>(sc, sp, so, has_origin, transient, T, S, bw, bo, stream);
      case 8: return launch_splat_ts<8>(sc, sp, so, has_origin, transient, T, S, bw, bo, stream);
      case 16: return launch_splat_ts<16>(sc, sp, so, has_origin, transient, T, S, bw, bo, stream);
      default: return fail(TOTRI_ERR_INVALID_ARGUMENT, "scan tile must be 1, 2, 4, 8 or 16");
    }
  }
  // Columns (splat_columns_kernel with 8 scan points per tile) for large meshes and
  // for middling ones over few points, from 1,024 points on (us, the tiles below
  // against it on spheres; 1,024, 2,304 and 4,096 points):
  //   20,448 faces, 1,024 bins  431/292  749/353  871/650; 2,048: 549/424 616/505 1091/924
  //                 3,000 bins  456/523  802/611 1240/1130; 8,000: 913/1124 1637/1325 2726/2441
  //   12,320 faces, 2,048 bins  376/331  436/382  747/658; 3,000: 330/419 580/482 897/825
  //    7,920 faces, 2,048 bins  273/239  320/277  553/508; 3,000: 242/307 446/354 693/649
  //    5,040 faces, 1,024 bins  147/132  235/146  277/265; 2,048: 206/209 240/230 421/414
  //                 3,000 bins  194/273  364/306  559/542; 8,000: 497/619 874/707 1434/1257
  //    3,024 faces, 1,024 bins  104/98   164/110  194/193; 2,048: 151/160 179/174 311/311
  //    1,520 faces, 1,024 bins   72/70   104/82   122/136; 2,048: 109/114 130/131 226/225
  //      700 faces, 512 bins     39/41    58/44    63/74
  // Boxes of 4,800 to 20,172 faces: 0.47 to 0.98 of the tiles' time up to 2,048 bins,
  // 0.80 to 1.04 above from 2,304 points, 1.13 to 1.55 there at 1,024. The spheres span 0.6
  // m of 5.12; meshes that span 3 m, 19,880 faces: 0.90-0.92 at 2,048 bins, 0.87-0.99 above
  // from 2,304 points; 5,040 faces: 1.02-1.08 and 0.87-1.07, which stay with the tiles.
  // Above 1,024 bins two CTAs share an SM, and a second wave that is nearly empty costs
  // as much as a full one (20,448 faces, 2,048 and 3,000 bins: 0.81 and 0.81 of the tiles'
  // time at 2,401 points, 0.99 waves; 1.08 and 1.31 at 2,500, 1.03 waves; 1.29 and 1.22 at
  // 2,704; 0.85 and 0.93 at 3,136; 0.86 and 0.92 at 4,096, 1.68 waves; at 1,024, 0.42 waves,
  // 0.79 and 1.16).
  // Below 1,024 points its tiles leave SMs idle (20,480 faces, 256 points: 123/262),
  // and small meshes spend the time on the rows. With 32 points per tile: 670, 669
  // and 574 us in the first row. "mesh.confocal.splat.columns" = 1 turns it off, 8
  // and 32 select a tile, ".window" its bins.
  const int cols = tune::get("mesh.confocal.splat.columns");
  const int64_t all = (int64_t)S * sc.B;
  const double waves = (double)ceil_div(all, 8) / (2 * tune::sm_count());
  const double filled = waves / std::ceil(waves);  // of all waves together
  const bool large = T <= 1024 ? sc.F >= 4096
                               : sc.F >= 7680 && (T <= 2048 ? waves <= 1.0 || filled >= 0.6
                                                            : filled >= 0.8);
  const bool few = sc.F >= 1024 && all <= 16 * tune::sm_count() && T <= 1024;
  const int ct = cols > 0 ? cols : all >= 1024 && (large || few) ? 8 : 0;
  // (its sides and windows run forwards in time)
  if (ct > 1 && bw > 0.f && (size_t)T * 4 <= budget && tune::get("mesh.confocal.splat.mode") != 1)
    return launch_confocal_columns(sc, sp, so, has_origin, ct, transient, T, S, bw, bo, stream);
  // Built-in choice: the widest scan tile that keeps the histogram within
  // 40 KB (several CTAs per SM) and still gives every SM tiles to work on.
  const size_t kTileBytes = 40 * 1024;
  if ((size_t)T * 8 * 4 <= kTileBytes && S >= 8 * 152)
    return launch_splat_ts<8>(sc, sp, so, has_origin, transient, T, S, bw, bo, stream);
  if ((size_t)T * 4 * 4 <= kTileBytes && S >= 4 * 152)
    return launch_splat_ts<4>(sc, sp, so, has_origin, transient, T, S, bw, bo, stream);
  if ((size_t)T * 2 * 4 <= kTileBytes && S >= 2 * 152)
    return launch_splat_ts<2>(sc, sp, so, has_origin, transient, T, S, bw, bo, stream);
  if ((size_t)T * 4 <= budget)
    return launch_splat_ts<1>(sc, sp, so, has_origin, transient, T, S, bw, bo, stream);
  return fail(TOTRI_ERR_UNSUPPORTED, "number of bins too large for the shared-memory tile");
}

int launch_confocal_grad(const Scene& sc, const View3f& sp, const View3f& so, int has_origin,
                         const float* tgrad, int T, int S, float bw, float bo,
                         const GradOut& out, cudaStream_t stream) {
  constexpr int kMaxSlice = 16384;  // 64 KB of mask words per CTA
  const int split =
      tune::grad_split("mesh.confocal.grad.split", (int64_t)sc.nch * sc.B, S, kMaxSlice);
  const size_t smem = sizeof(uint32_t) * (size_t)ceil_div(S, split);
  const auto kernel = bw > 0.f ? grad_kernel<true> : grad_kernel<false>;
  TOTRI_CUDA(tune::ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem));
  const dim3 grid((unsigned)sc.nch, (unsigned)sc.B, (unsigned)split);
  TOTRI_KERNEL("mesh confocal grad", stream,
               kernel<<<grid, 256, smem, stream>>>(sc, sp, so, has_origin, tgrad, T, S, bw, bo,
                                                   fixed_division(bw, bo), out));
  return TOTRI_OK;
}

}  // namespace mesh
}  // namespace totri
