// Tile-shape and kernel-variant overrides (see tune.cu); 0 (unset) takes the
// default. Keys:
//   "mesh.confocal.splat.ts"    scan points per confocal splat CTA (1,2,4,8,16)
//   "mesh.confocal.splat.mode"  confocal splat variant (at its launcher)
//   "mesh.confocal.exact"       1: every confocal sample takes the exact chain
//   "mesh.confocal.grad.split"  scan-point slices per confocal gradient chunk
//   "mesh.exhaustive.splat.lt"  laser points per exhaustive splat CTA (1,4,8,16,32)
//   "mesh.exhaustive.splat.mode", "mesh.exhaustive.splat.occupancy"
//                               exhaustive splat variant / 1: uncapped registers
//   "mesh.exhaustive.splat.cluster" 1: tiles under 8 lasers flush alone (default:
//                               through a cluster, in whole 32-byte sectors)
//   "mesh.exhaustive.exact"     1: every exhaustive sample takes the exact chain
//   "mesh.exhaustive.grad.mode" 1 per-lane mask tests, 2 compacted triples
//                               (default: per-face point records)
//   "mesh.confocal.splat.columns", ".window",
//   "mesh.exhaustive.splat.columns", ".window" 1: never the columns kernel, 8 or 32:
//                               its tile / bins per pass (at its launcher)
//   "mesh.exhaustive.grad.faces" faces per CTA of the point-record gradient (1)
//   "mesh.exhaustive.grad.occupancy" 4: that kernel capped for 4 CTAs/SM (64
//                               registers) instead of 3
//   "mesh.exhaustive.grad.lchunk", ".sslice" lasers / scan points per CTA of the
//                               point-record gradient (at most 256 each)
//   "mesh.exhaustive.grad.layout" 2: read transient_grad in place even when the
//                               workspace holds the bins-last scratch
//   "mesh.exhaustive.grad.chunk" most scan points per bins-last copy
//   "mesh.exhaustive.grad.split" scan-point slices per exhaustive gradient chunk
//   "mesh.visibility.mode"      1 per-lane BVH walk, 2 warp-packet walk, 7 one hull
//                               per target (at its launcher)
//   "mesh.visibility.queue"     1: queued BVH searches (visibility_queue_kernel)
//   "mesh.visibility.list", ".list.cap" 1: front-facing targets over candidate lists always,
//                               2: never (at its launcher) / most candidates in a list
//   "mesh.visibility.list.parts" runs of a face chunk in its walk kernel (1, 4)
//   "mesh.visibility.morton"    1: wall points in Morton order always
//   "mesh.build.small"          2: small meshes take the build of large ones too
//   "mesh.visibility.wide"      2: binary BVH search after the surface-walk prefix
//                               (the default is the 4-wide search)
//   "mesh.visibility.occupancy", ".chunks", ".seed", ".seed.steps", ".shaft.cap"
//                               visibility launch shape and prefix (at its launcher)
//   "volume.exact"              1: every volume sample takes the exact chain
//   "volume.forward.points", ".slices" points per CTA (4, 8, 16, 32; below 4: the built-in
//                               choice) and slices of the voxels, forward and
//                               measurement-point gradient
//   "volume.adjoint.mode"       0 lanes over 32 columns (default), 1 shared-memory
//                               atomics, 2 lane-owned cells (up to 256 cells)
//   "volume.adjoint.warps"      warps per CTA of the lanes-over-columns adjoint
//   "volume.adjoint.slabs"      z slabs of its columns (default: slabs of <= 64 cells)
//   "volume.exhaustive.lt"      laser points per exhaustive volume CTA (1,8,32)
//   "backprojection.velten.mode", ".vz", ".points"
//                               1: one voxel per thread without windows / voxels per
//                               thread (2, 4; 1 is taken as 2) / scan points per tile
//                               (8, 16, 32)
//   "backprojection.velten.pairs" 1: one voxel per thread in the exhaustive Velten
//   "rbf.cull"                  1: RBF kernels without the underflow cull
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace totri {
namespace tune {
int get(const char* key);  // 0 when unset
int sm_count();            // multiprocessors of the current device
// Slices of the scan-point loop for a gradient grid of `ctas` CTAs: enough for
// 32 CTAs per SM in total, at most one per 64 points (tuned value first),
// and never fewer than make each slice at most `max_slice` points long.
int grad_split(const char* key, int64_t ctas, int S, int max_slice);
// Raises the dynamic shared-memory limit of kernel `func` to at least `bytes`
// on the current device. The limit belongs to the (kernel, device) pair, so
// the value set is remembered per pair (under a lock: launches come from
// several host threads) and set again only when a launch needs more.
cudaError_t ensure_dynamic_smem(const void* func, size_t bytes);
}  // namespace tune
}  // namespace totri
