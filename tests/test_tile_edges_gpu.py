"""Kernels at the edges of their tiles and dispatch rules, against the oracle.

Where the inputs are small integers the sums are exact in FP32 below 2^24, so
the outputs must equal the oracle's bit for bit: one decision taken
differently changes an output by at least 1.
"""
import numpy as np
import pytest
import torch

import oracle
from totri_gb300.totri_cpp import reconstruct as K
from totri_gb300.totri_cpp import render as R

pytestmark = pytest.mark.gpu


def cu(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def points(g, n, z=0.0):
    return np.stack([g.uniform(-1, 1, n), g.uniform(-1, 1, n), np.full(n, z)], 1).astype(np.float32)


def rel(a, b):
    a = np.asarray(a, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


# (D, H, W), S, T, bin width: depths around the column of 4 voxels, one scan
# point to just past a tile of 8, one voxel row to several slices of the voxels,
# 512 and 1,024 threads per CTA (histograms below and above 100 KB)
ADJOINT = [((1, 1, 1), 1, 1, 0.02), ((3, 2, 5), 7, 40, 0.05), ((4, 1, 33), 8, 300, 0.01),
           ((5, 17, 3), 9, 300, 0.01), ((37, 40, 44), 17, 500, 0.008),
           ((9, 8, 70), 12, 3300, 0.0012), ((64, 48, 40), 3, 6400, 0.0006)]


@pytest.mark.parametrize("shape,S,T,bw", ADJOINT)
@pytest.mark.parametrize("origin", [False, True])
def test_velten_adjoint_edges(cuda_lib, shape, S, T, bw, origin):
    g = np.random.default_rng(S * 1000 + T)
    sp = points(g, S)
    so = points(g, S, -0.3) if origin else None
    st, en, bo = (-0.5, -0.4, 0.5), (0.45, 0.5, 1.4), 0.013
    # a single-voxel axis has no spacing (0 / 0): its voxels fall in no bin
    vol = g.integers(-3, 4, shape).astype(np.float64)
    ref = oracle.bp_confocal_velten_adjoint(vol, sp, so, T, st, en, bw, bo)
    out = torch.full((2, T, S), 7.0, device="cuda")
    both = np.stack([vol, 2 * vol]).astype(np.float32)
    so_t = cu(np.stack([so, so])) if origin else torch.empty((2, 0, 3), device="cuda")
    K.backprojection_confocal_velten_adjoint(cu(both), cu(np.stack([sp, sp])), so_t, out, st, en,
                                             bw, bo)
    got = out.double().cpu().numpy()
    assert np.array_equal(got[0], ref)
    assert np.array_equal(got[1], 2 * ref)


# (D, H, W), S, T, bin width, offset, z of the scan points: partial voxel
# blocks; one point, an odd count and counts around the tiles of 8, 16 and 32 and
# the batch of 256; bins of the whole volume before or past [0, T) and across its
# ends (rows staged as zeros); windows too small for a block (exact chain in
# place); scan points inside the volume (no window)
FORWARD = [((5, 3, 2), 1, 50, 0.05, 0.0, 0.0), ((16, 8, 8), 33, 300, 0.01, 0.0, 0.0),
           ((17, 9, 10), 255, 300, 0.01, 0.5, 0.0), ((30, 20, 12), 257, 200, 0.004, 1.2, 0.0),
           ((24, 24, 24), 47, 64, 0.02, 3.9, 0.0), ((24, 24, 24), 47, 64, 0.02, -1.5, 0.0),
           ((20, 20, 20), 31, 4000, 0.0008, 0.0, 0.0), ((9, 9, 9), 19, 4096, 0.0002, 1.0, 0.0),
           ((12, 11, 10), 21, 100, 0.02, 0.0, 0.9), ((1, 9, 9), 9, 100, 0.02, 0.0, 0.0)]


@pytest.mark.parametrize("shape,S,T,bw,bo,z", FORWARD)
@pytest.mark.parametrize("origin", [False, True])
def test_velten_forward_edges(cuda_lib, shape, S, T, bw, bo, z, origin):
    from totri_gb300 import autotune
    g = np.random.default_rng(S * 1000 + T)
    sp = points(g, S, z)
    so = points(g, S, -0.3) if origin else None
    st, en = (-0.5, -0.4, 0.5), (0.45, 0.5, 1.4)
    tr = g.integers(0, 16, (T, S)).astype(np.float32)
    ref = oracle.bp_confocal_velten(tr, sp, so, shape, st, en, bw, bo)
    so_t = cu(so[None]) if origin else torch.empty((1, 0, 3), device="cuda")
    try:
        for vz, n in ((0, 0), (2, 8), (4, 8), (4, 16), (4, 32)):
            autotune.set_tile("backprojection.velten.vz", vz)
            autotune.set_tile("backprojection.velten.points", n)
            out = torch.full((1,) + shape, 7.0, device="cuda")
            K.backprojection_confocal_velten_forward(cu(tr[None]), cu(sp[None]), so_t, out, st, en,
                                                     bw, bo)
            assert np.array_equal(out[0].double().cpu().numpy(), ref)
    finally:
        autotune.set_tile("backprojection.velten.vz", 0)
        autotune.set_tile("backprojection.velten.points", 0)


# (X, Y, Z), N, T, bin width, offset: one cell pair, columns around a slab of 64
# cells and past it, column tiles of 4 x 8 with remainders; runs of 8, 16 and 32
# points with a remainder; bin counts around the steps of 4 and chunks of 32
COLUMNS = [((1, 1, 2), 1, 700, 0.004, 0.0), ((4, 8, 64), 7, 161, 0.013, 0.0),
           ((5, 9, 65), 9, 162, 0.013, -0.4), ((3, 17, 20), 300, 131, 0.017, 0.0),
           ((13, 30, 130), 1100, 99, 0.02, 0.1), ((40, 41, 33), 2500, 64, 0.03, 0.3)]


@pytest.mark.parametrize("shape,N,T,bw,bo", COLUMNS)
def test_volume_adjoint_edges(cuda_lib, shape, N, T, bw, bo):
    """Against the exact FP64 adjoint, 1e-5 (columns of up to 200 cells)."""
    g = np.random.default_rng(N + T)
    mp = np.stack([g.uniform(-1, 1, N), g.uniform(-1, 1, N), g.uniform(0, 0.8, N)])
    mp = mp.astype(np.float32)
    org, size = (-0.5, -0.5, 0.5), (1.0, 1.0, 1.0)
    y = g.uniform(0.5, 1.5, (N, T)).astype(np.float32)
    ref = oracle.volume_confocal_adjoint(y, shape, mp, org, size, bw, bo)
    adj = torch.full(shape, 7.0, device="cuda")
    R.volume_confocal_adjoint(adj, cu(mp), cu(y), org, size, bw, bo)
    assert rel(adj.cpu().numpy(), ref) < 1e-5


# (D, H, W), S, L, T, bin width, offset: voxel blocks of 8 x 8 x 4 and laser groups
# of 8 with remainders; one scan point to several slices; bins that start before
# and end past [0, T); bins of one voxel in one bin, and past the staged 256
PAIRS = [((1, 1, 1), 1, 1, 300, 0.02, 0.0), ((5, 9, 3), 9, 7, 500, 0.01, 0.0),
         ((4, 8, 8), 33, 8, 120, 0.02, 1.3), ((9, 11, 17), 70, 9, 60, 0.05, 0.9),
         ((6, 7, 9), 5, 17, 3000, 0.0011, 0.5), ((6, 7, 9), 6, 3, 1500, 0.002, 1.0),
         ((7, 6, 5), 4, 2, 40, 0.4, -0.3)]


@pytest.mark.parametrize("shape,S,L,T,bw,bo", PAIRS)
def test_volume_pairs_edges(cuda_lib, shape, S, L, T, bw, bo):
    """Forward and gradient of the exhaustive volume render against the FP64
    oracle, 1e-5; the gradient with and without its workspace."""
    from totri_gb300 import _lib
    g = np.random.default_rng(S + T)
    sp, lp = points(g, S), points(g, L)
    vol = g.uniform(0.5, 1.5, (2,) + shape).astype(np.float32)
    st, en = (-0.5, -0.4, 0.5), (0.45, 0.5, 1.4)
    spt, lpt = (cu(np.stack([p.T, p.T])) for p in (sp, lp))
    none = torch.empty((2, 3, 0), device="cuda")
    out = torch.full((2, T, S, L), 7.0, device="cuda")
    R.volume_render_exhaustive_forward(cu(vol), spt, lpt, none, none, out, st, en, bw, bo)
    tg = g.uniform(0.5, 1.5, (2, T, S, L)).astype(np.float32)
    grad = torch.full((2,) + shape, 7.0, device="cuda")
    R.volume_render_exhaustive_grad_volume(cu(tg), spt, lpt, none, none, grad, st, en, bw, bo)
    inplace = torch.full((2,) + shape, 7.0, device="cuda")
    _lib.check(cuda_lib.totri_volume_exhaustive_grad_volume(
        *[_lib.array(t) for t in (cu(tg), spt, lpt, none, none, inplace)], _lib.vec3(st),
        _lib.vec3(en), bw, bo, _lib.stream_of(inplace.device)))
    for b in range(2):
        ref = oracle.volume_exhaustive_forward(vol[b], sp.T, lp.T, T, st, en, bw, bo)
        assert rel(out[b].cpu().numpy(), ref) < 1e-5
        ref = oracle.volume_exhaustive_adjoint(tg[b], shape, sp.T, lp.T, st, en, bw, bo)
        assert rel(grad[b].cpu().numpy(), ref) < 1e-5
        assert rel(inplace[b].cpu().numpy(), ref) < 1e-5


# (D, H, W), S, L, T, bin width, offset: voxel blocks of 8 x 8 x 16 and laser groups
# of 8 with remainders, one to several slices of the scan points, more bins than
# voxels (read in place), bins before and past [0, T), a single-voxel axis (no bin)
VELTEN_PAIRS = [((2, 2, 2), 1, 1, 200, 0.02, 0.0), ((17, 9, 10), 9, 7, 300, 0.01, 0.0),
                ((16, 8, 8), 5, 8, 64, 0.02, 1.9), ((33, 12, 7), 40, 17, 100, 0.02, 1.1),
                ((12, 10, 8), 6, 9, 2000, 0.0017, 0.0), ((1, 9, 9), 3, 2, 100, 0.03, -0.2)]


@pytest.mark.parametrize("shape,S,L,T,bw,bo", VELTEN_PAIRS)
@pytest.mark.parametrize("origin", [False, True])
def test_velten_pairs_edges(cuda_lib, shape, S, L, T, bw, bo, origin):
    from totri_gb300 import _lib
    g = np.random.default_rng(S + T)
    sp, lp = points(g, S), points(g, L)
    so, lo = (points(g, n, -0.3) if origin else None for n in (S, L))
    st, en = (-0.5, -0.4, 0.5), (0.45, 0.5, 1.4)
    tr = g.integers(0, 16, (2, T, S, L)).astype(np.float32)
    pair = [cu(np.stack([p, p])) for p in (sp, lp)]
    pair += [cu(np.stack([p, p])) if origin else torch.empty((2, 0, 3), device="cuda")
             for p in (so, lo)]
    out = torch.full((2,) + shape, 7.0, device="cuda")
    K.backprojection_exhaustive_velten_forward(cu(tr), *pair, out, st, en, bw, bo)
    inplace = torch.full((2,) + shape, 7.0, device="cuda")
    _lib.check(cuda_lib.totri_backprojection_exhaustive_velten_forward(
        *[_lib.array(t) for t in (cu(tr), *pair, inplace)], _lib.vec3(st), _lib.vec3(en), bw, bo,
        _lib.stream_of(inplace.device)))
    for b in range(2):
        ref = oracle.bp_exhaustive_velten(tr[b], sp, lp, so, lo, shape, st, en, bw, bo)
        assert np.array_equal(out[b].double().cpu().numpy(), ref)
        assert np.array_equal(inplace[b].double().cpu().numpy(), ref)


# (D, H, W), Gaussians, attributes: bricks of 16 x 16 x 8 (or 4) and 8 x 8 x 8 with
# remainders, single-voxel axes; Gaussian counts around the lane batches of 32,
# the shares of a brick (32, 64, 128) and the tiles of 256; every attribute
# specialisation (0-1, 2-4, 5-8)
RBF = [((1, 1, 1), 1, 1), ((9, 17, 18), 31, 0), ((8, 16, 16), 33, 1), ((5, 3, 40), 65, 2),
       ((12, 20, 9), 129, 4), ((17, 9, 33), 257, 1), ((7, 18, 15), 600, 5), ((11, 8, 8), 513, 8)]


@pytest.mark.parametrize("shape,N,A", RBF)
def test_rbf_edges(cuda_lib, shape, N, A):
    """Forward 1e-5 and gradient 1e-4 of the FP64 oracle."""
    from totri_gb300.totri_cpp import util as U
    g = np.random.default_rng(N + A)
    st, en = (-0.5, -0.5, 0.5), (0.5, 0.5, 1.5)
    rbf = np.concatenate([g.uniform(-0.5, 0.5, (N, 3)) + np.array([0, 0, 1.0]),
                          g.uniform(0.02, 0.3, (N, 1)), g.uniform(0.5, 1.5, (N, A))], 1)
    rbf = rbf.astype(np.float32)
    vol = torch.full((1, 1 + A) + shape, 7.0, device="cuda")
    U.rbf2volume_gaussian_forward(cu(rbf[None]), vol, st, en)
    ref = oracle.rbf2volume_forward(rbf, shape, st, en)
    assert rel(vol[0].cpu().numpy(), ref) < 1e-5
    vg = g.uniform(0.5, 1.5, (1 + A,) + shape).astype(np.float32)
    out = torch.zeros((1, N, 4 + A), device="cuda")
    U.rbf2volume_gaussian_grad(cu(rbf[None]), vol, cu(vg[None]), out, st, en)
    assert rel(out[0].cpu().numpy(), oracle.rbf2volume_grad(rbf, ref, vg, st, en)) < 1e-4


# (X, Y, Z), N, T, bin width, offset: tiles of 16, 8 and 4 points (by the bins that
# fit) with remainders, an odd bin count, one cell and two, slices of the voxels,
# negative bin centres, rows too long for shared memory (gradient only)
WALKS = [((1, 1, 1), 1, 900, 0.003, 0.0), ((3, 2, 2), 5, 901, 0.003, -0.2),
         ((20, 21, 40), 33, 333, 0.008, 0.0), ((30, 40, 50), 17, 200, 0.013, 0.05),
         ((4, 5, 9), 6, 4001, 0.0006, 0.0), ((4, 5, 9), 9, 6400, 0.0004, -0.1),
         ((4, 5, 9), 3, 9600, 0.00027, 0.0)]


@pytest.mark.parametrize("shape,N,T,bw,bo", WALKS)
def test_volume_walk_edges(cuda_lib, shape, N, T, bw, bo):
    """Forward 1e-5 and measurement-point gradient 1e-4 of the FP64 oracle (which
    takes the same FP32 cells)."""
    g = np.random.default_rng(N + T)
    mp = np.stack([g.uniform(-1, 1, N), g.uniform(-1, 1, N), g.uniform(0, 0.7, N)])
    mp = mp.astype(np.float32)
    org, size = (-0.5, -0.5, 0.5), (1.0, 1.0, 1.0)
    vol = g.uniform(0.5, 1.5, shape).astype(np.float32)
    if T * 32 <= 200 * 1024:
        ref = oracle.volume_confocal_forward(vol, mp, T, org, size, bw, bo)
        out = torch.full((N, T), 7.0, device="cuda")
        R.volume_confocal_forward(cu(vol), cu(mp), out, org, size, bw, bo)
        assert rel(out.cpu().numpy(), ref) < 1e-5
    y = g.uniform(0.5, 1.5, (N, T)).astype(np.float32)
    gm = torch.full((3, N), 7.0, device="cuda")
    R.volume_confocal_grad_measurement_points(gm, cu(vol), cu(mp), cu(y), org, size, bw, bo)
    ref = oracle.volume_confocal_grad_mp(vol, mp, y, org, size, bw, bo)
    assert rel(gm.cpu().numpy(), ref) < 1e-4


def _mesh(kind, faces, seed):
    from totri_gb300 import scenes
    if kind == "box":
        v, f, _ = scenes.random_box(faces, seed)
    elif kind == "sphere":
        v, f, _ = scenes.uv_sphere(faces, seed)
    else:  # a soup of large and tiny triangles, some degenerate
        g = np.random.default_rng(seed)
        c = g.uniform(-0.4, 0.4, (faces, 1, 3)) + np.array([0, 0, 1.0])
        v = c + g.normal(size=(faces, 3, 3)) * g.choice([0.2, 0.02, 0.0], (faces, 1, 1))
        v = torch.from_numpy(v.reshape(1, -1, 3).astype(np.float32))
        f = torch.arange(3 * faces, dtype=torch.int32).reshape(1, -1, 3)
    return v.cuda(), f.cuda()


# (mesh, faces, wall points): one point to just past blocks of 32, one face to past
# chunks of 32 and lists of 8
LISTS = [("soup", 1, 1), ("soup", 2, 33), ("soup", 31, 31), ("soup", 33, 64), ("soup", 300, 100),
         ("box", 300, 200), ("sphere", 700, 97), ("box", 3000, 300)]


@pytest.mark.parametrize("kind,faces,P", LISTS)
def test_visibility_lists_equal_brute_force(cuda_lib, kind, faces, P):
    """The candidate-list kernels give the brute-force masks bit for bit: the
    lists whole, capped so that groups and then single targets overflow to the
    BVH, the surface walk off, a wall 40 m away, and two items in a batch."""
    from totri_gb300 import autotune
    v, f = _mesh(kind, faces, faces + P)
    g = np.random.default_rng(P)
    near = points(g, P)
    far = points(g, P) * 20.0
    far[:, 2] = -40.0
    v2, f2 = torch.cat([v, v.flip(2)]), torch.cat([f, f])
    for sp in (near, far):
        pts = cu(np.stack([sp, sp]))
        bf = R.mesh_visibility(v2, f2, pts, brute_force=True)
        for cap, seed in ((0, 0), (40, 0), (1, 1)):
            keys = {"mesh.visibility.list": 1, "mesh.visibility.list.cap": cap,
                    "mesh.visibility.seed": seed}
            try:
                for k, x in keys.items():
                    autotune.set_tile(k, x)
                got = R.mesh_visibility(v2, f2, pts)
            finally:
                for k in keys:
                    autotune.set_tile(k, 0)
            assert torch.equal(got, bf), (cap, seed)


@pytest.mark.parametrize("faces", [1, 2, 31, 33, 320, 1024, 1025, 1535, 1536, 1537])
@pytest.mark.parametrize("P,B", [(1, 1), (33, 3), (2048, 1), (2049, 2)])
def test_small_build_equals_the_general_one(cuda_lib, faces, P, B):
    """Masks over the one-kernel build equal brute force over the general build:
    whole lists, a list cut short by an invalid face, 64-bit indices and a
    strided view, on both sides of the face limit and of the two point sorts."""
    from totri_gb300 import autotune
    g = np.random.default_rng(7 * faces + P)
    V = faces // 2 + 3
    verts = g.uniform(-1.0, 1.0, (B, V, 3)).astype(np.float32)
    verts[..., 2] += 2.0
    verts[:, V - 1] = verts[:, 0]  # a repeated vertex: equal Morton codes, degenerate faces
    fac = g.integers(0, V, (B, faces, 3))
    cut = fac.copy()
    cut[B - 1, faces // 2, 1] = -1
    pts = np.stack([points(g, P) for _ in range(B)])
    wide = torch.zeros((B, 2 * P, 3), device="cuda")
    wide[:, ::2] = cu(pts)
    for f in (cu(fac.astype(np.int32)), cu(cut.astype(np.int64))):
        v = cu(verts)
        try:
            autotune.set_tile("mesh.build.small", 2)
            want = R.mesh_visibility(v, f, cu(pts), brute_force=True)
        finally:
            autotune.set_tile("mesh.build.small", 0)
        assert torch.equal(R.mesh_visibility(v, f, cu(pts)), want)
        assert torch.equal(R.mesh_visibility(v, f, wide[:, ::2]), want)
        assert torch.equal(R.mesh_visibility(v, f, cu(pts), brute_force=True), want)


@pytest.mark.parametrize("faces,S,L", [(300, 1, 1), (300, 33, 32), (60, 2100, 3), (60, 3, 65)])
def test_joint_scan_and_laser_masks(cuda_lib, faces, S, L):
    """Exhaustive renders whose scan and laser masks come from one launch, against
    the oracle: sums of FP32 terms of one sign, a few per bin (the bound of the
    other exhaustive renders)."""
    g = np.random.default_rng(S + L)
    v, f = _mesh("soup", faces, S)
    m = torch.rand((1, v.shape[1], 1), device="cuda") + 0.5
    sp, lp = points(g, S), points(g, L)
    none = torch.empty((1, 0, 3), device="cuda")
    out = torch.empty((1, 200, S, L), device="cuda")
    R.mesh_exhaustive_forward(v, f, m, cu(sp[None]), cu(lp[None]), none, none, out, 0.05, 0.0, 0)
    vn, fn = v[0].cpu().numpy(), f[0].cpu().numpy()
    ref = oracle.mesh_exhaustive_forward(vn, fn, m[0].cpu().numpy(), sp, lp, None, None,
                                         oracle.mesh_visibility(vn, fn, sp),
                                         oracle.mesh_visibility(vn, fn, lp), 200, 0.05, 0.0)
    assert np.linalg.norm(ref) > 0.0 or faces < 60
    assert rel(out[0].cpu().numpy(), ref) < 1e-5


# S, L, bins, bin width, bin offset, origins: one point to just past tiles of 8 and
# 32 columns, fewer lasers than a tile has columns (many scan points in a tile),
# bins to just past windows, an odd bin count (padded rows), a first bin inside
# the mesh's returns (corners before bin 0) and a last one inside them
EXHAUSTIVE = [(1, 1, 1, 6.0, 0.0, False), (3, 11, 97, 0.06, 0.0, False),
              (33, 1, 64, 0.1, 0.0, True), (1, 40, 301, 0.012, 2.3, False),
              (7, 33, 60, 0.02, 1.9, True), (40, 6, 500, 0.011, 0.0, True),
              (36, 32, 1021, 0.0051, 0.3, False)]


def _exhaustive(shape, seed):
    S, L, T, bw, bo, origin = shape
    g = np.random.default_rng(seed)
    v, f = _mesh("soup", 90, seed)
    m = torch.rand((1, v.shape[1], 1), device="cuda") + 0.5
    sp, lp = points(g, S), points(g, L)
    so, lo = (points(g, S, -0.4), points(g, L, -0.6)) if origin else (None, None)
    n = [x[0].cpu().numpy() for x in (v, f, m)]
    vis = [oracle.mesh_visibility(n[0], n[1], p) for p in (sp, lp)]
    none = torch.empty((1, 0, 3), device="cuda")
    dev = [v, f, m, cu(sp[None]), cu(lp[None]), cu(so[None]) if origin else none,
           cu(lo[None]) if origin else none]
    return dev, (*n, sp, lp, so, lo, *vis, T, bw, bo)


@pytest.mark.parametrize("shape", EXHAUSTIVE)
@pytest.mark.parametrize("cols,window", [(8, 0), (8, 50), (32, 0), (32, 37), (32, 700)])
def test_exhaustive_columns_edges(cuda_lib, shape, cols, window):
    """Sums of a few FP32 terms of one sign per bin, as in the other exhaustive
    renders, whose bound this is."""
    from totri_gb300 import autotune
    S, L, T, bw, bo, _ = shape
    dev, ref = _exhaustive(shape, S + L)
    out = torch.full((1, T, S, L), 5.0, device="cuda")
    try:
        autotune.set_tile("mesh.exhaustive.splat.columns", cols)
        autotune.set_tile("mesh.exhaustive.splat.window", window)
        R.mesh_exhaustive_forward(*dev, out, bw, bo, 0)
    finally:
        autotune.set_tile("mesh.exhaustive.splat.columns", 0)
        autotune.set_tile("mesh.exhaustive.splat.window", 0)
    assert rel(out[0].cpu().numpy(), oracle.mesh_exhaustive_forward(*ref)) < 1e-5


@pytest.mark.parametrize("shape", EXHAUSTIVE)
@pytest.mark.parametrize("layout", [0, 2])
def test_exhaustive_grad_edges(cuda_lib, shape, layout):
    """Either side in the lanes, bins-last rows and the caller's order; the bound
    of the other exhaustive gradients."""
    from totri_gb300 import autotune
    S, L, T, bw, bo, _ = shape
    dev, ref = _exhaustive(shape, S + L)
    tg = np.random.default_rng(T).standard_normal((T, S, L)).astype(np.float32)
    vg, mg = torch.empty_like(dev[0]), torch.empty_like(dev[2])
    try:
        autotune.set_tile("mesh.exhaustive.grad.layout", layout)
        R.mesh_exhaustive_grad_verts(*dev, cu(tg[None]), vg, mg, bw, bo, 0)
    finally:
        autotune.set_tile("mesh.exhaustive.grad.layout", 0)
    rv, rm = oracle.mesh_exhaustive_grad(*ref, tg)
    assert rel(vg[0].cpu().numpy(), rv) < 1e-5
    assert rel(mg[0].cpu().numpy(), rm) < 1e-5


def test_exhaustive_grad_follows_the_decided_bins(cuda_lib):
    """Slivers with corners within rounding of a bin edge: the gradient splits each
    tent where the decided bins say (one that did not moved two vertices by 5e-4,
    the whole by 2.6e-5). FP32 sums over some 100 pairs per vertex: 2e-6."""
    from totri_gb300 import scenes
    v, f, m = [x.cuda() for x in scenes.uv_sphere(20000, 8, center=(0.03, -0.05, 1.0))]
    m = m.reshape(1, -1, 1)
    sp, lp = scenes.wall_grid(5)[0].numpy(), scenes.wall_grid(4)[0].numpy()
    T, bw = 2048, 0.0025
    tg = torch.randn((1, T, 25, 16), generator=torch.Generator().manual_seed(3))
    none = torch.empty((1, 0, 3), device="cuda")
    vg, mg = torch.empty_like(v), torch.empty_like(m)
    R.mesh_exhaustive_grad_verts(v, f, m, cu(sp[None]), cu(lp[None]), none, none, tg.cuda(), vg,
                                 mg, bw, 0.0, 0)
    vn, fn, mn = v[0].cpu().numpy(), f[0].cpu().numpy(), m[0].cpu().numpy()
    rv, rm = oracle.mesh_exhaustive_grad(vn, fn, mn, sp, lp, None, None,
                                         oracle.mesh_visibility(vn, fn, sp),
                                         oracle.mesh_visibility(vn, fn, lp), T, bw, 0.0,
                                         tg[0].numpy())
    assert rel(vg[0].cpu().numpy(), rv) < 2e-6
    assert rel(mg[0].cpu().numpy(), rm) < 2e-6


# S, T, bin width, bin offset, origin, mesh: corners before bin 0 and after the last,
# one point, tents of one bin and of many, slivers with corners at bin edges
@pytest.mark.parametrize("S,T,bw,bo,origin,kind", [
    (1, 1, 6.0, 0.0, False, "soup"), (33, 40, 0.02, 1.9, False, "soup"),
    (64, 97, 0.06, 0.0, True, "soup"), (31, 900, 0.004, 0.3, True, "soup"),
    (36, 2048, 0.0025, 0.0, False, "sphere")])
def test_confocal_grad_edges(cuda_lib, S, T, bw, bo, origin, kind):
    """FP32 sums over a vertex's few hundred pairs, as in the exhaustive gradients,
    whose bound this is."""
    g = np.random.default_rng(S + T)
    v, f = _mesh(kind, 20000 if kind == "sphere" else 90, S)
    m = torch.rand((1, v.shape[1], 1), device="cuda") + 0.5
    sp = points(g, S)
    so = points(g, S, -0.4) if origin else None
    none = torch.empty((1, 0, 3), device="cuda")
    tg = g.standard_normal((T, S)).astype(np.float32)
    vg, mg = torch.empty_like(v), torch.empty_like(m)
    R.mesh_confocal_grad_verts(v, f, m, cu(sp[None]), cu(so[None]) if origin else none,
                               cu(tg[None]), vg, mg, bw, bo, 0)
    vn, fn, mn = v[0].cpu().numpy(), f[0].cpu().numpy(), m[0].cpu().numpy()
    rv, rm = oracle.mesh_confocal_grad(vn, fn, mn, sp, so, oracle.mesh_visibility(vn, fn, sp), T,
                                       bw, bo, tg)
    assert rel(vg[0].cpu().numpy(), rv) < 1e-5
    assert rel(mg[0].cpu().numpy(), rm) < 1e-5


@pytest.mark.parametrize("S,T,bw,bo,origin", [
    (1, 1, 6.0, 0.0, False), (9, 40, 0.02, 1.9, False), (33, 97, 0.06, 0.0, True),
    (64, 1021, 0.0051, 0.3, True), (31, 301, 0.012, 2.3, False)])
@pytest.mark.parametrize("cols,window", [(8, 0), (8, 50), (32, 0), (32, 37), (32, 700)])
def test_confocal_columns_edges(cuda_lib, S, T, bw, bo, origin, cols, window):
    """Sums of a few FP32 terms of one sign per bin, as in the other renders, whose
    bound this is."""
    from totri_gb300 import autotune
    g = np.random.default_rng(S + T)
    v, f = _mesh("soup", 300, S)
    m = torch.rand((1, v.shape[1], 1), device="cuda") + 0.5
    sp = points(g, S)
    so = points(g, S, -0.4) if origin else None
    none = torch.empty((1, 0, 3), device="cuda")
    out = torch.full((1, T, S), 5.0, device="cuda")
    try:
        autotune.set_tile("mesh.confocal.splat.columns", cols)
        autotune.set_tile("mesh.confocal.splat.window", window)
        R.mesh_confocal_forward(v, f, m, cu(sp[None]), cu(so[None]) if origin else none, out, bw,
                                bo, 0)
    finally:
        autotune.set_tile("mesh.confocal.splat.columns", 0)
        autotune.set_tile("mesh.confocal.splat.window", 0)
    vn, fn, mn = v[0].cpu().numpy(), f[0].cpu().numpy(), m[0].cpu().numpy()
    ref = oracle.mesh_confocal_forward(vn, fn, mn, sp, so, oracle.mesh_visibility(vn, fn, sp), T,
                                       bw, bo)
    assert rel(out[0].cpu().numpy(), ref) < 1e-5


@pytest.mark.parametrize("kind,faces,P", LISTS)
@pytest.mark.parametrize("wall", ["plane", "tilted", "line", "space"])
def test_walk_runs_and_point_orders(cuda_lib, kind, faces, P, wall):
    """Masks are the brute-force ones whatever the runs of the walk kernel and the
    order of the points: a wall along two axes, one across all three, points on a
    line and in space, with repeated points."""
    from totri_gb300 import autotune
    v, f = _mesh(kind, faces, faces + P)
    g = np.random.default_rng(faces)
    pts = points(g, P)
    if wall == "tilted":
        pts[:, 2] = 0.7 * pts[:, 0] - 0.4 * pts[:, 1] - 0.5
    elif wall == "line":
        pts[:, 1:] = 0.0
    elif wall == "space":
        pts[:, 2] = g.uniform(-2.0, 0.0, P).astype(np.float32)
    pts[P // 2] = pts[0]
    pts = cu(pts[None])
    bf = R.mesh_visibility(v, f, pts, brute_force=True)
    for parts, morton, lists in ((1, 0, 1), (4, 0, 1), (4, 1, 1), (0, 0, 2)):
        keys = {"mesh.visibility.list": lists, "mesh.visibility.list.parts": parts,
                "mesh.visibility.morton": morton}
        try:
            for k, x in keys.items():
                autotune.set_tile(k, x)
            got = R.mesh_visibility(v, f, pts)
        finally:
            for k in keys:
                autotune.set_tile(k, 0)
        assert torch.equal(got, bf), keys
