"""Calls at the limits of what the entry points take: units, widths, counts and
values far from an ordinary scan's, repeated calls, several faces per block."""
import numpy as np
import pytest
import torch

import oracle
from totri_gb300 import _lib, autotune, scenes
from totri_gb300.totri_cpp import reconstruct as K
from totri_gb300.totri_cpp import render as R

pytestmark = pytest.mark.gpu

START, END = (-0.5, -0.4, 0.5), (0.45, 0.5, 1.4)


def cu(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def points(g, n, z=0.0):
    return np.stack([g.uniform(-1, 1, n), g.uniform(-1, 1, n), np.full(n, z)], 1).astype(np.float32)


def rel(a, b):
    a = np.asarray(a, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


class tuned:
    """Tuning keys set for a block."""

    def __init__(self, keys):
        self.keys = keys

    def __enter__(self):
        for k, v in self.keys.items():
            autotune.set_tile(k, v)

    def __exit__(self, *_):
        for k in self.keys:
            autotune.set_tile(k, 0)


def sphere(faces, seed):
    """A sphere in front of the wall: half of its faces are seen from behind."""
    v, f, m = scenes.uv_sphere(faces, seed, center=(0.03, -0.05, 1.0))
    return v.cuda(), f.cuda(), m.reshape(1, -1, 1).cuda()


def mesh_masks(v, f, *walls):
    vn, fn = v[0].cpu().numpy(), f[0].cpu().numpy()
    return [oracle.mesh_visibility(vn, fn, p, bvh=f.shape[1] > 4000) for p in walls]


@pytest.mark.parametrize("faces_per_block", [1, 2, 5, 32])
def test_exhaustive_gradient_of_unseen_faces(cuda_lib, faces_per_block):
    """Several faces per block, runs of them seen by no scan point (FP32 sums of a
    vertex's few hundred pairs: 1e-5, as in the other exhaustive gradients)."""
    g = np.random.default_rng(3)
    v, f, m = sphere(2000, 8)
    sp, lp = points(g, 40), points(g, 9)
    none = torch.empty((1, 0, 3), device="cuda")
    T, bw = 300, 0.02
    tg = g.standard_normal((T, 40, 9)).astype(np.float32)
    vn, fn, mn = (x[0].cpu().numpy() for x in (v, f, m))
    rv, rm = oracle.mesh_exhaustive_grad(vn, fn, mn, sp, lp, None, None,
                                         *mesh_masks(v, f, sp, lp), T, bw, 0.0, tg)
    vg, mg = torch.empty_like(v), torch.empty_like(m)
    with tuned({"mesh.exhaustive.grad.faces": faces_per_block}):
        R.mesh_exhaustive_grad_verts(v, f, m, cu(sp[None]), cu(lp[None]), none, none,
                                     cu(tg[None]), vg, mg, bw, 0.0, 0)
    assert rel(vg[0].cpu().numpy(), rv) < 1e-5
    assert rel(mg[0].cpu().numpy(), rm) < 1e-5


def test_visibility_keys_changed_by_another_thread(cuda_lib):
    """A call takes its visibility keys once: masks of one wall (mesh_visibility) and of
    two (the exhaustive render, whose sums are those of the same pairs: 1e-5) while
    another thread cycles the kernels that do and do not read the points in order."""
    import threading
    g = np.random.default_rng(5)
    v, f, m = sphere(1700, 4)
    sp, lp = cu(points(g, 200)[None]), cu(points(g, 35)[None])
    none = torch.empty((1, 0, 3), device="cuda")
    want = R.mesh_visibility(v, f, sp, brute_force=True)
    ref = torch.empty((1, 200, 200, 35), device="cuda")
    R.mesh_exhaustive_forward(v, f, m, sp, lp, none, none, ref, 0.03, 0.0, 0)
    stop = threading.Event()

    def cycle():
        while not stop.is_set():
            for mode in (3, 4, 1, 0):
                autotune.set_tile("mesh.visibility.mode", mode)
            for queue in (1, 0):
                autotune.set_tile("mesh.visibility.queue", queue)

    other = threading.Thread(target=cycle)
    other.start()
    try:
        for _ in range(200):
            assert torch.equal(R.mesh_visibility(v, f, sp), want)
            out = torch.full_like(ref, 7.0)
            R.mesh_exhaustive_forward(v, f, m, sp, lp, none, none, out, 0.03, 0.0, 0)
            assert float((out - ref).norm() / ref.norm()) < 1e-5
    finally:
        stop.set()
        other.join()
        autotune.set_tile("mesh.visibility.mode", 0)
        autotune.set_tile("mesh.visibility.queue", 0)


@pytest.mark.parametrize("seed", [1, 3, 7])
def test_volume_pairs_whose_offset_takes_most_of_the_path(cuda_lib, seed):
    """Bins of 2e-8 at a path of 2.26 less an offset of 2.26: the lengths' roundings are
    several bins, so a block's bins have no sound bounds. FP32 fractions of the
    oracle's bins: 1e-5, as in the other gradients."""
    g = np.random.default_rng(seed)
    a, b, r, q = g.uniform(0, 6.28, 24), g.uniform(0, 6.28, 9), 0.6, 0.45
    sp = np.stack([r * np.cos(a), r * np.sin(a), 0 * a], 1).astype(np.float32)
    lp = np.stack([q * np.cos(b), q * np.sin(b), 0 * b], 1).astype(np.float32)
    st, en = (0.0, 0.0, 1.0), (1e-6, 1e-6, 1.000001)
    T, bw, bo = 12000, 2e-8, float(np.sqrt(1 + r * r) + np.sqrt(1 + q * q) - 1e-4)
    tg = g.uniform(0.5, 1.5, (T, 24, 9)).astype(np.float32)
    none = torch.empty((1, 3, 0), device="cuda")
    out = torch.empty((1, 4, 4, 4), device="cuda")
    R.volume_render_exhaustive_grad_volume(cu(tg[None]), cu(sp.T[None]), cu(lp.T[None]), none,
                                           none, out, st, en, bw, bo)
    ref = oracle.volume_exhaustive_adjoint(tg, (4, 4, 4), sp.T, lp.T, st, en, bw, bo)
    assert np.linalg.norm(ref) > 0.0
    assert rel(out[0].cpu().numpy(), ref) < 1e-5


@pytest.mark.parametrize("bo", [2.5, 3.2, 6.5])
def test_volume_pairs_with_a_negative_bin_width(cuda_lib, bo):
    """Time running backwards, with voxels whose later end is past [0, T) and whose
    earlier one is inside: such a voxel adds nothing, in the forward and in the
    gradient alike (the two are adjoint: 1e-5 of the product of the norms)."""
    g = np.random.default_rng(11)
    shape, S, L, T = (6, 7, 9), 5, 9, 100
    sp, lp = (cu(points(g, n).T[None]) for n in (S, L))
    none = torch.empty((1, 3, 0), device="cuda")
    vol = cu(g.uniform(0.5, 1.5, (1,) + shape).astype(np.float32))
    y = cu(g.uniform(0.5, 1.5, (1, T, S, L)).astype(np.float32))
    out = torch.empty_like(y)
    R.volume_render_exhaustive_forward(vol, sp, lp, none, none, out, START, END, -0.04, bo)
    grad = torch.empty_like(vol)
    R.volume_render_exhaustive_grad_volume(y, sp, lp, none, none, grad, START, END, -0.04, bo)
    out, grad, vol, y = (t.double() for t in (out, grad, vol, y))
    assert bool(torch.isfinite(out).all()) and bool(torch.isfinite(grad).all())
    scale = float(out.norm() * y.norm() + grad.norm() * vol.norm())
    assert scale > 0.0
    assert abs(float((out * y).sum() - (grad * vol).sum())) < 1e-5 * scale


@pytest.mark.parametrize("unit", [1e6, 1e8, 1e-6, 1e-8])
@pytest.mark.parametrize("exact", [0, 1])
def test_volume_render_in_other_units(cuda_lib, unit, exact):
    """A scene of a metre in micrometres, tens of nanometres, megametres and light
    centiseconds: forward and adjoint 1e-5 of the FP64 oracle on the same FP32 inputs,
    as in metres, the measurement-point gradient 1e-4 (where FP32 holds it)."""
    g = np.random.default_rng(7)
    shape, N, T = (9, 8, 13), 20, 120
    mp = np.stack([g.uniform(-1, 1, N), g.uniform(-1, 1, N), np.zeros(N)]) * unit
    mp = mp.astype(np.float32)
    org, size, bw = (-0.5 * unit, -0.5 * unit, 0.5 * unit), (unit, unit, unit), 0.02 * unit
    vol = g.uniform(0.5, 1.5, shape).astype(np.float32)
    y = g.uniform(0.5, 1.5, (N, T)).astype(np.float32)
    out = torch.full((N, T), 7.0, device="cuda")
    adj = torch.full(shape, 7.0, device="cuda")
    gm = torch.full((3, N), 7.0, device="cuda")
    with tuned({"volume.exact": exact}):
        R.volume_confocal_forward(cu(vol), cu(mp), out, org, size, bw, 0.0)
        R.volume_confocal_adjoint(adj, cu(mp), cu(y), org, size, bw, 0.0)
        R.volume_confocal_grad_measurement_points(gm, cu(vol), cu(mp), cu(y), org, size, bw, 0.0)
    assert rel(out.cpu().numpy(), oracle.volume_confocal_forward(vol, mp, T, org, size, bw, 0.0)) < 1e-5
    assert rel(adj.cpu().numpy(), oracle.volume_confocal_adjoint(y, shape, mp, org, size, bw, 0.0)) < 1e-5
    ref = oracle.volume_confocal_grad_mp(vol, mp, y, org, size, bw, 0.0)
    if np.abs(ref).max() < 1e37 and np.abs(ref).max() > 1e-33:
        assert rel(gm.cpu().numpy(), ref) < 1e-4


def test_volume_pairs_gradient_of_infinite_elements(cuda_lib):
    """Infinite elements of transient_grad give the infinities (and the NaN where both
    signs meet) of the oracle, with the workspace and without."""
    g = np.random.default_rng(2)
    shape, S, L, T = (5, 6, 7), 4, 3, 200
    sp, lp = points(g, S), points(g, L)
    tg = g.uniform(0.5, 1.5, (T, S, L)).astype(np.float32)
    tg[120, 1, 1], tg[130, 2, 0] = np.inf, -np.inf
    ref = oracle.volume_exhaustive_adjoint(tg, shape, sp.T, lp.T, START, END, 0.02, 0.0)
    assert np.isposinf(ref).any() and np.isneginf(ref).any() and np.isfinite(ref).any()
    none = torch.empty((1, 3, 0), device="cuda")
    args = [cu(tg[None]), cu(sp.T[None]), cu(lp.T[None]), none, none]
    out, inplace = (torch.empty((1,) + shape, device="cuda") for _ in range(2))
    R.volume_render_exhaustive_grad_volume(*args, out, START, END, 0.02, 0.0)
    _lib.check(cuda_lib.totri_volume_exhaustive_grad_volume(
        *[_lib.array(t) for t in (*args, inplace)], _lib.vec3(START), _lib.vec3(END), 0.02, 0.0,
        _lib.stream_of(out.device)))
    for got in (out[0].cpu().numpy(), inplace[0].cpu().numpy()):
        for kind in (np.isnan, np.isposinf, np.isneginf):
            assert np.array_equal(kind(got), kind(ref))


def test_exhaustive_calls_of_two_million_bins(cuda_lib):
    """More tiles of 32 bins than a grid has rows: the exhaustive Velten backprojection
    equals its one-voxel-per-thread kernel bit for bit (one pair: each voxel is one
    bin), the volume gradient its in-place reads (1e-5)."""
    T, none = 1 << 21, torch.empty((1, 0, 3), device="cuda")
    p = cu(np.array([[[0.1, -0.2, 0.0]]], np.float32))
    tr = torch.rand((1, T, 1, 1), device="cuda")
    shape = (1, 128, 128, 128)  # as many voxels as bins: the layout copy is used
    got, want = torch.empty(shape, device="cuda"), torch.empty(shape, device="cuda")
    K.backprojection_exhaustive_velten_forward(tr, p, p, none, none, got, START, END, 2e-6, 0.0)
    with tuned({"backprojection.velten.pairs": 1}):
        K.backprojection_exhaustive_velten_forward(tr, p, p, none, none, want, START, END, 2e-6,
                                                   0.0)
    assert float(want.abs().sum()) > 0.0
    assert torch.equal(got, want)
    T = 2100000
    tg = torch.rand((1, T, 1, 1), device="cuda")
    q, none = p.transpose(1, 2).contiguous(), torch.empty((1, 3, 0), device="cuda")
    grad, inplace = (torch.empty((1, 4, 4, 4), device="cuda") for _ in range(2))
    R.volume_render_exhaustive_grad_volume(tg, q, q, none, none, grad, START, END, 2e-6, 0.0)
    _lib.check(cuda_lib.totri_volume_exhaustive_grad_volume(
        *[_lib.array(t) for t in (tg, q, q, none, none, inplace)], _lib.vec3(START),
        _lib.vec3(END), 2e-6, 0.0, _lib.stream_of(grad.device)))
    assert float(inplace.abs().sum()) > 0.0
    assert float((grad - inplace).norm() / inplace.norm()) < 1e-5


def test_exhaustive_gradient_of_black_and_degenerate_faces(cuda_lib):
    """Faces of albedo zero and negative, and faces whose squared area is below the FP32
    range: they add nothing to the oracle's gradient and nothing (no NaN) here."""
    g = np.random.default_rng(4)
    v, f, m = sphere(300, 2)
    half = m.shape[1] // 2
    m[:, half:] = 0.0
    m[:, -20:] = -0.5
    tiny = torch.tensor([[[0.0, 0.0, 0.4], [1e-12, 0.0, 0.4], [0.0, 1e-12, 0.4]]]).cuda()
    tri = torch.arange(3, device="cuda", dtype=f.dtype).reshape(1, 1, 3) + v.shape[1]
    v, f = torch.cat([v, tiny], 1), torch.cat([f, tri, tri.flip(2)], 1)
    m = torch.cat([m, torch.ones((1, 3, 1), device="cuda")], 1)
    sp, lp = points(g, 20), points(g, 7)
    none = torch.empty((1, 0, 3), device="cuda")
    tg = g.standard_normal((200, 20, 7)).astype(np.float32)
    vn, fn, mn = (x[0].cpu().numpy() for x in (v, f, m))
    rv, rm = oracle.mesh_exhaustive_grad(vn, fn, mn, sp, lp, None, None,
                                         *mesh_masks(v, f, sp, lp), 200, 0.03, 0.0, tg)
    assert np.isfinite(rv).all() and np.isfinite(rm).all()
    vg, mg = torch.empty_like(v), torch.empty_like(m)
    R.mesh_exhaustive_grad_verts(v, f, m, cu(sp[None]), cu(lp[None]), none, none, cu(tg[None]),
                                 vg, mg, 0.03, 0.0, 0)
    assert rel(vg[0].cpu().numpy(), rv) < 1e-5
    assert rel(mg[0].cpu().numpy(), rm) < 1e-5


@pytest.mark.parametrize("bw,bo", [(-0.02, 5.0), (-0.3, 5.0), (-2.0, 8.0), (0.02, 0.0)])
def test_mesh_gradients_with_a_negative_bin_width(cuda_lib, bw, bo):
    """Time running backwards: both gradients against the oracle (1e-5, as forwards)."""
    g = np.random.default_rng(6)
    v, f, m = sphere(2000, 8)
    sp, lp = points(g, 40), points(g, 5)
    none, T = torch.empty((1, 0, 3), device="cuda"), 300
    vn, fn, mn = (x[0].cpu().numpy() for x in (v, f, m))
    vs, vl = mesh_masks(v, f, sp, lp)
    vg, mg = torch.empty_like(v), torch.empty_like(m)
    tg = g.standard_normal((T, 40)).astype(np.float32)
    R.mesh_confocal_grad_verts(v, f, m, cu(sp[None]), none, cu(tg[None]), vg, mg, bw, bo, 0)
    rv, rm = oracle.mesh_confocal_grad(vn, fn, mn, sp, None, vs, T, bw, bo, tg)
    assert np.linalg.norm(rv) > 0.0
    assert rel(vg[0].cpu().numpy(), rv) < 1e-5
    assert rel(mg[0].cpu().numpy(), rm) < 1e-5
    tg = g.standard_normal((T, 40, 5)).astype(np.float32)
    rv, rm = oracle.mesh_exhaustive_grad(vn, fn, mn, sp, lp, None, None, vs, vl, T, bw, bo, tg)
    for layout in (0, 2):
        with tuned({"mesh.exhaustive.grad.layout": layout}):
            R.mesh_exhaustive_grad_verts(v, f, m, cu(sp[None]), cu(lp[None]), none, none,
                                         cu(tg[None]), vg, mg, bw, bo, 0)
        assert rel(vg[0].cpu().numpy(), rv) < 1e-5
        assert rel(mg[0].cpu().numpy(), rm) < 1e-5


@pytest.mark.parametrize("T", [300, 2048])
def test_large_mesh_renders_with_a_negative_bin_width(cuda_lib, T):
    """A mesh large enough for the columns kernel is rendered by the tiles: equal to
    them but for the order of the adds (terms of both signs: 1e-4)."""
    g = np.random.default_rng(6)
    v, f, m = sphere(20000, 8)
    sp = cu(points(g, 1100)[None])
    none = torch.empty((1, 0, 3), device="cuda")
    calls = [((1, T, 1100), lambda out: R.mesh_confocal_forward(v, f, m, sp, none, out, -0.3, 5.0, 0)),
             ((1, T, 40, 30), lambda out: R.mesh_exhaustive_forward(
                 v, f, m, sp[:, :40], sp[:, :30], none, none, out, -0.3, 5.0, 0))]
    for shape, call in calls:
        got, want = torch.empty(shape, device="cuda"), torch.empty(shape, device="cuda")
        call(got)
        with tuned({"mesh.confocal.splat.columns": 1, "mesh.exhaustive.splat.columns": 1}):
            call(want)
        assert float(want.abs().sum()) > 0.0
        assert float((got - want).norm() / want.norm()) < 1e-4


@pytest.mark.parametrize("want", [1, 2, 3, 5])
def test_volume_walks_with_other_point_counts(cuda_lib, want):
    """"volume.forward.points" below 4 leaves the built-in choice, a count in between
    takes the next lower tile (it divided by zero points): the oracle's values."""
    g = np.random.default_rng(9)
    shape, N, T, bw = (5, 6, 7), 21, 90, 0.02
    mp = np.stack([g.uniform(-1, 1, N), g.uniform(-1, 1, N), np.zeros(N)]).astype(np.float32)
    vol = g.uniform(0.5, 1.5, shape).astype(np.float32)
    y = g.uniform(0.5, 1.5, (N, T)).astype(np.float32)
    org, size = (-0.5, -0.5, 0.5), (1.0, 1.0, 1.0)
    out, gm = torch.full((N, T), 7.0, device="cuda"), torch.full((3, N), 7.0, device="cuda")
    with tuned({"volume.forward.points": want}):
        R.volume_confocal_forward(cu(vol), cu(mp), out, org, size, bw, 0.0)
        R.volume_confocal_grad_measurement_points(gm, cu(vol), cu(mp), cu(y), org, size, bw, 0.0)
    ref = oracle.volume_confocal_forward(vol, mp, T, org, size, bw, 0.0)
    assert rel(out.cpu().numpy(), ref) < 1e-5
    ref = oracle.volume_confocal_grad_mp(vol, mp, y, org, size, bw, 0.0)
    assert rel(gm.cpu().numpy(), ref) < 1e-4


def repeats(call, times=8):
    """Whether `call` gives the same bits each time."""
    first = call()
    return all(torch.equal(call(), first) for _ in range(times - 1))


@pytest.mark.parametrize("N", [20, 200, 256, 500, 512])
@pytest.mark.parametrize("shape", [(20, 21, 22), (9, 10, 65)])
def test_volume_adjoint_of_few_points_repeats(cuda_lib, N, shape):
    """Up to 512 points the adjoint's sums have a fixed order; against the FP64 oracle
    1e-5, as with more points."""
    g = np.random.default_rng(N)
    mp = np.stack([g.uniform(-1, 1, N), g.uniform(-1, 1, N), np.zeros(N)]).astype(np.float32)
    y = g.uniform(0.5, 1.5, (N, 150)).astype(np.float32)
    org, size = (-0.5, -0.5, 0.5), (1.0, 1.0, 1.0)
    mpc, yc = cu(mp), cu(y)

    def call():
        out = torch.full(shape, 7.0, device="cuda")
        R.volume_confocal_adjoint(out, mpc, yc, org, size, 0.02, 0.0)
        return out

    assert repeats(call)
    ref = oracle.volume_confocal_adjoint(y, shape, mp, org, size, 0.02, 0.0)
    assert rel(call().cpu().numpy(), ref) < 1e-5


@pytest.mark.parametrize("shape,S,L,T", [((24, 24, 24), 256, 36, 300), ((5, 9, 3), 41, 7, 400)])
def test_exhaustive_velten_repeats(cuda_lib, shape, S, L, T):
    """The slices of a launch are added in order; bins-last copies and in place."""
    g = np.random.default_rng(S)
    sp, lp = cu(points(g, S)[None]), cu(points(g, L)[None])
    none = torch.empty((1, 0, 3), device="cuda")
    tr = cu(g.uniform(0.5, 1.5, (1, T, S, L)).astype(np.float32))

    def call():
        out = torch.full((1,) + shape, 7.0, device="cuda")
        K.backprojection_exhaustive_velten_forward(tr, sp, lp, none, none, out, START, END, 0.02,
                                                   0.0)
        return out

    assert repeats(call)
    ref = oracle.bp_exhaustive_velten(tr[0].cpu().numpy(), sp[0].cpu().numpy(),
                                      lp[0].cpu().numpy(), None, None, shape, START, END, 0.02, 0.0)
    assert rel(call()[0].cpu().numpy(), ref) < 1e-5


@pytest.mark.parametrize("shape,S,L,T", [((24, 24, 24), 256, 36, 300), ((5, 9, 3), 41, 7, 400)])
def test_exhaustive_volume_gradient_repeats(cuda_lib, shape, S, L, T):
    """The slices of a launch are added in order; against the FP64 oracle 1e-5."""
    g = np.random.default_rng(S)
    sp, lp = cu(points(g, S).T[None]), cu(points(g, L).T[None])
    none = torch.empty((1, 3, 0), device="cuda")
    tg = cu(g.uniform(0.5, 1.5, (1, T, S, L)).astype(np.float32))

    def call():
        out = torch.full((1,) + shape, 7.0, device="cuda")
        R.volume_render_exhaustive_grad_volume(tg, sp, lp, none, none, out, START, END, 0.02, 0.0)
        return out

    assert repeats(call)
    ref = oracle.volume_exhaustive_adjoint(tg[0].cpu().numpy(), shape, sp[0].cpu().numpy(),
                                           lp[0].cpu().numpy(), START, END, 0.02, 0.0)
    assert rel(call()[0].cpu().numpy(), ref) < 1e-5


def _pair_calls(S, L, T, shape):
    """The exhaustive backprojection and volume gradient of the same sizes: (call, with
    the workspace's use in it) each of an output tensor."""
    g = np.random.default_rng(S)
    sp, lp = cu(points(g, S)[None]), cu(points(g, L)[None])
    tr = cu(g.integers(0, 16, (1, T, S, L)).astype(np.float32))
    n1, n3 = torch.empty((1, 0, 3), device="cuda"), torch.empty((1, 3, 0), device="cuda")
    return tr, {
        "velten": lambda out: K.backprojection_exhaustive_velten_forward(
            tr, sp, lp, n1, n1, out, START, END, 0.02, 0.0),
        "volume": lambda out: R.volume_render_exhaustive_grad_volume(
            tr, sp.transpose(1, 2), lp.transpose(1, 2), n3, n3, out, START, END, 0.02, 0.0)}


@pytest.mark.parametrize("kind", ["velten", "volume"])
def test_exhaustive_calls_without_memory_for_scratch(cuda_lib, kind, monkeypatch):
    """Where the scratch cannot be allocated the transient is read in place (integers
    and partial sums of a few hundred pairs: 1e-5)."""
    shape = (1, 9, 10, 11)
    _, calls = _pair_calls(33, 20, 200, shape)
    want, got = torch.empty(shape, device="cuda"), torch.empty(shape, device="cuda")
    calls[kind](want)
    empty = torch.empty

    def no_scratch(*args, **kw):
        if kw.get("dtype") == torch.uint8:
            raise torch.cuda.OutOfMemoryError("no memory")
        return empty(*args, **kw)

    monkeypatch.setattr(torch, "empty", no_scratch)
    calls[kind](got)
    assert float((got - want).norm() / want.norm()) < 1e-5


def test_exhaustive_velten_takes_no_copies_that_it_does_not_use(cuda_lib):
    """A volume of fewer voxels than bins is read in place: no copy of the transient."""
    shape = (1, 8, 8, 8)
    tr, calls = _pair_calls(100, 50, 2000, shape)
    out = torch.empty(shape, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    calls["velten"](out)
    assert torch.cuda.max_memory_allocated() - before < tr.numel() * 4 // 4


def test_exhaustive_calls_of_a_wrong_rank(cuda_lib):
    """Refused by the entry point, as every other wrong shape."""
    t = lambda *s: torch.zeros(s, device="cuda")
    none = t(1, 0, 3)
    with pytest.raises((ValueError, RuntimeError), match="dimensions"):
        K.backprojection_exhaustive_velten_forward(t(5), t(3), t(3), none, none, t(1, 4, 4, 4),
                                                   START, END, 0.02, 0.0)
    with pytest.raises((ValueError, RuntimeError), match="dimensions"):
        R.volume_render_exhaustive_grad_volume(t(1, 9, 2, 2), t(1, 3, 2), t(1, 3, 2),
                                               t(1, 3, 0), t(1, 3, 0), t(4, 4), START, END, 0.02,
                                               0.0)


@pytest.mark.parametrize("vz", [1, 2, 4])
@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("T,bw,bo", [(300, 0.01, 0.0), (700, 0.003, 1.0), (64, 0.02, 3.9)])
def test_every_tiled_velten_kernel_equals_the_untiled_one(cuda_lib, vz, tile, T, bw, bo):
    """Each voxels-per-thread and points-per-tile kernel sums the same bins in the same
    order as the kernel without windows: bit for bit, on real-valued transients."""
    g = np.random.default_rng(T)
    shape, S = (1, 19, 10, 21), 133
    sp, so = cu(points(g, S)[None]), cu(points(g, S, -0.2)[None])
    tr = cu(g.standard_normal((1, T, S)).astype(np.float32))
    got, want = torch.empty(shape, device="cuda"), torch.empty(shape, device="cuda")
    with tuned({"backprojection.velten.mode": 1}):
        K.backprojection_confocal_velten_forward(tr, sp, so, want, START, END, bw, bo)
    with tuned({"backprojection.velten.vz": vz, "backprojection.velten.points": tile}):
        K.backprojection_confocal_velten_forward(tr, sp, so, got, START, END, bw, bo)
    assert float(want.abs().sum()) > 0.0
    assert torch.equal(got, want)


def test_exhaustive_calls_over_several_ranges_of_scan_points(cuda_lib):
    """A transient above 2 GiB: bins-last copies of 512 and then 88 scan points. The
    backprojection of small integers (sums below 2^24) equals the one-voxel-per-thread
    kernel bit for bit; the volume gradient of 30 scan points across the two ranges is
    a sum of 27,000 FP32 terms of one sign in another order than the oracle's: 1e-4."""
    S, L, T, shape = 600, 900, 1024, (1, 16, 8, 8)
    g = np.random.default_rng(1)
    spn, lpn = points(g, S), points(g, L)
    sp, lp = cu(spn[None]), cu(lpn[None])
    none = torch.empty((1, 0, 3), device="cuda")
    tr = torch.randint(0, 16, (1, T, S, L), device="cuda", dtype=torch.uint8).float()
    got, want = torch.empty(shape, device="cuda"), torch.empty(shape, device="cuda")
    K.backprojection_exhaustive_velten_forward(tr, sp, lp, none, none, got, START, END, 0.005, 0.0)
    with tuned({"backprojection.velten.pairs": 1}):
        K.backprojection_exhaustive_velten_forward(tr, sp, lp, none, none, want, START, END, 0.005,
                                                   0.0)
    assert float(want.abs().sum()) > 0.0
    assert torch.equal(got, want)
    tr[:, :, :500] = 0.0
    tr[:, :, 530:] = 0.0
    none = torch.empty((1, 3, 0), device="cuda")
    R.volume_render_exhaustive_grad_volume(tr, sp.transpose(1, 2), lp.transpose(1, 2), none, none,
                                           got, START, END, 0.005, 0.0)
    part = tr[0, :, 500:530].cpu().numpy()
    ref = oracle.volume_exhaustive_adjoint(part, shape[1:], spn[500:530].T, lpn.T, START, END,
                                           0.005, 0.0)
    assert rel(got[0].cpu().numpy(), ref) < 1e-4


@pytest.mark.parametrize("T", [150, 4100])
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("bw,bo,far", [(1e-30, 0.0, 0.0), (0.02, -1e8, 0.0), (0.02, 0.0, 3e37),
                                       (0.02, 0.0, float("inf")), (1e-9, -3.0, 0.0)])
def test_volume_gradients_of_bins_out_of_reach(cuda_lib, T, mode, bw, bo, far):
    """First bins beyond 2^31 (a tiny bin width, an offset far below zero, points far
    away): empty spans, so the near points alone are in the adjoint (1e-5 of the FP64
    oracle) and the far ones get no gradient."""
    g = np.random.default_rng(12)
    shape, N = (5, 9, 40), 70
    mp = np.stack([g.uniform(-1, 1, N), g.uniform(-1, 1, N), np.zeros(N)]).astype(np.float32)
    y = g.uniform(0.5, 1.5, (N, T)).astype(np.float32)
    vol = g.uniform(0.5, 1.5, shape).astype(np.float32)
    org, size = (-0.5, -0.5, 0.5), (1.0, 1.0, 1.0)
    near = np.ones(N, bool)
    if far:
        near[::3] = False
        mp[0, ::3] = far
    adj, gm = torch.full(shape, 7.0, device="cuda"), torch.full((3, N), 7.0, device="cuda")
    with tuned({"volume.adjoint.mode": mode}):
        R.volume_confocal_adjoint(adj, cu(mp), cu(y), org, size, bw, bo)
    R.volume_confocal_grad_measurement_points(gm, cu(vol), cu(mp), cu(y), org, size, bw, bo)
    ref = oracle.volume_confocal_adjoint(y[near], shape, mp[:, near], org, size, bw, bo)
    assert rel(adj.cpu().numpy(), ref) < 1e-5
    assert not bool(gm[:, torch.as_tensor(~near).cuda()].any())


def test_volume_point_gradient_of_voxels_out_of_reach(cuda_lib):
    """An infinite voxel behind every point's samples adds nothing to their gradient
    (1e-4 of the FP64 oracle without it)."""
    g = np.random.default_rng(13)
    shape, N, T = (5, 6, 9), 40, 60
    mp = np.stack([g.uniform(-1, 1, N), g.uniform(-1, 1, N), np.zeros(N)]).astype(np.float32)
    y = g.uniform(0.5, 1.5, (N, T)).astype(np.float32)
    vol = g.uniform(0.5, 1.5, shape).astype(np.float32)
    vol[:, :, -1] = 0.0
    org, size = (-0.5, -0.5, 0.5), (1.0, 1.0, 1.0)
    ref = oracle.volume_confocal_grad_mp(vol, mp, y, org, size, 0.01, 0.0)  # bins to 0.6
    assert np.linalg.norm(ref) > 0.0
    vol[2, 3, -1] = np.inf
    gm = torch.full((3, N), 7.0, device="cuda")
    R.volume_confocal_grad_measurement_points(gm, cu(vol), cu(mp), cu(y), org, size, 0.01, 0.0)
    assert rel(gm.cpu().numpy(), ref) < 1e-4


def test_velten_of_no_bins(cuda_lib):
    """A transient [1, 0, S], which has no address, gives zeros."""
    out = torch.full((1, 5, 6, 7), 7.0, device="cuda")
    K.backprojection_confocal_velten_forward(
        torch.empty((1, 0, 9), device="cuda"), torch.zeros((1, 9, 3), device="cuda"),
        torch.empty((1, 0, 3), device="cuda"), out, START, END, 0.02, 0.0)
    assert not bool(out.any())


@pytest.mark.parametrize("unit", [1e-6, 1e-4, 1e3])
def test_mesh_gradients_in_other_units(cuda_lib, unit):
    """A scene of a metre in megametres, tens of kilometres and millimetres: both
    gradients 1e-5 of the oracle, as in metres."""
    g = np.random.default_rng(8)
    v, f, m = sphere(1600, 3)
    v = v * unit
    sp, lp = points(g, 70) * np.float32(unit), points(g, 12) * np.float32(unit)
    none, T, bw = torch.empty((1, 0, 3), device="cuda"), 150, 0.02 * unit
    vn, fn, mn = (x[0].cpu().numpy() for x in (v, f, m))
    vs, vl = mesh_masks(v, f, sp, lp)
    vg, mg = torch.empty_like(v), torch.empty_like(m)
    tg = g.standard_normal((T, 70)).astype(np.float32)
    R.mesh_confocal_grad_verts(v, f, m, cu(sp[None]), none, cu(tg[None]), vg, mg, bw, 0.0, 0)
    rv, rm = oracle.mesh_confocal_grad(vn, fn, mn, sp, None, vs, T, bw, 0.0, tg)
    assert np.linalg.norm(rv) > 0.0
    assert rel(vg[0].cpu().numpy(), rv) < 1e-5
    assert rel(mg[0].cpu().numpy(), rm) < 1e-5
    tg = g.standard_normal((T, 70, 12)).astype(np.float32)
    R.mesh_exhaustive_grad_verts(v, f, m, cu(sp[None]), cu(lp[None]), none, none, cu(tg[None]),
                                 vg, mg, bw, 0.0, 0)
    rv, rm = oracle.mesh_exhaustive_grad(vn, fn, mn, sp, lp, None, None, vs, vl, T, bw, 0.0, tg)
    assert np.linalg.norm(rv) > 0.0
    assert rel(vg[0].cpu().numpy(), rv) < 1e-5
    assert rel(mg[0].cpu().numpy(), rm) < 1e-5


@pytest.mark.parametrize("P", [32, 64, 1024, 2048, 4096])
@pytest.mark.parametrize("wall", ["grid", "jitter", "random", "line", "one"])
def test_power_of_two_walls(cuda_lib, P, wall):
    """Masks of 2^k wall points are the brute-force ones in either order of the points:
    a 2^a x 2^b grid, one with its points moved, random points, points on a line and
    all in one place; two items of different walls in a batch."""
    g = np.random.default_rng(P)
    v, f, _ = sphere(500, 3)
    a = 1 << ((P.bit_length() - 1) // 2)
    x, y = np.meshgrid(np.linspace(-1, 1, a), np.linspace(-1, 1, P // a), indexing="ij")
    grid = np.stack([x.ravel(), y.ravel(), 0 * x.ravel()], 1).astype(np.float32)
    pts = {"grid": grid, "random": points(g, P), "one": np.repeat(grid[:1], P, 0),
           "jitter": grid + points(g, P) * np.float32(0.5 / a),
           "line": grid * np.float32([1, 0, 0])}[wall]
    both = cu(np.stack([pts, points(g, P)]))
    v2, f2 = torch.cat([v, v]), torch.cat([f, f])
    want = R.mesh_visibility(v2, f2, both, brute_force=True)
    for lists in (0, 1):
        with tuned({"mesh.visibility.list": lists}):
            assert torch.equal(R.mesh_visibility(v2, f2, both), want)


@pytest.mark.parametrize("faces,S,T", [(7800, 1024, 2048), (7800, 2304, 4100)])
def test_confocal_columns_of_many_bins(cuda_lib, faces, S, T):
    """The built-in choice above 2,048 bins, against the oracle (sums of a few FP32
    terms of one sign per bin, as in the other renders: 1e-5)."""
    g = np.random.default_rng(T)
    v, f, m = sphere(faces, 5)
    sp, bw = points(g, S), 5.12 / T
    none = torch.empty((1, 0, 3), device="cuda")
    out = torch.full((1, T, S), 7.0, device="cuda")
    R.mesh_confocal_forward(v, f, m, cu(sp[None]), none, out, bw, 0.0, 0)
    vn, fn, mn = (x[0].cpu().numpy() for x in (v, f, m))
    ref = oracle.mesh_confocal_forward(vn, fn, mn, sp, None, *mesh_masks(v, f, sp), T, bw, 0.0)
    assert rel(out[0].cpu().numpy(), ref) < 1e-5


@pytest.mark.parametrize("faces,S,L,T", [(4200, 60, 20, 2049), (12300, 62, 119, 2049),
                                         (4200, 60, 20, 4096), (1600, 40, 30, 4500)])
def test_exhaustive_columns_of_many_bins(cuda_lib, faces, S, L, T):
    """As above for the exhaustive render: tiles of 8 and 32 columns, long rows."""
    g = np.random.default_rng(T)
    v, f, m = sphere(faces, 5)
    sp, lp, bw = points(g, S), points(g, L), 5.12 / T
    none = torch.empty((1, 0, 3), device="cuda")
    out = torch.full((1, T, S, L), 7.0, device="cuda")
    R.mesh_exhaustive_forward(v, f, m, cu(sp[None]), cu(lp[None]), none, none, out, bw, 0.0, 0)
    vn, fn, mn = (x[0].cpu().numpy() for x in (v, f, m))
    ref = oracle.mesh_exhaustive_forward(vn, fn, mn, sp, lp, None, None,
                                         *mesh_masks(v, f, sp, lp), T, bw, 0.0)
    assert rel(out[0].cpu().numpy(), ref) < 1e-5


@pytest.mark.parametrize("shape,S,L,T", [((8, 8, 8), 160, 64, 256), ((3, 2, 2), 160, 33, 300),
                                         ((8, 8, 8), 304, 5, 300), ((9, 7, 20), 61, 41, 900),
                                         ((20, 20, 9), 3, 7, 2000)])
@pytest.mark.parametrize("share", [0.002, 0.02, 0.2, 1.0])
def test_exhaustive_volume_tiles(cuda_lib, shape, S, L, T, share):
    """The built-in laser tiles (32, 8 and 1) with remainders and voxels shared by 1 to 32
    threads: forward 1e-5 of the FP64 oracle."""
    g = np.random.default_rng(S + L)
    sp, lp = points(g, S), points(g, L)
    vol = g.uniform(0.5, 1.5, shape) * (g.uniform(size=shape) < share)
    vol.flat[0] = 1.0
    vol, none = vol.astype(np.float32), torch.empty((1, 3, 0), device="cuda")
    out = torch.full((1, T, S, L), 7.0, device="cuda")
    R.volume_render_exhaustive_forward(cu(vol[None]), cu(sp.T[None]), cu(lp.T[None]), none, none,
                                       out, START, END, 5.12 / T, 0.0)
    ref = oracle.volume_exhaustive_forward(vol, sp.T, lp.T, T, START, END, 5.12 / T, 0.0)
    assert rel(out[0].cpu().numpy(), ref) < 1e-5


@pytest.mark.parametrize("N,T", [(1, 300), (5, 2048), (700, 1024), (700, 1025), (1300, 2049),
                                 (90, 4097), (19, 9600), (3, 28200)])
def test_point_gradient_tiles(cuda_lib, N, T):
    """Tiles of 16, 8 and 4 points by the points and bins, and bin tables past shared
    memory: 1e-4 of the FP64 oracle."""
    g = np.random.default_rng(N + T)
    shape, bw = (5, 6, 11), 3.0 / T
    mp = np.stack([g.uniform(-1, 1, N), g.uniform(-1, 1, N), np.zeros(N)]).astype(np.float32)
    vol = g.uniform(0.5, 1.5, shape).astype(np.float32)
    y = g.uniform(0.5, 1.5, (N, T)).astype(np.float32)
    org, size = (-0.5, -0.5, 0.5), (1.0, 1.0, 1.0)
    gm = torch.full((3, N), 7.0, device="cuda")
    R.volume_confocal_grad_measurement_points(gm, cu(vol), cu(mp), cu(y), org, size, bw, 0.0)
    ref = oracle.volume_confocal_grad_mp(vol, mp, y, org, size, bw, 0.0)
    assert rel(gm.cpu().numpy(), ref) < 1e-4


@pytest.mark.parametrize("value", [float("inf"), -float("inf"), 3e38, float("nan")])
def test_volume_adjoint_of_infinite_elements(cuda_lib, value):
    """Elements of the transient that are infinite or huge give the
    oracle's infinities and NaN (in FP32, as sums of the same products)."""
    g = np.random.default_rng(14)
    shape, N, T = (9, 10, 13), 40, 150
    mp = np.stack([g.uniform(-1, 1, N), g.uniform(-1, 1, N), np.zeros(N)]).astype(np.float32)
    y = g.uniform(0.5, 1.5, (N, T)).astype(np.float32)
    y[3, 60], y[17, 75] = value, value
    org, size = (-0.5, -0.5, 0.5), (1.0, 1.0, 1.0)
    out = torch.full(shape, 7.0, device="cuda")
    R.volume_confocal_adjoint(out, cu(mp), cu(y), org, size, 0.02, 0.0)
    got = out.cpu().numpy()
    ref = oracle.volume_confocal_adjoint(y, shape, mp, org, size, 0.02, 0.0)
    with np.errstate(over="ignore"):
        ref = ref.astype(np.float32)
    for kind in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(kind(got), kind(ref))
    assert np.isfinite(ref).any() and (np.isfinite(value) or not np.isfinite(ref).all())


@pytest.mark.parametrize("N,T,bo", [(256, 4097, 0.0), (1, 6001, 0.0), (7, 6400, -0.7),
                                    (256, 6003, 0.0), (257, 6400, 0.0), (6, 9386, 0.0),
                                    (6, 9387, 0.0)])
def test_point_gradient_long_rows(cuda_lib, N, T, bo):
    """Rows of few points in shared memory above 6,000 bins, as long as four fit: 1e-4 of
    the FP64 oracle."""
    g = np.random.default_rng(N + T)
    shape, bw = (5, 6, 7), (3.0 - bo) / T
    mp = np.stack([g.uniform(-1, 1, N), g.uniform(-1, 1, N), np.zeros(N)]).astype(np.float32)
    vol = g.uniform(0.5, 1.5, shape).astype(np.float32)
    y = g.uniform(0.5, 1.5, (N, T)).astype(np.float32)
    org, size = (-0.5, -0.5, 0.5), (1.0, 1.0, 1.0)
    gm = torch.full((3, N), 7.0, device="cuda")
    R.volume_confocal_grad_measurement_points(gm, cu(vol), cu(mp), cu(y), org, size, bw, bo)
    ref = oracle.volume_confocal_grad_mp(vol, mp, y, org, size, bw, bo)
    assert rel(gm.cpu().numpy(), ref) < 1e-4
