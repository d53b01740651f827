"""Performance cases: the calls that users of this framework make, over the sizes they use.

A case is a dict of plain values. ``prepare(case, seed)`` makes its inputs on the GPU,
``run(state)`` is one pass through the public entry points (an autograd function and,
where the case has gradients, its backward), ``work(case)`` counts what the pass cannot
do without, and ``exact(case, seed)`` restates the pass in 64 bits with plain torch.

Kinds:
  confocal        confocal mesh render (MeshRenderConfocal), with the vertex and albedo
                  gradients of a mean squared error when ``grad``
  exhaustive      laser x detector mesh render (MeshRenderExhaustive) and its gradients
                  for a given transient gradient
  volume          confocal voxel-volume render (VolumeRenderConfocal) and its volume
                  gradient (the exact adjoint); measurement-point gradient when ``points``
  volume_pairs    laser x detector voxel-volume render (VolumeRenderExhaustive) and its
                  volume gradient
  velten          confocal backprojection (BackprojectionConfocalVelten), with the
                  gradient of the transient when ``grad``
  velten_pairs    laser x detector backprojection (BackprojectionExhaustiveVelten)
  rbf             Gaussian RBFs to a volume (Rbf2VolumeGaussian) and the RBF gradient
"""
import math

import numpy as np
import torch

from totri_gb300 import scenes
from totri_gb300.data.util import make_wall_grid
from totri_gb300.reconstruct import (BackprojectionConfocalVelten,
                                     BackprojectionExhaustiveVelten)
from totri_gb300.render import (MeshRenderConfocal, MeshRenderExhaustive, VolumeRenderConfocal,
                                VolumeRenderExhaustive)
from totri_gb300.types import BinDef, VolumeDef
from totri_gb300.util.rbf2volume import Rbf2VolumeGaussian

DEV = torch.device("cuda")
SPAN = 5.12  # metres of path that the bins of a scan cover, in few or many bins
START, END = (-0.5, -0.5, 0.5), (0.5, 0.5, 1.5)  # the hidden volume


def listed():
    return [
        # One iteration of a pose fit: a 320-face mesh against a 32 x 32 scan, forward
        # and gradients. The smallest call; launches and host time count.
        dict(name="confocal_fit_320", kind="confocal", mesh="ico", faces=320, batch=1, scan_w=32,
             scan_h=32, bins=512, origin=False, grad=True),
        # The differentiable render of a fitted 20,480-face surface.
        dict(name="confocal_step_20k", kind="confocal", mesh="ico", faces=20480, batch=1,
             scan_w=64, scan_h=64, bins=1024, origin=False, grad=True),
        # A preview or measurement simulation: forward only, many fine bins, a scan grid
        # of odd sides and a laser that stands off the wall.
        dict(name="confocal_render_box", kind="confocal", mesh="box", faces=12288, batch=1,
             scan_w=101, scan_h=67, bins=2048, origin=True, grad=False),
        # One mesh of a non-confocal batch: laser grid x detector grid, 2,048 bins.
        dict(name="exhaustive_step_20k", kind="exhaustive", mesh="sphere", faces=20000, scan_w=20,
             scan_h=20, laser_w=12, laser_h=12, bins=2048, origin=False),
        # A small non-confocal fit with odd grids and both origins off the wall.
        dict(name="exhaustive_odd_small", kind="exhaustive", mesh="box", faces=768, scan_w=13,
             scan_h=11, laser_w=7, laser_h=5, bins=600, origin=True),
        # Volume render and its adjoint on the 128^3 grid of a full scan.
        dict(name="volume_step_128", kind="volume", x=128, y=128, z=128, fill=0.02, scan_w=128,
             scan_h=128, bins=1024, points=False),
        # A coarse volume being optimised together with its scan positions.
        dict(name="volume_odd_small", kind="volume", x=41, y=37, z=53, fill=0.1, scan_w=29,
             scan_h=31, bins=500, points=True),
        # Volume render between separate lasers and detectors.
        dict(name="volume_pairs_48", kind="volume_pairs", x=56, y=40, z=48, fill=0.02, scan_w=16,
             scan_h=16, laser_w=6, laser_h=6, bins=1024),
        # Reconstruction of a full scan into 128^3 voxels.
        dict(name="velten_128", kind="velten", x=128, y=128, z=128, scan_w=128, scan_h=128,
             bins=1024, origin=False, grad=False),
        # A finely binned scan of odd size into an odd volume, inside a differentiable
        # reconstruction: backprojection and its adjoint.
        dict(name="velten_fine_step", kind="velten", x=96, y=88, z=72, scan_w=72, scan_h=60,
             bins=4096, origin=True, grad=True),
        # Reconstruction from separate lasers and detectors.
        dict(name="velten_pairs_48", kind="velten_pairs", x=48, y=48, z=48, scan_w=16, scan_h=16,
             laser_w=8, laser_h=8, bins=1024),
        # A Gaussian scene splatted to 128^3 voxels, and the gradient of its parameters.
        dict(name="rbf_step_4096", kind="rbf", count=4096, attributes=1, x=128, y=128, z=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi, most):
    """A grid of w x h points with sides of lo to hi and at most `most` points."""
    w = _log(rng, lo, hi)
    h = max(1, min(_log(rng, max(lo, int(0.6 * w)), max(lo, int(1.5 * w))), hi, most // w))
    return w, h


def draw(rng):
    kind = rng.choice(["confocal", "confocal", "exhaustive", "volume", "volume_pairs", "velten",
                       "velten", "velten_pairs", "rbf"])
    if kind == "confocal":
        mesh = rng.choice(["ico", "sphere", "box"])
        faces = 20 * 4 ** rng.randint(2, 5) if mesh == "ico" else _log(rng, 320, 20480)
        batch = rng.choice([1, 1, 2, 3])
        w, h = _grid(rng, 16, 101, max(256, 80_000_000 // (faces * batch)))
        return dict(kind=kind, mesh=mesh, faces=faces, batch=batch, scan_w=w, scan_h=h,
                    bins=_log(rng, 400, 2048), origin=rng.random() < 0.4,
                    grad=rng.random() < 0.7)
    if kind == "exhaustive":
        faces = _log(rng, 500, 20000)
        lw, lh = _grid(rng, 4, 12, 144)
        w, h = _grid(rng, 8, 20, max(64, int(1.1e9) // (faces * lw * lh)))
        return dict(kind=kind, mesh=rng.choice(["sphere", "box"]), faces=faces, scan_w=w,
                    scan_h=h, laser_w=lw, laser_h=lh, bins=_log(rng, 500, 2048),
                    origin=rng.random() < 0.4)
    if kind == "volume":
        x, y, z = (_log(rng, 32, 128) for _ in range(3))
        w, h = _grid(rng, 24, 128, 16384)
        return dict(kind=kind, x=x, y=y, z=z, fill=round(0.005 * 10 ** rng.uniform(0, 1), 4),
                    scan_w=w, scan_h=h, bins=_log(rng, 400, 1024),
                    points=x * y * w * h < 4_000_000)
    if kind == "volume_pairs":
        x, y, z = (_log(rng, 16, 56) for _ in range(3))
        lw, lh = _grid(rng, 2, 6, 36)
        w, h = _grid(rng, 6, 16, 256)
        return dict(kind=kind, x=x, y=y, z=z, fill=round(0.02 * 5 ** rng.uniform(0, 1), 4),
                    scan_w=w, scan_h=h, laser_w=lw, laser_h=lh, bins=_log(rng, 500, 1024))
    if kind == "velten":
        x, y, z = (_log(rng, 48, 128) for _ in range(3))
        grad = rng.random() < 0.4
        w, h = _grid(rng, 24, 128, max(600, int(2.6e9 if grad else 3.4e10) // (x * y * z)))
        return dict(kind=kind, x=x, y=y, z=z, scan_w=w, scan_h=h, bins=_log(rng, 512, 4096),
                    origin=rng.random() < 0.4, grad=grad)
    if kind == "velten_pairs":
        x, y, z = (_log(rng, 16, 48) for _ in range(3))
        lw, lh = _grid(rng, 2, 8, 64)
        w, h = _grid(rng, 6, 16, 256)
        return dict(kind=kind, x=x, y=y, z=z, scan_w=w, scan_h=h, laser_w=lw, laser_h=lh,
                    bins=_log(rng, 500, 1024))
    x, y, z = (_log(rng, 32, 128) for _ in range(3))
    return dict(kind=kind, count=_log(rng, 100, 4096), attributes=rng.choice([1, 1, 1, 3]), x=x,
                y=y, z=z)


# ---------------------------------------------------------------------------
# Inputs

def _bins(case):
    return BinDef(SPAN / case["bins"], 0.0, case["bins"])


def _volume_def(case):
    return VolumeDef(START, END, (case["z"], case["y"], case["x"]))


def _wall(w, h):
    """[1, w h, 3] points of the relay wall, x fastest."""
    return make_wall_grid(-1.0, 1.0, w, -1.0, 1.0, h, device=DEV)[None].contiguous()


def _mesh(case, seed):
    """(verts [B, V, 3], faces [B, F, 3], albedo [B, V, 1]): a hidden object near (0, 0, 1)."""
    items = []
    for b in range(case.get("batch", 1)):
        g = scenes.rng(seed * 8 + b)
        centre = (float(g.uniform(-0.1, 0.1)), float(g.uniform(-0.1, 0.1)),
                  float(g.uniform(0.95, 1.05)))
        if case["mesh"] == "ico":
            level = int(round(math.log(case["faces"] / 20, 4)))
            make = scenes.jittered_sphere if level < 3 else scenes.displaced_sphere
            items.append(make(level, seed * 8 + b, center=centre))
        elif case["mesh"] == "sphere":
            items.append(scenes.uv_sphere(case["faces"], seed * 8 + b, center=centre))
        else:
            items.append(scenes.random_box(case["faces"], seed * 8 + b, center=centre))
    return [torch.cat([m[k] for m in items]).to(DEV) for k in range(3)]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _measured(shape, seed):
    """Photon counts of a scan: a dim floor with bright returns."""
    u = torch.rand(shape, device=DEV, generator=_generator(seed))
    return u * u * u * u


def _origins(n, seed, away):
    """A laser or detector on a stand: one position, [1, 1, 3]."""
    g = scenes.rng(seed + 101)
    p = [float(g.uniform(-0.3, 0.3)), float(g.uniform(-0.3, 0.3)), away]
    return torch.tensor(p, device=DEV).reshape(1, 1, 3)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "rbf":
        s["volume_def"] = _volume_def(case)
        rbf = scenes.rbf_set(case["count"], seed)
        extra = case["attributes"] - 1
        if extra:
            g = scenes.rng(seed + 13)
            more = g.uniform(0.0, 1.0, size=(1, case["count"], extra)).astype(np.float32)
            rbf = torch.cat([rbf, torch.from_numpy(more)], dim=2)
        s["rbf"] = rbf.to(DEV).contiguous().requires_grad_(True)
        shape = (1, 1 + case["attributes"], case["z"], case["y"], case["x"])
        s["volume_grad"] = torch.randn(shape, device=DEV, generator=_generator(seed + 1))
        return s
    bd = s["bin_def"] = _bins(case)
    s["scan_points"] = _wall(case["scan_w"], case["scan_h"])
    S = s["scan_points"].shape[1]
    s["scan_origin"] = _origins(S, seed, -0.4) if case.get("origin") else None
    if "laser_w" in case:
        s["laser_points"] = _wall(case["laser_w"], case["laser_h"])
        s["laser_origin"] = _origins(0, seed + 1, -0.6) if case.get("origin") else None
        L = s["laser_points"].shape[1]
    if kind in ("confocal", "exhaustive"):
        verts, s["faces"], albedo = _mesh(case, seed)
        s["verts"], s["albedo"] = verts.requires_grad_(True), albedo.requires_grad_(True)
        B = verts.shape[0]
        if kind == "confocal":
            s["scan_points"] = s["scan_points"].expand(B, -1, -1).contiguous()
            if s["scan_origin"] is not None:
                s["scan_origin"] = s["scan_origin"].expand(B, -1, -1).contiguous()
        if kind == "confocal" and case["grad"]:
            # the measurement: a returning front that decays
            near = torch.tensor((0.0, 0.0, 0.75), device=DEV)
            first = 2.0 * (s["scan_points"][:1] - near).norm(dim=2) / bd.width  # [1, S]
            t = torch.arange(bd.num, device=DEV, dtype=torch.float32)[None, :, None]
            late = (t - first[:, None]) * bd.width
            noise = torch.rand((B, bd.num, S), device=DEV, generator=_generator(seed))
            s["target"] = torch.where(late >= 0, torch.exp(-late.abs() / 0.2), 0.0 * late) * \
                (0.5 + noise) * (40.0 * bd.width)
        if kind == "exhaustive":
            s["transient_grad"] = torch.randn((1, bd.num, S, L), device=DEV,
                                              generator=_generator(seed))
        return s
    if kind in ("volume", "volume_pairs"):
        g = _generator(seed)
        shape = (case["x"], case["y"], case["z"]) if kind == "volume" else \
            (1, case["z"], case["y"], case["x"])
        vol = torch.rand(shape, device=DEV, generator=g)
        there = torch.rand(shape, device=DEV, generator=g) < case["fill"]
        s["volume"] = (vol * there).requires_grad_(True)
        s["volume_def"] = _volume_def(case)
        if kind == "volume":
            pts = s["scan_points"][0].T.contiguous()
            if case["points"]:  # scan positions that are being calibrated
                jitter = torch.randn(pts.shape, device=DEV, generator=g) * 0.002
                pts = (pts + jitter).requires_grad_(True)
            s["points"] = pts
            s["transient_grad"] = torch.randn((S, bd.num), device=DEV, generator=g)
        else:
            s["scan_points"] = s["scan_points"].transpose(1, 2).contiguous()
            s["laser_points"] = s["laser_points"].transpose(1, 2).contiguous()
            s["transient_grad"] = torch.randn((1, bd.num, S, L), device=DEV, generator=g)
        return s
    s["volume_def"] = _volume_def(case)
    shape = (1, bd.num, S) if kind == "velten" else (1, bd.num, S, L)
    s["transient"] = _measured(shape, seed)
    if case.get("grad"):
        s["transient"].requires_grad_(True)
        s["volume_grad"] = torch.randn((1, case["z"], case["y"], case["x"]), device=DEV,
                                       generator=_generator(seed + 1))
    return s


# ---------------------------------------------------------------------------
# One pass

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "confocal":
        tr = MeshRenderConfocal.apply(s["verts"], s["faces"], s["scan_points"], s["bin_def"],
                                      s["albedo"], s["scan_origin"])
        if not case["grad"]:
            return dict(transient=tr.detach())
        loss = torch.mean((tr - s["target"]) ** 2)
        gv, ga = torch.autograd.grad(loss, (s["verts"], s["albedo"]))
        return dict(transient=tr.detach(), verts=gv, albedo=ga)
    if kind == "exhaustive":
        tr = MeshRenderExhaustive.apply(s["verts"], s["faces"], s["scan_points"],
                                        s["laser_points"], s["bin_def"], s["albedo"],
                                        s["scan_origin"], s["laser_origin"])
        gv, ga = torch.autograd.grad(tr, (s["verts"], s["albedo"]), s["transient_grad"])
        return dict(transient=tr.detach(), verts=gv, albedo=ga)
    if kind == "volume":
        vd, bd = s["volume_def"], s["bin_def"]
        tr = VolumeRenderConfocal.apply(s["volume"], s["points"], vd.start, vd.extent(), bd.num,
                                        bd.width, bd.offset)
        if not case["points"]:
            gv, = torch.autograd.grad(tr, (s["volume"],), s["transient_grad"])
            return dict(transient=tr.detach(), volume=gv)
        gv, gp = torch.autograd.grad(tr, (s["volume"], s["points"]), s["transient_grad"])
        return dict(transient=tr.detach(), volume=gv, points=gp)
    if kind == "volume_pairs":
        tr = VolumeRenderExhaustive.apply(s["volume"], s["scan_points"], s["laser_points"],
                                          s["volume_def"], s["bin_def"])
        gv, = torch.autograd.grad(tr, (s["volume"],), s["transient_grad"])
        return dict(transient=tr.detach(), volume=gv)
    if kind == "velten":
        vol = BackprojectionConfocalVelten.apply(s["transient"], s["scan_points"],
                                                 s["volume_def"], s["bin_def"], s["scan_origin"])
        if not case["grad"]:
            return dict(volume=vol)
        gt, = torch.autograd.grad(vol, (s["transient"],), s["volume_grad"])
        return dict(volume=vol.detach(), transient=gt)
    if kind == "velten_pairs":
        return dict(volume=BackprojectionExhaustiveVelten.apply(
            s["transient"], s["scan_points"], s["laser_points"], s["volume_def"], s["bin_def"],
            s["scan_origin"], s["laser_origin"]))
    vol = Rbf2VolumeGaussian.apply(s["rbf"], s["volume_def"])
    gr, = torch.autograd.grad(vol, (s["rbf"],), s["volume_grad"])
    return dict(volume=vol.detach(), rbf=gr)


# ---------------------------------------------------------------------------
# Necessary work of one pass (add, multiply, compare 1; fused multiply-add 2)

def work(case):
    kind = case["kind"]
    S = case.get("scan_w", 0) * case.get("scan_h", 0)
    L = case.get("laser_w", 0) * case.get("laser_h", 0)
    T = case.get("bins", 0)
    if kind in ("confocal", "exhaustive"):
        F, B = case["faces"], case.get("batch", 1)
        ray = 40 * math.ceil(math.log2(F)) + 144  # a BVH walk and its triangle tests
        edge = 1.1 / math.sqrt(F)                 # of an object about 0.6 m across
        b = 2.0 + 1.5 * edge / (SPAN / T)         # bins of one (face, path)
        mesh_bytes = B * F * (12 + 8 + 2)
        if kind == "confocal":
            grad = case["grad"]
            seen = 0.4 * S * F * B
            flops = S * F * B * ray + seen * (116 + 10 * b)
            nbytes = mesh_bytes + 4.0 * B * T * S
            if grad:
                flops += seen * (190 + 60 * b)
                nbytes += 2 * 4.0 * B * T * S + mesh_bytes
            return dict(bytes=nbytes, flops=flops)
        seen = 0.2 * S * L * F
        return dict(bytes=2 * mesh_bytes + 2 * 4.0 * T * S * L,
                    flops=(S + L) * F * ray + seen * (14 + 10 * b + 45 + 60 * b))
    if kind == "rbf":
        V, N, C = case["x"] * case["y"] * case["z"], case["count"], 1 + case["attributes"]
        pairs = 0.5 * V * N  # those whose Gaussian is not zero in single precision
        return dict(bytes=4.0 * V * C * 3, flops=pairs * (6 + 2 * C + 10 + 4 * C))
    V = case["x"] * case["y"] * case["z"]
    if kind == "volume":
        run_bins = 0.7 / (SPAN / T)                 # bins of one (point, column)
        samples = case["x"] * case["y"] * S * run_bins
        per_voxel = 2.0 * run_bins / case["z"] + 1  # samples of one (point, voxel)
        flops = case["fill"] * V * S * (10 + 15 * per_voxel) + 15 * samples
        if case["points"]:
            flops += case["fill"] * V * S * (10 + 30 * per_voxel)
        return dict(bytes=4.0 * (2 * V + 2 * S * T), flops=flops)
    if kind == "volume_pairs":
        b = 2.0 + (1.5 / case["z"]) / (SPAN / T)
        return dict(bytes=4.0 * (2 * V + 2 * S * L * T),
                    flops=V * S * L * (20 + 2 * b) * (1 + case["fill"]))
    if kind == "velten":
        n = 2 if case["grad"] else 1
        return dict(bytes=n * 4.0 * (V + S * T), flops=n * 12.0 * V * S)
    return dict(bytes=4.0 * (V + S * L * T), flops=V * (8.0 * (S + L) + 6.0 * S * L))


# ---------------------------------------------------------------------------
# The same passes in 64 bits

def _d(t):
    return t.detach().double()


def _f32(v):
    return float(np.float32(v))


def _hidden(o, tri, target):
    """[n, F] bool: whether another triangle of tri [F, 3, 3] hides the face's centroid
    target [F, 3] from the points o [n, 3]."""
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    F = tri.shape[0]
    hidden = torch.zeros((o.shape[0], F), dtype=torch.bool, device=o.device)
    d = target[None] - o[:, None]  # [n, F, 3]; the target lies at t = 1
    own = torch.arange(F, device=o.device)
    step = max(1, int(2e7) // max(1, o.shape[0] * F))
    for g0 in range(0, F, step):
        g = slice(g0, min(F, g0 + step))
        p = torch.cross(d[:, :, None], e2[g][None, None], dim=3)
        det = (p * e1[g]).sum(3)
        inv = 1.0 / det
        s = (o[:, None] - v0[g][None])[:, None]  # [n, 1, G, 3]
        u = (p * s).sum(3) * inv
        q = torch.cross(s, e1[g][None, None], dim=3)
        v = (q * d[:, :, None]).sum(3) * inv
        t = (q * e2[g][None, None]).sum(3) * inv
        hit = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0) & (t < 1)
        hit &= (own[g][None, :] != own[:, None])[None]
        hidden |= hit.any(2)
    return hidden


def _tents(c, alpha, bins, column, columns):
    """[bins, columns]: for each row of c [n, 3] (corner bin coordinates, any order) a tent
    of area alpha [n] over them, added to its column."""
    c = c.sort(dim=1).values
    c0, c1, c2 = c[:, 0:1], c[:, 1:2], c[:, 2:3]
    tiny = 1e-30
    peak = 2.0 * alpha[:, None] / (c2 - c0).clamp_min(tiny)
    first = c0.detach().floor()
    count = int((c2.detach().floor() - first).max().item()) + 1 if c.shape[0] else 0

    def area(e):  # of the tent left of e
        a = e.clamp(c0, c1) - c0
        b = c2 - e.clamp(c1, c2)
        left = 0.5 * peak * a * a / (c1 - c0).clamp_min(tiny)
        right = 0.5 * peak * b * b / (c2 - c1).clamp_min(tiny)
        whole = alpha[:, None] - right
        return torch.where(e >= c2, alpha[:, None] + 0 * e, torch.where(e >= c1, whole, left))

    out = torch.zeros(bins * columns, dtype=torch.float64, device=c.device)
    before = 0.0 * first
    for k in range(count):
        after = area(first + (k + 1.0))
        t = first[:, 0].long() + k
        ok = (t >= 0) & (t < bins)
        out = out.index_add(0, (t.clamp(0, bins - 1) * columns + column), (after - before)[:, 0] *
                            ok)
        before = after
    return out.view(bins, columns)


def _mesh_exact(case, s):
    F = s["faces"].shape[1]
    S = s["scan_points"].shape[1]
    L = s["laser_points"].shape[1] if "laser_points" in s else 0
    B = s["verts"].shape[0]
    if B * (S + L) * F * F > 6e8 or (L and S * L * F > 1e7):
        return None
    bw, bo, T = _f32(s["bin_def"].width), _f32(s["bin_def"].offset), s["bin_def"].num
    verts, albedo = (_d(s[k]).requires_grad_(True) for k in ("verts", "albedo"))
    images = []
    for b in range(B):
        tri = verts[b][s["faces"][b].long()]  # [F, 3, 3]
        rho = albedo[b, s["faces"][b].long(), 0].mean(1)
        centre = tri.mean(1)
        n = torch.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0], dim=1)
        nn = (n * n).sum(1).sqrt()

        def side(points, origin, b=b, tri=tri, centre=centre):
            p = _d(points)[b]
            seen = torch.cat([~_hidden(q, tri.detach(), centre.detach())
                              for q in p.split(max(1, int(1e6) // F))])
            off = torch.zeros(p.shape[0], dtype=torch.float64, device=p.device)
            if origin is not None:
                off = (p - _d(origin)[b]).norm(dim=1)
            return p, seen, off

        p, seen, off = side(s["scan_points"], s["scan_origin"])
        if not L:
            i, f = seen.nonzero(as_tuple=True)
            r = centre[f] - p[i]
            rr = (r * r).sum(1)
            alpha = 100.0 * rho[f] * r[:, 2] ** 2 * (n[f] * r).sum(1) ** 2 / (nn[f] * rr ** 4)
            d = (tri[f] - p[i][:, None]).norm(dim=2)
            images.append(_tents((2 * d + 2 * off[i][:, None] - bo) / bw, alpha, T, i, S))
            continue
        q, lit, loff = side(s["laser_points"], s["laser_origin"])
        i, l, f = (seen[:, None] & lit[None]).nonzero(as_tuple=True)
        rs, rl = centre[f] - p[i], centre[f] - q[l]
        alpha = 100.0 * rho[f] * rs[:, 2] * rl[:, 2] * (n[f] * rs).sum(1).abs() * \
            (n[f] * rl).sum(1).abs() / (nn[f] * (rs * rs).sum(1) ** 2 * (rl * rl).sum(1) ** 2)
        d = (tri[f] - p[i][:, None]).norm(dim=2) + (tri[f] - q[l][:, None]).norm(dim=2)
        images.append(_tents((d + (off[i] + loff[l])[:, None] - bo) / bw, alpha, T, i * L + l,
                             S * L).view(T, S, L))
    tr = torch.stack(images)
    if case["kind"] == "confocal" and not case["grad"]:
        return dict(transient=tr.detach())
    if case["kind"] == "confocal":
        loss = torch.mean((tr - _d(s["target"])) ** 2)
        gv, ga = torch.autograd.grad(loss, (verts, albedo))
    else:
        gv, ga = torch.autograd.grad(tr, (verts, albedo), _d(s["transient_grad"]))
    return dict(transient=tr.detach(), verts=gv, albedo=ga)


def _centres(lo, size, n):
    return lo + (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) * (size / n)


def _volume_exact(case, s):
    X, Y, Z, T = case["x"], case["y"], case["z"], case["bins"]
    N = s["points"].shape[1]
    if X * Y * N * T > 4e9:
        return None
    bw, bo = _f32(s["bin_def"].width), _f32(s["bin_def"].offset)
    size = [e - a for a, e in zip(START, END)]
    x = _centres(START[0], size[0], X).view(X, 1).expand(X, Y).reshape(-1)
    y = _centres(START[1], size[1], Y).view(1, Y).expand(X, Y).reshape(-1)
    vol, pts = (_d(s[k]).requires_grad_(True) for k in ("volume", "points"))
    flat = vol.reshape(X * Y, Z)
    tc = torch.arange(T, device=DEV, dtype=torch.float64) * bw + bo
    cells = torch.arange(X * Y, device=DEV)
    gv, gp, rows = torch.zeros_like(vol), torch.zeros_like(pts), []
    for i0 in range(0, N, 16):
        i1 = min(N, i0 + 16)
        w = pts[:, i0:i1]
        rho2 = (w[0, :, None] - x) ** 2 + (w[1, :, None] - y) ** 2  # [n, XY]
        d2 = tc[None, :, None] ** 2 - rho2[:, None]
        with torch.no_grad():
            zh = (w[2, :, None, None] + d2.clamp_min(0).sqrt() - START[2]) * (Z / size[2]) - 0.5
            ok = (d2 > 0) & (zh.floor() >= 0) & (zh.floor() + 1 < Z)
            i, t, c = ok.nonzero(as_tuple=True)
        depth = d2[i, t, c].sqrt()
        zh = (w[2][i] + depth - START[2]) * (Z / size[2]) - 0.5
        fl = zh.detach().floor()
        fr, k = zh - fl, fl.long()
        value = (1 - fr) * flat[cells[c], k] + fr * flat[cells[c], k + 1]
        value = value * (depth / tc[t] ** 2) ** 4
        out = torch.zeros((i1 - i0) * T, dtype=torch.float64, device=DEV)
        out = out.index_add(0, i * T + t, value).view(i1 - i0, T)
        a, b = torch.autograd.grad(out, (vol, pts), _d(s["transient_grad"])[i0:i1],
                                   retain_graph=True)
        gv, gp = gv + a, gp + b
        rows.append(out.detach())
    got = dict(transient=torch.cat(rows), volume=gv)
    if case["points"]:
        got["points"] = gp
    return got


def _volume_pairs_exact(case, s):
    X, Y, Z, T = case["x"], case["y"], case["z"], case["bins"]
    p, q = _d(s["scan_points"])[0].T, _d(s["laser_points"])[0].T
    S, L, V = p.shape[0], q.shape[0], X * Y * Z
    if S * L * V > 2e9:
        return None
    bw, bo = _f32(s["bin_def"].width), _f32(s["bin_def"].offset)
    size = [e - a for a, e in zip(START, END)]
    z, y, x = torch.meshgrid(_centres(START[2], size[2], Z), _centres(START[1], size[1], Y),
                             _centres(START[0], size[0], X), indexing="ij")
    half = 0.5 * size[2] / Z
    ends = [torch.stack((x, y, z + h), 3).reshape(V, 3) for h in (-half, half)]
    far = [[torch.cdist(e, w, compute_mode="donot_use_mm_for_euclid_dist") for e in ends]
           for w in (p, q)]  # [V, S] and [V, L] to the voxel's lower and upper end
    vol = _d(s["volume"]).reshape(V)
    tg = _d(s["transient_grad"])[0].reshape(T, S * L)
    tr = torch.zeros(T * S * L, dtype=torch.float64, device=DEV)
    gv = torch.zeros(V, dtype=torch.float64, device=DEV)
    col = torch.arange(S * L, device=DEV)[None]
    for v0 in range(0, V, 4096):
        v = slice(v0, min(V, v0 + 4096))
        b = [((far[0][e][v][:, :, None] + far[1][e][v][:, None]).reshape(-1, S * L) - bo) / bw
             for e in (0, 1)]
        lo, hi = torch.minimum(*b), torch.maximum(*b)
        first = lo.floor()
        count = int((hi.floor() - first).max().item()) + 1
        span = hi - lo
        for k in range(count):
            a = first + k
            part = (torch.minimum(hi, a + 1) - torch.maximum(lo, a)).clamp_min(0) / span
            part = torch.where(hi.floor() == first, (a == first).double(), part)
            t = a.long()
            part = part * ((t >= 0) & (t < T))
            at = t.clamp(0, T - 1) * (S * L) + col
            tr.index_add_(0, at.reshape(-1), (part * vol[v][:, None]).reshape(-1))
            gv[v] += (part * tg.reshape(-1)[at]).sum(1)
    return dict(transient=tr.view(1, T, S, L), volume=gv.view(1, Z, Y, X))


def _nodes(case):
    """[V, 3] voxel positions of a backprojection, first and last on the volume's faces."""
    ax = [torch.linspace(START[i], END[i], case["xyz"[i]], device=DEV, dtype=torch.float64)
          for i in range(3)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return torch.stack((x, y, z), 3).reshape(-1, 3)


def _velten_exact(case, s):
    T = case["bins"]
    bw, bo = _f32(s["bin_def"].width), _f32(s["bin_def"].offset)
    at = _nodes(case)
    p = _d(s["scan_points"])[0]
    S, V = p.shape[0], at.shape[0]
    tr = _d(s["transient"])[0]
    vol = torch.zeros(V, dtype=torch.float64, device=DEV)
    L = 0
    if case["kind"] == "velten_pairs":
        q = _d(s["laser_points"])[0]
        L = q.shape[0]
        if S * L * V > 4e9:
            return None
        second = torch.cdist(at, q, compute_mode="donot_use_mm_for_euclid_dist")
        lasers = torch.arange(L, device=DEV)[None]
    elif S * V > 4e10:
        return None
    off = torch.zeros(S, dtype=torch.float64, device=DEV)
    if s["scan_origin"] is not None:
        off = 2 * (p - _d(s["scan_origin"])[0]).norm(dim=1)
    grad = torch.zeros_like(tr) if case.get("grad") else None
    vg = _d(s["volume_grad"]).reshape(-1) if case.get("grad") else None
    for i in range(S):
        one = (at - p[i]).norm(dim=1)
        if L:
            t = ((one[:, None] + second - bo) / bw + 0.5).floor().long()
            ok = (t >= 0) & (t < T)
            vol += (tr[t.clamp(0, T - 1), i, lasers] * ok).sum(1)
            continue
        t = ((off[i] + 2 * one - bo) / bw + 0.5).floor().long()
        ok = (t >= 0) & (t < T)
        t = t.clamp(0, T - 1)
        vol += tr[t, i] * ok
        if grad is not None:
            grad[:, i] = torch.zeros(T, dtype=torch.float64, device=DEV).index_add_(0, t, vg * ok)
    got = dict(volume=vol.view(1, case["z"], case["y"], case["x"]))
    if grad is not None:
        got["transient"] = grad[None]
    return got


def _rbf_exact(case, s):
    rbf = _d(s["rbf"]).requires_grad_(True)
    c, sigma, attr = rbf[0, :, :3], rbf[0, :, 3:4], rbf[0, :, 4:]
    k = -0.5 / sigma ** 2
    ax = [torch.linspace(START[i], END[i], case["xyz"[i]], device=DEV, dtype=torch.float64)
          for i in range(3)]
    ex, ey, ez = (torch.exp((ax[i][None] - c[:, i:i + 1]) ** 2 * k) for i in range(3))
    plane = (ey[:, :, None] * ex[:, None]).reshape(rbf.shape[1], -1)
    channels = [ez.T @ plane]
    norm = torch.where(channels[0] < 1e-8, torch.ones_like(channels[0]), channels[0])
    for a in range(attr.shape[1]):
        channels.append((ez * attr[:, a:a + 1]).T @ plane / norm)
    vol = torch.stack(channels).view(1, -1, case["z"], case["y"], case["x"])
    gr, = torch.autograd.grad(vol, (rbf,), _d(s["volume_grad"]))
    return dict(volume=vol.detach(), rbf=gr)


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind in ("confocal", "exhaustive"):
        return _mesh_exact(case, s)
    if kind == "volume":
        return _volume_exact(case, s)
    if kind == "volume_pairs":
        return _volume_pairs_exact(case, s)
    if kind in ("velten", "velten_pairs"):
        return _velten_exact(case, s)
    return _rbf_exact(case, s)
