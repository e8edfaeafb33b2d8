"""The work that programs built on this package have it do, as timed cases.

``listed()`` names the cases, ``draw(rng)`` makes more of the same ranges,
``prepare(case, seed)`` makes what a program holds before the call, ``run``
is one pass through the public entry points, ``work`` the bytes and floating
point operations a pass cannot do without, and ``exact`` what ``run`` returns
in 64-bit arithmetic, written in plain torch.

Grids of the query, contact and stepping cases hold the signed distance of a
torus or a box, sampled at the voxel centres (SdfOracle(SdfData) /
SdfOracle(SparseSdfData)); the build cases start from triangle meshes.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sdf-contact-module_b200"))

from sdfo import SdfGrid  # noqa: E402
from sdfo import meshes as M  # noqa: E402
from sdfo.autograd import sdf_query  # noqa: E402
from sdfo.batch import QueryBatch, pack_poses  # noqa: E402
from sdfo.be import BEStepper  # noqa: E402
from sdfo.contact import ContactBatch, pack_states  # noqa: E402


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # One contact body's quadrature points asked for through the engine's
        # NumPy grid interface (query_batch), as a contact loop in Python does
        # on every evaluation: the smallest call, host arrays in and out.
        dict(name="engine_points_960", kind="host", res=64, n=960, mode="trilinear"),
        # The headline query: 1M points near a part's surface on a dense 128
        # grid that fits in the second-level cache, value and gradient.
        dict(name="dense_tricubic_1m", kind="query", sparse=False, fp16=False, res=128, n=1_000_000,
             mode="tricubic", f64=False, extra=False),
        # A collision check over an unsorted point cloud of odd length on a
        # sparse grid kept in half precision, FP64 points, unit normals and
        # witness points asked for.
        dict(name="sparse_fp16_3m", kind="query", sparse=True, fp16=True, res=256, n=3_000_001,
             mode="tricubic", f64=True, extra=True),
        # The largest query: 16M points on a sparse 512 grid larger than the
        # second-level cache.
        dict(name="sparse_tricubic_16m", kind="query", sparse=True, fp16=False, res=512, n=16_000_000,
             mode="tricubic", f64=False, extra=False),
        # A training step that fits the stored field to samples of value and
        # gradient: forward and backward to points and payload.
        dict(name="train_sparse_2m", kind="train", sparse=True, res=256, n=2_000_000, mode="tricubic"),
        # A scene of many parts, each with its grid, pose and points, queried
        # in one launch.
        dict(name="posed_parts_48", kind="batch", parts=48, res=96, n=65_536, mode="tricubic"),
        # One time step of a small multi-body scene: forces with the engine's
        # broad phase and narrow filter, then the contact measure.
        dict(name="engine_contact_33", kind="cull", res=128, poses=33, major=192, minor=20),
        # Contact optimisation / implicit integration over many poses: forces
        # and the 6x6 pose Jacobian of a ring on a block.
        dict(name="contact_jacobian_4096", kind="contact", res=128, poses=4096, major=192, minor=20,
             mode="trilinear", jacobian=True),
        # Monte-Carlo drops: Backward-Euler steps of many scenes, some falling,
        # some already touching.
        dict(name="ring_drops_2048", kind="drops", res=128, scenes=2048, steps=2, major=192, minor=20),
        # SDF construction from a machined part's mesh, dense.
        dict(name="build_dense_128", kind="build_dense", res=128, n_az=512, n_vert=16),
        # SDF construction from a scanned free-form surface, sparse narrow
        # band.
        dict(name="build_sparse_512", kind="build_sparse", res=512, subdivisions=7, band=3),
        # A contact-aware grid (candidate lists per voxel) built from the part's
        # mesh with sharp corner normals, then asked for candidates near the
        # surface.
        dict(name="build_contact_aware_128", kind="build_ca", res=128, n_az=512, n_vert=16, n=100_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "query", "query", "query", "train", "batch", "cull", "contact", "drops",
                       "build_dense", "build_sparse", "build_ca"])
    mode = rng.choice(["tricubic", "tricubic", "trilinear"])
    ring = dict(major=rng.randint(48, 240), minor=rng.randint(8, 24))
    if kind == "host":
        return dict(kind=kind, res=rng.randint(32, 128), n=_log_int(rng, 1, 50_000), mode=mode)
    if kind == "query":
        sparse = rng.random() < 0.6
        return dict(kind=kind, sparse=sparse, fp16=sparse and rng.random() < 0.4,
                    res=rng.randint(48, 512) if sparse else rng.randint(32, 160),
                    n=_log_int(rng, 1_000, 12_000_000), mode=mode, f64=rng.random() < 0.25,
                    extra=rng.random() < 0.25)
    if kind == "train":
        sparse = rng.random() < 0.7
        return dict(kind=kind, sparse=sparse, res=rng.randint(48, 320) if sparse else rng.randint(32, 128),
                    n=_log_int(rng, 5_000, 3_000_000), mode=mode)
    if kind == "batch":
        return dict(kind=kind, parts=rng.randint(2, 48), res=rng.randint(40, 112), n=_log_int(rng, 100, 80_000),
                    mode=mode)
    if kind == "cull":
        return dict(kind=kind, res=rng.randint(48, 128), poses=_log_int(rng, 1, 300), **ring)
    if kind == "contact":
        return dict(kind=kind, res=rng.randint(48, 144), poses=_log_int(rng, 1, 4096), mode=mode,
                    jacobian=rng.random() < 0.6, **ring)
    if kind == "drops":
        return dict(kind=kind, res=rng.randint(48, 128), scenes=_log_int(rng, 8, 2048), steps=rng.randint(1, 2), **ring)
    if kind == "build_dense":
        return dict(kind=kind, res=rng.choice([32, 64, 96, 128]), n_az=rng.randint(24, 512), n_vert=rng.randint(2, 16))
    if kind == "build_sparse":
        return dict(kind=kind, res=rng.choice([64, 128, 192, 256, 384]), subdivisions=rng.randint(3, 7),
                    band=rng.randint(2, 4))
    return dict(kind=kind, res=rng.choice([32, 64, 96, 128]), n_az=rng.randint(24, 512), n_vert=rng.randint(2, 16),
                n=_log_int(rng, 1_000, 200_000))


# --------------------------------------------------------------------------
# fields and grids
# --------------------------------------------------------------------------
TORUS = (0.05, 0.016)  # ring and tube radius of the torus fields (metres)


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _torus_phin(p, shape=TORUS):
    """{phi, n} of a torus about z at the points p (N, 3)."""
    rho = torch.sqrt(p[:, 0] ** 2 + p[:, 1] ** 2).clamp_min(1e-12)
    a = rho - shape[0]
    d = torch.sqrt(a * a + p[:, 2] ** 2).clamp_min(1e-12)
    return torch.stack([d - shape[1], a / d * p[:, 0] / rho, a / d * p[:, 1] / rho, p[:, 2] / d], 1)


def _box_phin(p, half, top):
    """{phi, n} of a box of half extents `half` whose top face is z = top."""
    c = torch.tensor([0.0, 0.0, top - half[2]], dtype=p.dtype, device=p.device)
    h = torch.tensor(half, dtype=p.dtype, device=p.device)
    x = p - c
    sign = torch.where(x >= 0, 1.0, -1.0).to(p.dtype)
    q = x.abs() - h
    out = q.clamp_min(0.0)
    dist = out.norm(dim=1)
    inner = q.max(dim=1)
    n_out = out * sign / dist.clamp_min(1e-300)[:, None]
    n_in = torch.nn.functional.one_hot(inner.indices, 3).to(p.dtype) * sign
    outside = dist > 0
    phi = torch.where(outside, dist, inner.values)
    return torch.cat([phi[:, None], torch.where(outside[:, None], n_out, n_in)], 1)


def _spec(lo, hi, res):
    """A grid of `res` voxels along the longest side of the box lo..hi."""
    lo, hi = np.asarray(lo, np.float64), np.asarray(hi, np.float64)
    h = float((hi - lo).max() / res)
    shape = [int(math.ceil((hi[a] - lo[a]) / h - 1e-9)) for a in range(3)]
    return dict(bmin=lo, voxel=np.full(3, h), shape=shape)


def _torus_spec(res, shape=TORUS):
    xy, z = 1.25 * (shape[0] + shape[1]), 2.2 * shape[1]
    return _spec([-xy, -xy, -z], [xy, xy, z], res)


def _centres(spec, i, j, k):
    v = [torch.as_tensor(x, dtype=torch.float64) + 0.5 for x in (i, j, k)]
    return torch.stack([float(spec["bmin"][a]) + float(spec["voxel"][a]) * v[a] for a in range(3)], 1)


def _dense_payload(spec, field):
    """(N, 4) float64 {phi, n}, x fastest."""
    nx, ny, nz = spec["shape"]
    idx = torch.arange(nx * ny * nz, device=_dev())
    return field(_centres(spec, idx % nx, (idx // nx) % ny, idx // (nx * ny)))


def _sparse_payload(spec, field, band=3, halo=2, bd=8):
    """(ijk (B, 3), payload (B * bd^3, 4) float32, block table) of the narrow
    band, blocks and voxels in the builder's order."""
    dev = _dev()
    shape = spec["shape"]
    h = float(spec["voxel"][0])
    nb = [(s + bd - 1) // bd for s in shape]
    bl = torch.arange(nb[0] * nb[1] * nb[2], device=dev)
    b = torch.stack([bl % nb[0], (bl // nb[0]) % nb[1], bl // (nb[0] * nb[1])], 1)
    centre = torch.stack([float(spec["bmin"][a]) + h * (b[:, a].double() + 0.5) * bd for a in range(3)], 1)
    keep = field(centre)[:, 0].abs() <= (band + halo) * h + 0.5 * math.sqrt(3.0) * bd * h
    ijk = b[keep]
    B, V = len(ijk), bd ** 3
    loc = torch.arange(V, device=dev)
    v = [(ijk[:, a, None] * bd + l[None]).reshape(-1) for a, l in
         enumerate((loc % bd, (loc // bd) % bd, loc // (bd * bd)))]
    pay = torch.empty(B * V, 4, dtype=torch.float32, device=dev)
    for s in range(0, B * V, 1 << 22):
        e = min(B * V, s + (1 << 22))
        pay[s:e] = field(_centres(spec, v[0][s:e], v[1][s:e], v[2][s:e])).float()
    table = torch.full((len(bl),), -1, dtype=torch.int64, device=dev)
    table[bl[keep]] = torch.arange(B, device=dev)
    return ijk, pay, (table, nb, bd)


def _grid_dense(spec, field, mode):
    p = _dense_payload(spec, field).cpu().numpy()
    return SdfGrid.from_dense(spec, p[:, 0].copy(), p[:, 1:].copy(), mode=mode)


def _grid_sparse(spec, field, mode):
    ijk, pay, _ = _sparse_payload(spec, field)
    p = pay.cpu().numpy().reshape(len(ijk), 512, 4)
    return SdfGrid.from_sparse(spec, 8, ijk.cpu().numpy(), p[:, :, 0].copy(), p[:, :, 1:].copy(), mode=mode)


def _gen(seed, salt=0):
    return torch.Generator(device=_dev()).manual_seed(1_000_003 * int(seed) + salt)


def _torus_shape(seed):
    # scaled as a whole: another seed is another part on as many bricks
    f = np.random.default_rng([seed, 7]).uniform(0.8, 1.25)
    return (TORUS[0] * f, TORUS[1] * f)


def _torus_points(n, off, gen, shape):
    """n points about the torus surface in random order, offset along the
    normal by U(-off, off)."""
    u = torch.rand(n, 3, generator=gen, device=_dev(), dtype=torch.float64)
    a, b = 2 * math.pi * u[:, 0], 2 * math.pi * u[:, 1]
    r = shape[1] + off * (2 * u[:, 2] - 1)
    rho = shape[0] + r * torch.cos(b)
    return torch.stack([rho * torch.cos(a), rho * torch.sin(a), r * torch.sin(b)], 1)


def _query_inputs(case, seed, salt=0):
    shape = _torus_shape(seed)
    spec = _torus_spec(case["res"], shape)
    h = float(spec["voxel"][0])
    pts = _torus_points(case["n"], 3.0 * h, _gen(seed, salt), shape)
    return spec, (lambda p: _torus_phin(p, shape)), pts


def _rotations(rng, n, max_angle=math.pi):
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    a = max_angle * rng.uniform(0.0, 1.0, n)
    K = np.zeros((n, 3, 3))
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 0] = -d[:, 2], d[:, 1], d[:, 2]
    K[:, 1, 2], K[:, 2, 0], K[:, 2, 1] = -d[:, 0], -d[:, 1], d[:, 0]
    return np.eye(3) + np.sin(a)[:, None, None] * K + (1 - np.cos(a))[:, None, None] * (K @ K)


RING = (0.05, 0.01)  # contact ring: major and minor radius
LAW = dict(stiffness=1e11, order=2.0, damping=1e4, friction=0.3, regularizer=1e-4, activation_distance=1e-5)


def _ring(case):
    v, t = M.torus(*RING, case["major"], case["minor"])
    return M.centroid_quadrature(v, t)


def _ring_poses(n, seed):
    """Ring poses about the block's top face z = 0: some clear of it, some
    pressed in by up to the tube radius, tilted by at most 5 degrees."""
    rng = np.random.default_rng([seed, 11])
    phi = rng.uniform(0, 2 * np.pi, n)
    a = np.deg2rad(5.0) * rng.uniform(0, 1, n)
    c, s = np.cos(a), np.sin(a)
    x, y = np.cos(phi), np.sin(phi)
    R = np.empty((n, 3, 3))
    R[:, 0] = np.stack([c + x * x * (1 - c), x * y * (1 - c), y * s], 1)
    R[:, 1] = np.stack([x * y * (1 - c), c + y * y * (1 - c), -x * s], 1)
    R[:, 2] = np.stack([-y * s, x * s, c], 1)
    r = np.stack([rng.uniform(-0.002, 0.002, n), rng.uniform(-0.002, 0.002, n), rng.uniform(0.010, 0.020, n)], 1)
    return r, R, rng.uniform(-0.1, 0.1, (n, 3)), rng.uniform(-1, 1, (n, 3))


BLOCK = (0.05, 0.05, 0.05)
SLAB = (0.15, 0.15, 0.025)


def _block_spec(half, res):
    d = 0.1 * 2.0 * math.sqrt(sum(x * x for x in half))
    return _spec([-half[0] - d, -half[1] - d, -2 * half[2] - d], [half[0] + d, half[1] + d, d], res)


# --------------------------------------------------------------------------
# prepare and run
# --------------------------------------------------------------------------
def prepare(case, seed):
    return dict(case=case, **globals()["_prep_" + case["kind"]](case, seed))


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    return None if f is None else f(case, seed)


def work(case):
    b, f = globals()["_work_" + case["kind"]](case)
    return {"bytes": float(b), "flops": float(f)}


# --- host-array queries
def _prep_host(case, seed):
    spec, field, pts = _query_inputs(case, seed)
    return dict(grid=_grid_dense(spec, field, case["mode"]), pts=pts.cpu().numpy())


def _run_host(s):
    return s["grid"].query_batch(s["pts"])


def _exact_host(case, seed):
    spec, field, pts = _query_inputs(case, seed)
    gap, grad, ok = _interpolate(spec, _dense_payload(spec, field), None, pts, case["mode"])
    gn = grad.norm(dim=1)
    unit = torch.where((ok & (gn > 1e-30))[:, None], grad / gn.clamp_min(1e-300)[:, None],
                       torch.tensor([0.0, 0.0, 1.0], dtype=grad.dtype, device=grad.device))
    return tuple(x.cpu().numpy() for x in (gap, grad, gn, unit)) + (None,)


def _work_host(case):
    n = case["n"]
    return n * (24 + 8 + 24 + 8 + 24 + 1) + _touched(case, n, dense=True), n * _query_flops(case["mode"])


# --- device queries
def _prep_query(case, seed):
    spec, field, pts = _query_inputs(case, seed)
    grid = (_grid_sparse if case["sparse"] else _grid_dense)(spec, field, case["mode"])
    if case["fp16"]:
        grid = grid.to_fp16()
    return dict(grid=grid, pts=pts if case["f64"] else pts.float())


def _run_query(s):
    e = s["case"]["extra"]
    return s["grid"].query_tensors(s["pts"], unit=e, witness=e)


def _exact_query(case, seed):
    spec, field, pts = _query_inputs(case, seed)
    if not case["f64"]:
        pts = pts.float().double()
    if case["sparse"]:
        _, pay, table = _sparse_payload(spec, field)
    else:
        pay, table = _dense_payload(spec, field), None
    gap, grad, ok = _interpolate(spec, pay, table, pts, case["mode"])
    out = dict(gap=gap, grad=grad, valid=None)
    if case["extra"]:
        ln = grad.norm(dim=1, keepdim=True)
        x = torch.tensor([1.0, 0.0, 0.0], dtype=grad.dtype, device=grad.device)
        out["unit"] = torch.where(ok[:, None] & (ln > 1e-15), grad / ln.clamp_min(1e-300), x)
        out["witness"] = torch.where(ok[:, None], pts - gap[:, None] * out["unit"], torch.zeros_like(pts))
    return out


def _work_query(case):
    n = case["n"]
    per = (24 if case["f64"] else 12) + 4 + 12 + 1 + (24 if case["extra"] else 0)
    t = _touched(case, n, dense=not case["sparse"])
    return n * per + (t // 2 if case["fp16"] else t), n * _query_flops(case["mode"])


# --- training step: forward and backward to points and payload
def _prep_train(case, seed):
    spec, field, pts = _query_inputs(case, seed)
    grid = (_grid_sparse if case["sparse"] else _grid_dense)(spec, field, case["mode"])
    g = _gen(seed, 1)
    n = case["n"]
    return dict(grid=grid, pts=pts.float().requires_grad_(True), payload=grid.payload().requires_grad_(True),
                dgap=torch.randn(n, generator=g, device=_dev()),
                dgrad=0.1 * torch.randn(n, 3, generator=g, device=_dev()))


def _run_train(s):
    gap, grad = sdf_query(s["grid"], s["pts"], s["payload"], mode=s["case"]["mode"])
    dp, dv = torch.autograd.grad((gap, grad), (s["pts"], s["payload"]), (s["dgap"], s["dgrad"]))
    return gap.detach(), grad.detach(), dp, dv


def _exact_train(case, seed):
    spec, field, pts = _query_inputs(case, seed)
    pts = pts.float().double()
    if case["sparse"]:
        _, pay, table = _sparse_payload(spec, field)
    else:
        pay, table = _dense_payload(spec, field), None
    pay = pay.float().double()
    g = _gen(seed, 1)
    n = case["n"]
    dgap = torch.randn(n, generator=g, device=_dev()).double()
    dgrad = (0.1 * torch.randn(n, 3, generator=g, device=_dev())).double()
    gap, grad, dp = torch.empty(n).to(dgap), torch.empty(n, 3).to(dgap), torch.empty(n, 3).to(dgap)
    dv = torch.zeros_like(pay)
    for a in range(0, n, 1 << 18):
        b = min(n, a + (1 << 18))
        idx, ok, frac = _cells(spec, table, pts[a:b])
        corners = pay[idx].requires_grad_(True)
        frac = frac.requires_grad_(True)
        g0, g1 = _hermite_value(corners, frac, spec, case["mode"])
        gap[a:b], grad[a:b] = torch.where(ok, g0, 0.0 * g0).detach(), torch.where(ok[:, None], g1, 0.0 * g1).detach()
        up0, up1 = torch.where(ok, dgap[a:b], 0.0 * dgap[a:b]), torch.where(ok[:, None], dgrad[a:b], 0.0 * dgrad[a:b])
        dc, df = torch.autograd.grad((g0, g1), (corners, frac), (up0, up1))
        dp[a:b] = df / torch.as_tensor(spec["voxel"], device=df.device)
        dv.index_add_(0, idx.reshape(-1), dc.reshape(-1, 4))
    return gap, grad, dp, dv


def _work_train(case):
    n = case["n"]
    stored = _stored(case, dense=not case["sparse"])
    t = _touched(case, n, dense=not case["sparse"])
    # points, both upstream gradients, gap, grad, dL/dp; payload in, its gradient out
    return n * (12 + 4 + 12 + 4 + 12 + 12) + t + 16 * stored, n * 3 * _query_flops(case["mode"])


# --- many posed grids, one launch
def _parts(case, seed):
    fixed = np.random.default_rng([case["parts"], case["res"], case["n"]])
    res = [max(24, int(case["res"] * x)) for x in fixed.uniform(0.6, 1.0, case["parts"])]
    counts = [max(1, int(case["n"] * x)) for x in fixed.uniform(0.5, 1.0, case["parts"])]
    rng = np.random.default_rng([seed, 5])
    shapes = [(TORUS[0] * f, TORUS[1] * f) for f in rng.uniform(0.5, 1.5, case["parts"])]
    R, t = _rotations(rng, case["parts"]), rng.uniform(-1.0, 1.0, (case["parts"], 3))
    pts = []
    for g in range(case["parts"]):
        spec = _torus_spec(res[g], shapes[g])
        local = _torus_points(counts[g], 3.0 * float(spec["voxel"][0]), _gen(seed, 100 + g), shapes[g])
        pts.append(local @ torch.as_tensor(R[g].T, device=_dev()) + torch.as_tensor(t[g], device=_dev()))
    return res, shapes, counts, R, t, torch.cat(pts).float().contiguous()


def _prep_batch(case, seed):
    res, shapes, counts, R, t, pts = _parts(case, seed)
    grids = [_grid_sparse(_torus_spec(r, s), lambda p, s=s: _torus_phin(p, s), case["mode"])
             for r, s in zip(res, shapes)]
    return dict(batch=QueryBatch(grids, counts), pts=pts, poses=pack_poses(R, t))


def _run_batch(s):
    return s["batch"].run(s["pts"], s["poses"], mode=s["case"]["mode"])


def _exact_batch(case, seed):
    res, shapes, counts, R, t, pts = _parts(case, seed)
    gaps, grads, o = [], [], 0
    for g in range(case["parts"]):
        spec = _torus_spec(res[g], shapes[g])
        _, pay, table = _sparse_payload(spec, lambda p, s=shapes[g]: _torus_phin(p, s))
        Rg = torch.as_tensor(R[g], device=_dev())
        local = (pts[o:o + counts[g]].double() - torch.as_tensor(t[g], device=_dev())) @ Rg
        gap, grad, _ = _interpolate(spec, pay, table, local, case["mode"])
        gaps.append(gap)
        grads.append(grad @ Rg.T)
        o += counts[g]
    return torch.cat(gaps), torch.cat(grads), None


def _work_batch(case):
    n = 0.75 * case["n"]
    one = dict(case, res=0.8 * case["res"])
    return case["parts"] * (n * (12 + 17) + _touched(one, n, dense=False)), case["parts"] * n * (
        _query_flops(case["mode"]) + 36)


# --- contact forces
def _contact_setup(case, seed):
    qx, qw = _ring(case)
    r, R, v, w = _ring_poses(case["poses"], seed)
    return qx, qw, r, R, v, w


def _block_field(p):
    return _box_phin(p, BLOCK, 0.0)


def _prep_contact(case, seed, **kw):
    qx, qw, r, R, v, w = _contact_setup(case, seed)
    mode = case.get("mode", "trilinear")
    grid = _grid_dense(_block_spec(BLOCK, case["res"]), _block_field, mode)
    return dict(batch=ContactBatch(grid, qx, qw, mode=mode, **LAW, **kw), poses=pack_states(r, R, v, w),
                body=pack_states(np.zeros((1, 3)), np.eye(3)[None]))


def _run_contact(s):
    return s["batch"].evaluate(s["poses"], s["body"], jacobian=s["case"]["jacobian"])


def _exact_contact(case, seed, narrow=None):
    dev = _dev()
    qx, qw, r, R, v, w = _contact_setup(case, seed)
    t64 = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
    X, W = t64(qx).float().double(), t64(qw / qw.sum()).float().double()
    r, R, v, w = t64(r), t64(R), t64(v), t64(w)
    spec = _block_spec(BLOCK, case["res"])
    pay = _dense_payload(spec, _block_field).float().double()
    mode = case.get("mode", "trilinear")
    pose, point = [], []
    step = max(1, (1 << 22) // len(X))
    for a in range(0, len(r), step):  # the points in contact
        b = min(len(r), a + step)
        Y = torch.einsum("pij,qj->pqi", R[a:b], X) + r[a:b, None]
        gap, _, ok = _interpolate(spec, pay, None, Y.reshape(-1, 3), mode)
        on = ok & (LAW["stiffness"] * gap.clamp_max(0.0) ** 2 > 1e-30)
        if narrow is not None:
            on = on & (Y.reshape(-1, 3)[:, 2].abs() < narrow)
        k = torch.nonzero(on)[:, 0]
        pose.append(a + k // len(X))
        point.append(k % len(X))
    pose, point = torch.cat(pose), torch.cat(point)
    want_jac = case.get("jacobian", False)
    dx = torch.zeros(len(r), 3, dtype=torch.float64, device=dev, requires_grad=want_jac)
    dth = torch.zeros(len(r), 3, dtype=torch.float64, device=dev, requires_grad=want_jac)
    ft = torch.zeros(len(r), 6, dtype=torch.float64, device=dev)
    jac = torch.zeros(len(r), 6, 6, dtype=torch.float64, device=dev)
    for a in range(0, len(pose), 1 << 19):
        p, q = pose[a:a + (1 << 19)], point[a:a + (1 << 19)]
        off0 = torch.einsum("nij,nj->ni", R[p], X[q])
        off = off0 + torch.cross(dth[p], off0, dim=1)  # exp([dth]x) to first order
        Y = r[p] + dx[p] + off
        idx, _, frac = _cells(spec, None, Y.detach())
        h = torch.as_tensor(spec["voxel"], device=dev)
        frac = frac + (Y - Y.detach()) / h
        g, gl = _hermite_value(pay[idx], frac, spec, mode)
        d = (-g).clamp_min(0.0)
        pen = LAW["stiffness"] * d * d
        u = v[p] + torch.cross(w[p], off, dim=1)
        f = pen[:, None] * gl - LAW["damping"] * (u * gl).sum(1, keepdim=True) * gl
        gn = gl.norm(dim=1, keepdim=True)
        un = gl / gn
        ut = u - (u * un).sum(1, keepdim=True) * un
        den = torch.sqrt((ut * ut).sum(1, keepdim=True) + LAW["regularizer"] ** 2)
        f = f - LAW["friction"] * pen[:, None] * gn * ut / den
        wf = W[q, None] * torch.cat([f, torch.cross(off, f, dim=1)], 1)
        ft.index_add_(0, p, wf.detach())
        if want_jac:
            for i in range(6):
                jx, jt = torch.autograd.grad(wf[:, i].sum(), (dx, dth), retain_graph=i < 5)
                jac[:, i, :3] += jx
                jac[:, i, 3:] += jt
    return (ft, jac) if want_jac else ft


def _work_contact(case):
    nq = 2 * case["major"] * case["minor"]
    P = case["poses"]
    out = 6 + (36 if case.get("jacobian") else 0)
    # every point of every pose is placed in the grid's frame and compared
    # with the surface
    return nq * 16 + P * 8 * (18 + out) + 16 * case["res"] ** 3 // 8, P * nq * 40


def _prep_cull(case, seed):
    return _prep_contact(case, seed, narrow_margin=0.01)


def _run_cull(s):
    ft = s["batch"].evaluate(s["poses"], s["body"])
    return dict(ft=ft, **s["batch"].measure(s["poses"], s["body"]))


def _exact_cull(case, seed):
    return dict(ft=_exact_contact(case, seed, narrow=0.01), gap=None, penetration=None, normal_velocity=None,
                min_point_index=None, active_count=None, valid_count=None)


def _work_cull(case):
    b, f = _work_contact(case)
    return b + case["poses"] * 40, 2 * f


# --- Backward-Euler steps
def _prep_drops(case, seed):
    n = case["scenes"]
    qx, qw = _ring(case)
    rng = np.random.default_rng([seed, 13])
    _, R, _, _ = _ring_poses(n, seed)
    low = np.einsum("nij,qj->nqi", R[:, 2:3], qx)[:, :, 0].min(axis=1)
    # half of the rings fall from up to 0.3 mm, half already press in
    gap = np.where(rng.random(n) < 0.5, rng.uniform(0.0, 3e-4, n), -rng.uniform(1e-7, 5e-6, n))
    r = np.stack([rng.uniform(-0.05, 0.05, n), rng.uniform(-0.05, 0.05, n), gap - low], 1)
    v = np.stack([rng.uniform(-0.07, 0.07, n), rng.uniform(-0.07, 0.07, n), -rng.uniform(0.1, 0.3, n)], 1)
    Rr, rr, rho = RING[0], RING[1], 7800.0
    mass = rho * 2.0 * np.pi ** 2 * Rr * rr * rr
    inertia = np.diag([mass * (Rr * Rr / 2 + 5 * rr * rr / 8)] * 2 + [mass * (Rr * Rr + 3 * rr * rr / 4)])
    grid = _grid_dense(_block_spec(SLAB, case["res"]), lambda p: _box_phin(p, SLAB, 0.0), "trilinear")
    st = BEStepper(grid, qx, qw, mass, inertia, max_scenes=n, **dict(LAW, order=2))
    return dict(stepper=st, scenes=st.scenes(r, R, v, rng.uniform(-1, 1, (n, 3))))


def _run_drops(s):
    # the start states are kept, as a program that restarts its drops keeps them
    x = s["scenes"].clone()
    taken = [s["stepper"].step(x, 1e-3) for _ in range(s["case"]["steps"])]
    return x, taken


def _work_drops(case):
    nq = 2 * case["major"] * case["minor"]
    # each step measures the start and the end state and evaluates two residuals
    f = case["scenes"] * case["steps"] * nq * 4 * 40
    return case["scenes"] * case["steps"] * (2 * 208 + 16) + nq * 32 + 8 * case["res"] ** 3 // 8, f


# --- builds
def _placed(verts, tris, seed):
    """The mesh scaled, moved, its axes exchanged and its triangles in another
    order: other inputs whose narrow band has as many bricks."""
    rng = np.random.default_rng([seed, 3])
    v = rng.uniform(0.5, 2.0) * np.roll(verts, int(rng.integers(3)), axis=1) + rng.uniform(-0.1, 0.1, 3)
    return np.ascontiguousarray(v), np.ascontiguousarray(tris[rng.permutation(len(tris))])


def _cylinder(case, seed):
    f = np.random.default_rng([seed, 3]).uniform(0.9, 1.1, 3)
    return 0.05 * f[0], 0.04 * f[0] * f[1] ** 0.5, 0.02 * f[2]


def _prep_build_dense(case, seed):
    ro, ri, z = _cylinder(case, seed)
    v, t = M.hollow_cylinder(ro, ri, z, n_az=case["n_az"], n_vert=case["n_vert"], n_rad=1)
    return dict(verts=v, tris=t)


def _run_build_dense(s):
    r = s["case"]["res"]
    g = SdfGrid.build_dense(s["verts"], s["tris"], target_resolution=r, max_resolution=r)
    return g.payload()


def _exact_build_dense(case, seed):
    # the solid is an extruded ring of two regular polygons: its distance is
    # the planar distance to the polygons' edges combined with the height
    ro, ri, height = _cylinder(case, seed)
    n, res, dev = case["n_az"], case["res"], _dev()
    th = 2.0 * np.pi * np.arange(n) / n
    c, s = np.cos(th), np.sin(th)
    lo = np.array([(ro * c).min(), (ro * s).min(), 0.0])
    hi = np.array([(ro * c).max(), (ro * s).max(), height])
    pad = 0.1 * float(np.sqrt(((hi - lo) ** 2).sum()))
    bmin = lo - pad
    size = hi + pad - bmin
    h = float(size.max() / res)
    levels = [8, 16, 32, 64, 128, 256, 512, 1024, 2048]
    shape = [min(next(l for l in levels if l >= max(1, math.ceil(x / h)) or l >= res), res) for x in size]
    ctr = [torch.as_tensor(bmin[a] + h * (np.arange(shape[a]) + 0.5), device=dev) for a in range(3)]
    P = torch.stack(torch.meshgrid(ctr[1], ctr[0], indexing="ij"), -1).reshape(-1, 2).flip(1)
    best = torch.full((len(P),), float("inf"), dtype=torch.float64, device=dev)
    near = torch.zeros_like(P)
    inside = torch.ones(len(P), dtype=torch.bool, device=dev)
    for rad, outer in ((ro, True), (ri, False)):
        A = torch.as_tensor(np.stack([rad * c, rad * s], 1), device=dev)
        B = A.roll(-1, 0)
        inp = torch.ones(len(P), dtype=torch.bool, device=dev)
        for a0 in range(0, n, 64):
            a, b = A[a0:a0 + 64], B[a0:a0 + 64]
            e = b - a
            rel = P[:, None] - a[None]
            k = ((rel * e).sum(-1) / (e * e).sum(-1)).clamp(0.0, 1.0)
            foot = a[None] + k[..., None] * e
            d2 = ((P[:, None] - foot) ** 2).sum(-1)
            m = d2.min(dim=1)
            upd = m.values < best
            best = torch.where(upd, m.values, best)
            near = torch.where(upd[:, None], foot[torch.arange(len(P), device=dev), m.indices], near)
            inp &= ((e[None, :, 0] * rel[..., 1] - e[None, :, 1] * rel[..., 0]) >= 0).all(dim=1)
        inside &= inp if outer else ~inp
    d2 = torch.where(inside, -best.sqrt(), best.sqrt())
    away = torch.where(inside[:, None], near - P, P - near) / best.sqrt().clamp_min(1e-300)[:, None]
    nz = shape[2]
    dp = d2[None].expand(nz, -1)
    dz = torch.maximum(-ctr[2], ctr[2] - height)[:, None].expand(-1, len(P))
    sz = torch.where(ctr[2] > height / 2, 1.0, -1.0).to(torch.float64)[:, None].expand(-1, len(P))
    both = torch.sqrt(dp.clamp_min(0) ** 2 + dz.clamp_min(0) ** 2)
    phi = torch.where((dp > 0) | (dz > 0), both, torch.maximum(dp, dz))
    side = torch.where((dp > 0) | (dz > 0), dp.clamp_min(0) / both.clamp_min(1e-300), (dp >= dz).double())
    up = torch.where((dp > 0) | (dz > 0), dz.clamp_min(0) / both.clamp_min(1e-300), (dz > dp).double()) * sz
    out = torch.stack([phi, side * away[None, :, 0], side * away[None, :, 1], up], -1)
    return out.reshape(-1, 4)


def _work_build_dense(case):
    vox = case["res"] ** 3 / 2
    tri = 4 * case["n_az"] * (case["n_vert"] + 1)
    # one nearest triangle and one ray crossing per voxel, a descent to each
    return tri * 24 + vox * (16 + 16), vox * (60 + 30 + 2 * 20 * math.log2(max(tri, 2))) + tri * 40


def _prep_build_sparse(case, seed):
    v, t = _placed(*M.perturbed_icosphere(case["subdivisions"], 0.1, 0.002, 8, 1, 6, 4), seed)
    return dict(verts=v, tris=t)


def _run_build_sparse(s):
    c = s["case"]
    g = SdfGrid.build_sparse(s["verts"], s["tris"], target_resolution=c["res"], max_resolution=c["res"],
                             band_voxels=c["band"])
    return g.payload()


def _work_build_sparse(case):
    tri = 20 * 4 ** case["subdivisions"]
    vox = _band_voxels(4 * math.pi * 0.1 ** 2, 0.2 * 1.35 / case["res"], case["band"])
    # the payload and the Hessians the grid keeps
    return tri * 24 + vox * (16 + 24), vox * (60 + 30 + 2 * 20 * math.log2(tri)) + tri * 40


def _prep_build_ca(case, seed):
    ro, ri, z = _cylinder(case, seed)
    v, t = M.hollow_cylinder(ro, ri, z, n_az=case["n_az"], n_vert=case["n_vert"], n_rad=1)
    # points about the walls and the caps
    u = torch.rand(case["n"], 4, generator=_gen(seed), device=_dev(), dtype=torch.float64)
    a = 2 * math.pi * u[:, 0]
    rho = torch.where(u[:, 3] < 0.3, ri + 0 * a, torch.where(u[:, 3] < 0.7, ro + 0 * a, ri + (ro - ri) * u[:, 1]))
    h = torch.where(u[:, 3] < 0.7, z * u[:, 1], torch.where(u[:, 3] < 0.85, 0 * a, z + 0 * a))
    off = 0.002 * (2 * u[:, 2] - 1)
    side = (u[:, 3] < 0.7).double()
    pts = torch.stack([(rho + side * off) * torch.cos(a), (rho + side * off) * torch.sin(a), h + (1 - side) * off], 1)
    return dict(verts=v, tris=t, normals=M.corner_normals(v, t, "face"), pts=pts.float())


def _run_build_ca(s):
    r = s["case"]["res"]
    g = SdfGrid.build_contact_aware(s["verts"], s["tris"], s["normals"], target_resolution=r, max_resolution=r)
    return dict(payload=g.payload(), **g.query_candidates(s["pts"]))


def _work_build_ca(case):
    vox = case["res"] ** 3 / 2
    tri = 4 * case["n_az"] * (case["n_vert"] + 1)
    n = case["n"]
    b = tri * 96 + vox * (16 + 16 + 1 + 4 * 36) + n * (12 + 29 + 4 + 8 * 32)
    return b, vox * (4 * 90 + 2 * 20 * math.log2(max(tri, 2))) + n * 200


# --------------------------------------------------------------------------
# 64-bit interpolation and the sizes of grids
# --------------------------------------------------------------------------
def _cells(spec, table, pts):
    """Corner payload rows (N, 8) of each point's cell (corner di + 2 dj +
    4 dk; 0 where invalid), validity and the fractional position."""
    bmin = torch.as_tensor(spec["bmin"], dtype=torch.float64, device=pts.device)
    h = torch.as_tensor(spec["voxel"], dtype=torch.float64, device=pts.device)
    n = torch.tensor(spec["shape"], device=pts.device)
    f = (pts - bmin) / h - 0.5
    c = torch.floor(f)
    ok = ((c >= 0) & (c + 1 < n)).all(dim=1)
    lo = torch.where(ok[:, None], c, torch.zeros_like(c)).long()
    off = torch.tensor([[q & 1, (q >> 1) & 1, q >> 2] for q in range(8)], device=pts.device)
    v = lo[:, None, :] + off[None]
    if table is None:
        idx = v[..., 0] + n[0] * (v[..., 1] + n[1] * v[..., 2])
    else:
        tab, nb, bd = table
        b, l = v // bd, v % bd
        slot = tab[b[..., 0] + nb[0] * (b[..., 1] + nb[1] * b[..., 2])]
        ok = ok & (slot >= 0).all(dim=1)
        idx = slot.clamp_min(0) * bd ** 3 + l[..., 0] + bd * (l[..., 1] + bd * l[..., 2])
    return idx, ok, f - c


def _hermite_value(c, t, spec, mode):
    """Value and gradient of the cell interpolant: corners c (N, 8, 4)
    {phi, n}, position t (N, 3)."""
    h = [float(x) for x in spec["voxel"]]
    if mode == "trilinear":
        val = [[1 - t[:, a], t[:, a]] for a in range(3)]
        der = [[-torch.ones_like(t[:, a]), torch.ones_like(t[:, a])] for a in range(3)]
        slope = dslope = None
    else:
        val, der, slope, dslope = [], [], [], []
        for a in range(3):
            x = t[:, a]
            val.append([1 - x * x * (3 - 2 * x), x * x * (3 - 2 * x)])
            slope.append([x * (1 - x) ** 2, x * x * (x - 1)])
            der.append([-6 * x * (1 - x), 6 * x * (1 - x)])
            dslope.append([(1 - x) * (1 - 3 * x), x * (3 * x - 2)])

    def total(axis):
        b = [der[a] if a == axis else val[a] for a in range(3)]
        s = 0.0
        for q in range(8):
            d = (q & 1, (q >> 1) & 1, q >> 2)
            w = [b[a][d[a]] for a in range(3)]
            s = s + w[0] * w[1] * w[2] * c[:, q, 0]
            if slope is not None:
                for a in range(3):
                    sl = (dslope if a == axis else slope)[a][d[a]]
                    o = [w[e] for e in range(3) if e != a]
                    s = s + sl * o[0] * o[1] * h[a] * c[:, q, 1 + a]
        return s

    return total(-1), torch.stack([total(a) / h[a] for a in range(3)], 1)


def _interpolate(spec, pay, table, pts, mode):
    """gap, gradient (0 where invalid) and validity, in 64 bits."""
    gap = torch.zeros(len(pts), dtype=torch.float64, device=pts.device)
    grad = torch.zeros(len(pts), 3, dtype=torch.float64, device=pts.device)
    valid = torch.zeros(len(pts), dtype=torch.bool, device=pts.device)
    for a in range(0, len(pts), 1 << 20):
        b = min(len(pts), a + (1 << 20))
        idx, ok, frac = _cells(spec, table, pts[a:b])
        g0, g1 = _hermite_value(pay[idx].double(), frac, spec, mode)
        gap[a:b], grad[a:b], valid[a:b] = torch.where(ok, g0, 0.0 * g0), torch.where(ok[:, None], g1, 0.0 * g1), ok
    return gap, grad, valid


def _query_flops(mode):
    return 250 if mode == "tricubic" else 90


def _band_voxels(area, h, band, halo=2, bd=8):
    """Stored voxels of a narrow band about a surface of this area."""
    return area * 2.0 * ((band + halo) * h + 0.87 * bd * h) / h ** 3


def _stored(case, dense):
    spec = _torus_spec(max(int(case["res"]), 8))
    if dense:
        return spec["shape"][0] * spec["shape"][1] * spec["shape"][2]
    return _band_voxels(4 * math.pi ** 2 * TORUS[0] * TORUS[1], float(spec["voxel"][0]), 3)


def _touched(case, n, dense):
    """Bytes of the grid that n points within 3 voxels of the surface read."""
    h = float(_torus_spec(max(int(case["res"]), 8))["voxel"][0])
    near = min(_stored(case, dense), 4 * math.pi ** 2 * TORUS[0] * TORUS[1] * 8.0 * h / h ** 3)
    per = 4 if dense and case["mode"] == "trilinear" else 16
    return min(near * 16, n * 8 * per)
