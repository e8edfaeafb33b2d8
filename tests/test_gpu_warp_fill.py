"""The warp-wide fills against the per-thread traversal of the same tree, which
is pinned to the reference: equal bit for bit.  Meshes where the fast path can
go wrong: just below and at its smallest size, bricks that do not fill warps,
fans and symmetric shapes (many exactly equal distances), shapes about equally
far from much of the mesh, slivers (a few, and too many for the fast path),
coordinates far from the origin and in other units."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cull(on):
    from sdfo import _native as N

    t = N.Tuning()
    N.check(N.load().sdfo_get_tuning(ctypes.byref(t)))
    t.triangle_cull = 0 if on else 2
    N.check(N.load().sdfo_set_tuning(ctypes.byref(t)))


def _slivers(n):
    from sdfo import meshes as M

    v, t = M.hollow_cylinder(0.05, 0.04, 0.02, 64, 4, 1)
    a = 2.0 * np.pi * np.arange(n) / n
    c = np.stack([0.02 * np.cos(a), 0.02 * np.sin(a), np.full(n, 0.03)], 1)
    w = np.concatenate([c, c + [0.0, 0.0, 1e-6], c * [1.5, 1.5, 1.0]])
    s = len(v) + np.arange(n)
    return np.concatenate([v, w]), np.concatenate([t, np.stack([s, s + n, s + 2 * n], 1)]).astype(np.int32)


def _meshes():
    from sdfo import meshes as M

    q, _ = np.linalg.qr(np.random.default_rng(2).normal(size=(3, 3)))
    gear = M.gear_prism(23, 0.05, 0.01, 9000)
    ball = M.icosphere(4, 0.05)
    return {
        "torus_60": M.torus(0.05, 0.016, 6, 5),
        "torus_64": M.torus(0.05, 0.016, 8, 4),
        "cylinder": M.hollow_cylinder(0.05, 0.04, 0.02, 128, 8, 1),
        "gear": gear,
        "gear_turned": (gear[0] @ q.T, gear[1]),
        "gear_far": (gear[0] + [5.0, -3.0, 2.0], gear[1]),
        "gear_mm": (gear[0] * 1000.0, gear[1]),
        "ball": ball,
        "ball_twice": (ball[0], np.concatenate([ball[1], ball[1][:700]])),
        "slivers_3": _slivers(3),
        "slivers_40": _slivers(40),
    }


@pytest.mark.parametrize("name", ["torus_60", "torus_64", "cylinder", "gear", "gear_turned", "gear_far", "gear_mm",
                                  "ball", "ball_twice", "slivers_3", "slivers_40"])
def test_warp_fill_equals_per_thread_fill(cuda, name):
    from sdfo import SdfGrid

    v, t = _meshes()[name]
    out = []
    try:
        for on in (True, False):
            _cull(on)
            d = SdfGrid.build_dense(v, t, target_resolution=32, max_resolution=32).export_dense()
            s = [SdfGrid.build_sparse(v, t, target_resolution=48, max_resolution=48, band_voxels=2,
                                      block_dim=b).export_sparse() for b in (3, 5, 8)]
            out.append([d] + s)
    finally:
        _cull(True)
    for a, b in zip(*out):
        for k in a:
            assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("tile", [(3, 3), (2, 2), (5, 3), (1, 1)])
def test_warp_fill_of_every_tile_shape(cuda, port, tile):
    from sdfo import SdfGrid
    from sdfo import _native as N
    from sdfo import meshes as M

    v, t = M.torus(0.05, 0.016, 30, 13)
    P = port.build_dense(v, t, padding=0.1, target_resolution=28, max_resolution=28)
    tn = N.Tuning()
    N.check(N.load().sdfo_get_tuning(ctypes.byref(tn)))
    old = (tn.fill_tile_log2_x, tn.fill_tile_log2_y)
    tn.fill_tile_log2_x, tn.fill_tile_log2_y = tile
    N.check(N.load().sdfo_set_tuning(ctypes.byref(tn)))
    try:
        d = SdfGrid.build_dense(v, t, target_resolution=28, max_resolution=28).export_dense()
    finally:
        tn.fill_tile_log2_x, tn.fill_tile_log2_y = old
        N.check(N.load().sdfo_set_tuning(ctypes.byref(tn)))
    for k in ("phi", "normal", "witness"):
        assert np.array_equal(d[k], P[k]), k
