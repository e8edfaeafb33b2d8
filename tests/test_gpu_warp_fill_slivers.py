"""Near-degenerate triangles in the warp-wide fills, against the per-thread
traversal: as many as a lane's list holds, one more, the limit and one more,
among them triangles without area and repeated ones."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 8, 9, 31, 32, 33])
def test_slivers(cuda, n):
    from sdfo import SdfGrid
    from sdfo import _native as N
    from sdfo import meshes as M

    rng = np.random.default_rng(n)
    v, t = M.hollow_cylinder(0.05, 0.04, 0.02, 256, 4, 1)
    a = rng.uniform(-0.03, 0.03, (n, 3))
    d = rng.normal(size=(n, 3))
    b = a + 0.03 * d / np.linalg.norm(d, axis=1, keepdims=True)
    c = a + rng.uniform(0, 1, (n, 1)) * (b - a) + rng.choice([0.0, 1e-9, 1e-5], (n, 1)) * rng.normal(size=(n, 3))
    c[::5] = a[::5]
    a[1::6], b[1::6], c[1::6] = a[:1], b[:1], c[:1]
    s = len(v) + np.arange(n)
    verts = np.concatenate([v, a, b, c])
    tris = np.concatenate([t, np.stack([s, s + n, s + 2 * n], 1)]).astype(np.int32)
    tn = N.Tuning()
    N.check(N.load().sdfo_get_tuning(ctypes.byref(tn)))
    old = tn.triangle_cull
    out = []
    try:
        for cull in (0, 2):
            tn.triangle_cull = cull
            N.check(N.load().sdfo_set_tuning(ctypes.byref(tn)))
            out.append([SdfGrid.build_dense(verts, tris, target_resolution=48, max_resolution=48).export_dense(),
                        SdfGrid.build_sparse(verts, tris, target_resolution=64, max_resolution=64, band_voxels=2,
                                             block_dim=8).export_sparse()])
    finally:
        tn.triangle_cull = old
        N.check(N.load().sdfo_set_tuning(ctypes.byref(tn)))
    for p, q in zip(*out):
        for k in p:
            assert np.array_equal(p[k], q[k], equal_nan=True), k
