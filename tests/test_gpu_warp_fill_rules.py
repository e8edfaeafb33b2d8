"""Which way a fill takes, on both sides of each rule, against the per-thread
traversal: the number of triangles (256), of voxels (16 per SM), of patches for
the shorter search, and long thin triangles that crowd the ray's lists."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _split(mesh, times):
    v, t = np.asarray(mesh[0], float), np.asarray(mesh[1])
    for _ in range(times):
        a, b, c = v[t[:, 0]], v[t[:, 1]], v[t[:, 2]]
        n, m = len(v), len(t)
        v = np.concatenate([v, (a + b) / 2, (b + c) / 2, (c + a) / 2])
        ab, bc, ca = (n + k * m + np.arange(m) for k in range(3))
        t = np.concatenate([np.stack([t[:, 0], ab, ca], 1), np.stack([ab, t[:, 1], bc], 1),
                            np.stack([ca, bc, t[:, 2]], 1), np.stack([ab, bc, ca], 1)])
    return v, t.astype(np.int32)


def _meshes():
    from sdfo import meshes as M

    cube = M.cube(0.1)
    return {
        "torus_240": M.torus(0.05, 0.016, 15, 8),
        "torus_256": M.torus(0.05, 0.016, 16, 8),
        "ball": M.icosphere(2, 0.05),
        "rod": _split((cube[0] * [0.05, 0.05, 1.0], cube[1]), 3),
        "plate": _split((cube[0] * [1.0, 1.0, 0.05], cube[1]), 3),
        "pipe": M.hollow_cylinder(0.05, 0.04, 1.0, 128, 1, 1),
        "pipe_short": M.hollow_cylinder(0.05, 0.04, 0.15, 64, 1, 1),
    }


@pytest.mark.parametrize("res", [8, 16, 32, 64])
@pytest.mark.parametrize("name", ["torus_240", "torus_256", "ball", "rod", "plate", "pipe", "pipe_short"])
def test_fills_on_both_sides_of_the_rules(cuda, name, res):
    from sdfo import SdfGrid
    from sdfo import _native as N

    v, t = _meshes()[name]
    tn = N.Tuning()
    N.check(N.load().sdfo_get_tuning(ctypes.byref(tn)))
    old = tn.triangle_cull
    out = []
    try:
        for cull in (0, 2):
            tn.triangle_cull = cull
            N.check(N.load().sdfo_set_tuning(ctypes.byref(tn)))
            out.append([SdfGrid.build_dense(v, t, target_resolution=res, max_resolution=res).export_dense(),
                        SdfGrid.build_sparse(v, t, target_resolution=res, max_resolution=res, band_voxels=2,
                                             block_dim=8).export_sparse()])
    finally:
        tn.triangle_cull = old
        N.check(N.load().sdfo_set_tuning(ctypes.byref(tn)))
    for a, b in zip(*out):
        for k in a:
            assert np.array_equal(a[k], b[k]), k
