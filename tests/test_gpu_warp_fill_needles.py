"""Needles in the warp-wide fills.  Just past the tip of a needle (height just
above 1/1024 of its longest edge) the FP32 edge tests cannot tell inside from
outside, so the distance to its plane is no bound of the distance to the
triangle.  Each voxel here lies 1.0e-5 to 1.4e-5 past a tip, in the needle's
plane, with another triangle at 0.9 of that distance: the fill has to find the
other triangle, as the per-thread traversal does.  The seeds are those of
100,000 where FP32 puts the point inside the needle and the needle lies in the
cube."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEEDS = [2942, 3375, 8137, 8397, 13764, 26432, 30036, 43618, 43752, 45533, 52345, 54985, 55197, 64228, 65361,
         66614, 70303, 87383, 90803, 96546, 99276]
BMIN, VOXEL = -1.3464101615137753, 0.08415063509461096  # of a cube of side 2 at 32 voxels, padding 0.1


def _needle(seed):
    """(needle, other triangle, voxel indices, other triangle's distance)."""
    rng = np.random.default_rng(seed)
    ijk = rng.integers(8, 24, 3)
    p = BMIN + (ijk + 0.5) * VOXEL
    u = rng.normal(size=3)
    u /= np.linalg.norm(u)
    w = np.cross(u, rng.normal(size=3))
    w /= np.linalg.norm(w)
    angle, length, f, past = rng.uniform(0.00125, 0.00145), rng.uniform(0.4, 0.6), rng.uniform(0.8, 1), \
        rng.uniform(1.0e-5, 1.4e-5)
    t = rng.uniform(0, angle)
    c = p - past * (np.cos(t) * u + np.sin(t) * w)
    needle = np.stack([c - length * u, c - f * length * (np.cos(angle) * u + np.sin(angle) * w), c])
    s = p + 0.9 * past * np.cross(u, w)
    other = np.stack([s + 2e-3 * (np.cos(k) * u + np.sin(k) * w) for k in (0.3, 2.4, 4.5)])
    return needle, other, ijk, 0.9 * past


def test_nearest_triangle_past_a_needle_tip(cuda):
    from sdfo import SdfGrid
    from sdfo import _native as N
    from sdfo import meshes as M

    v, t = M.cube(2.0)
    b, bt = M.icosphere(3, 0.05)
    verts, tris = [v, b + [0.8, 0.8, 0.8]], [t, bt + len(v)]
    n = len(v) + len(b)
    for s in SEEDS:
        for tri in _needle(s)[:2]:
            verts.append(tri)
            tris.append([[n, n + 1, n + 2]])
            n += 3
    verts, tris = np.concatenate(verts), np.concatenate(tris).astype(np.int32)
    tn = N.Tuning()
    N.check(N.load().sdfo_get_tuning(ctypes.byref(tn)))
    old = tn.triangle_cull
    out = []
    try:
        for cull in (0, 2):
            tn.triangle_cull = cull
            N.check(N.load().sdfo_set_tuning(ctypes.byref(tn)))
            g = SdfGrid.build_dense(verts, tris, target_resolution=32, max_resolution=32)
            assert np.allclose(g.spec()["bmin"], BMIN, rtol=1e-15) and np.allclose(g.spec()["voxel"], VOXEL, rtol=1e-15)
            out.append(g.export_dense())
    finally:
        tn.triangle_cull = old
        N.check(N.load().sdfo_set_tuning(ctypes.byref(tn)))
    phi = out[0]["phi"].reshape(32, 32, 32)
    for s in SEEDS:
        _, _, (i, j, k), distance = _needle(s)
        # voxel centres and the triangle's corners are rounded to 2^-53
        assert abs(abs(phi[k, j, i]) - distance) < 1e-14, s
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
