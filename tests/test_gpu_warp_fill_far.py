"""The warp-wide fills of parts far from the origin, against the per-thread
traversal: FP32 sees points relative to the scene's middle, so only the FP64
rounding of the coordinates grows with the offset."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [10.0, 1e3, 1e5, 1e7])
@pytest.mark.parametrize("name", ["gear", "ball"])
def test_warp_fill_far_from_the_origin(cuda, name, offset):
    from sdfo import SdfGrid
    from sdfo import _native as N
    from sdfo import meshes as M

    q, _ = np.linalg.qr(np.random.default_rng(2).normal(size=(3, 3)))
    v, t = M.gear_prism(23, 0.05, 0.01, 9000) if name == "gear" else M.icosphere(4, 0.05)
    v = v @ q.T + offset * np.array([1.0, -0.6, 0.4])
    tn = N.Tuning()
    N.check(N.load().sdfo_get_tuning(ctypes.byref(tn)))
    old = tn.triangle_cull
    out = []
    try:
        for cull in (0, 2):
            tn.triangle_cull = cull
            N.check(N.load().sdfo_set_tuning(ctypes.byref(tn)))
            out.append([SdfGrid.build_dense(v, t, target_resolution=48, max_resolution=48).export_dense(),
                        SdfGrid.build_sparse(v, t, target_resolution=64, max_resolution=64, band_voxels=2,
                                             block_dim=8).export_sparse()])
    finally:
        tn.triangle_cull = old
        N.check(N.load().sdfo_set_tuning(ctypes.byref(tn)))
    for a, b in zip(*out):
        for k in a:
            assert np.array_equal(a[k], b[k]), k
