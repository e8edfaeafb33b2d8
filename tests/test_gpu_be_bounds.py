"""The shortcuts of a BE step's contact passes: the FP32 bounds of the measure
(from 1,536 points, and always with a warp per scene) and the points that a
cached evaluation leaves out.

The measure against the oracle's FP64 interpolation of every point, over
rotated bodies, grids far from the origin and point sets on both sides of each
limit.  Then the same scenes with points added outside the grid, without
weight, that switch the bounds on (1,535 -> 1,536 points) and the flags of the
cached evaluation off (33,000 points): states equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAW = dict(damping=1e3, friction=0.3, regularizer=1e-4)


def _rotations(rng, n):
    q = np.linalg.qr(rng.normal(size=(n, 3, 3)))[0]
    return q * np.sign(np.linalg.det(q))[:, None, None]


def _stepper(grid, x, w, n, tangent, threads, order, body_b=None):
    from sdfo.be import BEStepper, default_params

    return BEStepper(grid, x, w, 0.1, np.diag([1e-4, 1e-4, 2e-4]), 1e6, order=order, narrow_margin=None,
                     params=default_params(tangent=tangent), max_scenes=n, threads=threads, body_b=body_b, **LAW)


@pytest.mark.parametrize("threads", [32, 128, 256])
@pytest.mark.parametrize("nq", [1, 255, 257, 1535, 1536, 7680])
@pytest.mark.parametrize("offset", [0.0, 300.0])
def test_measured_gap_is_the_least_of_all_points(cuda, threads, nq, offset):
    import torch

    from oracle import interp_np
    from sdfo import SdfGrid
    from sdfo import meshes as M

    rng = np.random.default_rng(nq + threads)
    v, t = M.gear_prism(12, 0.05, 0.03, 900)
    shift = offset * np.array([1.0, -0.6, 0.4])
    grid = SdfGrid.build_dense(v + shift, t, target_resolution=32, max_resolution=32)
    phi = grid.export_dense()
    qx, qw = M.centroid_quadrature(*M.torus(0.03, 0.008, 192, 20))
    pick = rng.permutation(len(qx))[:nq]
    n = 48
    RB, rB = _rotations(rng, 1)[0], rng.normal(size=3)
    st = _stepper(grid, qx[pick], qw[pick], n, "reference", threads, 2, (rB, RB))
    # body A about the shifted gear, some at the edge of the grid, some outside
    local = shift + rng.uniform(-0.07, 0.07, (n, 3))
    R = _rotations(rng, n)
    scenes = st.scenes(rB + local @ RB.T, R, rng.uniform(-0.1, 0.1, (n, 3)), rng.uniform(-1, 1, (n, 3)))
    st.step(scenes, 1e-4)
    torch.cuda.synchronize()
    u = st.unpack(scenes)
    finite = 0
    for i in range(n):
        Y = qx[pick] @ (RB.T @ u["R"][i]).T + RB.T @ (u["r"][i] - rB)
        g, _, valid, _ = interp_np.query(grid.spec(), phi["phi"], phi["normal"], 2, Y)
        want = g[valid].min() if valid.any() else np.inf
        finite += np.isfinite(want)
        # coordinates of up to 400 are rounded to 2^-44 in Y, and so the gap;
        # a point that close to the grid's edge does not occur with these seeds
        assert u["last_gap"][i] == want or abs(u["last_gap"][i] - want) <= 1e-15 + 4e-15 * offset, i
        assert u["last_penetration"][i] == max(0.0, -u["last_gap"][i])
    assert finite > 0


@pytest.mark.parametrize("threads", [128, 256])
@pytest.mark.parametrize("tangent", ["reference", "exact"])
@pytest.mark.parametrize("order", [1, 2])
def test_points_without_effect_change_nothing(cuda, threads, tangent, order):
    import torch

    from sdfo import SdfGrid
    from sdfo import meshes as M

    rng = np.random.default_rng(3)
    v, t = M.cube(0.1)
    grid = SdfGrid.build_dense(v, t, target_resolution=32, max_resolution=32)
    qx, _ = M.centroid_quadrature(*M.torus(0.03, 0.008, 64, 12))
    qx = qx[rng.permutation(len(qx))[:1535]]
    qw = rng.integers(1, 9, 1535).astype(np.float64)  # sums without rounding
    n = 24
    r = np.stack([rng.uniform(-0.01, 0.01, n), rng.uniform(-0.01, 0.01, n), 0.058 + rng.uniform(-2e-4, 4e-4, n)], 1)
    out = []
    for total in (1535, 1536, 33000):
        x = np.concatenate([qx, np.full((total - 1535, 3), 1e3)])
        w = np.concatenate([qw, np.zeros(total - 1535)])
        st = _stepper(grid, x, w, n, tangent, threads, order)
        scenes = st.scenes(r, np.repeat(np.eye(3)[None], n, 0), np.tile([0.01, 0.0, -0.2], (n, 1)))
        steps = [st.step(scenes, 1e-3).clone() for _ in range(6)]
        torch.cuda.synchronize()
        out.append((scenes.cpu().numpy().view(np.int64), torch.stack(steps).cpu().numpy()))
        phases = st.unpack(scenes)["phase"]
    assert (phases != 0).any()
    for o in out[1:]:
        assert np.array_equal(o[0], out[0][0]) and np.array_equal(o[1], out[0][1])
