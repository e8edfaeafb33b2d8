"""Contact on a dense grid (points listed by the grid's touch bits) against the
same grid as a view, which has no bits and evaluates every point.  Same
arithmetic per point, so forces and Jacobians differ only by the order of FP64
sums over points, and the measure's integers and gap not at all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(n_poses, nq, seed=0):
    from sdfo import meshes as M
    from sdfo.contact import pack_states

    rng = np.random.default_rng(seed)
    v, t = M.torus(0.05, 0.01, 192, 20)
    qx, qw = M.centroid_quadrature(v, t)
    pick = rng.permutation(len(qx))[:nq] if nq <= len(qx) else np.arange(nq) % len(qx)
    a = rng.normal(size=(n_poses, 3, 3))
    R = np.linalg.qr(a)[0]
    r = rng.uniform(-0.06, 0.06, (n_poses, 3))
    r[::5] *= 40.0  # far outside the grid
    poses = pack_states(r, R, rng.uniform(-0.1, 0.1, (n_poses, 3)), rng.uniform(-1, 1, (n_poses, 3)))
    rb = np.linalg.qr(rng.normal(size=(3, 3)))[0]
    body = pack_states(np.array([[0.01, -0.02, 0.005]]), rb[None], np.full((1, 3), 0.02), np.full((1, 3), 0.3))
    return qx[pick], qw[pick], poses, body


@pytest.mark.parametrize("mode", ["trilinear", "tricubic"])
@pytest.mark.parametrize("nq,narrow", [(1, None), (255, None), (4097, None), (7680, 0.02), (9001, None)])
@pytest.mark.parametrize("order", [2.0, 1.5, 0.0])
def test_listed_points_give_what_all_points_give(cuda, mode, nq, narrow, order):
    import torch

    from sdfo import SdfGrid
    from sdfo import meshes as M
    from sdfo.contact import ContactBatch

    v, t = M.gear_prism(12, 0.05, 0.03, 900)
    grid = SdfGrid.build_dense(v, t, target_resolution=40, max_resolution=40)
    qx, qw, poses, body = _scene(23, nq)
    law = dict(stiffness=1e9, order=order, damping=1e3, friction=0.3, regularizer=1e-4)
    out = []
    for g in (grid, grid.view(grid.payload())):
        b = ContactBatch(g, qx, qw, mode=mode, narrow_margin=narrow, **law)
        ft = b.evaluate(poses, body)
        ft2, jac = b.evaluate(poses, body, jacobian=True)
        out.append((ft, ft2, jac, b.measure(poses, body)))
    a, b = out
    assert torch.isfinite(b[0]).all()
    if nq > 1 and order > 0:
        assert (b[0].abs().amax(1) > 0).any() and (b[0].abs().amax(1) == 0).any()
    # sums of at most 9,001 terms in another order: 9,001 ulp of the largest
    # partial sum, which 1e-9 of the largest entry covers with cancellation
    # (the Jacobian of an order-0 law is not finite: the same entries in both)
    for x, y in zip(a[:3], b[:3]):
        assert torch.equal(torch.isnan(x), torch.isnan(y))
        x, y = x.nan_to_num(0.0), y.nan_to_num(0.0)
        scale = y.abs().amax().clamp_min(1e-300)
        assert ((x - y).abs() <= 1e-9 * scale).all()
    for k in a[3]:
        assert torch.equal(a[3][k], b[3][k]), k
