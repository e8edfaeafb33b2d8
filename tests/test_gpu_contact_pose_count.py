"""Contact kernels on both sides of the number of poses where the threads per
pose change (the number of SMs): the same pose gives the same bits in any call,
and above the limit the points listed by touch bits give what a view, which
evaluates every point, gives."""
import pytest

from test_gpu_contact_touch import _scene

pytestmark = pytest.mark.gpu

LAW = dict(stiffness=1e9, order=2.0, damping=1e3, friction=0.3, regularizer=1e-4)


def _grid():
    from sdfo import SdfGrid
    from sdfo import meshes as M

    return SdfGrid.build_dense(*M.gear_prism(12, 0.05, 0.03, 900), target_resolution=40, max_resolution=40)


@pytest.mark.parametrize("mode", ["trilinear", "tricubic"])
@pytest.mark.parametrize("nq,narrow", [(255, None), (4097, 0.02), (9001, None)])
def test_a_pose_does_not_depend_on_the_others(cuda, mode, nq, narrow):
    import torch

    from sdfo.contact import ContactBatch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    qx, qw, poses, body = _scene(300, nq)
    b = ContactBatch(_grid(), qx, qw, mode=mode, narrow_margin=narrow, **LAW)
    meas = b.measure(poses, body)  # first: from then on the points are taken in the leaves' order
    ft, jac = b.evaluate(poses, body, jacobian=True)
    forward = b.evaluate(poses, body)
    assert torch.equal(forward, ft) and (ft.abs().amax(1) > 0).any()
    for n in (1, 23, sms, sms + 1):
        for first in (0, 300 - n):
            part = poses[first:first + n]
            f, j = b.evaluate(part, body, jacobian=True)
            m = b.measure(part, body)
            assert torch.equal(f, ft[first:first + n]) and torch.equal(b.evaluate(part, body), f)
            assert torch.equal(j, jac[first:first + n])
            for k in m:
                assert torch.equal(m[k], meas[k][first:first + n]), k


@pytest.mark.parametrize("mode", ["trilinear", "tricubic"])
@pytest.mark.parametrize("nq,narrow", [(1, None), (255, None), (4097, None), (7680, 0.02), (9001, None)])
def test_many_poses_against_all_points(cuda, mode, nq, narrow):
    import torch

    from sdfo.contact import ContactBatch

    grid = _grid()
    qx, qw, poses, body = _scene(301, nq, seed=1)
    out = []
    for g in (grid, grid.view(grid.payload())):
        b = ContactBatch(g, qx, qw, mode=mode, narrow_margin=narrow, **LAW)
        out.append((b.evaluate(poses, body), *b.evaluate(poses, body, jacobian=True), b.measure(poses, body)))
    # sums of at most 9,001 terms in another order: 9,001 ulp of the largest
    # partial sum, which 1e-9 of the largest entry covers with cancellation
    for x, y in zip(out[0][:3], out[1][:3]):
        assert torch.isfinite(y).all()
        assert ((x - y).abs() <= 1e-9 * y.abs().amax().clamp_min(1e-300)).all()
    for k in out[0][3]:
        assert torch.equal(out[0][3][k], out[1][3][k]), k
