"""A differentiable query's backward reads the gradient that it returned: a
caller that changes it in place gets an error, not a wrong dL/dp; changing the
gap, which the backward does not read, stays allowed."""
import pytest


@pytest.mark.gpu
def test_change_of_the_returned_gradient_is_noticed(cuda):
    import torch

    from sdfo import SdfGrid
    from sdfo import meshes as M
    from sdfo.autograd import sdf_query

    grid = SdfGrid.build_dense(*M.torus(0.05, 0.016, 24, 12), target_resolution=24, max_resolution=24)
    x = (0.04 * torch.rand(1000, 3, device="cuda")).requires_grad_(True)
    gap, grad = sdf_query(grid, x)
    loss = gap.sum() + grad.sum()
    want, = torch.autograd.grad(loss, x, retain_graph=True)
    with torch.no_grad():
        gap.mul_(2.0)
    again, = torch.autograd.grad(loss, x, retain_graph=True)
    assert torch.equal(again, want)
    with torch.no_grad():
        grad.div_(grad.norm(dim=1, keepdim=True) + 1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(loss, x)
