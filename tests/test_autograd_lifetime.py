"""A differentiable query's tensors are released with its results, without the
garbage collector: the node keeps no reference to its own outputs."""
import gc
import weakref

import pytest


@pytest.mark.gpu
def test_results_are_released_without_the_garbage_collector(cuda):
    import torch

    from sdfo import SdfGrid
    from sdfo import meshes as M
    from sdfo.autograd import sdf_query

    grid = SdfGrid.build_dense(*M.torus(0.05, 0.016, 24, 12), target_resolution=24, max_resolution=24)
    x = (0.04 * torch.rand(1000, 3, device="cuda")).requires_grad_(True)
    gc.collect()
    gc.disable()
    try:
        gap, grad = sdf_query(grid, x)
        node = weakref.ref(grad.grad_fn)
        dx, = torch.autograd.grad((gap.sum() + grad[:, 0].sum()), x)
        assert torch.isfinite(dx).all()
        del gap, grad, dx
        assert node() is None
    finally:
        gc.enable()
