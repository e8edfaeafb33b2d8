"""Points placed in FP32 ahead of the FP64 contact path, 2^33 voxels from the
grid's origin: there the FP64 coordinates themselves are rounded to 2^-20 of a
voxel, so a point 9.2e-7 voxels outside the grid's first voxel centre rounds to
the centre and counts as inside.  FP32 has to leave such points to FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FAR, H, N = 2.0 ** 23, 2.0 ** -10, 8


def _grid():
    from sdfo import SdfGrid

    phi = np.full((N, N, N), 1.0)
    phi[:2, :2, :2] = -1.0
    normal = np.tile([0.0, 0.0, 1.0], (N ** 3, 1))
    spec = dict(bmin=np.full(3, FAR), bmax=np.full(3, FAR + N * H), voxel=np.full(3, H), shape=(N, N, N))
    return SdfGrid.from_dense(spec, phi.ravel(), normal)


POINTS = np.array([[-0.9e-9, 0.0, 0.0], [0.0, 0.25 * H, 0.25 * H]])


def test_contact(cuda):
    import torch

    from sdfo.contact import ContactBatch, pack_states

    grid = _grid()
    pose = pack_states(np.full((1, 3), FAR + 0.5 * H), np.eye(3)[None])
    body = pack_states(np.zeros((1, 3)), np.eye(3)[None])
    out = []
    for g in (grid, grid.view(grid.payload())):
        b = ContactBatch(g, POINTS, np.ones(2), 1.0, order=1.0)
        out.append((b.evaluate(pose, body), b.measure(pose, body)))
    # the view places every point in FP64
    assert out[1][1]["valid_count"].item() == 2
    assert torch.equal(out[0][0], out[1][0])
    for k in out[0][1]:
        assert torch.equal(out[0][1][k], out[1][1][k]), k


@pytest.mark.parametrize("threads", [32, 256])
def test_be_step(cuda, threads):
    import torch

    from sdfo.be import BEStepper

    # 1,536 points: with FP32 bounds for every thread count
    st = BEStepper(_grid(), np.tile(POINTS[:1], (1536, 1)), np.ones(1536), 1.0, np.eye(3), 1e-3, order=1,
                   narrow_margin=None, gravity=(0.0, 0.0, 0.0), max_scenes=1, threads=threads)
    scenes = st.scenes(np.full((1, 3), FAR + 0.5 * H), np.eye(3)[None])
    st.step(scenes, 1e-5)
    torch.cuda.synchronize()
    assert st.unpack(scenes)["last_gap"][0] == -1.0
