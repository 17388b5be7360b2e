"""The Mandelbulb field where lanes take new points: grids of fewer points than a tile, a last tile of few points, more
tiles than blocks, and fields whose points all take no, one, every or mixed steps; each point's value is the one it has on
a grid of its own plane, whatever its neighbours."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 3, 2), (16, 16, 1), (257, 1, 1), (31, 33, 7), (201, 77, 41)])
@pytest.mark.parametrize("window", [(-1.0, 2.0), (-0.1, 0.2), (5.0, 0.2), (0.6, 0.1)])
def test_planes(dims, window):
    import torch
    from daxtoolkit_gb300 import cont
    lo, size = window
    step = size / 256  # a power of two times the size: the same coordinates for every shape of grid
    whole = cont.mandlebulb_field(cont.UniformGrid(dims, origin=(lo,) * 3, spacing=(step,) * 3))
    whole = whole.reshape(dims[2], -1)
    assert not torch.isnan(whole).any()
    for k in sorted({0, dims[2] // 2, dims[2] - 1}):
        plane = cont.UniformGrid(origin=(lo,) * 3, spacing=(step,) * 3)
        plane.SetExtent((0, 0, k), (dims[0] - 1, dims[1] - 1, k))
        assert torch.equal(cont.mandlebulb_field(plane).reshape(-1), whole[k])
