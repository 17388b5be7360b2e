"""The per-cell counts at the edges of a warp's run of 31 cells and of its rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 2, 2), (31, 9, 3), (32, 10, 2), (33, 8, 5), (63, 17, 4), (64, 2, 9), (257, 3, 3)])
def test_counts_of_every_cell(dims):
    import oracle
    import torch
    from daxtoolkit_gb300 import cont
    f = np.random.default_rng(dims[0]).uniform(0, 1, size=dims[0] * dims[1] * dims[2]).astype(np.float32)
    f[::7] = np.nan
    grid, fd = cont.UniformGrid(dims), torch.from_numpy(f).cuda()
    O, og = oracle.Oracle("port"), oracle.make_grid(dims)
    count = cont.DispatcherMapCell(cont.MarchingCubesCount(0.5)).Invoke(grid, fd)
    assert np.array_equal(count.cpu().numpy().ravel(), np.asarray(O.mc_count(og, f, 0.5)[0]).ravel())
    count = cont.DispatcherMapCell(cont.ThresholdCount(0.05, 0.95)).Invoke(grid, fd)
    assert np.array_equal(count.cpu().numpy().ravel(), np.asarray(O.threshold_count(og, f, 0.05, 0.95)).ravel())
