"""The threshold's masks at the edges of their walks: rows of one word, 31 words and as long as they get, ranges that end
inside a row, planes of two rows; dense and sparse intervals, in scratch that another threshold left."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [(0.0, 0.9), (0.4, 0.6), (-1.0, 2.0)])
@pytest.mark.parametrize("dims", [(2, 2, 2), (2, 2, 300), (3, 2, 1500), (33, 2, 90), (65, 41, 3), (992, 5, 7), (993, 7, 5),
                                  (8192, 2, 3), (8161, 9, 3), (70, 40, 40)])
def test_threshold(dims, lo, hi):
    import oracle
    import torch
    from daxtoolkit_gb300 import cont
    f = np.random.default_rng(dims[0]).uniform(0, 1, size=dims[::-1]).astype(np.float32)
    f[:, :, ::2] = 0.5  # pairs in range side by side, so that cells survive narrow intervals
    f[::2] = 0.5
    f = f.ravel()
    grid, O, og = cont.UniformGrid(dims), oracle.Oracle("port"), oracle.make_grid(dims)
    cont.threshold(grid, torch.from_numpy(1 - f).cuda(), 0.2, 0.8)
    out = cont.threshold(grid, torch.from_numpy(f).cuda(), lo, hi)
    ref = O.threshold_generate(og, f, O.threshold_count(og, f, lo, hi))
    assert np.array_equal(out["conn"].cpu().numpy(), ref["conn"])
    assert np.array_equal(out["coords"].cpu().numpy().view(np.uint32), ref["coords"].view(np.uint32))
    assert np.array_equal(out["field"].cpu().numpy().view(np.uint32), ref["field"].view(np.uint32))
