"""The radix sort where its blocks change: the block that sorts alone (8192), the sweep's tile (6144), and the sizes at
which the digit counts of one, several and all passes fit beside the tile states."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6143, 6145, 8192, 8193, 12288, 12289, 18433, 45056, 45057, 94208, 94209, 200_003])
@pytest.mark.parametrize("dtype,words", [("int32", 1), ("int32", 3), ("float32", 0), ("int64", 1), ("int64", 4)])
def test_sizes(dtype, words, n):
    import torch
    from daxtoolkit_gb300 import cont
    rng = np.random.default_rng(n)
    k = rng.normal(scale=40, size=n).astype(dtype)  # many equal keys: the order of their values shows stability
    keys, vals = torch.from_numpy(k.copy()).cuda(), None
    if words:
        v = rng.integers(0, 2 ** 31, size=(n, words)).astype(np.int32)
        vals = torch.from_numpy(v).cuda()
    cont.Algorithm.SortByKey(keys, vals)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(keys.cpu().numpy(), k[order])
    if words:
        assert np.array_equal(vals.cpu().numpy(), v[order])
