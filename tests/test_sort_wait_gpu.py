"""The radix sort when its waits for earlier tiles run out and their digits are counted from the keys."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls", [0, 1, 3])
@pytest.mark.parametrize("n", [8193, 12289, 100_003, 1_000_003])
def test_counts_from_the_keys(gb300, n, polls):
    import torch
    from daxtoolkit_gb300 import capi
    rng = np.random.default_rng(n)
    k = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    k[::3] &= 0xff00  # equal keys: the order of their values shows stability
    keys = torch.from_numpy(k.view(np.int32).copy()).cuda()
    vals = torch.arange(n, dtype=torch.int32, device="cuda")
    nb = capi.lib().dax_gb300_sort_scratch_bytes(n, capi.TYPE_U32, 4)
    scratch = torch.empty(nb, dtype=torch.uint8, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    capi.call("dax_gb300_selfcheck_sort_wait", p(keys), p(vals), n, polls, p(scratch), nb, None)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(keys.cpu().numpy().view(np.uint32), k[order])
    assert np.array_equal(vals.cpu().numpy(), order)
