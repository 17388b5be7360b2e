"""The single-pass scan when its waits run out: a timeout is reported, and no
element is written from a prefix that is not known; the next call is right."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TILE = 8192


def _scan(n, polls, lost, shift):
    from daxtoolkit_gb300 import capi
    x = np.random.default_rng(n).integers(1, 9, size=n).astype(np.int32)
    src = torch.zeros(n + shift, dtype=torch.int32, device="cuda")[shift:]
    src.copy_(torch.from_numpy(x))
    out = torch.full((n + shift,), -7, dtype=torch.int32, device="cuda")[shift:]
    nb = capi.lib().dax_gb300_scan_scratch_bytes(n)
    scratch = torch.empty(nb, dtype=torch.uint8, device="cuda")
    total = ctypes.c_int32(-1)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    st = capi.lib().dax_gb300_selfcheck_scan_wait(p(src), p(out), n, polls, lost, p(scratch), nb, ctypes.byref(total), None)
    return st, total.value, out.cpu().numpy(), np.cumsum(x, dtype=np.int32)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [TILE + 1, 40 * TILE, 152 * 8 * TILE + 5])
def test_a_tile_that_never_comes(gb300, n, shift):
    from daxtoolkit_gb300 import capi
    st, total, out, want = _scan(n, 2 ** 32 - 1, 1, shift)
    assert st == capi.ERROR_TIMEOUT and total == -1
    assert (out == -7).all()
    st, total, out, want = _scan(n, 2 ** 32 - 1, 0, shift)
    assert st == capi.SUCCESS and total == want[-1] and np.array_equal(out, want)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("polls", [1, 2, 50])
def test_short_waits(gb300, polls, shift):
    from daxtoolkit_gb300 import capi
    st, total, out, want = _scan(152 * 40 * TILE + 77, polls, 0, shift)
    assert st in (capi.SUCCESS, capi.ERROR_TIMEOUT)
    assert ((out == want) | (out == -7)).all()
    if st == capi.SUCCESS:
        assert total == want[-1] and np.array_equal(out, want)
