"""The count pass of marching tetrahedra when its waits for the connectivity
run out: every block leaves after its copies have landed, the totals are a
timeout, the generate pass writes nothing, and the next call is unaffected."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1, 160, 4096, 4096 * 1400 + 77])
def test_expired_wait(gb300, C):
    from daxtoolkit_gb300 import capi
    P = 500
    rng = np.random.default_rng(C)
    conn = torch.from_numpy(rng.integers(0, P, (C, 4), dtype=np.int32)).cuda()
    f = torch.from_numpy(rng.standard_normal(P).astype(np.float32)).cuda()
    pts = torch.zeros(P, 3, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    nb = capi.lib().dax_gb300_mt_scratch_bytes(C)
    scr = torch.empty(nb, dtype=torch.uint8, device="cuda")
    T = ctypes.c_int64(0)
    for _ in range(2):
        capi.call("dax_gb300_selfcheck_mt_wait", p(conn), C, p(f), P, 0.25, p(scr), nb, None)
        with pytest.raises(capi.DaxError) as err:
            capi.call("dax_gb300_mc_totals", p(scr), ctypes.byref(T), None, None)
        assert err.value.code == capi.ERROR_TIMEOUT
        verts = torch.full((6 * C, 3), 7.0, device="cuda")
        tri = torch.full((2 * C, 3), -5, dtype=torch.int32, device="cuda")
        capi.call("dax_gb300_mt_generate", p(pts), p(conn), C, p(f), P, 0.25, 0, p(scr), nb, None, 0, p(verts), 6 * C,
                  p(tri), 2 * C, None, None, None, None)
        assert bool((verts == 7.0).all()) and bool((tri == -5).all())
    capi.call("dax_gb300_mt_count", p(conn), C, p(f), P, 0.25, p(scr), nb, None)
    capi.call("dax_gb300_mc_totals", p(scr), ctypes.byref(T), None, None)
    inside = (f > 0.25)[conn.long()].sum(1)
    assert T.value == int(((inside == 1) | (inside == 3)).sum() + 2 * (inside == 2).sum())
