"""The threshold's connectivity into arrays at every offset from a 32-byte boundary: the same cells, and nothing beside
them."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", range(8))
@pytest.mark.parametrize("dims", [(70, 40, 40), (33, 9, 8)])
def test_offsets(dims, offset):
    import torch
    from daxtoolkit_gb300 import capi, cont
    grid = cont.UniformGrid(dims)
    f = torch.rand(dims[0] * dims[1] * dims[2], generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    f[: f.numel() // 2] = 0.5  # whole words of kept cells among the others
    scratch = cont.Scratch()
    want = cont.threshold(grid, f, 0.2, 0.9, scratch=scratch)
    K, U = want["conn"].shape[0], want["coords"].shape[0]
    buf = torch.full((8 * K + 24,), -3, dtype=torch.int32, device="cuda")
    assert buf.data_ptr() % 32 == 0
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    coords, g, s = torch.empty_like(want["coords"]), grid.desc(), scratch.buf
    capi.call("dax_gb300_threshold_generate", ctypes.byref(g), p(f), 0.2, 0.9, p(s), s.numel(),
              ctypes.c_void_p(buf.data_ptr() + 4 * (8 + offset)), K, p(coords), None, U, None)
    torch.cuda.synchronize()
    a = 8 + offset
    assert K > 100 and torch.equal(buf[a:a + 8 * K].view(K, 8), want["conn"]) and torch.equal(coords, want["coords"])
    assert bool((buf[:a] == -3).all()) and bool((buf[a + 8 * K:] == -3).all())
