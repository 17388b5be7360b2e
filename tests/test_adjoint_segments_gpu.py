"""CellGradient's adjoint on grids of more tiles than run at once, whose segments have the most planes, and on long thin
ones: a tile's planes must not depend on where its segment begins."""
import ctypes

import numpy as np
import pytest

from tests.test_grad_adjoint_edges_gpu import _want

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 2, 60001), (33, 9, 9001), (200, 3, 4099), (300, 260, 61), (31, 8, 25600)])
def test_segments(dims):
    import torch
    from daxtoolkit_gb300 import capi, cont
    nx, ny, nz = dims
    dg = np.random.default_rng(nz).normal(size=(nz - 1, ny - 1, nx - 1, 3)).astype(np.float32)
    d = torch.from_numpy(dg.ravel()).cuda()
    field, out = torch.zeros(nx * ny * nz, device="cuda"), torch.empty(nx * ny * nz, device="cuda")
    # adjacent coordinates differ by exactly 1 below 2^24
    g = cont.UniformGrid(dims).desc()
    capi.call("dax_gb300_field_adjoint", ctypes.byref(g), ctypes.c_void_p(field.data_ptr()), 0.5, None, 0, None,
              ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(out.data_ptr()),
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    want, mag = _want(dg, dims)
    # 24 terms, each rounded at most 12 times on its way into the sum (2^-24 each)
    assert (np.abs(out.cpu().numpy().reshape(want.shape) - want) <= 16 * 2.0 ** -24 * mag).all()
