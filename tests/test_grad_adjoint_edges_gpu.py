"""CellGradient's adjoint at the edges of its tiles (31 point columns, 8 point rows), in one segment of planes and in
several, from gradients at every offset from a 16-byte boundary."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _want(dg, dims):
    """dL/df in float64 for unit widths, and the sum of its terms' magnitudes."""
    nx, ny, nz = dims
    out, mag = np.zeros((nz, ny, nx)), np.zeros((nz, ny, nx))
    for c in range(3):
        for k in (0, 1):
            for j in (0, 1):
                for i in (0, 1):
                    t = 0.25 * dg[..., c].astype(np.float64)
                    at = np.s_[k:nz - 1 + k, j:ny - 1 + j, i:nx - 1 + i]
                    out[at] += t if (i, j, k)[c] else -t
                    mag[at] += np.abs(t)
    return out, mag


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("dims", [(2, 2, 2), (31, 8, 3), (32, 9, 13), (33, 17, 25), (63, 16, 40), (94, 30, 70), (125, 3, 2)])
def test_edges(dims, offset):
    import torch
    from daxtoolkit_gb300 import capi, cont
    nx, ny, nz = dims
    dg = np.random.default_rng(nx).normal(size=(nz - 1, ny - 1, nx - 1, 3)).astype(np.float32)
    buf = torch.full((dg.size + 8,), float("nan"), device="cuda")  # what lies around the gradients must not matter
    buf[offset:offset + dg.size] = torch.from_numpy(dg.ravel()).cuda()
    field, out = torch.zeros(nx * ny * nz, device="cuda"), torch.empty(nx * ny * nz, device="cuda")
    g = cont.UniformGrid(dims).desc()
    capi.call("dax_gb300_field_adjoint", ctypes.byref(g), ctypes.c_void_p(field.data_ptr()), 0.5, None, 0, None,
              ctypes.c_void_p(buf.data_ptr() + 4 * offset), ctypes.c_void_p(out.data_ptr()),
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    want, mag = _want(dg, dims)
    # 24 terms, each rounded at most 12 times on its way into the sum (2^-24 each)
    assert (np.abs(out.cpu().numpy().reshape(want.shape) - want) <= 16 * 2.0 ** -24 * mag).all()
