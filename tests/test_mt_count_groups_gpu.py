"""The count pass of marching tetrahedra where its copies and runs end: cell
counts one below, at and above a lane's run, a group, a chunk and a tile, more
tiles than resident blocks, connectivity off a 16-byte boundary, and bad ids in
whole and cut-off runs; counts identical to the oracle's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

P = 500


def _cells(C, seed):
    rng = np.random.default_rng(seed)
    conn = rng.integers(0, P, (C, 4), dtype=np.int32)
    return conn, rng.standard_normal(P).astype(np.float32)


def _grid(cont, conn, off):
    flat = torch.empty(conn.size + 4, dtype=torch.int32, device="cuda")
    flat[off:off + conn.size] = torch.from_numpy(conn.reshape(-1))
    view = flat[off:off + conn.size].view(-1, 4)
    assert (view.data_ptr() % 16 == 0) == (off == 0)
    return cont.UnstructuredGrid(torch.zeros(P, 3, device="cuda"), view)


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("C", [1, 4, 5, 6, 159, 160, 161, 319, 480, 481, 511, 512, 513, 4095, 4096,
                               4097, 4096 * 3 + 485, 4096 * 1400 + 77])
def test_count_at_group_ends(gb300, oracle_best, C, off):
    cont = gb300
    conn, f = _cells(C, C)
    ref = oracle_best.mt_count(conn, f, 0.25)
    count = cont.DispatcherMapCell(cont.MarchingTetrahedraCount(0.25)).Invoke(
        _grid(cont, conn, off), torch.from_numpy(f).cuda())
    assert np.array_equal(count.cpu().numpy(), ref)


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("bad", [P, -1, -2 ** 31, 2 ** 31 - 1])
@pytest.mark.parametrize("cell", [0, 4, 159, 480, 511, 512, 4096, 4098])
def test_bad_id_is_an_error(gb300, cell, bad, off):
    """Each corner in turn; the last cells lie in a run cut off by the end."""
    cont = gb300
    from daxtoolkit_gb300 import capi
    conn, f = _cells(4099, 7)
    conn[cell, cell % 4] = bad
    with pytest.raises(capi.ErrorControlBadValue):
        cont.DispatcherMapCell(cont.MarchingTetrahedraCount(0.25)).Invoke(
            _grid(cont, conn, off), torch.from_numpy(f).cuda())
