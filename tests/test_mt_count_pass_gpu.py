"""dax_gb300_mt_count, the count pass that marching tetrahedra runs: cell counts one below, at and above a lane's run, a
group, a chunk and a tile, and more tiles than resident blocks; runs of cells that lie together and apart; connectivity
on and off a 16-byte boundary; bad ids, the extreme ones among them, in whole and cut-off groups.  What it counts shows in
the totals and in the triangles generated from it, which are the oracle's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [1, 4, 5, 6, 31, 159, 160, 161, 319, 480, 481, 511, 512, 513, 4095, 4096, 4097, 4096 * 3 + 485, 4096 * 1400 + 77]


def _cells(C, seed, near):
    """near: the ids of cell c are c // 5 and up to seven more; else any of 500."""
    rng = np.random.default_rng(seed)
    P = C // 5 + 8 if near else 500
    conn = rng.integers(0, 8 if near else P, (C, 4), dtype=np.int32)
    if near:
        conn += (np.arange(C, dtype=np.int32) // 5)[:, None]
    return conn, rng.standard_normal(P).astype(np.float32), rng.random((P, 3)).astype(np.float32)


def _grid(cont, conn, pts, off):
    flat = torch.empty(conn.size + 4, dtype=torch.int32, device="cuda")
    flat[off:off + conn.size] = torch.from_numpy(conn.reshape(-1))
    view = flat[off:off + conn.size].view(-1, 4)
    assert (view.data_ptr() % 16 == 0) == (off == 0)
    return cont.UnstructuredGrid(torch.from_numpy(pts).cuda(), view)


@pytest.mark.parametrize("near", [True, False], ids=["together", "apart"])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("C", SIZES)
def test_count_at_group_ends(gb300, oracle_best, C, off, near):
    conn, f, pts = _cells(C, C, near)
    f[::11] = np.nan
    count = oracle_best.mt_count(conn, f, 0.25)
    ref = oracle_best.mt_generate(pts, conn, f, 0.25, count, False)
    out = gb300.marching_tetrahedra(_grid(gb300, conn, pts, off), torch.from_numpy(f).cuda(), 0.25, merge=False, records=True)
    assert out["conn"].shape[0] == int(count.sum())
    assert np.array_equal(out["rec_first"].cpu().numpy(), ref["rec_a"])
    assert np.array_equal(out["rec_second"].cpu().numpy(), ref["rec_b"])


@pytest.mark.parametrize("near", [True, False], ids=["together", "apart"])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("bad", ["P", -1, -2 ** 31, 2 ** 31 - 1])
@pytest.mark.parametrize("cell", [0, 4, 7, 31, 159, 160, 479, 480, 511, 512, 4096, 4098])
def test_bad_id_is_an_error(gb300, cell, bad, off, near):
    """Each corner in turn; the last cells lie in a group that the end cuts off."""
    from daxtoolkit_gb300 import capi
    conn, f, pts = _cells(4099, 7, near)
    for corner in range(4):
        c = conn.copy()
        c[cell, corner] = len(f) if bad == "P" else bad
        with pytest.raises(capi.ErrorControlBadValue):
            gb300.marching_tetrahedra(_grid(gb300, c, pts, off), torch.from_numpy(f).cuda(), 0.25, merge=False)


@pytest.mark.parametrize("order", ["cells", "points", "both"])
def test_mesh_in_no_order(gb300, order):
    """A large mesh gives the same triangles, up to their order, whatever the order of its cells and points."""
    n = 60
    grid = gb300.tetrahedralize(gb300.UniformGrid((n,) * 3))
    g = torch.Generator(device="cuda").manual_seed(5)
    f = torch.rand(n ** 3, generator=g, device="cuda")
    conn, pts, fx = grid.connectivity, grid.points, f
    if order != "points":
        conn = conn[torch.randperm(conn.shape[0], generator=g, device="cuda")].contiguous()
    if order != "cells":
        at = torch.randperm(n ** 3, generator=g, device="cuda")
        conn = at[conn.long()].to(torch.int32)
        pts, fx = torch.empty_like(pts), torch.empty_like(f)
        pts[at], fx[at] = grid.points, f
    a = gb300.marching_tetrahedra(grid, f, 0.5, merge=False)
    b = gb300.marching_tetrahedra(gb300.UnstructuredGrid(pts, conn), fx, 0.5, merge=False)
    assert a["conn"].shape == b["conn"].shape and a["conn"].shape[0] > 1_000_000
    if order == "cells":  # the same edges give the same bits
        a, b = (x["verts"].view(-1, 9).view(torch.int32).cpu().numpy() for x in (a, b))
        assert np.array_equal(a[np.lexsort(a.T)], b[np.lexsort(b.T)])
