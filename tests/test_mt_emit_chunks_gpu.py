"""The emit pass of marching tetrahedra over chunks with and without triangles
at the ends of a warp's round of chunks: single cells with triangles in otherwise
empty meshes, and meshes whose every cell has them, against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CHUNK, TILE = 512, 4096
# points 0..3 lie above the isovalue, 4..7 below
FIELD = np.array([1, 2, 3, 4, -1, -2, -3, -4], np.float32)
PTS = np.random.default_rng(3).random((8, 3)).astype(np.float32)


def _check(cont, oracle, conn, merge):
    count = oracle.mt_count(conn, FIELD, 0.0)
    ref = oracle.mt_generate(PTS, conn, FIELD, 0.0, count, merge)
    grid = cont.UnstructuredGrid(torch.from_numpy(PTS).cuda(), torch.from_numpy(conn).cuda())
    out = cont.marching_tetrahedra(grid, torch.from_numpy(FIELD).cuda(), 0.0, merge=merge,
                                   records=True)
    assert np.array_equal(out["conn"].cpu().numpy(), ref["conn"])
    assert np.array_equal(out["rec_first"].cpu().numpy(), ref["rec_a"])
    assert np.array_equal(out["rec_second"].cpu().numpy(), ref["rec_b"])
    assert np.array_equal(out["verts"].cpu().numpy().view(np.uint32), ref["verts"].view(np.uint32))


@pytest.mark.parametrize("merge", [True, False], ids=["merged", "unmerged"])
@pytest.mark.parametrize("C,cells", [
    (1, [0]),
    (CHUNK + 1, [CHUNK - 1, CHUNK]),
    (TILE, [0, 7 * CHUNK, TILE - 1]),
    (3 * TILE + 5, [CHUNK, TILE - 1, TILE, 2 * TILE + 5 * CHUNK, 3 * TILE + 4]),
    # several chunks for each resident warp
    (160 * 1024 * CHUNK // 4, [0, 5000 * CHUNK + 17, 9000 * CHUNK + 511, 40959 * CHUNK + 511]),
])
def test_few_cells(gb300, oracle_best, C, cells, merge):
    conn = np.tile(np.array([4, 5, 6, 7], np.int32), (C, 1))
    for k, c in enumerate(cells):
        conn[c] = [k % 4, 4 + k % 4, 4 + (k + 1) % 4, (k + 1) % 4 if k % 2 else 4 + (k + 2) % 4]
    _check(gb300, oracle_best, conn, merge)


@pytest.mark.parametrize("merge", [True, False], ids=["merged", "unmerged"])
@pytest.mark.parametrize("C", [CHUNK - 1, CHUNK, TILE + 1, 33 * CHUNK + 1])
def test_every_cell(gb300, oracle_best, C, merge):
    """Two triangles in every cell: the most entries and triangles of a chunk."""
    rng = np.random.default_rng(C)
    conn = np.stack([rng.permutation(4)[:2] for _ in range(C)], 0).astype(np.int32)
    low = np.stack([4 + rng.permutation(4)[:2] for _ in range(C)], 0).astype(np.int32)
    _check(gb300, oracle_best, np.ascontiguousarray(np.concatenate([conn, low], 1)), merge)
