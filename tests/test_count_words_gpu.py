"""The word count at the edges of its walks: rows of one word, rows as long as they get, ranges that
end inside a row, planes of two rows, and tiles that hold a few grids of a set or many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2, 2), (2, 2, 300), (3, 2, 1500), (33, 2, 90), (129, 41, 3), (8192, 2, 3), (8191, 3, 2), (8161, 9, 3),
          (70, 40, 40)]


def _field(dims, seed):
    return np.random.default_rng(seed).uniform(0, 1, size=dims[0] * dims[1] * dims[2]).astype(np.float32)


def _check(out, dims, f, iso, merge=True):
    import oracle
    O = oracle.Oracle("port")
    og = oracle.make_grid(dims)
    ref = O.mc_generate(og, f, iso, O.mc_count(og, f, iso)[0], merge=merge)
    assert np.array_equal(out[1], ref["conn"])
    assert np.array_equal(out[0].view(np.uint32), ref["verts"].view(np.uint32))


@pytest.mark.parametrize("iso", [0.5, 0.995])
@pytest.mark.parametrize("dims", SHAPES)
def test_counts_of_one_grid(dims, iso):
    import torch
    from daxtoolkit_gb300 import cont
    f = _field(dims, dims[0])
    out = cont.marching_cubes(cont.UniformGrid(dims), torch.from_numpy(f).cuda(), iso, merge=True)
    _check((out["verts"].cpu().numpy(), out["conn"].cpu().numpy()), dims, f, iso)


@pytest.mark.parametrize("sets", [SHAPES, [(5, 4, 4)] * 700, [(2, 2, 2)] * 40 + [(60, 50, 9)] * 3 + [(8192, 2, 2)]])
def test_counts_of_a_set(sets):
    import torch
    from daxtoolkit_gb300 import cont
    fields = [_field(d, i) for i, d in enumerate(sets)]
    batch = cont.MarchingCubesBatch([cont.UniformGrid(d) for d in sets], [torch.from_numpy(f).cuda() for f in fields],
                                    [0.5] * len(sets))
    verts, conn, tri, vert = batch.run(merge=True)
    verts, conn = verts.cpu().numpy(), conn.cpu().numpy()
    for i in list(range(0, len(sets), 1 + len(sets) // 12)) + [len(sets) - 1]:
        _check((verts[vert[i]:vert[i + 1]], conn[tri[i]:tri[i + 1]]), sets[i], fields[i], 0.5)


@pytest.mark.parametrize("iso", [0.5, 0.995])
@pytest.mark.parametrize("dims", SHAPES)
def test_unmerged_vertices_of_one_grid(dims, iso):
    import torch
    from daxtoolkit_gb300 import cont
    f = _field(dims, dims[0] + 1)
    out = cont.marching_cubes(cont.UniformGrid(dims), torch.from_numpy(f).cuda(), iso, merge=False)
    _check((out["verts"].cpu().numpy(), out["conn"].cpu().numpy()), dims, f, iso, merge=False)


def test_unmerged_vertices_of_a_set():
    import torch
    from daxtoolkit_gb300 import cont
    sets = SHAPES + [(5, 4, 4)] * 40
    fields = [_field(d, i) for i, d in enumerate(sets)]
    batch = cont.MarchingCubesBatch([cont.UniformGrid(d) for d in sets], [torch.from_numpy(f).cuda() for f in fields],
                                    [0.5] * len(sets))
    verts, conn, tri, _ = batch.run(merge=False)
    verts, conn = verts.cpu().numpy(), conn.cpu().numpy()
    for i, d in enumerate(sets):
        _check((verts[3 * tri[i]:3 * tri[i + 1]], conn[tri[i]:tri[i + 1]]), d, fields[i], 0.5, merge=False)


@pytest.mark.parametrize("dims", [(300, 40, 30), (161, 61, 43), (8192, 3, 3)])
def test_ids_across_words_without_edges(dims):
    """Sparse surfaces: a plane across x puts the only edges of long stretches of rows next to a word's last cell, whose
    far corners take their ids from the offset of a word that has none.  The scratch is dirtied by another surface."""
    import torch
    from daxtoolkit_gb300 import cont
    nx, ny, nz = dims
    grid, scratch = cont.UniformGrid(dims), cont.Scratch()
    cont.marching_cubes(grid, torch.from_numpy(_field(dims, 7)).cuda(), 0.5, scratch=scratch)
    x = np.arange(nx, dtype=np.float32)
    for cut in (31, 32, 63, 127, 128, nx - 2):
        f = np.broadcast_to(x + 0.003 * np.arange(ny, dtype=np.float32)[:, None], (nz, ny, nx)).astype(np.float32)
        f[1:, ::3] += 0.75
        f = np.ascontiguousarray(f.ravel())
        out = cont.marching_cubes(grid, torch.from_numpy(f).cuda(), cut + 0.5, scratch=scratch)
        _check((out["verts"].cpu().numpy(), out["conn"].cpu().numpy()), dims, f, cut + 0.5)
