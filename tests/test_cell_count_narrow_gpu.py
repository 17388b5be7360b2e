"""The per-cell counts of narrow grids, a cell a thread, and on both sides of the line to the kernel that takes rows: the
counts and cases of the oracle, and the clip count of a restatement in numpy float32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(2, 2, 3000), (2, 700, 5), (700, 2, 5), (3, 9, 400), (17, 3, 90), (22, 9, 30), (23, 9, 30), (24, 9, 30),
        (34, 34, 12), (32, 6, 20), (64, 64, 5), (65, 65, 5), (8192, 2, 3)]


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
def test_counts(dims):
    import oracle
    import torch
    from daxtoolkit_gb300 import cont
    nx, ny, nz = dims
    f = np.random.default_rng(nx).uniform(0, 1, size=nx * ny * nz).astype(np.float32)
    f[::7] = np.nan
    origin, spacing = (-0.5, 0.25, 1.0), (0.125, 0.5, 0.0625)
    grid, fd = cont.UniformGrid(dims, origin=origin, spacing=spacing), torch.from_numpy(f).cuda()
    O, og = oracle.Oracle("port"), oracle.make_grid(dims)
    want = [np.asarray(x).ravel() for x in O.mc_count(og, f, 0.5)]
    count, cases = cont.DispatcherMapCell(cont.MarchingCubesCount(0.5)).classify_cases(grid, fd)
    assert np.array_equal(count.cpu().numpy(), want[0]) and np.array_equal(cases.cpu().numpy(), want[1])
    count = cont.DispatcherMapCell(cont.ThresholdCount(0.05, 0.95)).Invoke(grid, fd)
    assert np.array_equal(count.cpu().numpy(), np.asarray(O.threshold_count(og, f, 0.05, 0.95)).ravel())
    # every product and sum below is a multiple of 2^-8 and less than 2^13: exact in float32
    normal, at = (0.25, -0.5, 1.0), (nx * 0.0625, ny * 0.25, 1.0 + nz * 0.03125)
    x, y, z = (np.float32(o) + np.float32(s) * np.arange(n, dtype=np.float32) for o, s, n in zip(origin, spacing, dims))
    t = ((normal[0] * (x - np.float32(origin[0])))[None, None, :] + (normal[1] * (y - np.float32(origin[1])))[None, :, None]
         + (normal[2] * (z - np.float32(origin[2])))[:, None, None])
    loc = sum(n * a for n, a in zip(normal, at))
    beyond = t > np.float32(loc)
    any_ = beyond[1:] | beyond[:-1]
    any_ = any_[:, 1:] | any_[:, :-1]
    any_ = any_[:, :, 1:] | any_[:, :, :-1]
    count = cont.DispatcherMapCell(cont.MandlebulbClipCount(origin, at, normal, 0.5)).Invoke(grid, fd)
    assert np.array_equal(count.cpu().numpy(), np.where(any_.ravel(), want[0], 0))
