"""The single-pass scan and compaction at the edges of a tile, of a block's ring of stages and of the grid, from
aligned arrays (bulk copies) and unaligned ones (element loads)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 8192
SIZES = [1, 31, TILE - 1, TILE, TILE + 1, 6 * TILE + 5, 152 * TILE, 152 * 3 * TILE + 1, 152 * 6 * TILE + TILE // 2]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dtype", ["int32", "int64"])
def test_scan(dtype, n, shift):
    import torch
    from daxtoolkit_gb300 import cont
    x = np.random.default_rng(n).integers(-5, 9, size=n + shift).astype(dtype)[shift:]
    buf = torch.empty(n + shift, dtype=getattr(torch, dtype), device="cuda")
    buf[shift:] = torch.from_numpy(x).cuda()
    total, out = cont.Algorithm.ScanInclusive(buf[shift:], torch.empty_like(buf)[shift:])
    want = np.cumsum(x, dtype=dtype)
    assert total == want[-1] and np.array_equal(out.cpu().numpy(), want)
    total, out = cont.Algorithm.ScanExclusive(buf[shift:], buf[shift:])
    assert total == want[-1] and np.array_equal(out.cpu().numpy(), want - x)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("words", [0, 1, 3])
def test_compact(n, words, shift):
    import torch
    from daxtoolkit_gb300 import cont
    rng = np.random.default_rng(n)
    s = rng.choice(np.array([0.0, -0.0, 1.0, -2.5, np.nan, 1e-42], np.float32), size=n + shift)
    if n % 2:
        s = (s > 0).astype(np.int32) << 31  # only the sign bit: not zero as an int
    stencil = torch.from_numpy(s).cuda()[shift:]
    if not words:
        got, want = cont.Algorithm.StreamCompact(stencil), np.nonzero(s[shift:])[0]
    else:
        v = rng.integers(0, 2 ** 31, size=(n + shift, words)).astype(np.int32)
        got, want = cont.Algorithm.StreamCompact(torch.from_numpy(v).cuda()[shift:], stencil), v[shift:][s[shift:] != 0]
    assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dtype", ["int32", "int64", "float32"])
def test_unique(dtype, n):
    import torch
    from daxtoolkit_gb300 import cont
    k = np.sort(np.random.default_rng(n).integers(0, max(1, n // 2), size=n)).astype(dtype)
    got = cont.Algorithm.Unique(torch.from_numpy(k).cuda())
    assert np.array_equal(got.cpu().numpy(), np.unique(k))
