"""StreamCompact of values of two to four words, whose kept rows leave a chunk of 128 elements at a time: chunks with no,
one, some and all elements kept, tiles with a ragged end, aligned and unaligned values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 8192


@pytest.mark.parametrize("words", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 127, 129, TILE - 1, TILE, TILE + 3, 7 * TILE + 130, 152 * 7 * TILE + 1])
@pytest.mark.parametrize("kept", [0.0, 0.01, 0.5, 1.0])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows(words, n, kept, shift):
    import torch
    from daxtoolkit_gb300 import cont
    rng = np.random.default_rng(n)
    s = (rng.random(n) < kept).astype(np.int32)
    s[n // 3:n // 2] = 1
    s[n // 2:n // 2 + n // 8] = 0
    v = rng.integers(0, 2 ** 31, size=n * words).astype(np.int32)
    buf = torch.zeros(n * words + shift, dtype=torch.int32, device="cuda")[shift:]
    buf.copy_(torch.from_numpy(v))
    rows = buf.view(n, words)
    got = cont.Algorithm.StreamCompact(rows, torch.from_numpy(s).cuda())
    assert np.array_equal(got.cpu().numpy(), v.reshape(n, words)[s != 0])
