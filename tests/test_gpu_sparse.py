"""The sparse encode at the edges of its tiles (32 or 128 output words per CTA, 16 warps over the positions, one or several
CTAs per tile) against the oracle: bytes, so equality."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

WORDS = [1, 2, 31, 33, 127, 512, 513, 640, 1000, 4096, 20001]


@pytest.mark.parametrize("weight", [1, 15, 17, 511, 513, 1025, 5000])
@pytest.mark.parametrize("words", WORDS)
def test_edges(ctx, words, weight):
    rng = np.random.default_rng(10007 * words + weight)
    n = 64 * words
    a_np = rng.integers(0, 1 << 64, words, dtype=np.uint64)
    pos = rng.integers(0, 2 * n + 3, weight, dtype=np.uint64)  # some beyond the range (ignored)
    pos[: weight // 3] %= np.uint64(n)
    a, pos_d = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a_np, pos))
    out = torch.full((words,), -1, dtype=torch.int64, device="cuda")
    ctx.qc_encode_sparse(a, pos_d, n, out)
    assert np.array_equal(out.cpu().numpy().view(np.uint64), oracle.qc_encode_sparse(a_np, pos, n))
    out.fill_(-1)
    ctx.qc_encode_sparse_r2(a, pos_d, n, out)
    exp = oracle.qc_encode_sparse(a_np, pos[(pos >= n) & (pos < 2 * n)] - np.uint64(n), n)
    for p in pos[pos < n]:
        exp[int(p) >> 6] ^= np.uint64(1 << (int(p) & 63))
    assert np.array_equal(out.cpu().numpy().view(np.uint64), exp)
