"""The PPRF's thread groups (256, 128 or 64 threads per tree, by tree count and
depth; 128-thread CTAs by tuning) in all four modes against the oracle, at
depths around the sizes that stay in shared memory and tree counts around the
rule's lines and a wave's end; and a batch whose trees mix depths and kinds."""
import numpy as np
import pytest

import oracle
from tests.util import delta_ferret, rng_blocks, to_dev, to_host

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# 444 resident CTAs of 256 threads: one tree each up to 444 trees, two up to
# 1,332 (or above depth 12), four beyond
SHAPES = [(1, 1), (3, 2), (2, 5), (5, 6), (2, 7), (3, 8), (2, 9), (444, 3), (445, 7), (889, 8), (1332, 2), (1333, 1),
          (1333, 6), (1777, 7), (1340, 9), (2, 13)]


def empty(m):
    return torch.empty((m, 16), dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("threads", [128, 256])
@pytest.mark.parametrize("t,h", SHAPES)
def test_all_modes(t, h, threads):
    import cuot_b200
    ctx = cuot_b200.Context(0)
    ctx.set_tuning(ctx.TUNE_PPRF_THREADS, threads)
    rng = np.random.default_rng(100 * t + h)
    roots, delta, choice = rng_blocks(rng, t), delta_ferret(rng), rng.integers(0, 2, t * h).astype(np.uint8)
    lv, ls, rs, ss, rl = empty(t << h), empty(t * h), empty(t * h), empty(t), empty(t << h)
    ctx.ferret_pprf_sender(to_dev(roots), h, delta, lv, ls, rs, ss)
    want = oracle.ferret_pprf_sender(roots, h, delta, threads=8)
    for got, w in zip((lv, ls, rs, ss), want):
        assert np.array_equal(to_host(got), w)
    mc = np.where(choice[:, None] == 0, want[1], want[2])
    ctx.ferret_pprf_recver(to_dev(mc), to_dev(choice), ss, h, rl)
    assert np.array_equal(to_host(rl), oracle.ferret_pprf_recver(mc, choice, want[3], h, threads=8))
    b0, b1 = rng_blocks(rng, t * h), rng_blocks(rng, t * h)
    m0, m1 = empty((h + 1) * t), empty((h + 1) * t)
    ctx.sot_pprf_sender(to_dev(roots), h, delta, to_dev(b0), to_dev(b1), lv, m0, m1)
    want = oracle.sot_pprf_sender(roots, h, delta, b0, b1, threads=8)
    for got, w in zip((lv, m0, m1), want):
        assert np.array_equal(to_host(got).reshape(w.shape), w)
    mc = np.where(choice[:, None] == 0, b0, b1)
    ctx.sot_pprf_recver(m0, m1, to_dev(mc), to_dev(choice), t, h, rl)
    assert np.array_equal(to_host(rl), oracle.sot_pprf_recver(want[1], want[2], mc, choice, t, h, threads=8))
    torch.cuda.synchronize()
    ctx.close()


@pytest.mark.parametrize("threads,count", [(0, 3), (0, 60), (0, 200), (128, 60)])
def test_batch_of_mixed_depths(ctx, threads, count):
    """Few trees (one per CTA), more (two) and many shallow ones (four)."""
    from cuot_b200.batch import KIND_FERRET, KIND_SOT, Batch, Instance
    insts = [Instance(ctx, KIND_FERRET, 1 + 13 * i % 23, 1 + i % 7, 70 + i, k=50) if i % 2 else
             Instance(ctx, KIND_SOT, 16 << i % 2, 6 + i % 2, 70 + i) for i in range(count)]
    s = torch.cuda.Stream()
    b = Batch(ctx, insts, pprf_threads=threads)
    b.run(s)
    b.run(s)
    torch.cuda.synchronize()
    got = [(to_host(i.v).copy(), to_host(i.w).copy()) for i in insts]
    b.run_plain(s)
    torch.cuda.synchronize()
    for i, (v, w) in zip(insts, got):
        assert np.array_equal(to_host(i.v), v) and np.array_equal(to_host(i.w), w)
    b.close()
