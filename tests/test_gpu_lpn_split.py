"""The d = 10 primal LPN (five lanes per 4-row group; six groups per warp) at
its edges: row counts around a warp's six groups and a CTA's round, row
windows, both roles below and above the size from which their kk are
interleaved (also with more kk than groups, and under stream capture), and the
batched engine's tasks -- against the oracle."""
import numpy as np
import pytest

import oracle
from tests.util import rng_blocks, to_dev, to_host

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

EDGE = [1, 4, 5, 8, 9, 23, 24, 27, 28, 29, 193, 197, 24 * 148 * 24 + 5]


@pytest.mark.parametrize("n", EDGE)
def test_one_role(ctx, n):
    rng = np.random.default_rng(n)
    seed, kk, e = rng_blocks(rng, 1)[0], rng_blocks(rng, 77), rng_blocks(rng, n)
    d = to_dev(e)
    ctx.lpn_primal(seed, to_dev(kk), d)
    want = oracle.lpn_primal(seed, kk, e, threads=8)
    assert np.array_equal(to_host(d), want)
    lo, hi = n // 3 // 4 * 4, n - n % 4
    if hi > lo:
        d = to_dev(e[lo:hi])
        ctx.lpn_primal_range(seed, to_dev(kk), d, lo, hi, n)
        assert np.array_equal(to_host(d), want[lo:hi])


@pytest.mark.parametrize("n,k", [(5, 3), (29, 1), (197, 5000), ((1 << 18) + 3, 65536), ((1 << 18) + 4, 65536),
                                 ((1 << 18) + 8, 65538), ((1 << 18) + 9, 12345)])
@pytest.mark.parametrize("captured", [False, True])
def test_both_roles(n, k, captured):
    import cuot_b200
    ctx = cuot_b200.Context(0)
    rng = np.random.default_rng(n + k)
    seed, kk = rng_blocks(rng, 1)[0], (rng_blocks(rng, k), rng_blocks(rng, k))
    e = (rng_blocks(rng, n), rng_blocks(rng, n))
    dk, de = [to_dev(x) for x in kk], [to_dev(x) for x in e]
    torch.cuda.synchronize()
    if captured:  # a context that has no scratch yet
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ctx.lpn_primal_dual(seed, dk[0], dk[1], de[0], de[1])
        g.replay()
    else:
        ctx.lpn_primal_dual(seed, dk[0], dk[1], de[0], de[1])
    torch.cuda.synchronize()
    for r in range(2):
        assert np.array_equal(to_host(de[r]), oracle.lpn_primal(seed, kk[r], e[r], threads=8)), r
    ctx.close()


def test_both_roles_keep_a_smaller_arena():
    """The context's scratch is too small for the interleaved copy: it stays (a graph may hold it)."""
    import cuot_b200
    ctx = cuot_b200.Context(0)
    n, k, t, h = (1 << 18) + 8, 65536, 3, 9
    rng = np.random.default_rng(3)
    roots, out = to_dev(rng_blocks(rng, t)), [torch.empty((m, 16), dtype=torch.uint8, device="cuda")
                                              for m in (t << h, t * h, t * h, t)]
    ctx.ferret_pprf_sender(roots, h, bytes(16), *out)
    seed, kk, e = rng_blocks(rng, 1)[0], rng_blocks(rng, 2 * k).reshape(2, k, 16), rng_blocks(rng, 2 * n).reshape(2, n, 16)
    de = [to_dev(x) for x in e]
    ctx.lpn_primal_dual(seed, to_dev(kk[0]), to_dev(kk[1]), de[0], de[1])
    for r in range(2):
        assert np.array_equal(to_host(de[r]), oracle.lpn_primal(seed, kk[r], e[r], threads=8)), r
    ctx.close()


@pytest.mark.parametrize("rows", [0, 4, 1000])
def test_batched_tasks(ctx, rows):
    from cuot_b200.batch import KIND_FERRET, Batch, Instance
    insts = [Instance(ctx, KIND_FERRET, t, h, 40 + i, k=k, d=d)
             for i, (t, h, k, d) in enumerate([(3, 1, 5, 10), (1, 3, 9, 10), (5, 9, 700, 10), (7, 8, 33, 6), (2, 12, 4096, 10)])]
    s = torch.cuda.Stream()
    b = Batch(ctx, insts, lpn_rows_per_task=rows)
    b.run(s)
    b.run(s)
    torch.cuda.synchronize()
    for i in insts:
        lv, ls, rs, ss = oracle.ferret_pprf_sender(i.roots, i.h, i.delta, threads=8)
        mc = np.where(i.choice[:, None] == 0, ls, rs)
        rl = oracle.ferret_pprf_recver(mc, i.choice, ss, i.h, threads=8)
        assert np.array_equal(to_host(i.v), oracle.lpn_primal(i.seed, i.kk_s, lv, d=i.d, threads=8))
        assert np.array_equal(to_host(i.w), oracle.lpn_primal(i.seed, i.kk_r, rl, d=i.d, threads=8))
    b.close()
