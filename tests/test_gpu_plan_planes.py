"""A plan whose dual LPN is ternary holds the FFT's transform of `a` only once
planes are encoded with it: memory, and first plane encodes after the caller's
`a` is gone, under capture, and in any order with dual LPNs."""
import numpy as np
import pytest

import oracle
from tests.util import rng_blocks, to_dev, to_host

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _ctx(backend=0):
    import cuot_b200
    c = cuot_b200.Context(0)
    c.set_tuning(c.TUNE_QC_BACKEND, backend)
    return c


@pytest.mark.parametrize("e", [20, 22])
def test_memory_of_plans(e):
    n, held = 1 << e, []
    a = to_dev(np.random.default_rng(e).integers(0, 1 << 63, n // 64, dtype=np.int64))
    for backend in (0, 2):
        c = _ctx(backend)
        plans = [c.qc_plan(a, n)]  # the context's tables and scratch
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        plans += [c.qc_plan(a, n) for _ in range(4)]
        torch.cuda.synchronize()
        held.append(free - torch.cuda.mem_get_info()[0])
        for p in plans:
            p.close()
        c.close()
    assert held[0] <= held[1] * 1.15 + 4 * (2 << 20)  # 17.1n bytes against 16n, in 2 MiB pages


@pytest.mark.parametrize("e,nplanes", [(14, 1), (17, 5), (20, 3), (22, 4)])
def test_first_plane_encode(e, nplanes):
    n = 1 << e
    rng = np.random.default_rng(300 + e)
    a_np, planes = (rng.integers(0, 1 << 64, s, dtype=np.uint64) for s in (n // 64, (nplanes, n // 64)))
    x = rng_blocks(rng, n)
    want = oracle.qc_encode(a_np, planes, n, threads=16)
    want2 = oracle.qc_encode(a_np, want, n, threads=16)
    c = _ctx()
    a, src = to_dev(a_np.view(np.int64)), to_dev(planes.view(np.int64))
    eager, captured = c.qc_plan(a, n), c.qc_plan(a, n)
    dual = to_dev(x)
    c.sot_dual_lpn(a, dual, n)
    a.fill_(-1)  # the plans keep their own
    c.reserve(1 << 28)
    d = torch.empty_like(src)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        d.copy_(src)
        captured.encode(d, nplanes)
        captured.encode(d, nplanes)
    check = lambda t, w: np.array_equal(to_host(t).view(np.uint64), w)
    for step in range(3):  # replayed before and after the plan's first call outside the graph
        d.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert check(d, want2), step
        for plan in (captured, eager):
            for w in (want, want2):
                t = src.clone() if w is want else t
                plan.encode(t, nplanes)
                assert check(t, w)
            b = to_dev(x)
            plan.dual_lpn(b)
            assert torch.equal(b, dual)
    torch.cuda.synchronize()
    del g
    eager.close()
    captured.close()
    c.close()
