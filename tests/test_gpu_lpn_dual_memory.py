"""Where both roles' LPN puts its interleaved kk: in memory of its own, whatever
arena the context has, beside captures on other streams and calls on other
streams; and the forms without it (captured, large k)."""
import numpy as np
import pytest

import oracle
from tests.util import rng_blocks, to_dev, to_host

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _case(n, k, seed=0):
    rng = np.random.default_rng(n + k + seed)
    s, kk, e = rng_blocks(rng, 1)[0], rng_blocks(rng, 2 * k).reshape(2, k, 16), rng_blocks(rng, 2 * n).reshape(2, n, 16)
    want = [oracle.lpn_primal(s, kk[r], e[r], threads=8) for r in range(2)]
    return s, [to_dev(x) for x in kk], [to_dev(x) for x in e], want


def _launches():
    import ctypes

    import cuot_b200
    lib = cuot_b200.load()
    lib.cuot_launch_count.restype = ctypes.c_ulonglong
    return lib.cuot_launch_count()


@pytest.mark.parametrize("reserved", [0, 4096, 1 << 24])
def test_the_arena_plays_no_part(reserved):
    import cuot_b200
    ctx = cuot_b200.Context(0)
    if reserved:
        ctx.reserve(reserved)
    s, kk, e, want = _case((1 << 18) + 8, 65536)
    torch.cuda.synchronize()
    before = _launches()
    ctx.lpn_primal_dual(s, kk[0], kk[1], e[0], e[1])
    assert _launches() - before == 2  # the copy and the LPN
    assert ctx.scratch_bytes() == reserved
    for r in range(2):
        assert np.array_equal(to_host(e[r]), want[r]), r
    ctx.close()


def test_beside_a_capture_and_on_two_streams():
    import cuot_b200
    ctx = cuot_b200.Context(0)
    cases = [_case(1 << 18, 60000, i) for i in range(2)]
    streams = [torch.cuda.Stream() for _ in range(3)]
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=streams[2]):
        x += 1
        for (s, kk, e, _), st in zip(cases, streams):
            ctx.lpn_primal_dual(s, kk[0], kk[1], e[0], e[1], stream=st)
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert x.cpu().tolist() == [2.0] * 8
    for _, _, e, want in cases:
        for r in range(2):
            assert np.array_equal(to_host(e[r]), want[r]), r
    ctx.close()


@pytest.mark.parametrize("n,k,launches", [((1 << 18) - 4, 65536, 1), (1 << 18, 65536, 2), (1 << 18, 131072, 2),
                                          (1 << 18, 131073, 1)])
def test_where_the_copy_is_made(n, k, launches):
    """n: rows in groups of four (the last four are not)."""
    import cuot_b200
    ctx = cuot_b200.Context(0)
    n += 4
    s, kk, e, want = _case(n, k)
    torch.cuda.synchronize()
    before = _launches()
    ctx.lpn_primal_dual(s, kk[0], kk[1], e[0], e[1])
    assert _launches() - before == launches
    for r in range(2):
        assert np.array_equal(to_host(e[r]), want[r]), r
    ctx.close()


@pytest.mark.parametrize("n,k", [((1 << 18) + 5, 2000000), ((1 << 18) + 5, 2000001), (29, 2000001)])
def test_large_k_in_turn(n, k):
    import cuot_b200
    ctx = cuot_b200.Context(0)
    s, kk, e, want = _case(n, k)
    ctx.lpn_primal_dual(s, kk[0], kk[1], e[0], e[1])
    for r in range(2):
        assert np.array_equal(to_host(e[r]), want[r]), r
    torch.cuda.synchronize()
    ctx.close()
