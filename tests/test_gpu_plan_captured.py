"""Small plans under capture: dual LPNs of 2^14 and 2^15 take the FFT there, if the
arena has its room, with the results of the ternary transform; larger ones do not."""
import ctypes

import numpy as np
import pytest

from tests.util import rng_blocks, to_dev

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

import cuot_b200  # noqa: E402


def _launches():
    lib = cuot_b200.load()
    lib.cuot_launch_count.restype = ctypes.c_ulonglong
    return lib.cuot_launch_count()


@pytest.mark.parametrize("e", [14, 15, 16])
@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("planes", [0, 16, 64])
def test_captured_dual_lpn(e, warm, planes):
    n = 1 << e
    rng = np.random.default_rng(40 + e)
    x = rng_blocks(rng, 2 * n)
    a = to_dev(rng.integers(0, 1 << 63, n // 64, dtype=np.int64))
    ref = cuot_b200.Context(0)
    want, want2 = to_dev(x[:n]), torch.empty((n, 16), dtype=torch.uint8, device="cuda")
    ref.sot_dual_lpn(a, want, n)
    ref.sot_dual_lpn_r2(a, to_dev(x), n, want2)
    ctx = cuot_b200.Context(0)
    ctx.set_tuning(ctx.TUNE_QC_PLANES, planes)
    if not warm:
        ctx.reserve(300 * n)  # the ternary transform's room, less than the FFT's for all planes
    plan = ctx.qc_plan(a, n)
    src, src2, d, d2 = to_dev(x[:n]), to_dev(x), torch.empty_like(want), torch.empty_like(want)
    count = _launches()
    if warm:
        d.copy_(src)
        plan.dual_lpn(d)
        plan.dual_lpn_r2(src2, d2)
        assert torch.equal(d, want) and torch.equal(d2, want2)
    eager = _launches() - count
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    count = _launches()
    with torch.cuda.graph(g):
        d.copy_(src)
        plan.dual_lpn(d)
        plan.dual_lpn_r2(src2, d2)
    captured = _launches() - count
    if warm and not planes:
        assert (captured < eager) == (e < 16)
    for _ in range(2):
        d.zero_()
        d2.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(d, want) and torch.equal(d2, want2)
    d.copy_(src)
    plan.dual_lpn(d)
    assert torch.equal(d, want)
    torch.cuda.synchronize()
    del g
    plan.close()
    ctx.close()
    ref.close()


@pytest.mark.parametrize("e", [14, 16, 17])
@pytest.mark.parametrize("room", ["warm", "reserved", "small"])
def test_captured_one_shot(e, room):
    """Also as a context's first call of the size: the FFT's tables are made beside the capture."""
    n = 1 << e
    rng = np.random.default_rng(90 + e)
    x = rng_blocks(rng, 2 * n)
    a = to_dev(rng.integers(0, 1 << 63, n // 64, dtype=np.int64))
    ref = cuot_b200.Context(0)
    ref.set_tuning(ref.TUNE_QC_BACKEND, 2)
    want, want2 = to_dev(x[:n]), torch.empty((n, 16), dtype=torch.uint8, device="cuda")
    ref.sot_dual_lpn(a, want, n)
    ref.sot_dual_lpn_r2(a, to_dev(x), n, want2)
    count = _launches()
    ref.sot_dual_lpn(a, to_dev(x[:n]), n)
    ref.sot_dual_lpn_r2(a, to_dev(x), n, torch.empty_like(want))
    fft = _launches() - count
    ctx = cuot_b200.Context(0)
    src, src2, d, d2 = to_dev(x[:n]), to_dev(x), torch.empty_like(want), torch.empty_like(want)
    if room == "warm":
        d.copy_(src)
        ctx.sot_dual_lpn(a, d, n)
        ctx.sot_dual_lpn_r2(a, src2, n, d2)
        assert torch.equal(d, want) and torch.equal(d2, want2)
    else:
        ctx.reserve(600 * n if room == "reserved" else 300 * n)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    count = _launches()
    with torch.cuda.graph(g):
        d.copy_(src)
        ctx.sot_dual_lpn(a, d, n)
        ctx.sot_dual_lpn_r2(a, src2, n, d2)
    assert (_launches() - count == fft) == (e < 17 and room != "small")
    for _ in range(2):
        d.zero_()
        d2.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(d, want) and torch.equal(d2, want2)
    d.copy_(src)
    ctx.sot_dual_lpn(a, d, n)
    assert torch.equal(d, want)
    torch.cuda.synchronize()
    del g
    ctx.close()
    ref.close()
