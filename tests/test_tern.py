"""The ternary-transform dual LPN (qc_tern.cu): its per-thread steps run on the
host against the oracle's product, and (GPU) the kernels against the FFT and
the oracle: every size, plan and one-shot, both rates, aliased outputs, the
heaviest and lightest inputs, and several jobs per launch."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle
from tests.util import rng_blocks, to_dev, to_host

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SIZES = range(14, 23)


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    so = str(tmp_path_factory.mktemp("tern") / "libtern_host.so")
    subprocess.check_call([nvcc, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                           os.path.join(ROOT, "tests", "cpp", "tern_host.cu"), "-o", so])
    return ctypes.CDLL(so)


def plane(words, k):
    return np.packbits(((words >> np.uint32(k)) & np.uint32(1)).astype(np.uint8), bitorder="little").view(np.uint64)


@pytest.mark.parametrize("e", SIZES)
def test_steps_on_host_match_oracle(host, e):
    n = 1 << e
    rng = np.random.default_rng(e)
    a = rng.integers(0, 1 << 64, n // 64, dtype=np.uint64)
    x = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    x &= ~np.uint32(6)          # planes 1, 2: empty and all ones
    x |= np.uint32(4)
    out = np.empty(n, np.uint32)
    ptr = lambda v: v.ctypes.data_as(ctypes.c_void_p)
    assert host.tern_host_dual(e, ptr(a), ptr(x), ptr(out)) == 0
    for k in (0, 1, 2, 31):
        assert np.array_equal(plane(out, k), oracle.gf2_cyclic_mul(a, plane(x, k), n)), k


def _ctx(backend=0):
    import cuot_b200
    c = cuot_b200.Context(0)
    c.set_tuning(c.TUNE_QC_BACKEND, backend)
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("e", SIZES)
def test_dual_lpn_equals_fft(e):
    torch = pytest.importorskip("torch")
    n = 1 << e
    rng = np.random.default_rng(50 + e)
    x = rng_blocks(rng, 2 * n)
    x[:, 3] = 0                 # empty planes
    x[:, 4] = 0xFF              # full planes
    polys = [rng.integers(0, 1 << 63, n // 64, dtype=np.int64), np.full(n // 64, -1, np.int64), np.zeros(n // 64, np.int64)]
    polys[2][-1] = -(1 << 63)   # x^(n-1) alone
    auto, fft = _ctx(), _ctx(2)
    for a_np in polys:
        a = to_dev(a_np)
        want = to_dev(x[:n])
        fft.sot_dual_lpn(a, want, n)
        plan, d = auto.qc_plan(a, n), to_dev(x[:n])
        plan.dual_lpn(d)
        assert torch.equal(d, want)
        d = to_dev(x[:n])
        auto.sot_dual_lpn(a, d, n)
        assert torch.equal(d, want)
        # rate 1/2, also into the first and into the second half of the input
        want = to_dev(x[:n])
        fft.sot_dual_lpn_r2(a, to_dev(x), n, want)
        out = torch.empty_like(want)
        plan.dual_lpn_r2(to_dev(x), out)
        assert torch.equal(out, want)
        for lo in (0, n):
            d = to_dev(x)
            auto.sot_dual_lpn_r2(a, d, n, d[lo:lo + n])
            assert torch.equal(d[lo:lo + n], want)
        # the same plan encodes planes with its FFT
        pl = rng.integers(0, 1 << 63, (5, n // 64), dtype=np.int64)
        p0, p1 = to_dev(pl), to_dev(pl)
        plan.encode(p0, 5)
        fft.qc_encode(a, p1, n, 5)
        assert torch.equal(p0, p1)
        del plan
    torch.cuda.synchronize()
    auto.close()
    fft.close()


@pytest.mark.gpu
@pytest.mark.parametrize("e,count", [(14, 3), (15, 9), (16, 9), (17, 4), (18, 3), (20, 2)])
def test_batched_jobs_equal_plain(e, count):
    """Several instances of one size share launches (e = 15, 16: 18 jobs, more than
    one launch holds); each equals its own plan's dual LPN, and a margin-
    recording context, which keeps to the FFT, agrees."""
    torch = pytest.importorskip("torch")
    from cuot_b200.batch import KIND_SOT, Batch, Instance
    outs = []
    for record in (0, 1):
        ctx = _ctx()
        ctx.set_tuning(ctx.TUNE_QC_RECORD_MARGIN, record)
        insts = [Instance(ctx, KIND_SOT, 1 << (e - 10), 10, 900 + i) for i in range(count)]
        s = torch.cuda.Stream()
        b = Batch(ctx, insts)
        # a batch keeps the transform it was made with
        ctx.set_tuning(ctx.TUNE_QC_RECORD_MARGIN, 1 - record)
        b.run(s)
        b.run(s)
        torch.cuda.synchronize()
        got = [(i.v.clone(), i.w.clone()) for i in insts]
        b.run_plain(s)
        torch.cuda.synchronize()
        for i, (v, w) in zip(insts, got):
            assert torch.equal(i.v, v) and torch.equal(i.w, w)
        outs.append(got)
        b.close()
        ctx.close()
    for (v, w), (v2, w2) in zip(*outs):
        assert torch.equal(v, v2) and torch.equal(w, w2)


@pytest.mark.gpu
def test_chained_launches_keep_the_order():
    """Small calls back to back on one stream (their kernels are chained), on two
    streams joined by events, and captured into a graph: every call sees the
    results of the one before."""
    import cuot_b200
    torch = pytest.importorskip("torch")
    t, h = 16, 10
    n = t << h
    rng = np.random.default_rng(99)
    ctxs = [cuot_b200.Context(0), cuot_b200.Context(0)]
    a = to_dev(rng.integers(0, 1 << 63, n // 64, dtype=np.int64))
    roots = [to_dev(rng_blocks(rng, t)) for _ in range(4)]
    kk, seed, delta = to_dev(rng_blocks(rng, 300)), bytes(range(16)), bytes(range(1, 17))
    e = lambda m: torch.empty((m, 16), dtype=torch.uint8, device="cuda")
    plans = [c.qc_plan(a, n) for c in ctxs]

    def chain(i, ctx, plan, v, s, sync):
        ls, rs, ss, out = e(t * h), e(t * h), e(t), e(t)
        for f in (lambda: ctx.ferret_pprf_sender(roots[i], h, delta, v, ls, rs, ss, stream=s),
                  lambda: ctx.lpn_primal(seed, kk, v, stream=s), lambda: plan.dual_lpn(v, stream=s),
                  lambda: plan.dual_lpn(v, stream=s), lambda: ctx.lpn_primal(seed, kk, v, stream=s),
                  lambda: ctx.ferret_chi_sum(v, h, ss, out, stream=s)):
            f()
            if sync:
                torch.cuda.synchronize()
        return out

    v = [e(n) for _ in range(2)]
    main = torch.cuda.current_stream()
    want = []
    for i in range(4):
        o = chain(i, ctxs[0], plans[0], v[0], main, True)
        want.append((v[0].clone(), o.clone()))
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for rep in range(3):
        got = []
        for i in range(4):  # alternate streams, each step after the one before
            s = side if i % 2 else main
            s.wait_stream(main if i % 2 else side)
            with torch.cuda.stream(s):
                o = chain(i, ctxs[i % 2], plans[i % 2], v[0], s, False)
                got.append((v[0].clone(), o))
        main.wait_stream(side)
        torch.cuda.synchronize()
        for (x, y), (x2, y2) in zip(want, got):
            assert torch.equal(x, x2) and torch.equal(y, y2), rep
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        o = chain(1, ctxs[0], plans[0], v[1], torch.cuda.current_stream(), False)
    for _ in range(3):
        v[1].zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(v[1], want[1][0]) and torch.equal(o, want[1][1])
    del plans
    torch.cuda.synchronize()
    for c in ctxs:
        c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("e", [16, 19, 21])
@pytest.mark.parametrize("streams", [1, 2])
def test_captured_and_streamed(e, streams):
    """Plans on one and two streams, one-shot and captured (also as a context's
    first call of the size), with work on the caller's stream before and after."""
    import cuot_b200
    torch = pytest.importorskip("torch")
    n = 1 << e
    rng = np.random.default_rng(70 + e)
    x = rng_blocks(rng, n)
    a = to_dev(rng.integers(0, 1 << 63, n // 64, dtype=np.int64))
    fft = _ctx(2)
    want = to_dev(x)
    fft.sot_dual_lpn(a, want, n)
    want ^= 0x5A
    ctx = _ctx()
    ctx.set_tuning(ctx.TUNE_QC_STREAMS, streams)
    ctx.reserve(1 << 30)
    src, d = to_dev(x), torch.empty((n, 16), dtype=torch.uint8, device="cuda")
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        d.copy_(src)
        ctx.sot_dual_lpn(a, d, n)
        d.bitwise_xor_(0x5A)
    plan = ctx.qc_plan(a, n)
    g2 = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g2):
        d.copy_(src)
        plan.dual_lpn(d)
        d.bitwise_xor_(0x5A)
    for run in (g.replay, g2.replay, g.replay):
        d.zero_()
        run()
        torch.cuda.synchronize()
        assert torch.equal(d, want)
    for _ in range(3):
        d.copy_(src)
        plan.dual_lpn(d)
        d.bitwise_xor_(0x5A)
    torch.cuda.synchronize()
    assert torch.equal(d, want)
    del plan
    torch.cuda.synchronize()
    ctx.close()
    fft.close()
