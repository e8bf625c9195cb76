"""A bounded number of planes per pass bounds the scratch of a ternary dual LPN:
its groups of 32 planes are then taken one or two at a time, with the results
of the FFT."""
import numpy as np
import pytest

from tests.util import rng_blocks, to_dev

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _ctx(backend=0, planes=0):
    import cuot_b200
    c = cuot_b200.Context(0)
    c.set_tuning(c.TUNE_QC_BACKEND, backend)
    c.set_tuning(c.TUNE_QC_PLANES, planes)
    return c


@pytest.mark.parametrize("e", [14, 15, 17, 20, 21])
@pytest.mark.parametrize("planes", [4, 16, 32, 64])
def test_scratch_is_no_more_than_the_ffts(e, planes):
    n = 1 << e
    rng = np.random.default_rng(e)
    a, x = to_dev(rng.integers(0, 1 << 63, n // 64, dtype=np.int64)), rng_blocks(rng, n)
    size, out = [], []
    for backend in (0, 2):
        for by_plan in (False, True):
            c = _ctx(backend, planes)
            d = to_dev(x)
            if by_plan:
                plan = c.qc_plan(a, n)
                plan.dual_lpn(d)
                torch.cuda.synchronize()
                plan.close()
            else:
                c.sot_dual_lpn(a, d, n)
            size.append(c.scratch_bytes())
            out.append(d)
            torch.cuda.synchronize()
            c.close()
    assert size[0] <= size[2] and size[1] <= size[3]
    assert all(torch.equal(o, out[0]) for o in out)


@pytest.mark.parametrize("e", range(14, 23))
@pytest.mark.parametrize("planes", [15, 16, 96])
def test_some_groups_at_a_time(e, planes):
    """One and two groups (and the FFT below 16 planes), on one stream and two, both rates, aliased outputs."""
    n = 1 << e
    rng = np.random.default_rng(80 + e)
    a, x = to_dev(rng.integers(0, 1 << 63, n // 64, dtype=np.int64)), rng_blocks(rng, 2 * n)
    fft = _ctx(2)
    want, want2 = to_dev(x[:n]), to_dev(x[:n])
    fft.sot_dual_lpn(a, want, n)
    fft.sot_dual_lpn_r2(a, to_dev(x), n, want2)
    for streams in (1, 2):
        c = _ctx(0, planes)
        c.set_tuning(c.TUNE_QC_STREAMS, streams)
        plan, d = c.qc_plan(a, n), to_dev(x[:n])
        plan.dual_lpn(d)
        assert torch.equal(d, want)
        d = to_dev(x[:n])
        c.sot_dual_lpn(a, d, n)
        assert torch.equal(d, want)
        for lo in (0, n):
            d = to_dev(x)
            plan.dual_lpn_r2(d, d[lo:lo + n])
            assert torch.equal(d[lo:lo + n], want2)
        plan.set_batch(128)
        d = to_dev(x[:n])
        plan.dual_lpn(d)
        assert torch.equal(d, want)
        torch.cuda.synchronize()
        plan.close()
        c.close()
    fft.close()


@pytest.mark.parametrize("planes", [8, 64, 300])
def test_batch_with_bounded_passes(ctx, planes):
    from cuot_b200.batch import KIND_SOT, Batch, Instance
    insts = [Instance(ctx, KIND_SOT, 1 << (e - 10), 10, 60 + i) for i, e in enumerate((14, 17, 17, 19))]
    s, got = torch.cuda.Stream(), []
    for p in (0, planes):
        b = Batch(ctx, insts, qc_planes_per_pass=p)
        b.run(s)
        torch.cuda.synchronize()
        got.append([(i.v.clone(), i.w.clone()) for i in insts])
        b.close()
    for (v, w), (v2, w2) in zip(*got):
        assert torch.equal(v, v2) and torch.equal(w, w2)
