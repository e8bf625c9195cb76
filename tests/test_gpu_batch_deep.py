"""Deep trees in a batch keep one scratch slot per CTA."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from cuot_b200.batch import KIND_FERRET, Batch, Instance  # noqa: E402


def test_scratch_of_deep_trees(ctx):
    h, trees = 16, 500
    insts = [Instance(ctx, KIND_FERRET, t, h, 5 + i, k=1000) for i, t in enumerate((250, 249, 1))]
    assert sum(i.t for i in insts) == trees
    ctas = 3 * torch.cuda.get_device_properties(0).multi_processor_count
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    b = Batch(ctx, insts)
    torch.cuda.synchronize()
    held = free - torch.cuda.mem_get_info()[0]
    assert held <= (min(ctas, trees) << h) * 16 + (64 << 20)
    s = torch.cuda.Stream()
    b.run(s)
    torch.cuda.synchronize()
    got = [(i.v.clone(), i.w.clone()) for i in insts]
    b.run_plain(s)
    torch.cuda.synchronize()
    for i, (v, w) in zip(insts, got):
        assert torch.equal(i.v, v) and torch.equal(i.w, w)
    b.close()
