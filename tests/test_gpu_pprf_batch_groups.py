"""A batch with enough shallow trees for four groups per CTA (64 threads per
tree), Ferret and SOT trees of mixed depths in one queue, against the oracle."""
import numpy as np
import pytest

import oracle
from tests.util import to_host

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from cuot_b200.batch import KIND_FERRET, KIND_SOT, Batch, Instance  # noqa: E402


def test_four_groups_per_cta(ctx):
    insts = [Instance(ctx, KIND_FERRET, 1 + 13 * i % 23, 1 + i % 7, 70 + i, k=50) if i % 2 else
             Instance(ctx, KIND_SOT, 16 << i % 2, 6 + i % 2, 70 + i) for i in range(340)]
    ctas = 3 * torch.cuda.get_device_properties(0).multi_processor_count
    assert sum(i.n for i in insts) >> max(i.h for i in insts) > 3 * ctas  # 64 threads (pprf_group_size)
    s = torch.cuda.Stream()
    b = Batch(ctx, insts)
    b.run(s)
    b.run(s)
    torch.cuda.synchronize()
    for i in insts:
        if i.kind == KIND_FERRET:
            lv, ls, rs, ss = oracle.ferret_pprf_sender(i.roots, i.h, i.delta, threads=8)
            mc = np.where(i.choice[:, None] == 0, ls, rs)
            rl = oracle.ferret_pprf_recver(mc, i.choice, ss, i.h, threads=8)
            want = [oracle.lpn_primal(i.seed, kk, x, d=i.d, threads=8) for kk, x in ((i.kk_s, lv), (i.kk_r, rl))]
        else:
            lv, m0, m1 = oracle.sot_pprf_sender(i.roots, i.h, i.delta, i.base0, i.base1, threads=8)
            rl = oracle.sot_pprf_recver(m0, m1, i.mc, i.choice, i.t, i.h, threads=8)
            a = to_host(i.a).view(np.uint64)
            want = [oracle.sot_dual_lpn(a, x, i.n, threads=8) for x in (lv, rl)]
        assert np.array_equal(to_host(i.v), want[0]) and np.array_equal(to_host(i.w), want[1]), (i.kind, i.t, i.h)
    b.close()
