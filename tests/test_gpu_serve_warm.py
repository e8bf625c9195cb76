"""What a server prepares for its slots: the encodes that requests run, and the
memory that those hold."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

import cuot_b200  # noqa: E402
from cuot_b200.serve import Server  # noqa: E402


def _launches():
    lib = cuot_b200.load()
    lib.cuot_launch_count.restype = ctypes.c_ulonglong
    return lib.cuot_launch_count()


def _created(max_log_n):
    before = _launches()
    srv = Server(slots=1, max_log_n=max_log_n)
    out = _launches() - before, srv.reserved_bytes()
    srv.close()
    return out


def test_slots_are_warmed_with_what_requests_run():
    small, large = _created(13), _created(16)
    ctx = cuot_b200.Context(0)
    before = _launches()
    for e in (14, 15, 16):
        n = 1 << e
        ctx.sot_dual_lpn(torch.zeros(n // 64, dtype=torch.int64, device="cuda"),
                         torch.zeros((n, 16), dtype=torch.uint8, device="cuda"), n)
    assert large[0] - small[0] == _launches() - before
    # the scratch arena grows by 24 bytes per block; ternary sizes have no tables
    assert large[1] - small[1] == 24 * ((1 << 16) - (1 << 13))
    torch.cuda.synchronize()
    ctx.close()
