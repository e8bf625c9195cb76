"""The autotuner's choices, with timings that need no device."""
import types

import pytest

from cuot_b200 import autotune, batch

torch = pytest.importorskip("torch")


def inst(kind=0, n=1 << 20, h=10):
    return types.SimpleNamespace(kind=kind, n=n, h=h, t=n >> h)


class FakeBatch:
    """Times what its configuration says (`fast`: the quickest one)."""

    def __init__(self, ctx, instances, **cfg):
        cfg.pop("use_graph")
        self.cfg = cfg

    def run(self, stream=None):
        return self.cfg

    def close(self):
        pass


@pytest.fixture
def fakes(monkeypatch):
    monkeypatch.setattr(batch, "Batch", FakeBatch)
    monkeypatch.setattr(torch.cuda, "Stream", lambda: None)

    def time_by(ms):
        monkeypatch.setattr(autotune, "_time", lambda fn, stream, reps: ms(fn(stream)))
    return time_by


def test_batch_may_keep_the_library_defaults(fakes, tmp_path):
    default = dict(pprf_threads=256, ctas_per_sm=3, lpn_rows_per_task=0)
    fakes(lambda cfg: 1.0 if cfg == default else 2.0)
    best, _ = autotune.tune_batch(None, [inst()], table=autotune.TuningTable(str(tmp_path / "t.json")))
    assert best == default
