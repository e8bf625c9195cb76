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


def test_winners_of_earlier_launch_rules_are_measured_again(fakes, tmp_path):
    import hashlib
    import json
    fakes(lambda cfg: 1.0 if cfg["pprf_threads"] == 256 else 2.0)
    table, old = autotune.TuningTable(str(tmp_path / "t.json")), {"config": dict(pprf_threads=128), "ms": 3.0}
    i = inst()
    sig = json.dumps([[i.kind, i.n, i.h]])  # keys without a version
    table.put("batch:" + hashlib.sha256(sig.encode()).hexdigest()[:16], old)
    table.put(f"ferret:{i.n}:{i.h}", old)
    best, _ = autotune.tune_batch(None, [i], table=table)
    assert best["pprf_threads"] == 256 and table.get(autotune.batch_key([i]))["config"] == best
    assert table.get(autotune.shape_key(i.kind, i.n, i.h)) is None


class FakeContext:
    TUNE_PPRF_THREADS, TUNE_QC_PLANES, TUNE_QC_BACKEND, TUNE_QC_RECORD_MARGIN = 1, 2, 3, 5

    def __init__(self, **tuning):
        self.tuning, self.calls = {getattr(self, k): v for k, v in tuning.items()}, []

    def set_tuning(self, key, value):
        self.tuning[key] = value

    def ferret_pprf_sender(self, *a, **kw):
        pass

    def sot_dual_lpn(self, *a, **kw):
        self.calls.append(self.tuning.get(self.TUNE_QC_PLANES))


@pytest.mark.parametrize("log_n,tuning,swept", [(13, {}, True), (14, {}, False), (22, {}, False), (23, {}, True),
                                                (20, dict(TUNE_QC_BACKEND=2), True), (20, dict(TUNE_QC_BACKEND=1), True),
                                                (20, dict(TUNE_QC_RECORD_MARGIN=1), True)])
def test_planes_are_tuned_where_a_pass_depends_on_them(fakes, monkeypatch, tmp_path, log_n, tuning, swept):
    """The ternary dual LPN takes all its planes at once unless the caller bounds its scratch."""
    fakes(lambda ret: 1.0)
    monkeypatch.setattr(torch, "empty", lambda *a, **kw: None)
    monkeypatch.setattr(autotune, "_time", lambda fn, stream, reps: fn(None) or 1.0)
    i = inst(kind=1, n=1 << log_n)
    i.a = i.v = i.d_roots = i.delta = None
    ctx = FakeContext(**tuning)
    hit = autotune.tune_single(ctx, i, table=autotune.TuningTable(str(tmp_path / "t.json")))
    assert ("qc_planes_per_pass" in hit) == swept == bool(ctx.calls)
    assert (ctx.TUNE_QC_PLANES in ctx.tuning) == swept
