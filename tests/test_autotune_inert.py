"""The autotuner times no setting of a knob that selects nothing, and keeps and
caches the values such knobs have."""
import json

import pytest

pytest.importorskip("torch")
try:
    from word2world_b200 import _C, autotune  # noqa: F401
except ImportError:
    pytest.skip("extension not built", allow_module_level=True)


def test_inert_knobs_are_not_timed(monkeypatch, tmp_path):
    before, seen = autotune.current(), []
    times = iter([1.0] + [0.5, 1.0] * 50)  # every other trial looks like a gain

    def timed(self, step):
        seen.append(autotune.current())
        return next(times)

    monkeypatch.setattr(autotune.Autotuner, "_cuda_time", timed)
    path = str(tmp_path / "tune.json")
    try:
        best = autotune.Autotuner(path=path).tune("bucket", step=None)
    finally:
        autotune.apply(before)
    assert all(k[i] == before[i] for k in seen for i in autotune.INERT)
    assert set(best) == set(before) and all(best[i] == before[i] for i in autotune.INERT)
    assert all(json.load(open(path))["bucket"][i] == before[i] for i in autotune.INERT)
    assert any(best[k] != before[k] for k in best)
