"""The autotuner times no setting of a knob that selects nothing, and keeps and
caches the values such knobs have."""
import json

import pytest

pytest.importorskip("torch")
try:
    from word2world_b200 import _C, autotune  # noqa: F401
except ImportError:
    pytest.skip("extension not built", allow_module_level=True)


@pytest.mark.parametrize("queue", [0, 1])  # the faster blend: per tile, or the queue-fed one that blend_warps shapes
def test_inert_knobs_are_not_timed(monkeypatch, tmp_path, queue):
    before, seen = autotune.current(), []

    def timed(self, step):  # every trial with the faster blend looks like a gain
        k = autotune.current()
        seen.append(k)
        return 1.0 - 0.02 * len(seen) + (0.0 if k["blend_queue"] == queue else 10.0)

    monkeypatch.setattr(autotune.Autotuner, "_cuda_time", timed)
    path = str(tmp_path / "tune.json")
    try:
        best = autotune.Autotuner(path=path).tune("bucket", step=None)
    finally:
        autotune.apply(before)
    assert all(k[i] == before[i] for k in seen for i in autotune.INERT)
    assert set(best) == set(before) and all(best[i] == before[i] for i in autotune.INERT)
    assert all(json.load(open(path))["bucket"][i] == before[i] for i in autotune.INERT)
    assert best["blend_queue"] == queue
    assert any(k["blend_warps"] != before["blend_warps"] for k in seen) == (queue == 1)
