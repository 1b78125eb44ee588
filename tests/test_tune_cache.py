"""A stored choice of knob values is taken only by a library whose values stand
for the same shapes, and the knob table tells different shapes apart."""
import json

from prtcl_gb300 import tune
from tests.test_tune import COSTS, UNROLL, FakeTarget


def test_choices_of_another_table_are_tuned_afresh(tmp_path, monkeypatch):
    path = tmp_path / "c.json"
    t = tune.Autotuner(cache_path=str(path), device="d")
    choice, _, _ = t.tune(FakeTarget(COSTS, UNROLL), "w")
    assert t.lookup("w") == choice
    monkeypatch.setattr(tune, "knob_fingerprint", lambda: "another")
    assert t.lookup("w") is None
    assert t.tune(FakeTarget(COSTS, UNROLL), "w")[1] == "tuned"
    assert t.tune(FakeTarget(COSTS, UNROLL), "w")[1] == "cache"


def test_choices_stored_without_their_table_are_tuned_afresh(tmp_path):
    path = tmp_path / "c.json"
    path.write_text(json.dumps({"d|w": {"choice": {"density": 1, "jacobi_unroll": 2}}}))
    assert tune.Autotuner(cache_path=str(path), device="d").lookup("w") is None


def test_the_table_tells_shapes_apart(gpu_lib):
    for k, text in tune.knob_table().items():
        if k not in tune.SWEEP_KNOBS:
            continue
        plain = text.split(" small:")[0].split(" unordered:")[0].split(" batched:")[0]
        shapes = [w.split("=")[1] for w in plain.split() if "=" in w]
        assert len(shapes) >= 4 and len(set(shapes)) == len(shapes), (k, text)
