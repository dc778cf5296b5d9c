"""The autotuner's choice, on timings made up here, and its cache: a rule is kept only
where it beats the library's defaults, the widths that the defaults use are among the
candidates, and a table of another device or library build is dropped."""

import json
from types import SimpleNamespace

import pytest

from helioselene_gb300 import autotune

CANDS = list(autotune.DEFAULT_CANDIDATES)


def timings(default, best, at_best, lone_default=100.0, lone=100.0):
    """batch and lone times: a valley at `best`, the defaults at `default`"""
    def batch(form):
        return default if form is None else at_best + abs(form[0] - best) + 0.1 * form[1]

    def single(form):
        return lone_default if form is None else lone
    return batch, single


def test_candidates_span_the_default_widths_of_batches():
    assert CANDS[0] <= 5 and CANDS[-1] >= 16


@pytest.mark.parametrize("best", [4, 5, 9, 16])
@pytest.mark.parametrize("start", [4, 8, 12])
def test_a_faster_width_is_found_and_kept(best, start):
    assert autotune._rule(*timings(50.0, best, 40.0), CANDS, start) == (best, {"c": best, "rounds": 0})


@pytest.mark.parametrize("default", [40.0, 40.5, 30.0])
def test_no_rule_that_does_not_beat_the_defaults(default):
    assert autotune._rule(*timings(default, 8, 40.0), CANDS, 8) == (8, None)


def test_no_rule_that_slows_one_msm():
    assert autotune._rule(*timings(50.0, 5, 40.0, lone_default=100.0, lone=120.0), CANDS, 8) == (5, None)


def test_cache_of_another_library_or_device(tmp_path, monkeypatch):
    torch = pytest.importorskip("torch")
    tuned, installed = [], []
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda d: "this")
    monkeypatch.setattr(autotune, "_library_id", lambda: "now")
    monkeypatch.setattr(autotune, "tune", lambda ctx, curve, **kw: tuned.append(curve) or {"64-127": {"c": 6, "rounds": 0}})
    ctx = SimpleNamespace(device=0, set_window=lambda *a: installed.append(a))
    path = tmp_path / "cache.json"
    old = {"n_max": 1 << 20, "helios": {"64-127": {"c": 8, "rounds": 0}}, "selene": {}}
    path.write_text(json.dumps({"this": old, "other": dict(old, library="now")}))
    autotune.load_or_tune(ctx, path)  # the entry names no library: tuned again
    assert tuned == [0, 1] and (0, 64, 127, 6, 0) in installed and (0, 64, 127, 8, 0) not in installed
    autotune.load_or_tune(ctx, path)  # now from the cache
    assert tuned == [0, 1]
    monkeypatch.setattr(autotune, "_library_id", lambda: "later")
    autotune.load_or_tune(ctx, path)
    assert tuned == [0, 1, 0, 1]
    assert "other" in json.loads(path.read_text())
