"""The tuning file (CPU): a choice kept from other passes is timed again, one of
these passes is taken, and what the file held stays in it."""
import json
import types

import pytest


@pytest.fixture
def tune(monkeypatch, tmp_path):
    from dftpy_gb300 import autotune
    path = tmp_path / "tune.json"
    monkeypatch.setenv("GBOFDFT_TUNE_CACHE", str(path))
    monkeypatch.setattr(autotune, "_CACHE", {})
    chosen = []
    monkeypatch.setattr(autotune, "schedules", lambda plan: 3)
    monkeypatch.setattr(autotune, "set_schedule", lambda plan, s: chosen.append(s))
    monkeypatch.setattr(autotune, "_time_schedules", lambda plan: [0.081, 0.099, 0.1])
    return autotune, path, chosen


def test_choice_of_earlier_passes_is_timed_again(tune):
    autotune, path, chosen = tune
    plan = types.SimpleNamespace(nr=(128, 128, 128), precision=0, full=False)
    old = {"128x128x128/0/0": {"schedule": 1, "ms": [0.102, 0.094, 0.1]}}
    path.write_text(json.dumps(old))
    assert autotune.tune(plan) == (0, [0.081, 0.099, 0.1]) and chosen[-1] == 0
    kept = json.loads(path.read_text())
    assert kept["128x128x128/0/0"] == old["128x128x128/0/0"] and len(kept) == 2
    # the new choice is taken from the file by another process
    autotune._CACHE.clear()
    assert autotune.tune(plan) == (0, None)
