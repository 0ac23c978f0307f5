"""Schedules that an earlier version tuned in another unit are not taken over (no GPU)."""

from types import SimpleNamespace

import pytest

from pyftle_b200 import batch as B


@pytest.mark.parametrize("unit,taken", [("", False), ("-blocks", True)])
def test_only_schedules_counted_in_blocks_are_taken_from_the_cache(monkeypatch, unit, taken):
    b = B.WindowBatch.__new__(B.WindowBatch)
    b.series = SimpleNamespace(grid=SimpleNamespace(dim=2), precision="fx16")
    b.kw, b.count = dict(integrator="rk4"), 2
    b.windows = [SimpleNamespace(num_steps=s, positions=SimpleNamespace(shape=(4 * 300, 2)))
                 for s in (3, 5)]
    tuned = {"d2-fx16-rk4-w2-g9-s5" + unit: {"schedule": {"ctas_per_sm": 2, "order": 2}}}
    monkeypatch.setattr(B, "_load_cache", lambda: dict(tuned))
    monkeypatch.setattr(b, "run", lambda schedule: 1 / 0)  # the candidates are timed
    if taken:
        assert b.autotune() == B.Schedule(2, 2) == b.schedule
    else:
        with pytest.raises(ZeroDivisionError):
            b.autotune()
