"""The autotuner's engine modes, on a fake engine (no device): what it sets by default, what
the rate beside a choice belongs to, and what a batch's lags are timed in."""
import pytest

import bk_b200 as bk
from bk_b200 import tune


class FakeEngine:
    device = 0

    def __init__(self):
        self.options, self.batches = {"engine_mode": 4}, []

    def set_option(self, name, value):
        self.options[name] = value

    def evolve_batch(self, instances, dt, n_steps, lag=0, **kw):
        self.batches.append((self.options["engine_mode"], lag))


@pytest.fixture
def eng(monkeypatch):
    monkeypatch.setattr(tune, "device_key", lambda device=0: "fake")
    return FakeEngine()


def test_defaults_are_the_engines_own_schedule(eng):
    tune.apply_config(eng, tune.DEFAULTS)
    assert eng.options["engine_mode"] == tune.TURNING == 4
    tune.apply_config(eng, {})
    assert eng.options["engine_mode"] == tune.TURNING


def test_saved_entry_without_a_mode_keeps_the_mode_it_was_timed_in(eng, tmp_path):
    path = str(tmp_path / "t.json")
    tune.save_cache({"fake": {"c64/n24": {"best": {"slab_lag": 2}, "amp_steps_per_s": 1.0}}}, path)
    assert tune.apply(eng, 24, bk.BK_C64, cache_path=path) == {"slab_lag": 2}
    assert (eng.options["engine_mode"], eng.options["slab_lag"]) == (0, 2)


@pytest.mark.parametrize("turning", [5.0, 50.0])
def test_rate_beside_a_choice_is_its_own(eng, tmp_path, monkeypatch, turning):
    rates = iter(range(1, 1000))
    monkeypatch.setattr(tune, "measure", lambda e, n, p, cfg, *a, **k: turning if cfg["engine_mode"] == tune.TURNING
                        else 10.0 + 0.01 * next(rates))
    e = tune.tune(eng, 22, bk.BK_C64, trap=(1, 1), cache_path=str(tmp_path / "t.json"))
    swept = max(c["amp_steps_per_s"] for c in e["candidates"])
    assert e["best_amp_steps_per_s"] == max(turning, swept)
    assert (e["best"]["engine_mode"] == tune.TURNING) == (turning > swept)
    assert e["best"]["engine_mode"] == eng.options["engine_mode"]


@pytest.mark.parametrize("fast", [(4, 0), (0, 6)])
def test_lags_of_a_batch_are_timed_where_they_apply(eng, tmp_path, monkeypatch, fast):
    def timer(e):
        def run(fn):
            fn()
            return 1.0 if e.batches[-1] == fast else 2.0
        return run

    monkeypatch.setattr(tune, "_timer", timer)
    path = str(tmp_path / "t.json")
    inst = [dict(n=16, s0=1, g=0.3)]
    e = tune.tune_batch(eng, inst, 0.02, 4, cache_path=path)
    assert {(c["engine_mode"], c["lag"]) for c in e["candidates"]} == {(4, 0)} | {(0, l) for l in (1, 2, 3, 4, 6, 8)}
    assert (e["best"]["engine_mode"], e["best"]["lag"]) == fast and eng.options["engine_mode"] == fast[0]
    eng.set_option("engine_mode", 1)
    assert tune.apply_batch(eng, inst, cache_path=path) == e["best"] and eng.options["engine_mode"] == fast[0]
    assert tune.batch_lag(eng, inst, cache_path=path) == fast[1]


def test_committed_rates_belong_to_the_committed_choices():
    for entries in tune.load_cache().values():
        for key, e in entries.items():
            if "turning_amp_steps_per_s" in e:
                own = "turning_amp_steps_per_s" if e["best"]["engine_mode"] == tune.TURNING else "amp_steps_per_s"
                assert e["best_amp_steps_per_s"] == e[own], key
            if key.startswith("batch/"):
                assert "engine_mode" in e["best"], key
