"""The autotuners' choices, with the timings made up."""
import types

import pytest

from transportse_b200 import autotune


class _Field:
    def clone(self):
        return self

    def copy_(self, other):
        return self


def _sim(max_blocks=0, index=0, shape=(40, 40, 40)):
    M = types.SimpleNamespace(precision="fp32dc", nx=shape[0], ny=shape[1], nz=shape[2], max_blocks=max_blocks,
                              device=types.SimpleNamespace(index=index), sweep_variant=None)
    return types.SimpleNamespace(M=M, S={"P": _Field()})


@pytest.fixture
def timings(monkeypatch):
    """us(max_blocks, variant) -> (us an iteration, the variant that ran)"""
    made = {}

    def timed(sim, variant, iters):
        us, ran = made["us"](sim.M.max_blocks, tuple(variant))
        return 1e-3 * us * iters, iters, ran

    monkeypatch.setattr(autotune, "_timed_solve", timed)
    monkeypatch.setattr(autotune.torch.cuda, "synchronize", lambda: None)
    monkeypatch.setattr(autotune, "_chosen", {})
    return made


def test_a_capped_models_choice_is_not_an_uncapped_ones(timings):
    """Under a block cap the grid streams, without one it is resident: each
    model gets its own choice, and so does another device's."""
    def us(cap, v):
        if any(v):
            return (7.0 if v == (256, 4, 1) else 8.0), v
        return (9.0, (512, 4, 2)) if cap else (2.0, (0, 0, 0))

    timings["us"] = us
    assert autotune.tune_sweep(_sim(max_blocks=8))["variant"] == (256, 4, 1)
    free = _sim()
    assert autotune.tune_sweep(free)["variant"] == (0, 0, 0) == free.M.sweep_variant
    assert autotune.tune_sweep(_sim())["cached"]
    assert "cached" not in autotune.tune_sweep(_sim(index=1))


def test_the_librarys_choice_keeps_its_name(timings):
    """Where asking for nothing wins, nothing is asked for later either, though
    a staged variant ran."""
    timings["us"] = lambda cap, v: (5.0, (512, 4, 2)) if not any(v) else (6.0, v)
    rec = autotune.tune_sweep(_sim())
    assert rec["variant"] == (0, 0, 0)
    assert min(rec["trials"], key=lambda t: t["us_per_iteration"])["chunk"] == 512


def test_the_ensemble_tuner_is_not_misled_by_a_first_run(monkeypatch):
    """The first run of a process is slow, and so is one in the middle; the set
    that is fastest when run again is chosen."""
    from transportse_b200 import ensemble
    true = {128: 69.0, 256: 70.0, 512: 73.0}
    runs = []

    class Runs:
        def __init__(self, configs, device=None, precision=None, **p):
            self.p = p

        def run(self, steps, keep=()):
            runs.append(self.p["dc_cycle"])
            slow = 0.3 if len(runs) in (1, 5) else 1.0
            return [], {"stepping_cell_updates_per_s": slow * true[self.p["dc_cycle"]], "cell_updates_per_s": 1.0}

    monkeypatch.setattr(ensemble, "Ensemble", Runs)
    best = ensemble.autotune([None], batched=True, clusters=(0,), cycles=(512, 256, 128))
    assert best["dc_cycle"] == 512 and [t["rate"] for t in best["trials"]] == [73.0, 70.0, 69.0]


@pytest.mark.parametrize("rates,chosen", [({128: 75.9, 256: 81.5, 512: 81.4}, 512), ({128: 82.0, 256: 70.0, 512: 60.0}, 128),
                                          ({128: 80.0, 256: 80.4, 512: 78.0}, 256)])
def test_the_ensemble_tuner_takes_the_longest_cycle_of_equals(rates, chosen, monkeypatch):
    """Rates within a sample's spread do not decide."""
    from transportse_b200 import ensemble

    class Runs:
        def __init__(self, configs, device=None, precision=None, **p):
            self.p = p

        def run(self, steps, keep=()):
            return [], {"stepping_cell_updates_per_s": rates[self.p["dc_cycle"]], "cell_updates_per_s": 1.0}

    monkeypatch.setattr(ensemble, "Ensemble", Runs)
    assert ensemble.autotune([None], batched=True, clusters=(0,), cycles=(128, 256, 512))["dc_cycle"] == chosen
