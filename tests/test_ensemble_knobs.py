"""CPU tests: the knobs that Ensemble.schedule() and the autotuner start from
are the ones a new ensemble has."""
import re

import pytest

from psyclonebench_gb300 import autotune, ensemble


class Lib:
    """Records the knob calls."""

    def __init__(self):
        self.calls = []

    def nl2d_ens_schedule(self, *a):
        self.calls.append(a)
        return 0

    def nl2d_ens_tile(self, *a):
        self.calls.append(a)
        return 0


class Ens(ensemble.Ensemble):
    def __init__(self, cost):
        self.lib = Lib()
        self.domains = [{"dims": (66, 66, 1, 64, 1, 64)}]
        self.cost = cost
        self.seen = []

    def run(self, istep0, nsteps, checksum_every=0):
        knobs = self.lib.calls[-2] + self.lib.calls[-1]
        self.seen.append(knobs)
        return self.cost(knobs) * nsteps, None

    def reset(self):
        pass


DEFAULTS = (2, 2, 4.0, 32, 8, 0)


def test_schedule_without_arguments_is_the_librarys_default():
    ens = Ens(lambda k: 1.0)
    ens.schedule()
    assert ens.lib.calls == [DEFAULTS[:3], DEFAULTS[3:]]
    # and the defaults are the ones the library states
    src = open(ensemble.__file__.replace("ensemble.py", "csrc/nl2d_ensemble.cu")).read()
    assert re.search(r"kDefaultCtas = 2, kDefaultPolicy = 2;", src)
    assert re.search(r"kDefaultWeight = 4\.0;", src)
    shapes = re.search(r"kShapes\[kNumShapes\]\[2\] = \{(.*)\};", src).group(1)
    k = int(re.search(r"kDefaultShape = (\d)", src).group(1))
    assert re.findall(r"\{(\d+), (\d+)\}", shapes)[k] == ("32", "8")
    assert re.search(r"int march_rows = 0;", src)


@pytest.mark.parametrize("precision", ["mixed", "df"])
def test_tuning_a_march_keeps_the_default_knobs_and_tries_its_own_rule(precision):
    ens = Ens(lambda k: 1.0 if k == DEFAULTS else 2.0)
    r = autotune.tune(ens, precision=precision, use_cache=False)
    assert {k[:5] for k in ens.seen} == {DEFAULTS[:5]}
    assert {k[5] for k in ens.seen} == {0, 8, 16, 32, 64}
    assert r["march_rows"] == 0 and ens.lib.calls[-2] + ens.lib.calls[-1] == DEFAULTS


def test_tuning_the_fp64_form_tries_the_defaults_and_leaves_the_strips_alone():
    ens = Ens(lambda k: 1.0)
    autotune.tune(ens, use_cache=False)
    assert {k[5] for k in ens.seen} == {0}
    assert (2, 2) + DEFAULTS[3:5] in {k[:2] + k[3:5] for k in ens.seen}


def test_choices_stored_for_other_kernels_are_not_used(tmp_path, monkeypatch):
    monkeypatch.setenv("NL2D_TUNE_CACHE", str(tmp_path))
    ens = Ens(lambda k: 1.0)
    autotune.tune(ens)
    assert autotune.tune(ens)["cached"]
    monkeypatch.setattr(autotune, "COSTS_VERSION", autotune.COSTS_VERSION + 1)
    assert not autotune.tune(ens)["cached"]
