"""The ensemble's schedule and tile knobs: what an ensemble starts with."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def domains():
    from psyclonebench_gb300.ensemble import build_domain
    from psyclonebench_gb300.workloads import ensemble_domains
    return [build_domain(s) for s in ensemble_domains(3, 5, 64, 128)]


def layout(ens):
    ens.run(1, 1)  # makes the schedule
    return ens.info()


def test_a_new_ensemble_starts_with_the_default_schedule(gpulib, domains):
    from psyclonebench_gb300.ensemble import Ensemble
    ens = Ensemble(domains, lib=gpulib)
    ens.schedule(1, 1, 0.0, (64, 8), 16)
    other = layout(ens)
    ens.close()
    ens = Ensemble(domains, lib=gpulib)
    cells, tiles, ctas = layout(ens)
    ens.close()
    assert ctas == tiles and other[2] != other[1]  # one unit per CTA, not a grid per SM
    ens = Ensemble(domains, lib=gpulib)  # without a close between: the same
    ens.schedule(1, 0, 0.0, (32, 32))
    ens = Ensemble(domains, lib=gpulib)
    assert layout(ens) == (cells, tiles, ctas)
    ens.close()


@pytest.mark.parametrize("precision", [1, 2])
def test_the_strip_rule_can_be_had_back(gpulib, domains, precision):
    import numpy as np
    from psyclonebench_gb300.ensemble import Ensemble
    ens = Ensemble(domains, lib=gpulib)
    ens.set_precision(precision)
    ens.run(1, 20)
    want = ens.read(1)
    for rows in (16, 0):
        assert gpulib.nl2d_ens_tile(32, 8, rows) == 0
        ens.reset()
        ens.run(1, 20)
        assert all(np.array_equal(a, b) for a, b in zip(ens.read(1), want))
    for rows in (-1, 1, 7, 24, 128):
        assert gpulib.nl2d_ens_tile(32, 8, rows) != 0
    ens.close()
