"""Ensembles with much land under every tile shape and assignment policy:
bit-identical to the oracle (each kernel instance takes the cells beside land
by its own copy of the code)."""
import pytest

import nl2d_testlib as T
from test_gpu_ensemble_masks import domain
from test_oracle import bits_equal

pytestmark = pytest.mark.gpu

NSTEPS = 20


@pytest.fixture(scope="module")
def problem(oracle):
    doms = [domain(nx, ny, side, land, seed)
            for seed, (nx, ny, side, land) in enumerate(
                [(5, 4, "S", 0.1), (33, 9, "N", 0.1), (70, 20, "W", 0.5), (41, 67, "E", 0.03),
                 (130, 40, "S", 0.0)])]
    return doms, [T.ensemble_oracle_run(d, NSTEPS, oracle=oracle)[0] for d in doms]


@pytest.mark.parametrize("tile", [(32, 16), (32, 8), (16, 16), (64, 8), (32, 32)])
@pytest.mark.parametrize("ctas,policy,weight", [(1, 0, 0.0), (2, 0, 16.0), (2, 1, 4.0), (2, 2, 4.0)])
def test_land_under_every_schedule(gpulib, problem, tile, ctas, policy, weight):
    from psyclonebench_gb300.ensemble import Ensemble
    doms, want = problem
    e = Ensemble(doms, lib=gpulib)
    e.schedule(ctas, policy, weight, tile)
    e.run(1, NSTEPS)
    got = [e.read(k) for k in range(len(doms))]
    e.close()
    for d, r, w in zip(doms, got, want):
        assert all(bits_equal(a, w.f[k]) for a, k in zip(r, ("sshn_t", "un", "vn"))), d["dims"]
