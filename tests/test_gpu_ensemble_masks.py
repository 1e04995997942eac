"""What an ensemble's set-up makes of a domain's mask: which masks it takes,
and the split of the cells between the march and the exact code."""
import numpy as np
import pytest

import nl2d_testlib as T
from test_gpu_ensemble_df import REL_L2, run_pair, worst_rel_l2
from test_oracle import bits_equal

pytestmark = pytest.mark.gpu


def takes(m, dims):
    """The rule, face by face: no Flather face takes its value from outside
    the arrays or from a face that is itself a Flather face."""
    w, h, xs, xe, ys, ye = dims

    def flather(a, b):
        return a + b > -1 and (a < 0 or b < 0)

    for j in range(ys - 1, ye + 2):
        for i in range(xs - 1, xe + 1):
            if flather(m[j, i], m[j, i + 1]):
                nb = i + 1 if m[j, i] < 0 else i - 1
                if nb < 0 or xs - 1 <= nb <= xe and flather(m[j, nb], m[j, nb + 1]):
                    return False
    for j in range(ys - 1, ye + 1):
        for i in range(xs - 1, xe + 2):
            if flather(m[j, i], m[j + 1, i]):
                nb = j + 1 if m[j, i] < 0 else j - 1
                if nb < 0 or ys - 1 <= nb <= ye and flather(m[nb, i], m[nb + 1, i]):
                    return False
    return True


def domain(nx, ny, side="S", land=0.0, seed=0):
    from psyclonebench_gb300.ensemble import build_domain
    d = build_domain({"nx": nx, "ny": ny, "depth_seed": seed, "open_side": side,
                      "tide_amp": 0.2, "tide_period_h": 12.42})
    w, h, xs, xe, ys, ye = d["dims"]
    rng = np.random.default_rng(seed)
    t = d["tmask"][ys:ye + 1, xs:xe + 1]
    t[rng.uniform(size=t.shape) < land] = 0
    return d


def test_masks_taken_and_refused(gpulib):
    """Random masks of open, land and sea cells: taken or refused as the
    rule says, a refusal naming the domain."""
    from psyclonebench_gb300.ensemble import Ensemble
    rng = np.random.default_rng(3)
    seen = set()
    for k in range(60):
        d = domain(int(rng.integers(1, 6)), int(rng.integers(1, 6)))
        p = rng.choice([0.02, 0.1, 0.3])
        d["tmask"][:] = rng.choice([-1, 0, 1, 2], size=d["tmask"].shape,
                                   p=[p, 0.1, 0.8 - p, 0.1])
        want = takes(d["tmask"], d["dims"])
        seen.add(want)
        try:
            Ensemble([d], lib=gpulib).close()
            got = True
        except RuntimeError as e:
            assert "set_domain(0)" in str(e)
            got = False
        assert got == want, d["tmask"]
    assert seen == {False, True}


@pytest.mark.parametrize("which", ["hu", "hv"])
def test_depths_refused(gpulib, which):
    from psyclonebench_gb300.ensemble import Ensemble
    for bad in (0.0, -1.0, np.nan):
        d = domain(5, 4)
        d[which] = d[which].copy()
        d[which][-1, -1] = bad
        with pytest.raises(RuntimeError):
            Ensemble([d], lib=gpulib)


def test_every_cell_is_stepped(gpulib, oracle):
    """Thin domains and domains with land: the FP64 form bit-identical to
    the oracle after 40 steps, the FP64-equivalent form within its bound of
    it (a cell that neither the march nor the exact code took would stay at
    rest)."""
    doms = [domain(nx, ny, side, land, seed)
            for seed, (nx, ny, side, land) in enumerate(
                [(1, 1, "S", 0), (2, 2, "N", 0), (3, 3, "E", 0), (2, 9, "W", 0), (9, 2, "S", 0),
                 (4, 9, "N", 0), (33, 5, "S", 0), (34, 35, "E", 0.02), (70, 20, "W", 0.1),
                 (20, 40, "S", 0.01)])]
    ref, _, got, _ = run_pair(gpulib, doms, 40)
    for d, r in zip(doms, ref):
        want, _ = T.ensemble_oracle_run(d, 40, oracle=oracle)
        assert all(bits_equal(a, want.f[k]) for a, k in zip(r, ("sshn_t", "un", "vn"))), d["dims"]
    assert worst_rel_l2(doms, ref, got) <= REL_L2
