"""The FP64 fused step over the sizes, values and constants where its tile
code changes form: interiors around a tile's edge (16 x 8 tiles for small
grids, 32 x 8 for large ones), interiors too thin for any tile, fields inside
and outside the range of the straight-line arithmetic (zeros, subnormals,
2^-200, 2^200), grid spacings with and without a short significand or outside
the constants' range, and land.  Bit-identical to the oracle, all 13 fields:
every form rounds each operation as IEEE does, so the tolerance is zero."""
import numpy as np
import pytest

import nl2d_testlib as T
from test_oracle import bits_equal


def scales(rng, shape, lo, hi, zeros=0.0):
    """+-m * 2^k with k uniform in [lo, hi], some of them zero."""
    a = np.ldexp(rng.uniform(1.0, 2.0, shape), rng.integers(lo, hi + 1, shape))
    a *= rng.choice([-1.0, 1.0], shape)
    a[rng.uniform(size=shape) < zeros] = 0.0
    return a


def edges(rng, shape):
    """The first and last values of the straight-line range and their
    neighbours outside it."""
    lo = 2.0 ** -200
    return rng.choice([lo, -lo, np.nextafter(lo, 0), -np.nextafter(lo, 0), 0.0, -0.0, 0.25,
                       5e-324], shape)


# name -> (ssh, velocity) of the start state
VALUES = {
    "plain": (lambda r, s: r.uniform(-0.3, 0.3, s), lambda r, s: r.uniform(-0.1, 0.1, s)),
    "scales": (lambda r, s: scales(r, s, -260, -2, 0.2), lambda r, s: scales(r, s, -260, -3, 0.2)),
    "tiny": (lambda r, s: scales(r, s, -1073, -500, 0.1), lambda r, s: scales(r, s, -1073, -500)),
    "edges": (edges, edges),
    # (the first step squares the velocities: the second, fused one reads 2^150 .. 2^220)
    "huge": (lambda r, s: r.uniform(-0.3, 0.3, s), lambda r, s: scales(r, s, 90, 112, 0.5)),
}
SPACING = {"short": (1000.0, 1000.0), "long": (987.654321, 1234.56789),
           "big": (2.0 ** 41 * 1.1, 2.0 ** 40), "vast": (1e60, 1e59)}


def build(inner, values, spacing, land, seed, oracle):
    """inner: cells strictly inside the internal region's outermost ring,
    which the tiles cover (-1: the region is one cell across)."""
    dx, dy = SPACING[spacing]
    m = T.make_model(inner[0] + 4, inner[1] + 4, dx=dx, dy=dy, oracle=oracle)
    rng = np.random.default_rng(seed)
    ssh, vel = VALUES[values]
    m.f["sshn_t"][:] = ssh(rng, m.f["sshn_t"].shape)
    m.f["un"][:] = vel(rng, m.f["un"].shape)
    m.f["vn"][:] = vel(rng, m.f["vn"].shape)
    if land:
        t = m.grid["tmask"][m.ys:m.ye + 1, m.xs:m.xe + 1]
        t[rng.uniform(size=t.shape) < 0.1] = 0
    return m


NSTEPS = {"huge": 2}

CASES = [((w, h), "plain", "short", False) for w in (-1, 0, 1, 15, 16, 17) for h in (0, 7, 8, 9)]
CASES += [((33, 19), v, s, l) for v in VALUES for s, l in
          (("short", False), ("long", True), ("big", False), ("vast", True))]
# 608 or more 32 x 8 tiles
CASES += [((33, 2433), v, "short", v == "plain") for v in VALUES]
CASES += [((31, 4857), "plain", "long", False), ((19457, 7), "scales", "short", True),
          ((64, 2439), "tiny", "long", True)]


def test_oracle_stays_finite(oracle):
    """The start states are ones whose bits can be compared: no infinity or
    NaN within the steps taken."""
    for values in VALUES:
        for spacing in SPACING:
            m = build((33, 19), values, spacing, True, 5, oracle)
            T.run(oracle.oracle_invoke_time_step, m, NSTEPS.get(values, 3))
            assert all(np.isfinite(m.f[k]).all() for k in T.FIELDS), (values, spacing)


@pytest.mark.gpu
@pytest.mark.parametrize("inner,values,spacing,land", CASES)
def test_fused_tiles_match_oracle(gpulib, oracle, inner, values, spacing, land):
    m = build(inner, values, spacing, land, 5, oracle)
    want = m.copy()
    n = NSTEPS.get(values, 3)
    T.run(oracle.oracle_invoke_time_step, want, n)
    paths = T.gpu_run_calls(gpulib, m, n)
    gpulib.nl2d_finalize()
    assert paths[-1] == 2, paths  # the fused step
    bad = [k for k in T.FIELDS if not bits_equal(m.f[k], want.f[k])]
    assert not bad, bad
