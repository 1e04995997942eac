"""The FP64 fused step's cells beside land and open water inside the domain:
by the tile's staged values, or, where a Flather face reads two cells on, by
the arrays.  Bit-identical to the oracle, all 13 fields."""
import numpy as np
import pytest

import nl2d_testlib as T
from test_oracle import bits_equal

pytestmark = pytest.mark.gpu


def build(nx, ny, dry, pools, seed, oracle):
    m = T.make_model(nx, ny, oracle=oracle)
    rng = np.random.default_rng(seed)
    m.f["sshn_t"][:] = rng.uniform(-0.3, 0.3, m.f["sshn_t"].shape)
    m.f["un"][:] = rng.uniform(-0.1, 0.1, m.f["un"].shape)
    m.f["vn"][:] = rng.uniform(-0.1, 0.1, m.f["vn"].shape)
    t = m.grid["tmask"]
    inner = np.zeros(t.shape, bool)
    inner[m.ys:m.ye + 1, m.xs:m.xe + 1] = True
    t[inner & (rng.uniform(size=t.shape) < dry)] = 0
    if pools:  # single open cells, six apart: every place in a tile and at its edges
        t[m.ys + 5:m.ye - 4:6, m.xs + 5:m.xe - 4:7] = -1
    return m


@pytest.mark.parametrize("nx,ny,dry,pools", [
    (45, 61, 0.03, True), (45, 61, 0.3, True), (45, 61, 0.7, False),   # 16 x 8 tiles
    (85, 41, 0.0, True),
    (37, 2437, 0.05, True), (1031, 157, 0.5, True), (1031, 157, 0.0, True),  # 32 x 8 tiles
])
def test_cells_beside_land_and_pools_match_oracle(gpulib, oracle, nx, ny, dry, pools):
    m = build(nx, ny, dry, pools, nx + ny, oracle)
    want = m.copy()
    T.run(oracle.oracle_invoke_time_step, want, 4)
    assert all(np.isfinite(want.f[k]).all() for k in T.FIELDS)
    paths = T.gpu_run_calls(gpulib, m, 4)
    gpulib.nl2d_finalize()
    assert paths[-1] == 2, paths  # the fused step
    bad = [k for k in T.FIELDS if not bits_equal(m.f[k], want.f[k])]
    assert not bad, bad
