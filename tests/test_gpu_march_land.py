"""The single-domain column marches where many cells lie beside land, which the
mixed form's strip heights depend on: every row against the FP64 form."""
import numpy as np
import pytest

import nl2d_testlib as T
from test_gpu_march_strips import BOUND, NSTEPS
from test_gpu_mixed import run_form

pytestmark = pytest.mark.gpu


# mixed: one wave up to 14 592 general cells, shorter strips of several waves beyond
@pytest.mark.parametrize("nx,ny,land", [
    (61, 500, 0.1), (1501, 1103, 0.0002), (1501, 1103, 0.01), (2901, 2500, 0.0001),
    (2901, 2500, 0.001),
])
@pytest.mark.parametrize("precision", [1, 2])
def test_every_row_is_stepped_beside_land(gpulib, oracle, nx, ny, land, precision):
    m = T.make_model(nx + 2, ny + 2, oracle=oracle)
    rng = np.random.default_rng(12)
    for k, a in (("sshn_t", 0.3), ("un", 0.1), ("vn", 0.1)):
        m.f[k][:] = rng.uniform(-a, a, m.f[k].shape)
    t = m.grid["tmask"][m.ys:m.ye + 1, m.xs:m.xe + 1]
    t[rng.uniform(size=t.shape) < land] = 0
    run_form(gpulib, m, 1, 0)  # the forms agree from a state that a step leaves
    gpulib.nl2d_finalize()
    ref = run_form(gpulib, m.copy(), NSTEPS, 0)
    gpulib.nl2d_finalize()
    got = run_form(gpulib, m, NSTEPS, precision)
    gpulib.nl2d_finalize()
    worst = {}
    for k in ("sshn_t", "un", "vn"):
        a, b = got.f[k][:, :nx + 2], ref.f[k][:, :nx + 2]
        rows = np.linalg.norm(a - b, axis=1) / np.maximum(np.linalg.norm(b, axis=1), 1e-3)
        worst[k] = float(rows.max())
    assert max(worst.values()) <= BOUND[precision], worst
