"""The strip heights that the single-domain column marches choose: one wave
of strips of any height, strips at their shortest, several waves, and ragged
last strips.  Every row is held to the FP64 form, which is bit-identical to the
reference, so that a row left out or taken twice shows."""
import numpy as np
import pytest

import nl2d_testlib as T
from test_gpu_mixed import run_form

pytestmark = pytest.mark.gpu

NSTEPS = 5
# relative, per row: the mixed form rounds about 100 operations per step and
# cell in FP32 (5 * 100 * 2^-24 = 3e-5), the FP64-equivalent one holds 1e-10
BOUND = {1: 1e-4, 2: 1e-10}


def model(gpulib, nx, ny, oracle):
    """A random state after one FP64 step: the forms agree only from a state
    that a step leaves (land at rest, sshn_u and sshn_v those of sshn_t)."""
    m = T.make_model(nx + 2, ny + 2, oracle=oracle)
    rng = np.random.default_rng(11)
    for k, a in (("sshn_t", 0.3), ("un", 0.1), ("vn", 0.1)):
        m.f[k][:] = rng.uniform(-a, a, m.f[k].shape)
    run_form(gpulib, m, 1, 0)
    gpulib.nl2d_finalize()
    return m


# columns: 3 (8 rows), 20 (ragged 9), 34 x 1500 (22 rows), 51 (a ragged last
# strip), 101 (128 rows at the limit, several waves of 64 beyond it)
@pytest.mark.parametrize("nx,ny", [(3, 3), (61, 500), (600, 1029), (1000, 1500), (1501, 1103),
                                   (3000, 3070), (3000, 3071), (3000, 3200)])
@pytest.mark.parametrize("precision", [1, 2])
def test_every_row_is_stepped(gpulib, oracle, nx, ny, precision):
    base = model(gpulib, nx, ny, oracle)
    ref = run_form(gpulib, base.copy(), NSTEPS, 0)
    gpulib.nl2d_finalize()
    got = run_form(gpulib, base, NSTEPS, precision)
    gpulib.nl2d_finalize()
    worst = {}
    for k in ("sshn_t", "un", "vn"):
        a, b = got.f[k][:, :nx + 2], ref.f[k][:, :nx + 2]
        rows = np.linalg.norm(a - b, axis=1) / np.maximum(np.linalg.norm(b, axis=1), 1e-3)
        worst[k] = float(rows.max())
    assert max(worst.values()) <= BOUND[precision], worst
