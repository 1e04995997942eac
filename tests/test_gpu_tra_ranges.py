"""The tracer kernels at the edges of their tiles and runs of levels, and on
inputs at and beyond the range their straight-line forms take: every bit of
the field against the oracle."""
import numpy as np
import pytest

from test_gpu_tra_adv import gpu_compute, gpu_field, oracle_field
from test_tra_oracle import random_inputs

pytestmark = pytest.mark.gpu


def check(lib, f, niter):
    want = oracle_field(f, niter)
    gpu_compute(lib, f, niter)
    got = gpu_field(lib, want.shape)
    lib.tra_adv_finalize()
    np.testing.assert_array_equal(got.view(np.int64), want.view(np.int64))


# interiors of one tile (32 x 8) and one point more or less; runs of levels of
# the column march from one to many
@pytest.mark.parametrize("dims", [(3, 3, 2), (33, 10, 3), (34, 9, 5), (35, 11, 8), (66, 18, 31),
                                  (40, 30, 75)])
def test_tile_and_run_edges(gpulib, oracle, dims):
    check(gpulib, random_inputs(*dims, seed=sum(dims)), 4)


@pytest.mark.parametrize("kind", ["land", "tiny", "huge", "mixed", "wide velocity"])
def test_ranges(gpulib, oracle, kind):
    f = random_inputs(45, 29, 9, seed=17)
    rng = np.random.default_rng(23)
    m = f["mydomain"]
    if kind == "land":  # 0 / 1 masks, zeros of either sign on land
        sea = (rng.random(m.shape) > 0.3).astype(float)
        for n in ("tmask", "umask", "vmask"):
            f[n][:] = sea
        for n in ("pun", "pvn", "pwn"):
            f[n] *= sea
        m *= np.where(sea > 0, 1.0, rng.choice([0.0, -0.0], m.shape))
    elif kind == "tiny":  # around 2^-400 and down to subnormals
        m *= 2.0 ** rng.integers(-1070, -390, m.shape)
    elif kind == "huge":  # around 2^700
        m *= 2.0 ** rng.integers(690, 710, m.shape)
    elif kind == "mixed":  # a few points out of range, the rest ordinary
        at = rng.random(m.shape) < 0.01
        m[at] *= 2.0 ** -900
    else:  # one input out of range
        f["pun"][3, 5, 7] = 2.0 ** -150
    check(gpulib, f, 3)
