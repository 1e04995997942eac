"""Registrations that only just fit the GPU's memory: what the faster forms
keep beside the caller's arrays is left out then, and the bits are the same."""
import numpy as np
import pytest

import nl2d_testlib as T
from test_oracle import bits_equal

pytestmark = pytest.mark.gpu

MB = 1 << 20


class Filled:
    """Holds GPU memory so that about `left` bytes are free."""

    def __init__(self, left):
        self.left, self.held = left, []

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        for _ in range(4):
            more = torch.cuda.mem_get_info()[0] - self.left
            if more < 4 * MB:
                break
            self.held.append(torch.empty(more // (2 * MB) * 2 * MB, dtype=torch.uint8,
                                         device="cuda"))
        return self

    def __exit__(self, *exc):
        import torch
        self.held = []
        torch.cuda.empty_cache()


def problem(oracle, region=None):
    m = T.make_model(2902, 2402, oracle=oracle)
    if region:  # a few cells of large arrays: the other tile form
        m.xs, m.xe, m.ys, m.ye = region
    rng = np.random.default_rng(3)
    for k, lo, hi in (("sshn_t", -0.3, 0.3), ("un", -0.1, 0.1), ("vn", -0.1, 0.1),
                      ("hu", 90, 110), ("hv", 90, 110), ("ssha_u", 0, 1), ("ssha_v", 0, 1)):
        m.f[k][:] = rng.uniform(lo, hi, m.f[k].shape)
    return m


@pytest.mark.parametrize("precision,region", [(0, None), (0, (40, 150, 60, 140)), (2, None)])
def test_registration_without_room_for_the_depth_sums(gpulib, oracle, precision, region):
    import torch
    start = problem(oracle, region)
    points = start.width * start.height
    arrays = 31 * 8 * points + 4 * points  # FP64 arrays and the mask

    def go():
        m = start.copy()
        gpulib.nl2d_set_precision(precision)
        free = torch.cuda.mem_get_info()[0]
        T.gpu_register(gpulib, m)
        taken = free - torch.cuda.mem_get_info()[0]
        out = np.zeros(3)
        import psyclonebench_gb300 as P
        P.check(gpulib.nl2d_run_steps(1, 3, 0, T.dptr(out)), "run")
        T.gpu_read_all(gpulib, m)
        gpulib.nl2d_finalize()
        gpulib.nl2d_set_precision(0)
        return m, taken

    want, taken = go()
    assert taken > arrays + 15 * points  # with the sums: 16 bytes per point more
    # FP64: room for the arrays alone; FP64-equivalent: and for that form's
    with Filled(arrays + (44 * points if precision else 8 * points) + 16 * MB):
        got, taken = go()
    assert taken < arrays + 8 * points
    bad = [k for k in T.FIELDS if not bits_equal(got.f[k], want.f[k])]
    assert not bad, bad
    if precision == 0:
        T.run(oracle.oracle_invoke_time_step, start, 3)
        assert all(bits_equal(got.f[k], start.f[k]) for k in ("sshn_t", "un", "vn"))


def test_tracer_without_room_for_the_courant_factors(gpulib, oracle):
    import torch
    from test_gpu_tra_adv import gpu_compute, gpu_field, oracle_field
    from test_tra_oracle import random_inputs
    f = random_inputs(300, 200, 40, seed=5)
    size = f["mydomain"].nbytes

    def go():
        free = torch.cuda.mem_get_info()[0]
        gpu_compute(gpulib, f, 3)
        taken = free - torch.cuda.mem_get_info()[0]
        got = gpu_field(gpulib, f["mydomain"].shape)
        gpulib.tra_adv_finalize()
        return got, taken

    want, taken = go()
    assert taken > 11 * size
    with Filled(11 * size + 16 * MB):  # nine fields and what the registration needs for a while
        got, taken = go()
    assert taken < 10 * size
    np.testing.assert_array_equal(got.view(np.int64), want.view(np.int64))
    np.testing.assert_array_equal(got.view(np.int64), oracle_field(f, 3).view(np.int64))
