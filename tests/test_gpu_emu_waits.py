"""The convolution kernels whose roles' waits for one another run out: the
launch ends, says so, and leaves the GPU as it was.  With limits from none to
far above what a row takes, the wait that gives up first is another one each
time, in the middle of rows that other warps and lanes have finished."""
import pytest

pytestmark = pytest.mark.gpu

LIMITS = [0, 50, 200, 500, 1000, 2000, 4000, 8000, 20000, 100000]


@pytest.mark.parametrize("wgrad,cin,cout", [(0, 16, 16), (0, 48, 48), (0, 64, 64),
                                            (1, 16, 24), (1, 48, 48), (1, 48, 128)])
def test_waits_that_run_out(gpulib, wgrad, cin, cout):
    import torch
    batch, h, w = 2, 1216, 128  # 16 rows per CTA: every ring turns
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn(batch, h, w, cin, generator=g, device="cuda").to(torch.bfloat16)
    shape = (batch, h, w, cout) if wgrad else (9, cout, cin)
    b = (torch.randn(shape, generator=g, device="cuda") * 0.1).to(torch.bfloat16)

    def launch(limit):
        out = torch.zeros((9, cout, cin) if wgrad else (batch, h, w, cout), device="cuda")
        db = torch.zeros(cout, device="cuda")
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        assert gpulib.nl2d_selftest_emu_wait(wgrad, x.data_ptr(), b.data_ptr(), out.data_ptr(),
                                             db.data_ptr(), batch, h, w, cin, cout, limit,
                                             err.data_ptr()) == 0
        torch.cuda.synchronize()
        return out, db, int(err.item())

    out, db, err = launch(1 << 31)
    assert err == 0
    codes = []
    for limit in LIMITS:
        o, d, code = launch(limit)
        codes.append(code)
        if code == 0:
            assert torch.equal(o, out) and torch.equal(d, db)
    assert codes[0] == 1 and set(codes) <= {0, 1}
    o, d, code = launch(1 << 31)
    assert code == 0 and torch.equal(o, out) and torch.equal(d, db)
