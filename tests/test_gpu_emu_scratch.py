"""The weight gradients' scratch, kept between calls, is given back by
nl2d_finalize; calls after it are as before."""
import pytest

pytestmark = pytest.mark.gpu

SHAPE = (152, 4, 128, 48, 128)  # 34 MB of partial sums on 152 SMs


def test_finalize_gives_the_scratch_back(gpulib):
    import torch
    batch, h, w, cin, cout = SHAPE
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randint(-2, 3, (batch, h, w, cin), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randint(-2, 3, (batch, h, w, cout), generator=g, device="cuda").to(torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    dw = torch.zeros(9, cout, cin, device="cuda")
    db = torch.zeros(cout, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(6)]

    def gradient(stream):
        assert gpulib.nl2d_emu_conv_wgrad(x.data_ptr(), dy.data_ptr(), dw.data_ptr(),
                                          db.data_ptr(), batch, h, w, cin, cout, err.data_ptr(),
                                          stream) == 0

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    def on_all_streams():  # four keep a buffer each, two share the pool
        for s in streams:
            dw.zero_()
            db.zero_()
            torch.cuda.synchronize()
            gradient(s.cuda_stream)
            torch.cuda.synchronize()
            assert torch.equal(dw, want[0]) and torch.equal(db, want[1])

    gpulib.nl2d_finalize()
    gradient(None)
    torch.cuda.synchronize()
    want = dw.clone(), db.clone()
    assert int(err.item()) == 0 and float(want[0].abs().max()) > 0
    on_all_streams()
    gpulib.nl2d_finalize()
    before = free()
    on_all_streams()
    assert before - free() > 100e6
    gpulib.nl2d_finalize()
    assert before - free() < 8e6
