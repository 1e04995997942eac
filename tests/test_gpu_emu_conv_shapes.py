"""The convolution kernel where its ring of accumulator blocks, its ring of
input rows and its row shares change: every channel count's ring, single rows,
interior columns of pixels, both outputs, outputs on a 16-byte boundary only."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,h,w,cin,cout,relu,outs,offset", [
    (1, 1, 128, 16, 16, 0, "32", 0),       # one row: one output block, no interior tap
    (1, 2, 128, 48, 16, 1, "16", 0),
    (1, 3, 384, 16, 64, 0, "both", 0),     # four blocks; a column with both neighbours
    (2, 7, 256, 64, 64, 1, "both", 8),     # the widest; 16-byte aligned BF16 output
    (1, 41, 128, 32, 32, 0, "32", 4),      # eight blocks; 16-byte aligned FP32 output
    (3, 333, 128, 48, 48, 1, "16", 0),     # shares that cut columns, the ring many times round
    (1, 1300, 128, 16, 48, 0, "32", 0),
])
def test_convolution_shapes(gpulib, batch, h, w, cin, cout, relu, outs, offset):
    import torch
    g = torch.Generator(device="cuda").manual_seed(h * 100 + cin + cout)
    x = torch.randn(batch, h, w, cin, generator=g, device="cuda").to(torch.bfloat16)
    wt = torch.randn(9, cout, cin, generator=g, device="cuda").to(torch.bfloat16)
    bias = torch.randn(cout, generator=g, device="cuda") if relu else None
    n = batch * h * w * cout
    y16 = torch.zeros(n + offset, dtype=torch.bfloat16, device="cuda")[offset:]
    y32 = torch.zeros(n + offset, device="cuda")[offset:]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert gpulib.nl2d_emu_conv3x3(
        x.data_ptr(), wt.data_ptr(), bias.data_ptr() if relu else None,
        y16.data_ptr() if outs != "32" else None, y32.data_ptr() if outs != "16" else None,
        batch, h, w, cin, cout, relu, err.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    p = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    taps = [p[:, t // 3:t // 3 + h, t % 3:t % 3 + w].reshape(-1, cin) for t in range(9)]
    want = sum(t @ wt[k].double().t() for k, t in enumerate(taps))
    mag = sum(t.abs() @ wt[k].double().abs().t() for k, t in enumerate(taps))
    if relu:
        want = (want + bias.double()).relu_()
        mag = mag + bias.double().abs()
    # FP32 accumulation of 9 cin exact products, then one BF16 rounding
    tol = (9 * cin + 2) * 2.0 ** -24 * mag
    if outs != "16":
        assert bool(((y32.double().reshape(want.shape) - want).abs() <= tol).all())
    if outs != "32":
        assert bool(((y16.double().reshape(want.shape) - want).abs() <=
                     tol + want.abs() * 2.0 ** -8).all())
