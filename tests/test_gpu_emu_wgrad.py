"""The weight-gradient kernel on the shapes where its two forms (rows stacked
in pairs up to 64 output channels, single rows above), its ring and its row
shares change: against the sum in float64."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,h,w,cin,cout", [
    (1, 1, 128, 16, 8),      # one row: both neighbours outside the image
    (1, 3, 128, 48, 16),     # fewer rows than the ring has slots
    (2, 37, 256, 32, 48),    # two columns of pixels, shares that cut columns
    (3, 153, 128, 48, 64),   # the widest pair, more rows than CTAs
    (1, 20, 128, 48, 72),    # the narrowest single-row form
    (2, 9, 256, 48, 128),    # four slots, two rows in flight
    (1, 700, 128, 16, 24),   # several rows per CTA in one column
])
def test_weight_gradient_shapes(gpulib, batch, h, w, cin, cout):
    import torch
    g = torch.Generator(device="cuda").manual_seed(batch * 1000 + h * 10 + cin + cout)
    x = torch.randn(batch, h, w, cin, generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(batch, h, w, cout, generator=g, device="cuda").to(torch.bfloat16)
    dw = torch.full((9, cout, cin), 0.5, device="cuda")  # the gradient is added
    db = torch.full((cout,), -1.0, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert gpulib.nl2d_emu_conv_wgrad(x.data_ptr(), dy.data_ptr(), dw.data_ptr(), db.data_ptr(),
                                      batch, h, w, cin, cout, err.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    p = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    d = dy.double().reshape(-1, cout)
    want = torch.stack([d.t() @ p[:, t // 3:t // 3 + h, t % 3:t % 3 + w].reshape(-1, cin)
                        for t in range(9)])
    # every product of BF16 pairs is exact in FP32; n additions in FP32 lose at
    # most n 2^-24 of the sum of magnitudes (a generous bound for any order)
    n = batch * h * w
    mag = torch.stack([d.abs().t() @ p[:, t // 3:t // 3 + h, t % 3:t % 3 + w].reshape(
        -1, cin).abs() for t in range(9)])
    assert bool(((dw.double() - 0.5 - want).abs() <= (n + 200) * 2.0 ** -24 * (mag + 1)).all())
    assert bool(((db.double() + 1.0 - d.sum(0)).abs() <=
                 (n + 200) * 2.0 ** -24 * (d.abs().sum(0) + 1)).all())
