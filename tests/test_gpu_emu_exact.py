"""The convolution and the weight gradient on small whole numbers, whose
products and sums FP32 holds exactly: every row and tap counted once gives
equality, a lost or doubled one does not.  Batches long enough that each
CTA's rings turn several times."""
import pytest

pytestmark = pytest.mark.gpu


def _whole(shape, g):
    import torch
    return torch.randint(-2, 3, shape, generator=g, device="cuda").to(torch.bfloat16)


# rows per SM: 28 and more (8 slots paired, 4 slots of single rows)
@pytest.mark.parametrize("batch,h,w,cin,cout", [
    (1, 1, 128, 16, 8), (2, 37, 256, 32, 48), (3, 153, 128, 48, 64), (1, 700, 128, 16, 24),
    (1, 20, 128, 48, 72),
    (17, 251, 128, 48, 64),   # paired, columns cut between CTAs
    (9, 239, 256, 16, 16),    # paired, the narrowest
    (17, 251, 128, 48, 128),  # single rows, the fewest slots
    (9, 239, 256, 32, 72),
])
def test_weight_gradient_counts_every_row_once(gpulib, batch, h, w, cin, cout):
    import torch
    g = torch.Generator(device="cuda").manual_seed(batch + h + cin + cout)
    x, dy = _whole((batch, h, w, cin), g), _whole((batch, h, w, cout), g)
    assert 4 * batch * h * w < 2 ** 24  # no partial sum leaves FP32's whole numbers
    dw = torch.full((9, cout, cin), 3.0, device="cuda")
    db = torch.full((cout,), -1.0, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert gpulib.nl2d_emu_conv_wgrad(x.data_ptr(), dy.data_ptr(), dw.data_ptr(), db.data_ptr(),
                                      batch, h, w, cin, cout, err.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    p = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    d = dy.double().reshape(-1, cout)
    for t in range(9):
        want = d.t() @ p[:, t // 3:t // 3 + h, t % 3:t % 3 + w].reshape(-1, cin)
        assert torch.equal(dw[t].double() - 3.0, want)
    assert torch.equal(db.double() + 1.0, d.sum(0))


@pytest.mark.parametrize("batch,h,w,cin,cout", [
    (1, 1, 128, 16, 16), (17, 251, 128, 48, 48), (9, 239, 256, 64, 64), (9, 239, 256, 16, 32),
])
def test_convolution_counts_every_tap_once(gpulib, batch, h, w, cin, cout):
    import torch
    g = torch.Generator(device="cuda").manual_seed(batch + h + cin + cout)
    x, k = _whole((batch, h, w, cin), g), _whole((9, cout, cin), g)
    y = torch.empty(batch, h, w, cout, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert gpulib.nl2d_emu_conv3x3(x.data_ptr(), k.data_ptr(), None, None, y.data_ptr(), batch, h,
                                   w, cin, cout, 0, err.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    p = torch.nn.functional.pad(x.float(), (0, 0, 1, 1, 1, 1))
    want = torch.zeros(batch, h, w, cout, dtype=torch.float64, device="cuda")
    for t in range(9):
        want += p[:, t // 3:t // 3 + h, t % 3:t % 3 + w].double() @ k[t].double().t()
    assert torch.equal(y.double(), want)
