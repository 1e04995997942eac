"""The weight gradient of inputs with infinities and NaN: non-finite where the
sum over the pixels is (zero padding counted as zeros), finite and equal
elsewhere, at the image's edges above all."""
import pytest

pytestmark = pytest.mark.gpu

INF = float("inf")


@pytest.mark.parametrize("batch,h,w,cin,cout", [
    (1, 1, 128, 16, 8), (2, 37, 256, 32, 48), (3, 153, 128, 48, 64),  # rows stacked in pairs
    (1, 20, 128, 48, 72),                                             # single rows
])
@pytest.mark.parametrize("where", ["x", "dy"])
def test_gradient_of_non_finite_inputs(gpulib, batch, h, w, cin, cout, where):
    import torch
    g = torch.Generator(device="cuda").manual_seed(batch + h + cin + cout)
    x = torch.randint(-2, 3, (batch, h, w, cin), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randint(1, 4, (batch, h, w, cout), generator=g, device="cuda").to(torch.bfloat16)
    odd = x if where == "x" else dy
    # a channel each: the image's first and last row and column, inside, NaN, zeros beside
    odd[0, 0, 5, 0] = INF
    odd[-1, h - 1, 70, 1] = -INF
    odd[0, h // 2, 0, 2] = INF
    odd[-1, h // 2, w - 1, 3] = -INF
    odd[0, h // 3, w // 2, 4] = INF
    odd[0, h // 4, 9, 5] = float("nan")
    if where == "x":
        dy[-1, h - 1, 70, 7] = 0.0  # 0 x inf
    dw = torch.full((9, cout, cin), 3.0, device="cuda")
    db = torch.full((cout,), -1.0, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert gpulib.nl2d_emu_conv_wgrad(x.data_ptr(), dy.data_ptr(), dw.data_ptr(), db.data_ptr(),
                                      batch, h, w, cin, cout, err.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    p = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    d = dy.double()
    for t in range(9):
        xs = p[:, t // 3:t // 3 + h, t % 3:t % 3 + w]
        want = torch.stack([(d[..., c:c + 1] * xs).sum((0, 1, 2)) for c in range(cout)]) + 3.0
        got = dw[t].double()
        bad = ~((got == want) | (got.isnan() & want.isnan()))
        assert not bool(bad.any()), (t, got[bad][:8], want[bad][:8])
    want = d.sum((0, 1, 2)) - 1.0
    assert bool(((db.double() == want) | (db.isnan() & want.isnan())).all())
