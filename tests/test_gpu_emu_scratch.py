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


@pytest.mark.parametrize("other", [False, True])
def test_scratch_made_during_a_capture(gpulib, other):
    """After calls on one stream: the first captured one, or (other) one on a
    new stream while another captures."""
    import torch
    batch, h, w, cin, cout = 2, 96, 128, 48, 48
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randint(-2, 3, (batch, h, w, cin), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randint(-2, 3, (batch, h, w, cout), generator=g, device="cuda").to(torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    sums = [(torch.zeros(9, cout, cin, device="cuda"), torch.zeros(cout, device="cuda"))
            for _ in range(3)]
    here, beside = torch.cuda.Stream(), torch.cuda.Stream()

    def gradient(k, stream):
        assert gpulib.nl2d_emu_conv_wgrad(x.data_ptr(), dy.data_ptr(), sums[k][0].data_ptr(),
                                          sums[k][1].data_ptr(), batch, h, w, cin, cout,
                                          err.data_ptr(), stream.cuda_stream) == 0

    torch.cuda.synchronize()
    gpulib.nl2d_finalize()
    gradient(0, here)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        if other:
            gradient(2, beside)
            sums[1][0].add_(1.0)
        else:
            gradient(1, torch.cuda.current_stream())
    gpulib.nl2d_finalize()  # a graph's memory is its own
    graph.replay()
    torch.cuda.synchronize()
    assert int(err.item()) == 0 and float(sums[0][0].abs().max()) > 0
    if other:
        assert torch.equal(sums[1][0], torch.ones_like(sums[1][0]))
    for a, b in zip(sums[0], sums[2 if other else 1]):
        assert torch.equal(a, b)
