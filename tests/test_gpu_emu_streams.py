"""Weight gradients on several streams and threads at once: each call's partial
sums are its own, so the bits are those of the calls made one after another."""
import threading

import pytest

pytestmark = pytest.mark.gpu

# more streams than keep a buffer of their own
SHAPES = [(2, 96, 128, 48, 48), (3, 40, 256, 16, 64), (2, 30, 128, 48, 128)] * 2


def _inputs(shape):
    import torch
    batch, h, w, cin, cout = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.randn(batch, h, w, cin, generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(batch, h, w, cout, generator=g, device="cuda").to(torch.bfloat16)
    return x, dy


def _gradient(lib, shape, x, dy, stream):
    import torch
    batch, h, w, cin, cout = shape
    dw = torch.zeros(9, cout, cin, device="cuda")
    db = torch.zeros(cout, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert lib.nl2d_emu_conv_wgrad(x.data_ptr(), dy.data_ptr(), dw.data_ptr(), db.data_ptr(),
                                   batch, h, w, cin, cout, err.data_ptr(), stream) == 0
    return dw, db, err


def _same(got, want):
    import torch
    return all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("threads", [False, True])
def test_gradients_on_several_streams(gpulib, threads):
    import torch
    inputs = [_inputs(s) for s in SHAPES]
    want = [_gradient(gpulib, s, x, dy, None) for s, (x, dy) in zip(SHAPES, inputs)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in SHAPES]
    got = [[] for _ in SHAPES]

    def call(k):
        with torch.cuda.stream(streams[k]):
            got[k].append(_gradient(gpulib, SHAPES[k], *inputs[k], streams[k].cuda_stream))

    if threads:
        def many(k):
            for _ in range(20):
                call(k)
        ts = [threading.Thread(target=many, args=(k,)) for k in range(len(SHAPES))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    else:
        for _ in range(20):
            for k in range(len(SHAPES)):
                call(k)
    torch.cuda.synchronize()
    for k in range(len(SHAPES)):
        assert len(got[k]) == 20
        assert int(want[k][2].item()) == 0 and float(want[k][0].abs().max()) > 0
        assert all(_same(r, want[k]) for r in got[k])


def test_gradient_in_a_captured_graph(gpulib):
    import torch
    shape = SHAPES[0]
    x, dy = _inputs(shape)
    want = _gradient(gpulib, shape, x, dy, None)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _gradient(gpulib, shape, x, dy, torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        graph.replay()
        torch.cuda.synchronize()
        assert _same(got, want)
