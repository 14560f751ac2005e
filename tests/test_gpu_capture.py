"""Launches that overlap the kernel before them (programmatic dependent launch)
recorded into a CUDA graph: the replay must give the direct call's bits, from
fresh inputs, for one tile launch after another, for multi-pass pipelines with
and without forked lanes, for the RFFT's split and pre-step, and for the STFT
and its inverse."""
import numpy as np
import pytest

import zldsp_fft_b200 as Z

pytestmark = pytest.mark.gpu


def _chain(kind, order, batch):
    """(run, inputs, outputs): forward then backward of `batch` transforms."""
    import torch
    n = 1 << order
    plan = Z.Plan(kind, order, np.float32)
    if kind == Z.C2C:
        x, y, z = (torch.zeros((batch, n, 2), device="cuda") for _ in range(3))
    else:
        x, z = (torch.zeros((batch, n), device="cuda") for _ in range(2))
        y = torch.zeros((batch, n // 2 + 1, 2), device="cuda")

    def run(st):
        plan.exec_device(Z.FORWARD, Z.AOS, Z.AOS, x.data_ptr(), None, y.data_ptr(), None, batch, stream=st)
        plan.exec_device(Z.BACKWARD, Z.AOS, Z.AOS, y.data_ptr(), None, z.data_ptr(), None, batch, stream=st)
    return run, [x], [y, z], plan


def _stft_chain():
    import torch
    n, hop, frames = 2048, 512, 700
    plan = Z.Plan(Z.R2C, 11, np.float32)
    x = torch.zeros((frames - 1) * hop + n, device="cuda")
    w = torch.hann_window(n, device="cuda")
    y = torch.zeros((frames, n // 2 + 1, 2), device="cuda")
    z = torch.zeros_like(x)

    def run(st):
        plan.stft(Z.FORWARD, Z.AOS, x.data_ptr(), hop, w.data_ptr(), y.data_ptr(), None, frames, stream=st)
        plan.istft(Z.AOS, y.data_ptr(), None, hop, frames, z.data_ptr(), window=w.data_ptr(), stream=st)
    return run, [x], [y, z], (plan, w)


@pytest.mark.parametrize("what", [(Z.C2C, 10, 1), (Z.C2C, 12, 700), (Z.R2C, 12, 33), (Z.C2C, 16, 1), (Z.C2C, 16, 300),
                                  (Z.R2C, 17, 250), (Z.C2C, 20, 2), "stft"])
def test_captured_equals_direct(what):
    import torch
    run, ins, outs, keep = _stft_chain() if what == "stft" else _chain(*what)
    g = torch.Generator(device="cuda").manual_seed(31)

    def fill():
        for t in ins:
            t.copy_(torch.rand(t.shape, generator=g, device="cuda") * 2 - 1)
    fill()
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        run(st.cuda_stream)  # first use: scratch, streams
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        run(torch.cuda.current_stream().cuda_stream)
    for _ in range(3):
        fill()
        for t in outs:
            t.fill_(7)
        graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in outs]
        for t in outs:
            t.fill_(7)
        run(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        for a, b in zip(got, outs):
            assert torch.equal(a, b)


def test_back_to_back_calls_share_scratch():
    """Calls of one plan on one stream, each reading what the one before wrote,
    with no synchronisation between them."""
    import torch
    for kind, order, batch in ((Z.C2C, 11, 900), (Z.C2C, 17, 70), (Z.R2C, 17, 70)):
        run, (x,), (y, z), keep = _chain(kind, order, batch)
        g = torch.Generator(device="cuda").manual_seed(32)
        x.copy_(torch.rand(x.shape, generator=g, device="cuda") * 2 - 1)
        scale = float(1 << (order if kind == Z.C2C else order - 1))
        st = torch.cuda.current_stream().cuda_stream
        run(st)
        torch.cuda.synchronize()
        want = (z / scale).clone()
        for _ in range(20):
            run(st)
            torch.div(z, scale, out=z)
        torch.cuda.synchronize()
        assert torch.equal(z, want)
