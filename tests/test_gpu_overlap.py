"""Launches that overlap the kernel before them: a call in a chain of calls takes
no longer than the same call with a memset between (which lets nothing
overlap), and gives the same bits, also where the CTAs ask for an even share of
an SM's shared memory or a pass begins only when the one before it is done."""
import numpy as np
import pytest

import zldsp_fft_b200 as Z
from tests import gpu_util as G

pytestmark = pytest.mark.gpu


def _us_per_call(run, between):
    import torch
    flag = torch.zeros(64, device="cuda")
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        run(st.cuda_stream)
        flag.zero_()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        for _ in range(24):
            if between:
                flag.zero_()
            run(torch.cuda.current_stream().cuda_stream)
    times = []
    for _ in range(12):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        graph.replay()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b) * 1e3 / 24)
    return sorted(times)[5]


@pytest.mark.parametrize("kind,order,dtype,batch", [
    (Z.C2C, 19, np.float32, 1),     # one item per SM and less
    (Z.C2C, 18, np.float32, 2), (Z.C2C, 16, np.float32, 8), (Z.C2C, 15, np.float64, 8),
    (Z.C2C, 9, np.float32, 1040),   # 260 tiles: two on most SMs
    (Z.C2C, 6, np.float32, 296 * 32),
    (Z.R2C, 16, np.float64, 8)])    # split or pre-step between the passes
def test_chained_call_is_not_slower_than_alone(kind, order, dtype, batch):
    import torch
    n = 1 << order
    dt = torch.float32 if dtype == np.float32 else torch.float64
    plan = Z.Plan(kind, order, dtype)
    x = torch.rand(batch * (2 * n if kind == Z.C2C else n), dtype=dt, device="cuda")
    y = torch.zeros(batch * (2 * n if kind == Z.C2C else n + 2), dtype=dt, device="cuda")

    def run(st):
        plan.exec_device(Z.FORWARD, Z.AOS, Z.AOS, x.data_ptr(), None, y.data_ptr(), None, batch, stream=st)
    chained, alone = _us_per_call(run, False), _us_per_call(run, True)
    assert chained <= alone, (chained, alone)


# grids of three CTAs per SM where more would fit, of a few ragged waves, of single items
@pytest.mark.parametrize("kind,order,batch", [
    (Z.C2C, 6, 444 * 32 - 5), (Z.C2C, 9, 370 * 4 - 1), (Z.C2C, 11, 440), (Z.R2C, 12, 400), (Z.R2C, 7, 443 * 32 + 3),
    (Z.C2C, 16, 16), (Z.C2C, 16, 40), (Z.C2C, 19, 5), (Z.C2C, 21, 1), (Z.R2C, 19, 2), (Z.R2C, 17, 9),
    (Z.C2C, 8, 1184 * 8 - 1), (Z.R2C, 7, 888 * 32 + 1),  # short tiles, a second wave not full
    (Z.C2C, 16, 300), (Z.R2C, 18, 200)])                 # more than two chunks on two streams
def test_bits_of_chained_calls(oracle, kind, order, batch):
    """Each call reads what the one before wrote, with nothing between them;
    the inputs change from round to round, so a call that reads too early finds
    other values than those it should."""
    import torch
    n = 1 << order
    rng = np.random.default_rng(9200 + order)
    plan = Z.Plan(kind, order, np.float32)
    ins = [torch.from_numpy(rng.uniform(-1, 1, (batch, 2 * n if kind == Z.C2C else n)).astype(np.float32)).cuda()
           for _ in range(3)]
    bins = [torch.full((batch, 2 * n if kind == Z.C2C else n + 2), 7.0, device="cuda") for _ in range(2)]
    outs = [torch.zeros_like(ins[0]) for _ in range(3)]
    torch.cuda.synchronize()
    st = torch.cuda.current_stream().cuda_stream
    for i in range(3):  # bins[0], bins[1] and bins[0] again: other values each time
        plan.exec_device(Z.FORWARD, Z.AOS, Z.AOS, ins[i].data_ptr(), None, bins[i & 1].data_ptr(), None, batch, stream=st)
        plan.exec_device(Z.BACKWARD, Z.AOS, Z.AOS, bins[i & 1].data_ptr(), None, outs[i].data_ptr(), None, batch, stream=st)
    torch.cuda.synchronize()
    rows = sorted({0, batch // 3, batch - 1})
    for i in range(3):
        x = G.host(ins[i])[rows]
        if kind == Z.C2C:
            want = oracle.cfft_port(oracle.cfft_port(x.view(np.complex64), True), False).view(np.float32)
        else:
            want = oracle.rfft_backward_port(oracle.rfft_forward_port(x))
        assert np.array_equal(G.host(outs[i])[rows], want), i
    assert plan.device_status() == 0
