"""Tile kernels that run two transforms per thread or read their tables from
shared memory: batches around the tile size (a last tile with one of its two
transforms missing), odd strides that rule out bulk copies, and unaligned
bases, against the oracle (FP32 bit for bit) and the FP64 bar."""
import numpy as np
import pytest

import zldsp_fft_b200 as Z
from tests import gpu_util as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [10, 11, 12, 13])
@pytest.mark.parametrize("batch,pad", [(1, 0), (2, 2), (3, 0), (5, 6), (1185, 2)])
def test_rfft_ragged_tiles(oracle, order, batch, pad):
    import torch
    n, nb = 1 << order, (1 << order) // 2 + 1
    rng = np.random.default_rng(8000 + order + batch)
    x = rng.uniform(-1, 1, (batch, n)).astype(np.float32)
    xi = torch.zeros((batch, n + pad), dtype=torch.float32, device="cuda")
    xi[:, :n] = G.dev(x)
    plan = Z.Plan(Z.R2C, order, np.float32)
    sq = torch.full((batch, nb + 1), 7.0, dtype=torch.float32, device="cuda")
    plan.exec_device(Z.FORWARD_SQR_MAG, Z.AOS, Z.AOS, xi.data_ptr(), None, sq.data_ptr(), None, batch, n + pad, nb + 1)
    X = torch.full((batch, nb + 1, 2), 7.0, dtype=torch.float32, device="cuda")
    plan.exec_device(Z.FORWARD, Z.AOS, Z.AOS, xi.data_ptr(), None, X.data_ptr(), None, batch, n + pad, nb + 1)
    back = torch.full((batch, n + pad), 7.0, dtype=torch.float32, device="cuda")
    plan.exec_device(Z.BACKWARD, Z.AOS, Z.AOS, X.data_ptr(), None, back.data_ptr(), None, batch, nb + 1, n + pad)
    torch.cuda.synchronize()
    assert plan.device_status() == 0
    rows = sorted({0, batch // 2, batch - 2 if batch > 1 else 0, batch - 1})
    Xh = G.host(X[:, :nb].contiguous()).view(np.complex64).reshape(batch, nb)
    assert np.array_equal(Xh[rows], oracle.rfft_forward_port(x[rows]))
    assert np.array_equal(G.host(sq)[rows, :nb], oracle.rfft_forward_port(x[rows], sqr_mag=True))
    assert np.array_equal(G.host(back)[rows, :n], oracle.rfft_backward_port(Xh[rows]))
    for t, w in ((sq, nb), (X, nb), (back, n)):  # nothing written past a row
        assert bool((t[:, w:] == 7.0).all())


@pytest.mark.parametrize("order,hop", [(10, 102), (11, 512), (12, 1026), (12, 4096)])
@pytest.mark.parametrize("frames", [1, 2, 7, 1185])
def test_stft_ragged_tiles(oracle, order, hop, frames):
    import torch
    n, nb = 1 << order, (1 << order) // 2 + 1
    rng = np.random.default_rng(8100 + order + frames)
    sig = rng.uniform(-1, 1, (frames - 1) * hop + n).astype(np.float32)
    win = rng.uniform(0, 1, n).astype(np.float32)
    ts, tw = G.dev(sig), G.dev(win)
    plan = Z.Plan(Z.R2C, order, np.float32)
    fr = np.stack([sig[f * hop:f * hop + n] * win for f in range(frames)])
    rows = sorted({0, frames // 2, frames - 1})
    sq = torch.zeros((frames, nb), dtype=torch.float32, device="cuda")
    plan.stft(Z.FORWARD_SQR_MAG, Z.AOS, ts.data_ptr(), hop, tw.data_ptr(), sq.data_ptr(), None, frames)
    X = torch.zeros((frames, nb, 2), dtype=torch.float32, device="cuda")
    plan.stft(Z.FORWARD, Z.AOS, ts.data_ptr(), hop, tw.data_ptr(), X.data_ptr(), None, frames)
    torch.cuda.synchronize()
    assert np.array_equal(G.host(sq)[rows], oracle.rfft_forward_port(fr[rows], sqr_mag=True))
    assert np.array_equal(G.host(X).view(np.complex64).reshape(frames, nb)[rows], oracle.rfft_forward_port(fr[rows]))


@pytest.mark.parametrize("order", [9, 10, 11, 12, 13])
def test_cfft_f64_tables(oracle, order):
    rng = np.random.default_rng(8200 + order)
    n = 1 << order
    x = rng.uniform(-1, 1, (307, 2 * n)).view(np.complex128)
    for mode in (Z.MODE_PLAIN, Z.MODE_FAST):
        plan = Z.Plan(Z.C2C, order, np.float64, mode=mode)
        y = G.run_c2c(plan, x, True)
        assert oracle.rel_l2(y, oracle.cfft_fp64(x)).max() <= oracle.tolerance(order, "f64")
        assert oracle.rel_l2(G.run_c2c(plan, y, False), n * x).max() <= 2 * oracle.tolerance(order, "f64")
