"""Squared magnitudes and STFT frames with one or two transforms per thread, by
the size of the batch: the oracle's bits on both sides of each line and with a
last tile that is not full."""
import numpy as np
import pytest

import zldsp_fft_b200 as Z
from tests import gpu_util as G

pytestmark = pytest.mark.gpu


def _lines(order):
    """Batches on both sides of the rule's lines: tiles that fill the GPU with
    one transform per thread (5 CTAs of 128 threads per SM), and with two (4)."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per_tile = 128 // ((1 << (order - 1)) // 16)
    one, two = 5 * sms * per_tile, 8 * sms * per_tile
    return [1, per_tile + 1, one, one + 1, two - 1, two + 1, 2 * one + 3]


@pytest.mark.parametrize("order", [10, 11, 12])
def test_bits_on_both_sides_of_the_lines(oracle, order):
    import torch
    n, nb = 1 << order, (1 << order) // 2 + 1
    rng = np.random.default_rng(9300 + order)
    plan = Z.Plan(Z.R2C, order, np.float32)
    big = max(_lines(order))
    x = rng.uniform(-1, 1, (big, n)).astype(np.float32)
    xd = G.dev(x)
    win = rng.uniform(0, 1, n).astype(np.float32)
    wd, hop = G.dev(win), n // 4
    flat = x.reshape(-1)
    for batch in _lines(order):
        rows = sorted({0, batch // 2, max(0, batch - 2), batch - 1})
        sq = torch.full((batch + 1, nb), 7.0, device="cuda")
        plan.exec_device(Z.FORWARD_SQR_MAG, Z.AOS, Z.AOS, xd.data_ptr(), None, sq.data_ptr(), None, batch)
        assert np.array_equal(G.host(sq)[rows], oracle.rfft_forward_port(x[rows], sqr_mag=True)), batch
        assert bool((sq[batch] == 7.0).all())
        frames = np.stack([flat[r * hop:r * hop + n] * win for r in rows])
        for op in (Z.FORWARD_SQR_MAG, Z.FORWARD):
            c = 1 if op == Z.FORWARD_SQR_MAG else 2
            out = torch.full((batch + 1, nb * c), 7.0, device="cuda")
            plan.stft(op, Z.AOS, xd.data_ptr(), hop, wd.data_ptr(), out.data_ptr(), None, batch)
            got = G.host(out)
            want = oracle.rfft_forward_port(frames, sqr_mag=c == 1)
            assert np.array_equal(got[rows] if c == 1 else got.view(np.complex64)[rows], want), (batch, op)
            assert bool((got[batch] == 7.0).all())
    assert plan.device_status() == 0
