"""Inverse STFT of few frames without overlap: CTAs of one group each. The
sequential loop's bits on both sides of the rule (one wave of groups, one frame
each), with and without filter and window, AoS and split bins."""
import numpy as np
import pytest

import zldsp_fft_b200 as Z
from tests import gpu_util as G

pytestmark = pytest.mark.gpu
# groups per SM of the kernel that shares its tables, by (frame order, precision)
GROUPS = {(10, "f32"): 21, (11, "f32"): 10, (12, "f32"): 5, (13, "f32"): 2, (14, "f32"): 1, (11, "f64"): 7}


def _frames(oracle, plan, bins, filt, win, n, prec):
    """Each frame by itself through the plan's backward transform, filtered and windowed."""
    x = bins if filt is None else bins.astype(bins.dtype)
    if filt is not None:  # products rounded operation by operation
        re = x.real * filt.real - x.imag * filt.imag
        im = x.real * filt.imag + x.imag * filt.real
        x = (re + 1j * im).astype(bins.dtype)
    y = oracle.rfft_backward_port(x) if prec == "f32" else G.run_c2r(plan, x)
    return y if win is None else y * win


@pytest.mark.parametrize("order,prec", list(GROUPS))
@pytest.mark.parametrize("extras,layout", [(False, Z.AOS), (True, Z.AOS), (True, Z.SOA)])
def test_bits_on_both_sides(oracle, order, prec, extras, layout):
    import torch
    dt = np.float32 if prec == "f32" else np.float64
    cdt = np.complex64 if prec == "f32" else np.complex128
    n = 1 << order
    nb = n // 2 + 1
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    full = sms * GROUPS[order, prec]
    rng = np.random.default_rng(9400 + order)
    plan = Z.Plan(Z.R2C, order, dt)
    filt = (rng.uniform(-1, 1, nb) + 1j * rng.uniform(-1, 1, nb)).astype(cdt) if extras else None
    win = rng.uniform(0, 1, n).astype(dt) if extras else None
    fd, wd = (None if a is None else G.dev(a.view(dt)) for a in (filt, win))
    for count in sorted({1, 3, full // 2 + 1, full, full + 1}):
        bins = (rng.uniform(-1, 1, (count, nb)) + 1j * rng.uniform(-1, 1, (count, nb))).astype(cdt)
        if layout == Z.AOS:
            a, b = G.dev(bins.view(dt)), None
        else:
            a, b = G.dev(np.ascontiguousarray(bins.real)), G.dev(np.ascontiguousarray(bins.imag))
        out = torch.full((count * n + 2,), 7.0, dtype=a.dtype, device="cuda")
        plan.istft(layout, a.data_ptr(), None if b is None else b.data_ptr(), n, count, out.data_ptr(),
                   filter=None if fd is None else fd.data_ptr(), window=None if wd is None else wd.data_ptr())
        got = G.host(out)
        assert np.all(got[count * n:] == 7.0)
        rows = sorted({0, count // 2, count - 1})
        want = _frames(oracle, plan, bins[rows], filt, win, n, prec)
        if prec == "f32":
            assert np.array_equal(got[:count * n].reshape(count, n)[rows], want), count
        else:
            assert oracle.rel_l2(got[:count * n].reshape(count, n)[rows], want).max() <= oracle.tolerance(order, prec)
    # one frame, overlapping hop: each block of the output is a run of its own
    bins = (rng.uniform(-1, 1, (1, nb)) + 1j * rng.uniform(-1, 1, (1, nb))).astype(cdt)
    a = G.dev(bins.view(dt))
    out = torch.full((n,), 7.0, dtype=a.dtype, device="cuda")
    plan.istft(Z.AOS, a.data_ptr(), None, n // 4, 1, out.data_ptr())
    if prec == "f32":
        assert np.array_equal(G.host(out), oracle.rfft_backward_port(bins)[0])
    assert plan.device_status() == 0
