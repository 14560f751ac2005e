"""What the autotuner times is what a plan made from the entry runs: the same
number of kernels per call, for batches of more than two chunks (where the
default splits a call into smaller chunks), with and without an entry of the
size in the table, and the default's own rule (chunk 0) among the candidates."""
import ctypes

import numpy as np
import pytest

import zldsp_fft_b200 as Z

pytestmark = pytest.mark.gpu
C = Z._capi


@pytest.fixture(autouse=True)
def _clean_table():
    Z.tuning_clear()
    yield
    Z.tuning_clear()


def _load(tmp_path, kind, prec, order, chunk, streams):
    import torch
    prop = torch.cuda.get_device_properties(0)
    path = tmp_path / "entry.txt"
    path.write_text(f"gpu {prop.name.replace(' ', '_')} sms {prop.multi_processor_count}\n"
                    f"entry {kind} {prec} {order} {chunk} {streams} 1 0 0 -1 0 0\n")
    Z.tuning_clear()
    assert Z.tuning_load(str(path)) == 1


def _timed(kind, prec, order, chunk, streams, batch):
    t = C.Tuning(chunk_mb=chunk, streams=streams, tma=1, form=Z.MODE_PLAIN, split_fused=0, store_tma=-1)
    n = ctypes.c_size_t()
    C.check(C.lib().zlfft_selftest_tune_launches(-1, kind, prec, order, ctypes.byref(t), batch, ctypes.byref(n)))
    return n.value


def _planned(kind, prec, order, batch):
    import torch
    dt = np.float32 if prec == Z.F32 else np.float64
    plan = Z.Plan(kind, order, dt, mode=Z.MODE_TUNED)
    n = 1 << order
    td = torch.float32 if prec == Z.F32 else torch.float64
    x = torch.zeros(batch * (2 * n if kind == Z.C2C else n), dtype=td, device="cuda")
    y = torch.zeros(batch * (2 * n if kind == Z.C2C else n + 2), dtype=td, device="cuda")
    plan.take_launch_count()
    plan.exec_device(Z.FORWARD, Z.AOS, Z.AOS, x.data_ptr(), None, y.data_ptr(), None, batch)
    torch.cuda.synchronize()
    return plan.take_launch_count()


@pytest.mark.parametrize("kind,prec,order", [(Z.C2C, Z.F32, 16), (Z.C2C, Z.F64, 16), (Z.R2C, Z.F32, 18),
                                             (Z.C2C, Z.F32, 20), (Z.C2C, Z.F32, 12)])
@pytest.mark.parametrize("chunk,streams", [(0, 2), (16, 2), (32, 2), (48, 2), (48, 1)])
def test_candidate_and_plan_launch_the_same(tmp_path, kind, prec, order, chunk, streams):
    es = 4 if prec == Z.F32 else 8
    batch = (256 << 20) // (es << (order + (kind == Z.C2C)))
    alone = _timed(kind, prec, order, chunk, streams, batch)
    _load(tmp_path, kind, prec, order, chunk, streams)
    assert _planned(kind, prec, order, batch) == alone
    # another entry of the size does not leak into the candidate
    _load(tmp_path, kind, prec, order, 192 if chunk != 192 else 16, 1)
    assert _timed(kind, prec, order, chunk, streams, batch) == alone


def test_default_rule_is_a_candidate(tmp_path):
    """A plan of an entry with chunk 0 splits its calls as an untuned one does."""
    batch = (256 << 20) // (8 << 16)
    untuned = _planned(Z.C2C, Z.F32, 16, batch)
    _load(tmp_path, Z.C2C, Z.F32, 16, 0, 2)
    assert _planned(Z.C2C, Z.F32, 16, batch) == untuned == _timed(Z.C2C, Z.F32, 16, 0, 2, batch)
    Z.tuning_clear()
    Z.autotune(Z.C2C, 16, 16, np.float32)
    t = Z.tuning(Z.C2C, 16, np.float32)
    assert t["chunk_mb"] in (0, 16, 32, 48, 96, 192) and t["gbs"] >= t["gbs_default"] > 0
