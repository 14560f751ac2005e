"""Mixed batches of sizes whose tuning entry asks for the fast-twiddle form:
every schedule gives the same bits, and complex orders up to 13 the plain
form's (in FP32 the oracle's)."""
import numpy as np
import pytest

import zldsp_fft_b200 as Z
from tests.test_gpu_mixed import Packed, _oracle, _run, _single

pytestmark = pytest.mark.gpu


@pytest.fixture
def fast_entries(tmp_path):
    """A tuning table that picks the fast form for every size used here."""
    import torch
    prop = torch.cuda.get_device_properties(0)
    lines = [f"gpu {prop.name.replace(' ', '_')} sms {prop.multi_processor_count}"]
    for kind in (0, 1):
        for prec in (0, 1):
            for order in range(9, 17):
                lines.append(f"entry {kind} {prec} {order} 0 2 1 {Z.MODE_FAST} 0 -1 0 0")
    path = tmp_path / "fast.txt"
    path.write_text("\n".join(lines) + "\n")
    Z.tuning_clear()
    assert Z.tuning_load(str(path)) == len(lines) - 1
    yield
    Z.tuning_clear()


def test_schedules_agree_and_small_orders_stay_plain(oracle, fast_entries):
    rng = np.random.default_rng(9100)
    specs = []
    for prec in (Z.F32, Z.F64):
        for order in range(10, 16):
            for _ in range(2):
                specs += [(Z.C2C, order, Z.FORWARD, prec), (Z.C2C, order, Z.BACKWARD, prec)]
                specs += [(Z.R2C, order, op, prec) for op in (Z.FORWARD, Z.BACKWARD, Z.FORWARD_SQR_MAG)]
    pk = Packed(rng, specs)
    res = {s: _run(pk, s)[1] for s in (Z.SCHED_PER_ORDER, Z.SCHED_PERSISTENT, Z.SCHED_GRAPH)}
    for s in (Z.SCHED_PERSISTENT, Z.SCHED_GRAPH):
        for i, spec in enumerate(specs):
            assert np.array_equal(res[s][i], res[Z.SCHED_PER_ORDER][i]), (s, spec)
    for i, spec in enumerate(specs):
        kind, order, _, prec = spec
        if order - (kind == Z.R2C) > 13:
            continue
        assert np.array_equal(res[Z.SCHED_GRAPH][i], _single(spec, pk.x[i])), spec  # (a plain plan of that size)
        if prec == Z.F32:
            assert np.array_equal(res[Z.SCHED_GRAPH][i], _oracle(oracle, spec, pk.x[i])), spec
