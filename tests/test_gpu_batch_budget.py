"""The FP64 batch's face scratch lives in the batch's budget: what the
instances leave of capacity_bytes, whatever is added or removed, with the
same bits, and it is given back."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLACK = 40 << 20   # tables and the allocator's granularity


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


def test_scratch_stays_within_the_budget(ctx):
    from cfd_gb300 import cases, runtime
    c = cases.taylor_green(n=64)
    need = runtime.Batch.instance_bytes(0, c.sd_node)
    ample = runtime.Batch(ctx, 0)
    slot = ample.add(c)
    ample.step(1)
    want = ample.get_flow(slot)
    ample.close()

    before = _free()
    b = runtime.Batch(ctx, 0, capacity_bytes=3 * need)
    slots = [b.add(c)]
    b.step(1)                                    # one instance: a round of everything fits
    assert before - _free() <= 3 * need + SLACK
    slots += [b.add(c) for _ in range(2)]        # the budget is full: the scratch gives way
    assert before - _free() <= 3 * need + SLACK
    for s in slots:
        b.set_flow(s, c.arrays["flow"])
    b.step(1)
    assert before - _free() <= 3 * need + SLACK
    assert b.info().device_bytes == 3 * need
    for s in slots:
        assert np.array_equal(b.get_flow(s), want)
    for s in slots:
        b.remove(s)
    assert before - _free() <= SLACK
    b.close()


@pytest.mark.parametrize("shape", [(5, 4, 3), (33, 29, 31)])
def test_a_budget_filled_to_the_last_byte(ctx, shape):
    from cfd_gb300 import cases, runtime
    c = cases.isentropic_vortex(shape=shape)
    need = runtime.Batch.instance_bytes(0, c.sd_node)
    got = []
    for capacity in (0, 2 * need):
        b = runtime.Batch(ctx, 0, capacity_bytes=capacity)
        slots = [b.add(c) for _ in range(2)]
        b.step(2)
        got.append([b.get_flow(s) for s in slots])
        b.close()
    for x, y in zip(*got):
        assert np.array_equal(x, y)
