"""Tuning a batch whose instances are all held times nothing and changes
nothing: the tiling stays and later steps still replay a CUDA graph."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_tune_with_every_instance_held(ctx, precision):
    from cfd_gb300 import cases, runtime
    c = cases.taylor_green(n=12)
    b = runtime.Batch(ctx, precision)
    slot = b.add(c)
    b.step(1)
    before = b.info()
    assert before.graph
    b.set_hold(slot, True)
    b.tune(1)
    b.set_hold(slot, False)
    b.step(1)
    after = b.info()
    assert after.graph and after.tile_nodes == before.tile_nodes
    other = runtime.Batch(ctx, precision)
    s = other.add(c)
    other.step(2)
    assert np.array_equal(other.get_flow(s), b.get_flow(slot))
    b.close()
    other.close()
