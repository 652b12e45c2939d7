"""A CUDA error that other code left pending on the thread (a refused
allocation, say) is not a batch's: its steps run and replay a graph."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _leave_an_error_pending(ctx):
    from cfd_gb300 import abi
    with pytest.raises(abi.CfdError) as e:
        ctx.alloc(1 << 46)                       # 64 TB
    assert e.value.status == abi.ENOMEM


def _take_it_back(ctx, c):
    """cfd_batch_add reports and clears whatever is pending."""
    from cfd_gb300 import abi, runtime
    b = runtime.Batch(ctx, 1)
    try:
        b.add(c)
    except abi.CfdError:
        pass
    b.close()


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_steps_after_a_refused_allocation(ctx, precision, use_graph):
    from cfd_gb300 import cases, runtime
    c = cases.taylor_green(n=16)                 # whole tiles
    out = []
    for pending in (False, True):
        b = runtime.Batch(ctx, precision)
        slot = b.add(c)
        b.set_tiling(0, 0, use_graph)
        if pending:
            _leave_an_error_pending(ctx)
        try:
            b.step(1)
        finally:
            _take_it_back(ctx, c)
        assert b.info().graph == use_graph
        out.append(b.get_flow(slot))
        b.close()
    assert np.array_equal(*out)
