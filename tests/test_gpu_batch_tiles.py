"""The reduced batch's face tiles (FLAT tiles of three widths along i, chosen
by extents) against the solver's: the same bits on extents that pad, wrap
and split them differently."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("shape", [(3, 4, 5), (7, 9, 3), (8, 8, 8), (13, 17, 11), (16, 5, 33), (33, 8, 7), (40, 31, 9),
                                   (64, 6, 6)])
def test_batch_faces_equal_the_solvers(ctx, precision, shape):
    from cfd_gb300 import cases, runtime
    c = cases.taylor_green(shape=shape)
    own = slice(1, c.sd_node + 1)
    s = runtime.Solver(ctx, c, precision=precision)
    s.set_flow(c.arrays["flow"])
    s.step(c.dt, 2)
    want = s.get_flow()[own]
    s.close()
    b = runtime.Batch(ctx, precision)
    slots = [b.add(c) for _ in range(2)]
    b.step(2)
    for slot in slots:
        assert np.array_equal(b.get_flow(slot)[own], want)
    b.close()
