"""The reduced forms' fluxes in one launch (small lattices) against the
kernels they are timed as (profile_stage launches each on its own): the same
arithmetic from other tiles, so the state has the same bits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("name,shape", [("tgv", (7, 5, 6)), ("tgv", (33, 17, 9)), ("vortex", (32, 16, 16)),
                                        ("channel", (18, 12, 7)), ("tgv", (58, 58, 59)), ("tgv", (59, 59, 59))])
def test_one_launch_equals_separate_launches(ctx, precision, name, shape):
    """198,476 and 205,379 nodes lie either side of the line."""
    from cfd_gb300 import cases, runtime
    if name == "tgv":
        c = cases.taylor_green(shape=shape)
    elif name == "vortex":
        c = cases.isentropic_vortex(shape=shape)
    else:
        c = cases.channel(*shape)
    got = []
    for profiled in (False, True):
        s = runtime.Solver(ctx, c, precision=precision)
        assert s.info().path == "structured"
        s.set_flow(c.arrays["flow"])
        for _ in range(2):
            if profiled:
                for j in range(3):
                    s.profile_stage(j, c.dt)
            else:
                s.step(c.dt, 1)
        got.append((s.get_u0(), s.get_flow()))
        s.close()
    own = slice(1, c.sd_node + 1)
    assert np.array_equal(got[0][0][own], got[1][0][own])
    assert np.array_equal(got[0][1][own], got[1][1][own])
