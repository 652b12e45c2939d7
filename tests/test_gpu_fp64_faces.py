"""The FP64 face pass's kernels at the edges of their launches: more nodes
than one round of their scratch, odd extents down to a single warp, and
register budgets that differ per direction -- U0 after a step has the bits of
the gather path (the drop-in kernels) or the oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,budgets", [((7, 5, 6), None), ((33, 7, 9), (2, 3, 4)), ((20, 18, 22), (4, 2, 2))])
def test_small_and_odd_lattices_equal_the_oracle(ctx, oracle_mod, shape, budgets):
    from cfd_gb300 import cases, runtime
    from helpers import copy_arrays
    c = cases.isentropic_vortex(shape=shape)
    a = copy_arrays(c.arrays)
    oracle_mod.rk3_steps(a, c.g_node, c.sd_node, c.params, c.dt, 2)
    s = runtime.Solver(ctx, c)
    if budgets:
        s.set_face_blocks(*budgets)
    s.set_flow(c.arrays["flow"])
    s.step(c.dt, 2)
    assert np.array_equal(s.get_u0()[1:c.sd_node + 1], a["U0"][1:c.sd_node + 1])
    s.close()


def test_rounds_of_the_face_scratch_equal_the_gather_path(ctx):
    """2,129,920 nodes: two rounds of the face kernels (2^21 nodes each)."""
    from cfd_gb300 import cases, runtime
    c = cases.isentropic_vortex(shape=(130, 128, 128))
    got = []
    for path in (1, 0):
        s = runtime.Solver(ctx, c, force_path=path)
        s.set_flow(c.arrays["flow"])
        s.step(c.dt, 1)
        got.append(s.get_u0()[1:])   # row 0 is the layout's dummy row, not a node
        s.close()
    assert np.array_equal(got[0], got[1])
