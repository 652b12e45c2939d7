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


@pytest.mark.parametrize("shape", [(40, 40, 40), (40, 40, 41)])
def test_product_forms_have_the_same_bits(ctx, shape):
    """64,000 and 65,600 nodes: either side of the line up to which the
    solver's and the drop-in's per-node kernels take their products on the
    FP64 pipe; the batch takes them on the integer pipe at every size.  FLOW
    is compared: the batch's U0 is already the next stage's."""
    from cfd_gb300 import cases, runtime
    c = cases.taylor_green(shape=shape)
    b = runtime.Batch(ctx, 0)
    slot = b.add(c)
    b.step(2)
    want = b.get_flow(slot)[1:c.sd_node + 1]
    b.close()
    for path in (1, 0):
        s = runtime.Solver(ctx, c, force_path=path)
        s.set_flow(c.arrays["flow"])
        s.step(c.dt, 2)
        assert np.array_equal(s.get_flow()[1:c.sd_node + 1], want)
        s.close()


def test_batch_rounds_equal_the_solver(ctx):
    """Five instances of 216,000 nodes: two rounds of the batch's face
    scratch (2^20 nodes each), the last instance in the second."""
    from cfd_gb300 import cases, runtime
    c = cases.taylor_green(n=60)
    s = runtime.Solver(ctx, c)
    s.set_flow(c.arrays["flow"])
    s.step(c.dt, 1)
    want = s.get_flow()[1:c.sd_node + 1]
    s.close()
    b = runtime.Batch(ctx, 0)
    slots = [b.add(c) for _ in range(5)]
    b.step(1)
    for slot in slots:
        assert np.array_equal(b.get_flow(slot)[1:c.sd_node + 1], want)
    b.close()
