"""cfd_viscous around its two launches: rows whose neighbour chain leaves the
table are skipped whole, and no memory but the call's own is used."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import copy_arrays

pytestmark = pytest.mark.gpu

OUT = ("F", "E", "G", "Fv", "Ev", "Gv")


def _viscous(ctx, dev, c, n_items):
    ctx.viscous(dev["U0"], dev["F"], dev["E"], dev["G"], dev["Fv"], dev["Ev"], dev["Gv"], dev["grid"], dev["metric"],
                dev["det"], dev["flow"], n_items, c.params)


@pytest.mark.parametrize("reuse", [True, False])
def test_rows_with_a_bad_chain_are_left_as_they_were(ctx, reuse):
    from cfd_gb300 import abi, cases
    c = cases.isentropic_vortex(shape=(12, 6, 5))
    a = copy_arrays(c.arrays)
    ctx.set_face_reuse(reuse)
    dev = ctx.upload_case(a)
    try:
        ctx.uq(dev["U0"], dev["Q"], dev["grid"], dev["det"], dev["flow"], dev["roe"], c.g_node + 1)
        g = a["grid"]
        plus = g["N1"].copy()                    # the next row along i
        g["N1"][29] = c.g_node + 7               # outside [0, n_rows)
        ctx.write(dev["grid"], g)
        bad = np.array([29 in (r, plus[r], plus[plus[r]]) for r in range(c.g_node + 1)])
        assert 3 <= bad.sum() < len(bad)
        for k in OUT:
            a[k][...] = -7.25
            ctx.write(dev[k], a[k])
        with pytest.raises(abi.CfdError) as e:
            _viscous(ctx, dev, c, c.g_node + 1)
        assert e.value.status == abi.EINVAL
        for k in OUT:
            got = ctx.download(dev, k, a[k])
            assert np.all(got[bad] == -7.25), f"{k}: a skipped row was written"
            assert np.all(got[1:][~bad[1:]][:, 1:] != -7.25), f"{k}: a row was left out"
    finally:
        ctx.set_face_reuse(True)
        for p in dev.values():
            ctx.free(p)


@pytest.mark.parametrize("les", [0, 1, 2])
def test_the_scratch_of_the_other_kernels_is_not_used(ctx, les):
    """The face scratch belongs to cfd_uq and cfd_weno, which may run for
    another table on another stream: with and without it cfd_viscous makes
    the same two launches and the same bits."""
    import dataclasses

    from cfd_gb300 import cases
    c = cases.taylor_green(shape=(9, 8, 7))
    c = dataclasses.replace(c, params=dataclasses.replace(c.params, les=les))
    out, launches = [], []
    for reuse in (True, False):
        ctx.set_face_reuse(reuse)
        a = copy_arrays(c.arrays)
        dev = ctx.upload_case(a)
        try:
            ctx.uq(dev["U0"], dev["Q"], dev["grid"], dev["det"], dev["flow"], dev["roe"], c.g_node + 1)
            n = ctx.launch_count
            _viscous(ctx, dev, c, c.g_node + 1)
            launches.append(ctx.launch_count - n)
            out.append([ctx.download(dev, k, a[k]) for k in OUT + ("flow",)])
        finally:
            ctx.set_face_reuse(True)
            for p in dev.values():
                ctx.free(p)
    assert launches == [2, 2]
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64))
