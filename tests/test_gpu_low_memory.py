"""Little free device memory: the scratch that the face passes work through
in rounds gives way, so what fits without it (plus a few MB) still runs, with
the same bits."""
from __future__ import annotations

import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLACK = 48 << 20   # allocation granularity and the smallest rounds


@contextlib.contextmanager
def free_memory(nbytes):
    """All but about nbytes of the device's memory taken."""
    import torch
    torch.cuda.empty_cache()
    hog = None
    for spare in range(0, 8):   # free memory may be in pieces
        free, _ = torch.cuda.mem_get_info()
        try:
            hog = torch.empty((free - nbytes - (spare << 23)) >> 21 << 21, dtype=torch.uint8, device="cuda")
            break
        except torch.cuda.OutOfMemoryError:
            torch.cuda.empty_cache()
    if hog is None:
        pytest.skip("the device's memory cannot be taken in one piece")
    try:
        yield
    finally:
        del hog
        torch.cuda.empty_cache()


def _advance(solver, c):
    solver.set_flow(c.arrays["flow"])
    solver.step(c.dt, 1)
    flow = solver.get_flow()
    solver.close()
    return flow


def test_gather_path(ctx):
    from cfd_gb300 import cases, runtime
    c = cases.taylor_green(n=64)
    rows = c.g_node + 1
    s = runtime.Solver(ctx, c, force_path=0)
    need = s.info().device_bytes - 1152 * min(rows, 1 << 18)   # without the rounds
    want = _advance(s, c)
    with free_memory(need + SLACK):
        got = _advance(runtime.Solver(ctx, c, force_path=0), c)
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))


def test_drop_in_kernels(ctx):
    """cfd_ctx_set_rows with memory for 252 bytes per row still shares the
    faces (more than one launch of cfd_weno)."""
    from cfd_gb300 import cases, runtime
    from helpers import copy_arrays
    c = cases.taylor_green(n=64)
    rows = c.g_node + 1
    out = []
    for little in (False, True):
        own = runtime.Context(0)
        dev = {k: own.alloc(v.nbytes) for k, v in c.arrays.items()}
        a = copy_arrays(c.arrays)
        for k, v in a.items():
            own.write(dev[k], np.ascontiguousarray(v))
        with free_memory(252 * rows + SLACK) if little else contextlib.nullcontext():
            own.set_rows(rows)
        P, d = c.params, dev
        own.uq(d["U0"], d["Q"], d["grid"], d["det"], d["flow"], d["roe"], rows)
        own.viscous(d["U0"], d["F"], d["E"], d["G"], d["Fv"], d["Ev"], d["Gv"], d["grid"], d["metric"], d["det"],
                    d["flow"], rows, P)
        n = own.launch_count
        own.weno(0, P.mach, c.dt, d["deter"], d["det"], d["U0"], d["U1"], d["U2"], d["grid"], d["Q"], d["metric"],
                 d["roe"], d["Fv"], d["Ev"], d["Gv"], d["F"], d["E"], d["G"], d["flow"], c.sd_node + 1, P)
        assert own.launch_count - n > 1
        out.append([own.download(dev, k, a[k]) for k in ("U1", "flow")])
        own.close()
    for x, y in zip(*out):
        assert np.array_equal(x.view(np.uint64), y.view(np.uint64))


@pytest.mark.parametrize("maker", ["periodic", "walls"])
def test_structured_fp64_solver(ctx, maker):
    """The solver's arrays take 116 doubles per node; 117, as much as before
    the face pass had scratch, are enough."""
    from cfd_gb300 import cases, runtime
    c = cases.taylor_green(n=64) if maker == "periodic" else cases.channel(ni=64, nj=58, nk=60)
    n = c.g_node
    s = runtime.Solver(ctx, c)
    assert s.info().path == "structured"
    assert s.info().device_bytes <= 8 * n * (117 + 126) + 8 * n      # index and loc codes
    want = _advance(s, c)
    assert np.array_equal(want[0], c.arrays["flow"][0])              # the dummy row as it was set
    with free_memory(8 * n * 117 + 6 * n + SLACK):
        s = runtime.Solver(ctx, c)
        assert s.info().device_bytes < 8 * n * (117 + 126 // 2)
        got = _advance(s, c)
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
