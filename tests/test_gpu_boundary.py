"""The boundary routine on the GPU and the lattice path with ghost layers.

* cfd_boundary_fill against the golden vectors of the reference's own
  routine (bit-exact: copies and the reference's formulas, compiled without
  FMA contraction);
* the wall-bounded channel (periodic x/z, walls and inlet/outlet in y) on the
  face-based lattice path with the routine after every stage, against the
  oracle (FP64: relative L2 <= 1e-12), against the drop-in gather path, and
  in the mixed form (<= 1e-6 against FP64)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_l2
from test_oracle_boundary import golden_inputs

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("initial", [1, 0])
def test_boundary_fill_matches_reference_golden(ctx, initial):
    from cfd_gb300 import runtime
    z, a, bc = golden_inputs()
    bnd = runtime.Boundary(ctx, a["grid"], bc)
    dev = ctx.alloc(a["flow"].nbytes)
    try:
        ctx.write(dev, a["flow"])
        bnd.fill(dev, float(z["mach"]), initial, int(z["sd_node"]))
        out = np.empty_like(a["flow"])
        ctx.read(out, dev)
    finally:
        ctx.free(dev)
        bnd.close()
    assert np.array_equal(out, z[f"out_flow_initial{initial}"])


@pytest.mark.parametrize("variant,launches", [("channel", 1), ("channel_shared_row", 3), ("golden", 4)])
def test_independent_lists_fill_in_one_launch(ctx, oracle_mod, variant, launches):
    """Lists that touch no row another list writes (the channel's outlet,
    inlet and walls) run as one launch over all entries.  A row in two lists
    (written by both, so list order decides), or lists that read each
    other's rows (the golden box), keep one launch per list in list order.
    Every variant matches the oracle's routine bit for bit."""
    from cfd_gb300 import cases, runtime
    if variant == "golden":
        z, a, bc = golden_inputs()
        mach, sd_node = float(z["mach"]), int(z["sd_node"])
    else:
        c = cases.channel(ni=16, nj=12, nk=8)
        a, bc = c.copy().arrays, c.bc
        a["flow"][1:] = np.random.default_rng(3).uniform(0.5, 1.5, a["flow"][1:].shape)
        mach, sd_node = c.params.mach, c.sd_node
        if variant == "channel_shared_row":
            bc = cases.BoundaryLists(outlet=bc.outlet, inlet=bc.inlet, boundary=bc.boundary,
                                     wall=np.concatenate([bc.wall, bc.outlet[:1]]))
    bnd = runtime.Boundary(ctx, a["grid"], bc)
    dev = ctx.alloc(a["flow"].nbytes)
    try:
        ctx.write(dev, a["flow"])
        n0 = ctx.launch_count
        bnd.fill(dev, mach, 1, sd_node)
        n = ctx.launch_count - n0
        out = np.empty_like(a["flow"])
        ctx.read(out, dev)
    finally:
        ctx.free(dev)
        bnd.close()
    oracle_mod.boundary_fill(a, bc, mach, 1, sd_node)
    assert np.array_equal(out, a["flow"])
    assert n == launches


@pytest.mark.parametrize("ghost_chain", ["apart", "second_ghost_again", "back_to_the_node", "into_the_interior"])
def test_entries_with_coinciding_nodes_fill_in_order(ctx, oracle_mod, ghost_chain):
    """An entry's targets are written side by side only where its node,
    ghosts and sources all differ; chains that name a node twice (here one
    wall node's, rewired) give what the routine's own order gives."""
    from cfd_gb300 import cases, runtime
    c = cases.channel(ni=16, nj=12, nk=8)
    a, bc = c.copy().arrays, c.bc
    a["flow"][1:] = np.random.default_rng(7).uniform(0.5, 1.5, a["flow"][1:].shape)
    g, b = a["grid"], int(bc.wall[len(bc.wall) // 2])
    slot = next(f"N{k}" for k in range(6) if int(g[b][f"N{k}"]) > c.sd_node)   # towards the ghosts
    inward = next(f"N{k}" for k in range(6) if k % 2 == int(slot[1]) % 2 and f"N{k}" != slot
                  and int(g[b][f"N{k}"]) <= c.sd_node)
    g1 = int(g[b][slot])
    if ghost_chain == "second_ghost_again":
        g2 = int(g[g1][slot])
        g[slot][g2] = g2
    elif ghost_chain == "back_to_the_node":
        g[slot][g1] = b
    elif ghost_chain == "into_the_interior":
        g[slot][g1] = int(g[b][inward])
    bnd = runtime.Boundary(ctx, g, bc)
    dev = ctx.alloc(a["flow"].nbytes)
    try:
        ctx.write(dev, a["flow"])
        bnd.fill(dev, c.params.mach, 1, c.sd_node)
        out = np.empty_like(a["flow"])
        ctx.read(out, dev)
    finally:
        ctx.free(dev)
        bnd.close()
    oracle_mod.boundary_fill(a, bc, c.params.mach, 1, c.sd_node)
    assert np.array_equal(out, a["flow"])


def test_singular_wall_node_is_unsupported(ctx):
    from cfd_gb300 import abi, runtime
    z, a, bc = golden_inputs()
    a["grid"]["ID"][bc.wall[0]] = 10
    with pytest.raises(abi.CfdError) as e:
        runtime.Boundary(ctx, a["grid"], bc)
    assert e.value.status == abi.EUNSUPPORTED


def _assert_flow_close(got, want, tol=TOL):
    """Rows 1.. (row 0 is the reference's dummy row, which the lattice path
    does not process); names the worst rows and fields on failure."""
    g, w = got[1:], want[1:]
    err = rel_l2(g, w)
    if not err <= tol:
        d = np.abs(g - w)
        rows = np.argsort(d.max(axis=1))[::-1][:5] + 1
        fields = np.argsort(d.max(axis=0))[::-1][:3]
        raise AssertionError(f"rel L2 {err:.3e}; worst rows {rows.tolist()}, fields {fields.tolist()}")


def _channel():
    from cfd_gb300 import cases
    return cases.channel(ni=16, nj=12, nk=8)


def test_channel_takes_the_lattice_path(ctx):
    from cfd_gb300 import runtime
    c = _channel()
    s = runtime.Solver(ctx, c)
    info = s.info()
    s.close()
    assert info.path == "structured" and tuple(info.shape) == (16, 18, 8)


def test_channel_fp64_lattice_matches_oracle(ctx, oracle_mod):
    """RHS of the first stage and three steps with the boundary routine."""
    from cfd_gb300 import runtime
    c = _channel()
    own = slice(1, c.sd_node + 1)
    s = runtime.Solver(ctx, c)
    s.set_flow(c.arrays["flow"])
    Lg = s.stage(0, c.dt)
    a = c.copy().arrays
    Lo = oracle_mod.stage(a, c.g_node, c.sd_node, c.params, 0, c.dt, want_L=True)
    oracle_mod.boundary_fill(a, c.bc, c.params.mach, 1, c.sd_node)
    flow = s.get_flow()
    s.close()
    assert rel_l2(Lg[own], Lo[own]) <= TOL
    _assert_flow_close(flow, a["flow"])
    s = runtime.Solver(ctx, c)
    s.set_flow(c.arrays["flow"])
    s.step(c.dt, 3)
    flow = s.get_flow()
    s.close()
    a = c.copy().arrays
    oracle_mod.rk3_steps_bc(a, c.g_node, c.sd_node, c.params, c.dt, 3, c.bc)
    _assert_flow_close(flow, a["flow"])


def test_channel_lattice_equals_gather_path(ctx):
    from cfd_gb300 import runtime
    c = _channel()
    out = []
    for force in (1, 0):
        s = runtime.Solver(ctx, c, force_path=force)
        s.set_flow(c.arrays["flow"])
        s.step(c.dt, 4)
        out.append(s.get_flow())
        s.close()
    _assert_flow_close(out[0], out[1])


def test_channel_mixed_error_budget(ctx):
    from cfd_gb300 import runtime
    c = _channel()
    res = []
    for prec in (0, 1):
        s = runtime.Solver(ctx, c, precision=prec)
        s.set_flow(c.arrays["flow"])
        s.step(c.dt, 10)
        res.append(s.get_flow()[1:c.sd_node + 1])
        s.close()
    assert np.isfinite(res[1]).all()
    assert rel_l2(res[1], res[0]) <= 1e-6


def test_ghost_box_gather_path_with_boundary(ctx, oracle_mod):
    """A table that is not a lattice with single-valued faces (ghosts carry
    their own node metrics) runs the drop-in kernels; the boundary routine
    follows every stage there too."""
    from cfd_gb300 import cases, runtime
    c = cases.ghost_box(shape=(7, 6, 5), seed=2, bc=True)
    s = runtime.Solver(ctx, c)
    assert s.info().path == "gather"
    s.set_flow(c.arrays["flow"])
    s.step(c.dt, 1)
    flow = s.get_flow()
    s.close()
    a = c.copy().arrays
    oracle_mod.rk3_steps_bc(a, c.g_node, c.sd_node, c.params, c.dt, 1, c.bc)
    _assert_flow_close(flow, a["flow"])


def test_naca0012_ogrid_fp64_matches_oracle_and_mixed_budget(ctx, oracle_mod):
    """The NACA0012 O-grid case at a reduced size: the O-grid on the lattice path with
    the wall and inlet/outlet far field filled after every stage, FP64
    against the oracle, and the mixed form's density and pressure."""
    from cfd_gb300 import cases, layout, runtime
    c = cases.naca0012(ni=64, nj=24, nk=4)
    flow0 = c.copy().arrays
    oracle_mod.boundary_fill(flow0, c.bc, c.params.mach, 1, c.sd_node)
    res = {}
    for prec in (0, 1):
        s = runtime.Solver(ctx, c, precision=prec)
        assert s.info().path == "structured"
        s.set_flow(flow0["flow"])
        s.step(c.dt, 3)
        res[prec] = s.get_flow()
        s.close()
    a = {k: v.copy() for k, v in flow0.items()}
    oracle_mod.rk3_steps_bc(a, c.g_node, c.sd_node, c.params, c.dt, 3, c.bc)
    _assert_flow_close(res[0], a["flow"])
    own = slice(1, c.sd_node + 1)
    for name in ("rho", "p"):
        k = layout.FLOW[name]
        assert rel_l2(res[1][own, k], res[0][own, k]) <= 1e-6


def test_duct_edges_on_the_lattice_path(ctx, oracle_mod):
    """Walls on four sides: face and edge codes in one wall list; FP64
    lattice path against the oracle, the gather path, and the mixed form."""
    from cfd_gb300 import cases, runtime
    c = cases.duct()
    assert {15, 17, 19, 21} <= set(c.arrays["grid"]["loc"][c.bc.wall].tolist())
    out = {}
    for key, kw in (("lattice", {}), ("gather", {"force_path": 0}), ("mixed", {"precision": 1})):
        s = runtime.Solver(ctx, c, **kw)
        assert s.info().path == ("gather" if key == "gather" else "structured")
        s.set_flow(c.arrays["flow"])
        s.step(c.dt, 3)
        out[key] = s.get_flow()
        s.close()
    a = c.copy().arrays
    oracle_mod.rk3_steps_bc(a, c.g_node, c.sd_node, c.params, c.dt, 3, c.bc)
    _assert_flow_close(out["lattice"], a["flow"])
    _assert_flow_close(out["gather"], a["flow"])
    # the mixed form derives FLOW from its state; the reference's edge and
    # corner rules leave the sound speed `a` of those nodes stale (no kernel
    # reads it), so compare the fields the next stage reads
    from cfd_gb300 import layout
    own = slice(1, c.sd_node + 1)
    cols = [layout.FLOW[k] for k in ("rho", "u", "v", "w", "p")]
    assert rel_l2(out["mixed"][own][:, cols], out["lattice"][own][:, cols]) <= 1e-6
    a = layout.FLOW["a"]
    stale = np.abs(out["mixed"][own, a] - out["lattice"][own, a]) > 1e-6 * np.abs(out["lattice"][own, a])
    assert set(c.arrays["grid"]["loc"][1:c.sd_node + 1][stale].tolist()) <= set(range(7, 27))


def test_channel_stages_out_of_order_and_profiled(ctx):
    """Stages called out of the usual order (each stage's U_Q then comes from
    the current state, copied into the stage's slot, ghosts included) and a
    profiled stage (the boundary routine is one timed entry): the mixed form
    tracks the FP64 form through the same calls."""
    from cfd_gb300 import layout, runtime
    c = _channel()
    seq = (0, 0, 1, 2, 1, 2, 0)
    out = {}
    for prec in (0, 1):
        s = runtime.Solver(ctx, c, precision=prec)
        s.set_flow(c.arrays["flow"])
        for j in seq:
            s.stage(j, c.dt, want_L=False)
        names = [n for n, _ in s.profile_stage(1, c.dt)]
        assert names[-1] == "boundary"
        out[prec] = s.get_flow()
        s.close()
    own = slice(1, c.sd_node + 1)
    cols = [layout.FLOW[k] for k in ("rho", "u", "v", "w", "p")]
    assert np.isfinite(out[1][own]).all()
    assert rel_l2(out[1][own][:, cols], out[0][own][:, cols]) <= 1e-6
