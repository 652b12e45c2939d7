"""Slow departures of the reduced forms from the FP64 form that the error of
the whole state (most of it pressure and energy) does not show."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _after(ctx, c, precision, steps):
    from cfd_gb300 import runtime
    s = runtime.Solver(ctx, c, precision=precision)
    s.set_flow(c.arrays["flow"])
    s.step(c.dt, steps)
    flow = s.get_flow()[1:c.sd_node + 1]
    s.close()
    return flow


def test_the_split_form_does_not_dissipate_by_its_rounding(ctx):
    """Kinetic energy of a Taylor-Green vortex after 200 steps within one FP32
    rounding (2^-24) of the FP64 form's: rounding errors of either sign leave
    some 1e-8, a first-order dissipation of 1e-8 of its full strength 1.7e-7."""
    from cfd_gb300 import cases
    c = cases.taylor_green(n=32)
    det = c.arrays["det"][1:c.sd_node + 1]
    ke = [float(np.sum(0.5 * det * f[:, 5] * (f[:, 0] ** 2 + f[:, 1] ** 2 + f[:, 2] ** 2)))
          for f in (_after(ctx, c, p, 200) for p in (0, 2))]
    assert abs(ke[1] - ke[0]) <= 2.0 ** -24 * ke[0]


def test_velocities_of_the_mixed_form(ctx):
    """u after 200 steps of a Taylor-Green vortex at Mach 0.1, whose pressure
    noise the velocities take up: 4.6e-6 with the eigenvectors applied as
    matrices; no form of applying them may be 10 % worse."""
    from cfd_gb300 import cases
    c = cases.taylor_green(n=64)
    a, b = _after(ctx, c, 0, 200), _after(ctx, c, 1, 200)
    assert np.linalg.norm(b[:, 0] - a[:, 0]) <= 5.1e-6 * np.linalg.norm(a[:, 0])
