"""The plugin's BGK step on flows of tiny velocity, against extended precision."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble
CX, CY = (0, 1, 0, -1, 0, 1, -1, -1, 1), (0, 0, 1, 0, -1, 1, 1, -1, -1)
W = [LD(4) / 9] + [LD(1) / 9] * 4 + [LD(1) / 36] * 4


def relax(h, omega):
    d = h.sum(0)
    jx, jy = (sum(c[q] * h[q] for q in range(9)) for c in (CX, CY))
    out = []
    for q in range(9):
        cj = CX[q] * jx + CY[q] * jy
        eq = W[q] * (d + 3 * cj + (LD(4.5) * cj * cj - LD(1.5) * (jx * jx + jy * jy)) / (1 + d))
        out.append(h[q] + omega * (eq - h[q]))
    return np.array(out)


@pytest.mark.parametrize("u0", [1e-3, 1e-6, 1e-8, 1e-9, 1e-10, 1e-13])
def test_velocity_of_a_decaying_vortex(gpu_lib, u0):
    """Error of the velocity in the mean square, 60 steps.  Cells with |h| of 2^-27 and more are held in units
    of 2^-59, whose bracket errs by up to 2^-57 per population: of velocities of u0, 3 x 2^-57 / u0 per
    step, independent from step to step, and 2^-52 of the velocity itself; below, 2^-50 of
    max |h|, a third of u0.  The units of 2^-59 alone would give 7e-9 and more from 1e-9 down.
    (Default arithmetic: the hybrid plugin starts from an equilibrium in those units.)"""
    from plbm.plugin import SimPlugin, make_params
    nx, ny, steps, omega = 40, 36, 60, 1.6
    x, y = np.arange(nx)[:, None] * 2 * math.pi / nx, np.arange(ny)[None, :] * 2 * math.pi / ny
    u = np.stack([-u0 * np.cos(x) * np.sin(y), u0 * np.sin(x) * np.cos(y)], axis=2)
    sim = SimPlugin()
    sim.init((nx, ny), 1.0, np.zeros((nx, ny), order="F"), np.asfortranarray(u), params=make_params(kind="bgk", math="fma"))
    sim.steps(omega, steps)
    got = sim.vars()[1]
    ux, uy = u[..., 0].astype(LD), u[..., 1].astype(LD)
    h = np.array([W[q] * (3 * (CX[q] * ux + CY[q] * uy) + LD(4.5) * (CX[q] * ux + CY[q] * uy) ** 2
                          - LD(1.5) * (ux * ux + uy * uy)) for q in range(9)])
    for _ in range(steps):
        h = relax(h, LD(omega))
        h = np.array([np.roll(h[q], (CX[q], CY[q]), (0, 1)) for q in range(9)])
    d = 1 + h.sum(0)
    want = np.stack([sum(c[q] * h[q] for q in range(9)) / d for c in (CX, CY)], axis=2)
    err = float(np.sqrt(((got - want) ** 2).sum() / (want ** 2).sum()))
    per_step = 2.0 ** -50 if u0 < 2e-8 else 3 * 2.0 ** -57 / u0 + 2.0 ** -52
    assert err <= 3 * math.sqrt(steps) * per_step + steps * 2.0 ** -53, err
