"""Many binary64 reverse steps against extended precision: what every step rounds
alike adds up to more than the rounding of the cells."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble
CX, CY = (0, 1, 0, -1, 0, 1, -1, -1, 1), (0, 0, 1, 0, -1, 1, 1, -1, -1)
W = [LD(4) / 9] + [LD(1) / 9] * 4 + [LD(1) / 36] * 4


def feq(rho, ux, uy):
    out = []
    for cx, cy, w in zip(CX, CY, W):
        cu = cx * ux + cy * uy
        out.append(w * rho * (1 + 3 * cu + LD(4.5) * cu * cu - LD(1.5) * (ux * ux + uy * uy)))
    return np.array(out)


def moments(f):
    rho = f.sum(0)
    return rho, (f[1] - f[3] + f[5] - f[6] - f[7] + f[8]) / rho, (f[2] - f[4] + f[5] + f[6] - f[7] - f[8]) / rho


def gradient(u0, target, omega, steps):
    """dL/du0 of L = sum (u_T - target)^2 / 2."""
    omega, states = LD(omega), []
    f = feq(np.ones_like(u0[0]), u0[0], u0[1])
    for _ in range(steps):
        g = np.array([np.roll(f[q], (CX[q], CY[q]), (0, 1)) for q in range(9)])
        states.append(g)
        f = g + omega * (feq(*moments(g)) - g)
    rho, ux, uy = moments(f)
    rx, ry = ux - target[0], uy - target[1]
    lam = np.array([(rx * (CX[q] - ux) + ry * (CY[q] - uy)) / rho for q in range(9)])
    for g in reversed(states):
        rho, ux, uy = moments(g)
        a, bx, by = 0, 0, 0
        for q in range(9):
            cu, wl = CX[q] * ux + CY[q] * uy, W[q] * lam[q]
            a = a + wl * (1 + 3 * cu + LD(4.5) * cu * cu - LD(1.5) * (ux * ux + uy * uy))
            bx, by = (b + wl * (3 * c + 9 * cu * c - 3 * u) for b, c, u in ((bx, CX[q], ux), (by, CY[q], uy)))
        lam = np.array([np.roll((1 - omega) * lam[p] + omega * (a + bx * (CX[p] - ux) + by * (CY[p] - uy)),
                                (-CX[p], -CY[p]), (0, 1)) for p in range(9)])
    gx, gy = 0, 0
    for q in range(9):
        cu, wl = CX[q] * u0[0] + CY[q] * u0[1], W[q] * lam[q]
        gx, gy = (b + wl * (3 * c + 9 * cu * c - 3 * u) for b, c, u in ((gx, CX[q], u0[0]), (gy, CY[q], u0[1])))
    return np.array([gx, gy])


@pytest.mark.parametrize("tau", [0.52, 0.6, 0.7, 0.8])
def test_velocity_gradient_after_many_steps(gpu_lib, tau):
    """Mean-square bound: a step's roundings, four of 2^-53 of lambda, are independent from step
    to step and cell to cell: 4 sqrt(steps) 2^-53 = 6.9e-15.  (A rate off by 2^-53 in every
    step would give 2.7e-14 by itself.)"""
    import torch
    from plbm.autograd import velocity_misfit
    nx, ny, steps = 44, 36, 240
    rng = np.random.default_rng(2)
    x, y = np.meshgrid(np.arange(nx) * 2 * math.pi / nx, np.arange(ny) * 2 * math.pi / ny, indexing="ij")
    u0 = 0.04 * np.stack([np.sin(y), np.sin(x)]) + 1e-3 * rng.standard_normal((2, nx, ny))
    target = 0.04 * np.stack([np.cos(y), -np.cos(x)]) + 1e-3 * rng.standard_normal((2, nx, ny))
    u = torch.from_numpy(u0).cuda().requires_grad_(True)
    t = torch.tensor(tau, dtype=torch.float64, device="cuda", requires_grad=True)
    loss = velocity_misfit(u, t, torch.from_numpy(target).cuda(), steps)
    got = torch.autograd.grad(loss, u)[0].cpu().numpy()
    want = gradient(u0.astype(LD), target.astype(LD), np.float64(1) / np.float64(tau), steps)
    err = float(np.sqrt(((got - want) ** 2).sum() / (want ** 2).sum()))
    assert err <= 4 * math.sqrt(steps) * 2.0 ** -53, err
