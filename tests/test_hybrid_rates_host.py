"""Relaxation rates outside (0, 2) in the fixed-point collisions (csrc/hybrid.cuh),
from the host build of tests/hybrid_cells_host.cpp: a cell is either right or reported."""
import ctypes
import math
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
CX = np.array((0, 1, 0, -1, 0, 1, -1, -1, 1.0))
CY = np.array((0, 0, 1, 0, -1, 1, 1, -1, -1.0))
W = np.array((4 / 9,) + (1 / 9,) * 4 + (1 / 36,) * 4)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("hc") / "hc.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off",
                    "-I", str(ROOT / "periodic-lbm_gb300" / "csrc"), str(ROOT / "tests" / "hybrid_cells_host.cpp"),
                    "-o", str(so)], check=True)
    h = ctypes.CDLL(str(so))
    h.hc_collide.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_double, ctypes.c_double]
    return h


def hermite_rr(f, omega):
    """The recursive-regularized collision of f, binary64 (|f'| of order 1: a few 1e-16 per unit of omega)."""
    rho, ux, uy = f.sum(), (CX * f).sum() / f.sum(), (CY * f).sum() / f.sum()
    hxx, hyy, hxy = CX * CX - 1 / 3, CY * CY - 1 / 3, CX * CY
    hxxy, hyyx, hxxyy = hxx * CY, hyy * CX, hxx * hyy

    def expand(xx, xy, yy, xxy, yyx, xxyy):
        return (4.5 * (hxx * xx + 2 * hxy * xy + hyy * yy) + 13.5 * (hxxy * xxy + hyyx * yyx) + 20.25 * hxxyy * xxyy)

    feq = W * rho * (1 + 3 * (CX * ux + CY * uy) + expand(ux * ux, ux * uy, uy * uy, ux * ux * uy, uy * uy * ux,
                                                          ux * ux * uy * uy))
    d = f - feq
    axx, axy, ayy = (hxx * d).sum(), (hxy * d).sum(), (hyy * d).sum()
    axxy, ayyx = 2 * ux * axy + uy * axx, 2 * uy * axy + ux * ayy
    axxyy = 2 * (ux * ayyx + uy * axxy) - ux * ux * ayy - uy * uy * axx - 4 * ux * uy * axy
    return feq + W * (1 - omega) * expand(axx, axy, ayy, axxy, ayyx, axxyy)


def state(rng):
    f = W * (1 + 0.02 * rng.standard_normal(9)) + W * 3 * 0.03 * (CX + CY)
    return f


@pytest.mark.parametrize("shifted", [0, 1])
@pytest.mark.parametrize("omega", [-3.0, -1e-9, 2.0 + 1e-9, 2.05, 2.5, 5.0, 1e3, math.inf, -math.inf, math.nan])
def test_rr_reports_a_rate_that_has_no_fixed_point(lib, omega, shifted):
    rng = np.random.default_rng(5)
    for _ in range(8):
        a = np.ascontiguousarray(state(rng) - W * shifted)
        assert lib.hc_collide(2, shifted, a.ctypes.data, omega, 1.0) == 1


@pytest.mark.parametrize("omega", [0.0, 1e-9, 0.7, 1.0, 1.99, 2.0])
def test_rr_rates_in_range(lib, omega):
    """Bound: the operands' and the comparison's own roundings, 40 of 2^-53 for values below one."""
    rng = np.random.default_rng(6)
    for _ in range(8):
        a = state(rng)
        want = hermite_rr(a, omega)
        assert lib.hc_collide(2, 0, a.ctypes.data, omega, 1.0) == 0
        assert np.max(np.abs(a - want)) <= 40 * 2.0 ** -53
