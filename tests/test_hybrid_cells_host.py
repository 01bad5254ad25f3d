"""The fixed-point binary64 collisions (csrc/hybrid.cuh, csrc/fixed.cuh) from a
host build of the kernels' header, against exact rational arithmetic."""
import ctypes
import math
import subprocess
from fractions import Fraction as Fr
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
CX = (0, 1, 0, -1, 0, 1, -1, -1, 1)
CY = (0, 0, 1, 0, -1, 1, 1, -1, -1)
W = (Fr(4, 9),) + (Fr(1, 9),) * 4 + (Fr(1, 36),) * 4
OPP = (0, 3, 4, 1, 2, 7, 8, 5, 6)
KINDS = {"bgk": 0, "trt": 1, "rr": 2}


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("hc") / "hc.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off",
                    "-I", str(ROOT / "periodic-lbm_gb300" / "csrc"), str(ROOT / "tests" / "hybrid_cells_host.cpp"),
                    "-o", str(so)], check=True)
    h = ctypes.CDLL(str(so))
    h.hc_collide.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_double, ctypes.c_double]
    h.hc_collide_quick.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_double, ctypes.c_double]
    h.hc_mulh64.restype = h.hc_recip.restype = ctypes.c_int64
    h.hc_mulh64.argtypes = [ctypes.c_int64, ctypes.c_int64]
    h.hc_recip.argtypes = [ctypes.c_int64]
    return h


def exact_collide(kind, f, omega, ld):
    """The collision of the rational populations f (unshifted), true weights."""
    rho = sum(f)
    jx, jy = sum(c * v for c, v in zip(CX, f)), sum(c * v for c, v in zip(CY, f))
    if kind == "trt":
        out = []
        for q in range(9):
            cj = CX[q] * jx + CY[q] * jy
            even = W[q] * (rho + Fr(9, 2) * cj * cj - Fr(3, 2) * (jx * jx + jy * jy))
            s, a = (f[q] + f[OPP[q]]) / 2 - even, (f[q] - f[OPP[q]]) / 2 - W[q] * 3 * cj
            out.append(f[q] - omega * s - ld * a)
        return out, rho, jx, jy
    ux, uy = jx / rho, jy / rho
    if kind == "bgk":
        feq = []
        for q in range(9):
            cu = CX[q] * ux + CY[q] * uy
            feq.append(W[q] * rho * (1 + 3 * cu + Fr(9, 2) * cu * cu - Fr(3, 2) * (ux * ux + uy * uy)))
        return [v + omega * (e - v) for v, e in zip(f, feq)], rho, jx, jy
    t = Fr(1, 3)
    herm = [(CX[q] ** 2 - t, CX[q] * CY[q], CY[q] ** 2 - t) for q in range(9)]
    herm = [(xx, xy, yy, xx * CY[q], yy * CX[q], xx * yy) for q, (xx, xy, yy) in enumerate(herm)]
    fac = (Fr(9, 2), Fr(9), Fr(9, 2), Fr(27, 2), Fr(27, 2), Fr(81, 4))
    eq = (ux * ux, ux * uy, uy * uy, ux * ux * uy, uy * uy * ux, ux * ux * uy * uy)

    def expand(q, m):
        return sum(k * h * v for k, h, v in zip(fac, herm[q], m))

    feq = [W[q] * rho * (1 + 3 * (CX[q] * ux + CY[q] * uy) + expand(q, eq)) for q in range(9)]
    axx, axy, ayy = (sum(herm[q][i] * (f[q] - feq[q]) for q in range(9)) for i in range(3))
    axxy, ayyx = 2 * ux * axy + uy * axx, 2 * uy * axy + ux * ayy
    a = (axx, axy, ayy, axxy, ayyx,
         2 * (ux * ayyx + uy * axxy) - ux * ux * ayy - uy * uy * axx - 4 * ux * uy * axy)
    return [feq[q] + W[q] * (1 - omega) * expand(q, a) for q in range(9)], rho, jx, jy


def cells(n, umax, seed, noise):
    rng = np.random.default_rng(seed)
    for _ in range(n):
        u, th = umax * rng.uniform(), 2 * math.pi * rng.uniform()
        ux, uy, rho = u * math.cos(th), u * math.sin(th), 1 + 0.02 * rng.standard_normal()
        f = []
        for q in range(9):
            cu = CX[q] * ux + CY[q] * uy
            f.append(float(W[q]) * (rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * (ux * ux + uy * uy))
                                    + noise * rng.standard_normal()))
        yield f, float(rng.uniform(0.6, 1.95))


@pytest.mark.parametrize("shifted", [0, 1])
@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("umax,noise", [(1e-4, 1e-7), (0.05, 1e-4), (0.14, 1e-3), (0.14, 0.03)])
def test_collision_within_the_derived_error(lib, kind, shifted, umax, noise):
    """|f' - exact| per population: the final rounding (half a spacing); the
    fixed-point terms.  Unshifted loads are exact and the integer brackets are
    off by the roundings of the nonlinear terms alone, at most 14 units of 2^-59
    times 4 omega / 36: below 2^-57.  Shifted loads add half a unit each, 36 units in
    the rest bracket: below 2^-56.  The bracket's conversion and the rounded
    relaxation constant: 2^-51 of the change.  The reference weights' drift that
    the rest and axis brackets restore: omega 2^-54 of rho and |j|."""
    for f, omega in cells(60, umax, 17 + shifted, noise):
        ld = (4.0 - 2.0 * omega) / (4.0 * 0.25 * omega + 2.0 - omega)
        if shifted:
            f = [v - float(w) for v, w in zip(f, W)]
        a = np.array(f)
        assert lib.hc_collide(KINDS[kind], shifted, a.ctypes.data, omega, ld) == 0
        base = [Fr(v) + (w if shifted else 0) for v, w in zip(f, W)]
        ref, rho, jx, jy = exact_collide(kind, base, Fr(omega), Fr(ld))
        for q in range(9):
            want = ref[q] - (W[q] if shifted else 0)
            rate = max(omega, ld, 1.0)
            drift = rate * 2.0 ** -54 * float(rho if q == 0 else (abs(jx) + abs(jy) if q < 5 else 0))
            tol = (0.5 * math.ulp(abs(a[q])) + 2.0 ** (-56 if shifted else -57) + drift
                   + 2.0 ** -51 * abs(a[q] - f[q]))
            assert abs(float(Fr(a[q]) - want)) <= tol, (q, float(Fr(a[q]) - want), tol)


@pytest.mark.parametrize("kind", list(KINDS))
def test_cells_out_of_range_are_reported(lib, kind):
    """Negative, large and non-finite populations, and densities outside the
    reciprocal's range, report the cell instead of a wrapped result."""
    w = np.array([float(v) for v in W])
    for rho in (0.2, 2.6, 5.0, 1e3, 1e300):
        a = w * rho
        assert lib.hc_collide(KINDS[kind], 0, a.ctypes.data, 1.2, 1.0) == (0 if kind == "trt" and rho == 0.2 else 1)
    for q in range(9):
        for v in (-0.01, 1.5, math.inf, -math.inf, math.nan):
            for shifted in (0, 1):
                if shifted and v == -0.01:
                    continue
                a = np.zeros(9) if shifted else w.copy()
                a[q] = v
                assert lib.hc_collide(KINDS[kind], shifted, a.ctypes.data, 1.2, 1.0) == 1, (q, v, shifted)


def test_small_populations_and_rest(lib):
    """Populations below 2^-7 take the out-of-line load; a rest state of shifted
    populations stays exactly at rest."""
    for kind in KINDS.values():
        a = np.zeros(9)
        assert lib.hc_collide(kind, 1, a.ctypes.data, 1.2, 1.0) == 0 and not a.any()
    f = [float(w) for w in W]
    f[5] = 2.0 ** -8 + 2.0 ** -50
    f[6] = 0.0
    for name, kind in KINDS.items():
        a = np.array(f)
        assert lib.hc_collide(kind, 0, a.ctypes.data, 1.2, 1.0) == 0
        ref, rho, _, _ = exact_collide(name, [Fr(v) for v in f], Fr(1.2), Fr(1.0))
        assert max(abs(float(Fr(x) - r)) for x, r in zip(a, ref)) <= 2.0 ** -53 * 1.2 + 2.0 ** -54


def test_product_and_reciprocal(lib):
    """mulh64 within 2 units of a b / 2^64; recip_fixed within 2^-59 relative."""
    rng = np.random.default_rng(3)
    for _ in range(2000):
        a, b = (int(rng.integers(-2 ** 62, 2 ** 62)) >> int(rng.integers(0, 40)) for _ in range(2))
        assert abs(Fr(lib.hc_mulh64(a, b)) - Fr(a * b, 2 ** 64)) < 2
    lo, hi = (0x2000001 << 32), 2 ** 61 - 1
    for R in [lo, hi, 2 ** 59, 2 ** 59 - 1, 2 ** 60 + 1] + [int(v) for v in rng.integers(lo, hi, 2000)]:
        assert abs(Fr(lib.hc_recip(R)) * R / 2 ** 120 - 1) < Fr(1, 2 ** 59)


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("case", ["calm", "noisy", "binade", "small"])
def test_finish_in_the_populations_last_places(lib, kind, case):
    """The branch-free last operations: the bounds of
    test_collision_within_the_derived_error and the product's two units of 2^-59.
    binade: populations a few spacings from a power of two, which the collision
    moves across it; small: one below 2^-7, and one zero."""
    states = list(cells(60, 0.05, 23, 1e-4) if case == "calm" else cells(60, 0.14, 29, 0.03))
    for i, (f, omega) in enumerate(states):
        if case == "binade":
            f = [float(w) for w in W]
            f[1 + i % 4] = 0.125 + (i - 30) * 2.0 ** -55
            f[5 + i % 4] = 0.03125 + (30 - i) * 2.0 ** -57
        elif case == "small":
            f[5 + i % 4], f[1 + i % 4] = (2.0 ** -8 + i * 2.0 ** -60, 0.0)
        ld = (4.0 - 2.0 * omega) / (4.0 * 0.25 * omega + 2.0 - omega)
        a = np.array(f)
        assert lib.hc_collide_quick(KINDS[kind], a.ctypes.data, omega, ld) == 0
        ref, rho, jx, jy = exact_collide(kind, [Fr(v) for v in f], Fr(omega), Fr(ld))
        for q in range(9):
            drift = max(omega, ld, 1.0) * 2.0 ** -54 * float(rho if q == 0 else (abs(jx) + abs(jy) if q < 5 else 0))
            tol = (0.5 * math.ulp(abs(a[q])) + 2.0 ** -57 + 2.0 ** -58 + drift + 2.0 ** -51 * abs(a[q] - f[q])
                   + (2.0 ** -58 if case == "small" else 0))  # populations below 2^-7 are rounded by the load
            assert abs(float(Fr(a[q]) - ref[q])) <= tol, (q, float(Fr(a[q]) - ref[q]), tol)
