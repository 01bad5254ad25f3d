"""Single operations of the fixed-point collisions from a host build of their headers."""
import ctypes
import subprocess
from fractions import Fraction as Fr
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("fx") / "fx.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off",
                    "-I", str(ROOT / "periodic-lbm_gb300" / "csrc"), str(ROOT / "tests" / "fixed_host.cpp"),
                    "-o", str(so)], check=True)
    h = ctypes.CDLL(str(so))
    h.fx_to_double.restype = ctypes.c_double
    h.fx_bgk_shifted.argtypes = [ctypes.c_void_p, ctypes.c_double]
    h.fx_load_shifted.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    h.fx_to_double.argtypes = [ctypes.c_int64, ctypes.c_int]
    return h


def integers(n, seed):
    """Of every length, both signs, and the neighbours of the powers of two."""
    rng = np.random.default_rng(seed)
    out = [0] + [s * (2 ** k + d) for k in range(1, 62) for d in (-1, 0, 1) for s in (1, -1)]
    return out + [int(v) >> int(k) for v, k in zip(rng.integers(-2 ** 62, 2 ** 62, n), rng.integers(0, 60, n))]


def test_conversion_to_binary64(lib):
    """Up to 53 bits: exact with EXACT, else within one unit, on the side of zero; above, truncated to
    53 bits."""
    for t in integers(4000, 1):
        exact, near = (Fr(lib.fx_to_double(t, e)) * 2 ** 59 for e in (1, 0))
        ulp = Fr(2) ** max(0, abs(t).bit_length() - 53)
        assert (exact == t if ulp == 1 else 0 <= abs(t) - abs(exact) < ulp), t
        assert 0 <= abs(t) - abs(near) < ulp + 1, t


CX, CY = (0, 1, 0, -1, 0, 1, -1, -1, 1), (0, 0, 1, 0, -1, 1, 1, -1, -1)
W = (Fr(4, 9),) + (Fr(1, 9),) * 4 + (Fr(1, 36),) * 4


def exact_shifted_bgk(h, omega):
    rho1, jx, jy = sum(h), sum(c * v for c, v in zip(CX, h)), sum(c * v for c, v in zip(CY, h))
    rho = 1 + rho1
    out = []
    for q in range(9):
        cj = CX[q] * jx + CY[q] * jy
        eq = W[q] * (rho1 + 3 * cj + (Fr(9, 2) * cj * cj - Fr(3, 2) * (jx * jx + jy * jy)) / rho)
        out.append(h[q] + omega * (eq - h[q]))
    return out, abs(rho1), abs(jx) + abs(jy)


@pytest.mark.parametrize("exponent", [-27, -28, -29, -30, -31, -33, -40, -60, -61, -80, -300, -1000])
def test_shifted_cells_of_tiny_deviations(lib, exponent):
    """A cell whose largest |h| is below 2^-27 is held in units 2^-54 of that and finer: the load rounds to
    a unit, the brackets add up 36 of them at 4 omega / 36, as in the shifted collision's test with
    half a unit, 2^-55 in units of which max |h| is 2^-6 and more."""
    rng = np.random.default_rng(-exponent)
    for _ in range(40):
        omega = float(rng.uniform(0.6, 1.95))
        h = np.ldexp(rng.uniform(-1, 1, 9), exponent)
        h[rng.integers(0, 9)] = np.ldexp(rng.choice([-1, 1]) * rng.uniform(0.5, 1.0), exponent)
        a = h.copy()
        assert lib.fx_bgk_shifted(a.ctypes.data, omega) == 1
        want, rho1, j = exact_shifted_bgk([Fr(float(v)) for v in h], Fr(omega))
        unit = Fr(2) ** -49 * max(abs(Fr(float(v))) for v in h)
        for q in range(9):
            drift = max(omega, 1.0) * Fr(2) ** -54 * (rho1 if q == 0 else (j if q < 5 else 0))
            tol = (Fr(float(np.spacing(abs(a[q])))) / 2 + unit + drift + Fr(2) ** -51 * abs(Fr(float(a[q])) - Fr(float(h[q]))))
            assert abs(Fr(float(a[q])) - want[q]) <= tol, q


def test_cells_at_rest_and_false_hints(lib):
    """Zeros stay at rest, negative ones too; two small populations beside larger ones take the
    fixed point out of line, not the binary64 operator."""
    for zero in (0.0, -0.0):
        a = np.full(9, zero)
        assert lib.fx_bgk_shifted(a.ctypes.data, 1.3) < 2 and not a.any()
    h = np.array([0.01, 1e-10, -1e-10, 0.02, 0.003, -0.004, 0.005, 0.006, -0.007])
    a = h.copy()
    assert lib.fx_bgk_shifted(a.ctypes.data, 1.3) == 1
    want, _, _ = exact_shifted_bgk([Fr(float(v)) for v in h], Fr(1.3))
    assert max(abs(Fr(float(x)) - y) for x, y in zip(a, want)) <= 2.0 ** -55
    h[3] = 0.2  # past the limit
    assert lib.fx_bgk_shifted(h.ctypes.data, 1.3) == 2


@pytest.mark.parametrize("top", [-5, -20, -27, -28, -29, -45, -57, -58, -59, -60, -61, -62, -100, -1022])
def test_shifted_load_rounds_to_nearest(lib, top):
    """Every deviation that the fixed point takes, of either sign and of every size: within half a
    unit of 2^-59, zeros of either sign zero."""
    rng = np.random.default_rng(-top)
    F = np.zeros(9, np.int64)
    for _ in range(60):
        h = np.ldexp(rng.choice([-1, 1], 9) * rng.uniform(0.5, 1.0, 9), top)
        h[rng.integers(0, 9)] = rng.choice([0.0, -0.0])
        assert lib.fx_load_shifted(h.ctypes.data, F.ctypes.data)
        for q in range(9):
            assert abs(Fr(float(h[q])) * 2 ** 59 - int(F[q])) <= Fr(1, 2), (q, h[q])
