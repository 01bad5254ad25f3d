"""The binary32 operators of csrc/f32x2.cuh and the reciprocals under them, from a host
build with reciprocal seeds at and an ulp to either side of the rounded quotient (the
hardware's are within one), against exact or binary64 arithmetic."""
import ctypes as C
import subprocess
from fractions import Fraction as Fr
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
CX = np.array((0, 1, 0, -1, 0, 1, -1, -1, 1.0))
CY = np.array((0, 0, 1, 0, -1, 1, 1, -1, -1.0))
W = np.array((4 / 9,) + (1 / 9,) * 4 + (1 / 36,) * 4)


@pytest.fixture(scope="module", params=[-1, 0, 1])
def lib(request, tmp_path_factory):
    so = tmp_path_factory.mktemp("pk") / "pk.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", f"-DSEED_ULPS={request.param}",
                    "-I", str(ROOT / "periodic-lbm_gb300" / "csrc"), str(ROOT / "tests" / "packed_host.cpp"),
                    "-o", str(so)], check=True)
    h = C.CDLL(str(so))
    h.pk_recip_fixed.restype, h.pk_recip_fixed.argtypes = C.c_int64, [C.c_int64]
    h.pk_bgk.argtypes = [C.c_void_p, C.c_float, C.c_int]
    return h


def ptr(a):
    return C.c_void_p(a.ctypes.data)


def ulp(a):
    return np.spacing(np.abs(a).astype(np.float32)).astype(np.float64)


def test_reciprocal_and_quotient(lib):
    """1 / x within one ulp, a / x within half an ulp and a fiftieth, x over three octaves."""
    rng = np.random.default_rng(1)
    n = 400_000
    x = np.concatenate([np.linspace(0.5, 4.0, n, dtype=np.float32), np.float32(1) + np.float32(2.0 ** -23) * np.arange(-2000, 2000, dtype=np.float32)])
    a = (rng.uniform(-1, 1, x.size) * 2.0 ** rng.integers(-20, 3, x.size)).astype(np.float32)
    r, q = np.empty_like(x), np.empty_like(x)
    lib.pk_rcp(ptr(x), ptr(r), C.c_long(x.size))
    lib.pk_quot(ptr(a), ptr(x), ptr(q), C.c_long(x.size))
    x64, a64 = x.astype(np.float64), a.astype(np.float64)
    assert np.max(np.abs(r - 1 / x64) / ulp(r)) <= 1.0
    assert np.max(np.abs(q - a64 / x64) / ulp(q)) <= 0.52


def test_fixed_point_reciprocal(lib):
    """2^61 / rho within 2^-59, rho between 1/4 and 4."""
    rng = np.random.default_rng(3)
    lo, hi = (0x2000001 << 32), 2 ** 61 - 1
    for R in [lo, hi, 2 ** 59, 2 ** 59 - 1, 2 ** 59 + 1, 2 ** 60 + 1] + [int(v) for v in rng.integers(lo, hi, 4000)]:
        assert abs(Fr(lib.pk_recip_fixed(R)) * R / 2 ** 120 - 1) < Fr(1, 2 ** 59)


@pytest.mark.parametrize("f16", [0, 1])
@pytest.mark.parametrize("umax,noise", [(1e-4, 1e-6), (0.05, 1e-4), (0.15, 0.02)])
def test_bgk_of_a_cell(lib, f16, umax, noise):
    """Against binary64 on the same h: the last operations round the new and the relaxed value once
    each, the terms under the weight take at most ten roundings of the moments' terms, each below
    3 sum |h| (binary16: h scaled by 2^15, and a division within 2 ulp: fourteen)."""
    rng = np.random.default_rng(5)
    scale = 32768.0 if f16 else 1.0
    for _ in range(300):
        omega = np.float32(rng.uniform(0.6, 1.95))
        u, th, rho = umax * rng.uniform(), 2 * np.pi * rng.uniform(), 1 + 0.02 * rng.standard_normal()
        cu = u * (CX * np.cos(th) + CY * np.sin(th))
        h = W * (rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * u * u) - 1 + noise * rng.standard_normal(9))
        H = (h * scale).astype(np.float16 if f16 else np.float32).astype(np.float32)
        h = H.astype(np.float64) / scale
        d, jx, jy = h.sum(), CX @ h, CY @ h
        cj = CX * jx + CY * jy
        heq = W * (d + 3 * cj + (4.5 * cj * cj - 1.5 * (jx * jx + jy * jy)) / (1 + d))
        want = h + float(omega) * (heq - h)
        lib.pk_bgk(H.ctypes.data, omega, f16)
        tol = 2.0 ** -24 * (np.abs(want) + 2 * float(omega) * (np.abs(h) + np.abs(heq))
                            + float(omega) * W * (14 if f16 else 10) * 3 * np.abs(h).sum())
        assert np.all(np.abs(H / scale - want) <= tol)
