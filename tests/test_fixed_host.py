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
