"""The finite-difference schemes' fixed-point kernel (k_step_scheme_fixed) at the
edges of its tiles (32 rows by 4, 8 or 16 columns), its range and its rule."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_schemes import KIND, gpu_grid, relinf, state

pytestmark = pytest.mark.gpu

# Three steps; the oracle's own evaluation rounds about ten times per step and
# population at 2^-53 of values below the largest one: 3 x 10 x 1.1e-16 < 1e-14.
TOL = 1e-14


def compare(nx, ny, scheme, kind, mode, dt, f0, steps=3):
    g = gpu_grid(nx, ny, scheme, kind, mode, dt, 0.05, f0)
    om, magic = g.omega, g.properties()["trt_magic"]
    g.perform_lbm_step(steps)
    got = g.download(g.iold)
    g.close()
    f2 = np.stack([np.zeros_like(f0), f0.copy()])
    iold, _ = O.perform_step_scheme(f2, ny, 2, 1, scheme, dt, KIND[kind], om, magic, steps)
    assert relinf(got[:, :, :ny], f2[iold - 1][:, :, :ny]) <= TOL


@pytest.mark.parametrize("scheme,kind", [("fdm_bardow", "bgk"), ("fvm_bardow", "rr"), ("fdm_sofonea", "trt"),
                                         ("fdm_bardow_iso", "bgk"), ("fdm_bardow_wls", "trt")])
@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 3), (3, 31), (2, 32), (5, 33), (16, 64), (17, 65), (300, 200),
                                   (1300, 1201)])
def test_tile_edges(gpu_lib, scheme, kind, nx, ny):
    compare(nx, ny, scheme, kind, "fma", 0.3, state(nx, ny), steps=2 if nx > 1000 else 3)


@pytest.mark.parametrize("scheme", ["fdm_bardow", "fdm_sofonea", "fdm_bardow_iso"])
@pytest.mark.parametrize("mode", ["fma", "hybrid"])
def test_range_and_rule(gpu_lib, scheme, mode):
    """Cells past the fixed point's range (density 3, 0.1, and a patch of it among
    ordinary cells), populations below 2^-7, and a time step past the rule."""
    nx, ny = 40, 70
    f0 = state(nx, ny)
    for factor in (3.0, 0.1):
        compare(nx, ny, scheme, "bgk", mode, 0.3, f0 * factor)
    patch = f0.copy()
    patch[:, 18:23, 30:36] *= 2.6
    compare(nx, ny, scheme, "rr", mode, 0.3, patch)
    small = f0.copy()
    small[5, 10, 10] = small[2, 35, 60] = 1e-3
    compare(nx, ny, scheme, "bgk", mode, 0.3, small)
    compare(nx, ny, scheme, "bgk", mode, 1.5, f0, steps=1)
