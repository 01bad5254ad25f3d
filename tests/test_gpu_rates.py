"""Relaxation rates outside (0, 2) through the entry points that take one per call
(plbm_launch_step, the plugin's step): the strict operator's result, or NaN where it
gives NaN."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KINDS = {"bgk": 0, "trt": 1, "rr": 2}
W = np.array((4 / 9,) + (1 / 9,) * 4 + (1 / 36,) * 4)
RATES = [-1.0, 0.0, 1.9, 2.0, 2.05, 2.5, 4.6, 5.0, 100.0, math.nan]


def bound(omega):
    """Two binary64 evaluations of f + omega (feq - f), values below one: 32 roundings of 2^-53 each
    way, in the terms that omega scales too."""
    return 64 * 2.0 ** -53 * (1 + abs(omega))


@pytest.mark.parametrize("math_", [0, 2])  # FMA, HYBRID
@pytest.mark.parametrize("nx,ny", [(33, 47), (160, 161)])  # the branch-free last operations, and above them
@pytest.mark.parametrize("kind", KINDS)
def test_launch_step(gpu_lib, kind, nx, ny, math_):
    import torch
    ld = (ny + 15) // 16 * 16
    rng = np.random.default_rng(ny)
    f = torch.from_numpy(W[:, None, None] * (1 + 0.02 * rng.standard_normal((9, nx, ld)))).cuda()
    for omega in RATES:
        out = [torch.zeros_like(f) for _ in range(2)]
        for o, m in zip(out, (1, math_)):
            assert gpu_lib.plbm_launch_step(0, m, KINDS[kind], nx, ny, ld, C.c_void_p(f.data_ptr()),
                                            C.c_void_p(o.data_ptr()), omega, 0.25, None) == 0
        torch.cuda.synchronize()
        want, got = (o[:, :, :ny].cpu().numpy() for o in out)
        assert np.array_equal(np.isnan(want), np.isnan(got)), omega
        if not math.isnan(omega):
            assert np.max(np.abs(got - want)) <= bound(omega), omega


@pytest.mark.parametrize("math_", ["fma", "hybrid"])
@pytest.mark.parametrize("kind", ["rr"])
def test_plugin_step(gpu_lib, kind, math_):
    """One step from a flow's equilibrium (moments, of sums of nine populations)."""
    from plbm.plugin import SimPlugin, make_params
    nx, ny = 37, 29
    rng = np.random.default_rng(8)
    p = np.asfortranarray(0.01 * rng.standard_normal((nx, ny)))
    u = np.asfortranarray(0.05 * rng.standard_normal((nx, ny, 2)))
    for omega in RATES:
        out = []
        for m in ("strict", math_):
            sim = SimPlugin()
            sim.init((nx, ny), 1.0, p, u, params=make_params(kind=kind, math=m, trt_magic=0.25))
            sim.steps(omega, 2)
            out.append(sim.vars())
        for want, got in zip(*out):
            assert np.array_equal(np.isnan(want), np.isnan(got)), omega
            if not math.isnan(omega):
                assert np.max(np.abs(got - want)) <= 9 * (1 + abs(omega)) * bound(omega), omega
