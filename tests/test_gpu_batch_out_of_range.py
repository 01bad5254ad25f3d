"""Batched cells outside the fixed point's range (hybrid.cuh) take the binary64
operator, in both launch modes, beside ordinary cells of the same tile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fields(nx, ny, seed):
    """Density 1 with a patch of density 3 (f_0 > 1) and one of 0.2 (the reciprocal's range)."""
    rng = np.random.default_rng(seed)
    rho = 1 + 0.01 * rng.standard_normal((nx, ny))
    rho[nx // 4:nx // 2, ny // 3:2 * ny // 3] = 3.0
    rho[-3:, :5] = 0.2
    return rho, 0.02 * rng.standard_normal((nx, ny)), 0.02 * rng.standard_normal((nx, ny))


@pytest.mark.parametrize("threads,persistent", [(256, 1), (512, 1), (128, 0), (256, 0)])
@pytest.mark.parametrize("math", ["fma", "hybrid"])
@pytest.mark.parametrize("steps", [1, 2, 5])
def test_against_the_strict_grid(gpu_lib, math, threads, persistent, steps):
    """One step of either operator rounds within 4 spacings of values below 4 (3.6e-15);
    differences grow with the flow's gradients by at most a factor of two per step
    around the patches: 2^steps - 1 of them."""
    from plbm import LatticeGrid
    from plbm.batched import BatchedGrids, GridSpec, Schedule
    sizes = [(37, 45), (96, 130)]
    specs = [GridSpec(nx, ny, kind, 1.4, 0.25) for nx, ny in sizes for kind in ("bgk", "trt")]
    with BatchedGrids(specs, "f64", math) as b:
        b.schedule = Schedule.from_dict({"threads": threads, "ctas_per_sm": 0, "persistent": persistent,
                                         "ty": [32] * 5})
        for i, s in enumerate(specs):
            b.set_equilibrium(i, *fields(s.nx, s.ny, i))
        b.run(steps)
        for i, s in enumerate(specs):
            with LatticeGrid(s.nx, s.ny, collision=s.kind, math="strict") as g:
                g.set_relaxation(s.omega, s.trt_magic)
                g.set_pdf_to_equilibrium(*fields(s.nx, s.ny, i))
                g.perform_lbm_step(steps)
                want = g.download(g.iold)[:, :, :s.ny]
            got = b.download(i)[:, :, :s.ny]
            assert np.max(np.abs(got - want)) <= 3.6e-15 * (2 ** steps - 1), (i, s.kind)
