"""Deviation storage on grids of either side of the sizes that are marched
(step_march.cu): a lattice of repeated copies of a small one evolves as its copies."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(nx, ny, storage, math, state, steps):
    from plbm import LatticeGrid
    with LatticeGrid(nx, ny, collision="bgk", storage=storage, math=math) as g:
        g.set_relaxation(1 / 0.6, 0.25)
        g.set_pdf_to_equilibrium(*state)
        g.perform_lbm_step(steps)
        return g.download(g.iold)[:, :, :ny]


@pytest.mark.parametrize("math", ["fma", "hybrid"])
@pytest.mark.parametrize("nx,ny,cx,cy", [
    (128, 128, 8, 10),   # 1024 x 1280, marched, strips of whole pairs
    (131, 101, 8, 16),   # 1048 x 1616, marched, 101 odd and 1616 even: pairs and single cells
    (129, 201, 12, 7),   # 1548 x 1407, marched, odd rows on both
    (101, 131, 11, 9),   # 1111 x 1179, above 2^20 cells and not marched
])
def test_binary16_copies_evolve_as_the_small_lattice(gpu_lib, nx, ny, cx, cy, math):
    """Bit for bit: binary16 BGK, plain and compensated, is one operator, however many cells, cells per thread
    or steps per pass.  (Another rounding inside the operator shows as one unit of
    binary16, 2^-11 of a population's deviation, within a few steps.)"""
    rng = np.random.default_rng(nx + cy)
    state = [1 + 0.01 * rng.standard_normal((nx, ny)), 0.05 * rng.standard_normal((nx, ny)),
             0.05 * rng.standard_normal((nx, ny))]
    small = run(nx, ny, "f16dev", math, state, 14)
    large = run(nx * cx, ny * cy, "f16dev", math, [np.tile(s, (cx, cy)) for s in state], 14)
    assert np.array_equal(large, np.tile(small, (1, cx, cy)))
