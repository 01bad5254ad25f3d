"""Schemes in the stencil form (step_hybrid.cu) on grids of many sizes: a lattice of repeated copies
of a small one evolves as its copies."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(nx, ny, kind, state):
    from plbm import LatticeGrid
    with LatticeGrid(nx, ny, collision=kind, math="hybrid", streaming="fdm_bardow_wls_gauss_v1") as g:
        g.set_properties(0.05, 0.3)
        g.set_pdf_to_equilibrium(*state)
        g.perform_lbm_step(5)
        return g.download(g.iold)[:, :, :ny]


@pytest.mark.parametrize("kind", ["bgk", "trt", "rr"])
@pytest.mark.parametrize("nx,ny,cx,cy", [(1, 1, 3, 5), (5, 3, 7, 11), (3, 32, 17, 8), (10, 257, 30, 1), (19, 32, 16, 8),
                                         (31, 33, 33, 31)])
def test_copies_evolve_as_the_small_lattice(gpu_lib, nx, ny, cx, cy, kind):
    """Bit for bit, in blocks of every size, with and without a share of its own for each SM."""
    rng = np.random.default_rng(nx + ny)
    state = [1 + 0.01 * rng.standard_normal((nx, ny)), 0.03 * rng.standard_normal((nx, ny)),
             0.03 * rng.standard_normal((nx, ny))]
    small = run(nx, ny, kind, state)
    large = run(nx * cx, ny * cy, kind, [np.tile(s, (cx, cy)) for s in state])
    assert np.array_equal(large, np.tile(small, (1, cx, cy)))
