"""The two forms of the fixed-point lattice step beside the one-cell-per-thread one
(step_hybrid.cu): columns copied ahead on large grids, branch-free last operations
on small ones.  A lattice that repeats a small one's state evolves as copies of
it, so either form is compared with the one-cell form of another size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grid(nx, ny, kind, math, tile, reps=(1, 1)):
    from plbm import LatticeGrid
    g = LatticeGrid(nx, ny, collision=kind, math=math)
    g.set_relaxation(1 / 0.6, 0.25)
    g.set_pdf_to_equilibrium(*(np.tile(t, reps) for t in tile))
    return g


def tile_state(nx, ny, patch):
    rng = np.random.default_rng(nx * ny)
    rho = 1 + 0.01 * rng.standard_normal((nx, ny))
    if patch:  # past the fixed point's range, among ordinary cells and at the edges
        rho[: min(3, nx), -2:] = 3.0
        rho[nx // 2, ny // 3:ny // 3 + 5] = 3.0
    return rho, 0.03 * rng.standard_normal((nx, ny)), 0.03 * rng.standard_normal((nx, ny))


# (tile, repetitions): the tile itself between the small grids' form and the
# columns-ahead one; repeated, past its line: rows below, at and past a multiple of
# 128 and the fewest taken; columns that the segments of 4 and 8 divide and not.
@pytest.mark.parametrize("kind,math,patch", [("bgk", "fma", False), ("bgk", "hybrid", True), ("trt", "fma", True)])
@pytest.mark.parametrize("nx,ny,rx,ry", [(1031, 64, 65, 1), (517, 127, 65, 1), (520, 128, 65, 1), (511, 129, 66, 1),
                                         (300, 300, 7, 7), (299, 317, 19, 19)])
def test_columns_ahead_equal_one_cell_per_thread(gpu_lib, kind, math, patch, nx, ny, rx, ry):
    tile = tile_state(nx, ny, patch)
    a, b = grid(nx, ny, kind, math, tile), grid(nx * rx, ny * ry, kind, math, tile, (rx, ry))
    for g in (a, b):
        g.perform_lbm_step(3)
    fa, fb = (g.download(g.iold)[:, :, :g.ny] for g in (a, b))
    a.close()
    b.close()
    for j in range(ry):
        for i in range(rx):
            assert np.array_equal(fb[:, i * nx:(i + 1) * nx, j * ny:(j + 1) * ny], fa), (i, j)


@pytest.mark.parametrize("kind", ["bgk", "trt", "rr"])
@pytest.mark.parametrize("nx,ny", [(1, 1), (3, 2), (31, 33), (64, 64), (128, 128)])
def test_small_grid_form(gpu_lib, kind, nx, ny):
    """Three steps; either form rounds a population once per step at 2^-53 of values
    below 1 and the streaming and collision pass differences on at most fourfold:
    3 x 2 x 1.1e-16 x 4 < 3e-15."""
    tile = tile_state(nx, ny, nx > 3)
    rx, ry = (300 // nx + 1, 300 // ny + 1) if nx < 128 else (2, 1)
    a, b = grid(nx, ny, kind, "fma", tile), grid(nx * rx, ny * ry, kind, "fma", tile, (rx, ry))
    for g in (a, b):
        g.perform_lbm_step(3)
    fa, fb = (g.download(g.iold)[:, :nx, :ny] for g in (a, b))
    a.close()
    b.close()
    assert np.abs(fa - fb).max() <= 3e-15
