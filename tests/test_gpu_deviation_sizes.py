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


@pytest.mark.parametrize("nx,ny", [(1025, 1031), (1026, 1029), (1449, 730), (2047, 513)])
def test_column_pairs_of_the_compensated_step(gpu_lib, nx, ny):
    """Two columns per thread, from 2^20 cells, odd and even column counts: the same grid with its
    columns rolled by one, which pairs them differently, gives the same bits."""
    rng = np.random.default_rng(nx)
    state = [1 + 0.01 * rng.standard_normal((nx, ny)), 0.03 * rng.standard_normal((nx, ny)),
             0.03 * rng.standard_normal((nx, ny))]
    a = run(nx, ny, "f32dev", "hybrid", state, 3)
    b = run(nx, ny, "f32dev", "hybrid", [np.roll(s, 1, axis=0) for s in state], 3)
    assert np.array_equal(np.roll(a, 1, axis=1), b)


# 2^20 = 1024^2: binary32 takes other operators from there on, in single steps and marched
@pytest.mark.parametrize("nx,ny", [(1021, 1024), (1027, 1024), (1203, 1201)])
@pytest.mark.parametrize("storage,math", [("f32dev", "fma"), ("f32dev", "hybrid"), ("f16dev", "fma"), ("f16dev", "hybrid")])
def test_either_side_of_the_line_against_binary64(gpu_lib, storage, math, nx, ny):
    """Twelve steps of one flow, largest distance of a population from the strict binary64 grid's.  A step
    rounds a population's deviation, below 1/16, to storage (2^-24 or 2^-11 of it), and the plain
    operators round rho = 1 + sum h and its products, 4 x 2^-24 of populations below 1/2; the flow
    does not amplify them more than twice over these steps.  One bound for all sizes."""
    rng = np.random.default_rng(11)
    x, y = np.arange(nx)[:, None] * 2 * np.pi / nx, np.arange(ny)[None, :] * 2 * np.pi / ny
    state = [1 + 0 * x * y, 0.04 * np.cos(x) * np.sin(y) + 1e-3 * rng.standard_normal((nx, ny)),
             -0.04 * np.sin(x) * np.cos(y) + 1e-3 * rng.standard_normal((nx, ny))]
    got = run(nx, ny, storage, math, state, 12)
    want = run(nx, ny, "f64", "strict", state, 12)
    store = (2.0 ** -24 if storage == "f32dev" else 2.0 ** -11) / 16
    assert np.max(np.abs(got - want)) <= 2 * 12 * (store + 4 * 2.0 ** -24 / 2)


@pytest.mark.parametrize("storage,math", [("f32dev", "strict"), ("f16dev", "strict"), ("f32dev", "df64"), ("f16dev", "df64")])
@pytest.mark.parametrize("nx,ny,cx,cy", [(1, 1, 3, 5), (5, 3, 7, 11), (3, 32, 17, 8), (10, 257, 30, 1), (31, 33, 33, 31)])
def test_binary64_collisions_of_copies(gpu_lib, nx, ny, cx, cy, storage, math):
    """Collisions in binary64 and double-float: a lattice of copies evolves as its copies bit for bit, in
    blocks of every size, rows that fill them and rows that do not."""
    rng = np.random.default_rng(nx + ny)
    state = [1 + 0.01 * rng.standard_normal((nx, ny)), 0.05 * rng.standard_normal((nx, ny)),
             0.05 * rng.standard_normal((nx, ny))]
    small = run(nx, ny, storage, math, state, 6)
    large = run(nx * cx, ny * cy, storage, math, [np.tile(s, (cx, cy)) for s in state], 6)
    assert np.array_equal(large, np.tile(small, (1, cx, cy)))
