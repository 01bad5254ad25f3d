"""Several steps of a deviation-storage grid in one pass over memory
(step_march.cu): the bits and the buffers of single steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grid(nx, ny, storage, math, state):
    from plbm import LatticeGrid
    g = LatticeGrid(nx, ny, collision="bgk", storage=storage, math=math)
    g.set_relaxation(1 / 0.6, 0.25)
    g.set_pdf_to_equilibrium(*state)
    return g


@pytest.mark.parametrize("storage,math", [("f32dev", "fma"), ("f16dev", "fma"), ("f32dev", "hybrid")])
@pytest.mark.parametrize("nx,ny", [(64, 33000), (16400, 130), (1500, 1401), (1201, 1792), (1449, 1456)])
def test_marched_steps_equal_single_steps(gpu_lib, storage, math, nx, ny):
    """Both lattices and the buffer indices after every count of steps a plan can
    split differently; rows that fill strips of 56 and 60 exactly and not, odd row
    counts (whose edge strips wrap at an odd row), the fewest columns and rows."""
    rng = np.random.default_rng(nx + ny)
    state = (1 + 0.01 * rng.standard_normal((nx, ny)), 0.03 * rng.standard_normal((nx, ny)),
             0.03 * rng.standard_normal((nx, ny)))
    a, b = grid(nx, ny, storage, math, state), grid(nx, ny, storage, math, state)
    for n in (4, 5, 6, 11, 12):
        a.perform_lbm_step(n)
        for _ in range(n):
            b.perform_lbm_step(1)
        assert a.indices == b.indices
    for i in (1, 2):
        assert np.array_equal(a.download(i)[:, :, :ny], b.download(i)[:, :, :ny])
    a.close()
    b.close()


def test_march_inside_a_stream_capture(gpu_lib):
    """A caller's own capture records the passes; replaying it advances the grid."""
    import torch
    nx, ny = 1100, 1024
    rng = np.random.default_rng(4)
    state = (np.ones((nx, ny)), 0.03 * rng.standard_normal((nx, ny)), 0.03 * rng.standard_normal((nx, ny)))
    a, b = grid(nx, ny, "f32dev", "fma", state), grid(nx, ny, "f32dev", "fma", state)
    s = torch.cuda.Stream()
    a.set_stream(s)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=s):
        a.perform_lbm_step(8)
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    b.perform_lbm_step(16)
    assert np.array_equal(a.download(a.iold)[:, :, :ny], b.download(b.iold)[:, :, :ny])
    a.close()
    b.close()


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 3), (17, 13), (33, 64), (64, 65)])
def test_compensated_step_in_column_pairs(gpu_lib, nx, ny):
    """Two columns per thread: every storage of the compensated collision against the
    same grid with its columns rolled by one, which pairs them differently."""
    rng = np.random.default_rng(9)
    state = [1 + 0.01 * rng.standard_normal((nx, ny)), 0.03 * rng.standard_normal((nx, ny)),
             0.03 * rng.standard_normal((nx, ny))]
    for storage in ("f32dev", "f16dev"):
        a = grid(nx, ny, storage, "hybrid", state)
        b = grid(nx, ny, storage, "hybrid", [np.roll(s, 1, axis=0) for s in state])
        for g in (a, b):
            g.perform_lbm_step(3)
        assert np.array_equal(np.roll(a.download(a.iold)[:, :, :ny], 1, axis=1), b.download(b.iold)[:, :, :ny])
        a.close()
        b.close()
