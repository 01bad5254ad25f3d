"""Steps whose threads are laid over the cells row after row (plbm_launch.h): rows
shorter and longer than a block, of every remainder, at the sizes where the launch
changes its blocks, its order of cells or the shared memory that limits an SM's
blocks.  A lattice rolled along the rows evolves as the rolled lattice, with its cells
in other threads; a lattice of two copies evolves as the one, in another launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 300), (300, 1), (2, 31), (77, 33), (64, 64), (129, 63), (200, 129), (257, 257), (300, 300), (450, 330),
         (641, 500), (1000, 65), (1030, 1021)]
MODES = [("rr", "f64", "fma"), ("bgk", "f64", "hybrid"), ("trt", "f64", "strict"), ("rr", "f32dev", "fma"),
         ("bgk", "f16dev", "fma"), ("trt", "f16dev", "fma"), ("bgk", "f32dev", "hybrid")]


def state(nx, ny):
    rng = np.random.default_rng(nx * 10000 + ny)
    return [1 + 0.01 * rng.standard_normal((nx, ny)), 0.03 * rng.standard_normal((nx, ny)),
            0.03 * rng.standard_normal((nx, ny))]


def run(nx, ny, mode, fields, steps=3):
    from plbm import LatticeGrid
    g = LatticeGrid(nx, ny, collision=mode[0], storage=mode[1], math=mode[2])
    g.set_relaxation(1 / 0.7, 0.25)
    g.set_pdf_to_equilibrium(*fields)
    for _ in range(steps):
        g.perform_lbm_step(1)
    f = g.download(g.iold)[:, :, :ny]
    g.close()
    return f


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("nx,ny", SIZES)
def test_rolled_lattice_steps_to_the_rolled_result(gpu_lib, mode, nx, ny):
    fields = state(nx, ny)
    a = run(nx, ny, mode, fields)
    for shift in ((0, 1), (nx // 2, ny // 3)):
        b = run(nx, ny, mode, [np.roll(f, shift, axis=(0, 1)) for f in fields])
        assert np.array_equal(np.roll(a, shift, axis=(1, 2)), b)


@pytest.mark.parametrize("mode", [MODES[2], MODES[3], MODES[4]])
@pytest.mark.parametrize("nx,ny", [(1, 300), (129, 63), (300, 300), (450, 330)])
def test_two_copies_step_to_two_copies(gpu_lib, mode, nx, ny):
    fields = state(nx, ny)
    a, b = run(nx, ny, mode, fields), run(nx, 2 * ny, mode, [np.tile(f, (1, 2)) for f in fields])
    assert np.array_equal(b[:, :, :ny], a) and np.array_equal(b[:, :, ny:], a)


@pytest.mark.parametrize("kind,storage,math", [("bgk", "f64", "hybrid"), ("rr", "f64", "fma"), ("trt", "f64", "strict"),
                                               ("rr", "f32dev", "fma")])
@pytest.mark.parametrize("nx,ny", [(1, 300), (300, 1), (33, 77), (300, 300), (641, 500)])
def test_plugin_rolled(gpu_lib, kind, storage, math, nx, ny):
    from plbm.plugin import SimPlugin, make_params
    rng = np.random.default_rng(nx + ny)
    p, u = 0.003 * rng.standard_normal((nx, ny)), 0.03 * rng.standard_normal((nx, ny, 2))
    out = []
    for shift in ((0, 0), (nx // 2, ny // 3)):
        sim = SimPlugin()
        sim.init((nx, ny), 1.0, np.asfortranarray(np.roll(p, shift, axis=(0, 1))),
                 np.asfortranarray(np.roll(u, shift, axis=(0, 1))),
                 params=make_params(kind=kind, storage=storage, math=math, trt_magic=0.25))
        sim.steps(1 / 0.7, 3)
        out.append([np.array(v) for v in sim.vars()])
    for a, b in zip(*out):
        assert np.array_equal(np.roll(a, (nx // 2, ny // 3), axis=(0, 1)), b)


@pytest.mark.parametrize("storage,math", [("f64", "fma"), ("f32dev", "fma"), ("f32dev", "hybrid")])
@pytest.mark.parametrize("nx,ny,copies", [(3, 128, 2), (5, 85, 3), (2, 51, 5), (40, 150, 2)])
def test_reverse_steps_of_copies(gpu_lib, storage, math, nx, ny, copies):
    """The reverse step in rows (256, 255 rows) and over flat cells: the gradient of
    copies is the copies of the gradient, dL/domega their sum (binary64 sums of equal
    terms in another order: 1e-12 of the terms' size, at most 40 x 300 of them)."""
    import torch
    from plbm.autograd import Adjoint
    rng = np.random.default_rng(nx + ny)
    u, g = 0.03 * rng.standard_normal((2, nx, ny)), rng.standard_normal((2, nx, ny))
    out = []
    for k in (1, copies):
        a = Adjoint(nx, ny * k, 4, checkpoint_every=2, storage=storage, math=math)
        a.forward(torch.tensor(np.tile(u, (1, 1, k)), device="cuda"), 1.4)
        gu, dom = a.backward(torch.tensor(np.tile(g, (1, 1, k)), device="cuda"))
        out.append((gu.cpu().numpy(), dom / k))
        a.close()
    assert np.array_equal(np.tile(out[0][0], (1, 1, copies)), out[1][0])
    assert abs(out[0][1] - out[1][1]) <= 1e-12 * nx * ny
