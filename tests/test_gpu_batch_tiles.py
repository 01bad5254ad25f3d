"""The batch's tiles (consecutive cells of strips of rows) at their edges: strips of
every remainder, grids narrower than a tile, CTAs with more tiles than their table
holds, both launch modes and storages, against grids stepped alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 40), (40, 1), (2, 31), (3, 32), (5, 33), (7, 47), (4, 48), (9, 49), (3, 63), (6, 64), (5, 65),
         (33, 96), (2, 97), (31, 127), (8, 128), (2, 129), (3, 383), (2, 384), (5, 385), (1, 511), (2, 512), (3, 513),
         (2, 767), (1, 768), (2, 1025), (200, 300), (701, 650)]


def state(nx, ny):
    rng = np.random.default_rng(nx * 1000 + ny)
    return (1 + 0.01 * rng.standard_normal((nx, ny)), 0.03 * rng.standard_normal((nx, ny)),
            0.03 * rng.standard_normal((nx, ny)))


# 64 threads, one CTA per SM: over 32 tiles per CTA.
@pytest.mark.parametrize("threads,ctas,persistent,ty", [(256, 0, 1, [32, 64, 128, 256, 256]), (64, 1, 1, [32] * 5),
                                                        (512, 0, 1, [512] * 5), (128, 0, 0, [32, 64, 128, 128, 128]),
                                                        (96, 0, 1, [32] * 5)])
@pytest.mark.parametrize("storage", ["f64", "f32dev"])
def test_tile_edges(gpu_lib, storage, threads, ctas, persistent, ty):
    """Three steps.  Binary64: a grid of at most 2^14 cells ends its collisions with
    another rounding of the same values, 3 x 2 x 1.1e-16 x 4 < 3e-15; binary32: the same
    operations, up to the order of a fused multiply-add, 3 x 6e-8 x 4 of values below 1."""
    from plbm import LatticeGrid
    from plbm.batched import BatchedGrids, GridSpec, Schedule
    specs = [GridSpec(nx, ny, ("bgk", "trt")[i % 2], 1 / (0.55 + 0.05 * (i % 7)), 0.25)
             for i, (nx, ny) in enumerate(SIZES)]
    b = BatchedGrids(specs, storage, "fma")
    b.schedule = Schedule.from_dict({"threads": threads, "ctas_per_sm": ctas, "persistent": persistent, "ty": ty})
    for i, (nx, ny) in enumerate(SIZES):
        b.set_equilibrium(i, *state(nx, ny))
    b.run(2)
    b.run(1)
    b.synchronize()
    for i, (nx, ny) in enumerate(SIZES):
        g = LatticeGrid(nx, ny, collision=specs[i].kind, storage=storage, math="fma")
        g.set_relaxation(specs[i].omega, 0.25)
        g.set_pdf_to_equilibrium(*state(nx, ny))
        g.perform_lbm_step(3)
        d = np.abs(b.download(i)[:, :, :ny] - g.download(g.iold)[:, :, :ny]).max()
        g.close()
        assert d <= (3e-15 if storage == "f64" else 7e-7), (nx, ny, d)
    b.close()
