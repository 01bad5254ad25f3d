"""Every CTA size that a batch schedule may ask for, and batches of different sizes
side by side: the persistent kernel's shared memory grows with the threads, its limit
belongs to the kernel and not to the batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(40, 33), (64, 100), (17, 200), (130, 96)]
THREADS = [64, 96, 128, 160, 192, 224, 256, 288, 320, 352, 384, 416, 448, 480, 512]


def batch(threads, persistent=1):
    from plbm.batched import BatchedGrids, GridSpec, Schedule
    specs = [GridSpec(nx, ny, ("bgk", "trt")[i % 2], 1.3 + 0.1 * i, 0.25) for i, (nx, ny) in enumerate(SIZES)]
    b = BatchedGrids(specs, "f64", "fma")
    b.schedule = Schedule.from_dict({"threads": threads, "ctas_per_sm": 0, "persistent": persistent, "ty": [32] * 5})
    for i, (nx, ny) in enumerate(SIZES):
        rng = np.random.default_rng(i)
        b.set_equilibrium(i, 1 + 0.01 * rng.standard_normal((nx, ny)), 0.03 * rng.standard_normal((nx, ny)),
                          0.03 * rng.standard_normal((nx, ny)))
    return b


def lattices(b):
    return [b.download(i)[:, :, :ny] for i, (_, ny) in enumerate(SIZES)]


def test_every_thread_count(gpu_lib):
    """The cells' operations do not depend on the schedule: the same bits."""
    want = None
    for threads in THREADS:
        for persistent in (0, 1):
            with batch(threads, persistent) as b:
                b.run(5)
                got = lattices(b)
            want = want or got
            assert all(np.array_equal(w, g) for w, g in zip(want, got)), (threads, persistent)


def test_batches_of_different_thread_counts_side_by_side(gpu_lib):
    """Schedules applied from large to small, all batches run afterwards."""
    with batch(128, 0) as b:
        b.run(6)
        want = lattices(b)
    many = [batch(t) for t in (512, 384, 320, 352, 64)]
    for _ in range(2):
        for b in many:
            b.run(3)
    for b in many:
        assert all(np.array_equal(w, g) for w, g in zip(want, lattices(b)))
        b.close()
