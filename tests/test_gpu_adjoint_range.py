"""The binary64 reverse step at the edges of its launch and of the fixed point's
range, against the CPU adjoint."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,amp", [(1, 1, 0.02), (3, 257, 0.02), (24, 40, 0.45), (40, 31, 0.38)])
def test_reverse_step_against_the_cpu_adjoint(gpu_lib, nx, ny, amp):
    """Amplitudes 0.38 and 0.45 put cells past 7.5 rho |u|^2 = 1, which take the
    binary64 expressions; four steps stay far from instability.  Bound as for the
    ordinary case (the gradients are sums of O(100) products in binary64 on both
    sides): 1e-9."""
    import torch
    from plbm.autograd import Adjoint
    steps, omega = 4, 1.1
    rng = np.random.default_rng(12)
    x, y = (np.arange(nx) + 0.5)[:, None] / nx, (np.arange(ny) + 0.5)[None, :] / ny
    ux = amp * np.sin(2 * np.pi * y) * np.cos(2 * np.pi * x) + 1e-3 * rng.standard_normal((nx, ny))
    uy = -amp * np.cos(2 * np.pi * y) * np.sin(2 * np.pi * x) + 1e-3 * rng.standard_normal((nx, ny))
    u_t, v_t = O.forward_bgk(ux, uy, omega, steps)
    gx_t, gy_t = rng.standard_normal((2, nx, ny))
    _, (gx, gy), gom = O.adjoint_bgk(ux, uy, omega, steps, gx_t, gy_t)
    a = Adjoint(nx, ny, steps, checkpoint_every=2, storage="f64")
    got = a.forward(torch.tensor(np.stack([ux, uy]), device="cuda"), omega).cpu().numpy()
    g0, dom = a.backward(torch.tensor(np.stack([gx_t, gy_t]), device="cuda"))
    a.close()
    g0 = g0.cpu().numpy()
    assert np.max(np.abs(got - np.stack([u_t, v_t]))) <= 1e-12 * max(np.max(np.abs(u_t)), np.max(np.abs(v_t)))
    scale = max(np.max(np.abs(gx)), np.max(np.abs(gy)))
    assert max(np.max(np.abs(g0[0] - gx)), np.max(np.abs(g0[1] - gy))) <= 1e-9 * scale
    assert abs(dom - gom) <= 1e-9 * max(abs(gom), scale)
