"""The MIXED adjoint's error against the FP64 form's gradient is the one it had
with the symmetric reverse of HLLC in FP32, measured when every face went
through it: no more than 2 % above that (other roundings of the forward run)."""
import numpy as np
import pytest

from test_gpu_adjoint import cuda, smooth_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,steps,err_rho,err_gamma", [(64, 48, 20, 4.948e-6, 3.165e-7),
                                                           (96, 128, 30, 5.831e-6, 8.584e-7),
                                                           (200, 64, 40, 6.721e-6, 2.170e-6)])
def test_error_of_the_mixed_gradient(gpu_lib, nx, ny, steps, err_rho, err_gamma):
    import torch

    from zephyr_b200.adjoint import Adjoint
    z = cuda(*smooth_state(nx, ny, 7))
    out = []
    for precision in (0, 1):
        adj = Adjoint(nx, ny, box=(0.0, nx / 64.0, 0.0, ny / 64.0))
        prm = Adjoint.params(steps=steps, dt=0.2 / 64.0, limiter_eps=1e-8, precision=precision,
                             probe=(0.2, 0.6, 0.2, 0.6))
        g = torch.empty_like(z[0])
        _, dg = adj.gradient(prm, *z, g)
        out.append((g.cpu().numpy(), dg))
        adj.close()
    (g64, d64), (gmx, dmx) = out
    assert np.linalg.norm(gmx - g64) <= 1.02 * err_rho * np.linalg.norm(g64)
    assert abs(dmx - d64) <= 1.02 * err_gamma * abs(d64)
