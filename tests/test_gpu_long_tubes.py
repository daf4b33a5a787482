"""Rectangles of many rows: more row tiles than a grid's second dimension has
blocks (65535).  The PARITY second-order step against the oracle bit for bit;
the adjoint's forward run against one period of the same data, the mean
pressure to the rounding of its sum (the same cells, each many times)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme,flux", [(0, 3), (1, 2)])
def test_parity_second_order(gpu_lib, scheme, flux):
    Z, nx = gpu_lib, 800_003
    box, bounds = (0.0, 800.0, 0.0, 0.001), (1, 2, 1, 1)
    gen = Z.Rectangle(*box)
    gen.set_boundaries(Z.Boundaries(*bounds))
    gen.set_sizes(nx, 1)
    mesh = Z.EuMesh(gen)
    eos = Z.IdealGas(1.4)
    solver = Z.SmFluid(eos)
    solver.set_accuracy(2)
    solver.set_CFL(0.4)
    solver.set_limiter("MC")
    solver.set_method(Z.Fluxes(flux))
    solver.set_scheme(Z.Scheme(scheme))
    solver.add_types(mesh)
    osv = O.Solver(O.Mesh(nx, 1, *box, bounds=bounds), eos_kind=eos.kind, gamma=1.4, P0=0.0, e0=0.0, flux=flux,
                   limiter=3, accuracy=2, scheme=scheme, CFL=0.4, threads=4)
    rng = np.random.default_rng(1)
    rho, p, u = 1.0 + rng.random(nx), 1.0 + rng.random(nx), rng.standard_normal(nx)
    z = [rho, u, np.zeros(nx), p, eos.energy_rP(rho, p)]
    mesh.set_state(*z)
    osv.set_state(*z)
    for _ in range(2):
        solver.update(mesh)
        assert solver.dt() == osv.step()
    for a, b in zip(mesh.get_state(), osv.state()):
        assert np.array_equal(a, b)
    mesh.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_adjoint_forward(gpu_lib, precision):
    import torch

    from zephyr_b200.adjoint import Adjoint
    n, copies, ny = 1024, 900, 4  # 921 600 rows of 1/1024
    x = (np.arange(n) + 0.5) / n
    one = [1.0 + 0.2 * np.sin(2 * np.pi * x), 0.3 * np.cos(2 * np.pi * x), 0.0 * x, 1.0 + 0.1 * np.sin(4 * np.pi * x)]
    out = []
    for k in (1, copies):
        z = [torch.tensor(np.repeat(np.tile(a, k), ny), dtype=torch.float64, device="cuda") for a in one]
        adj = Adjoint(k * n, ny, box=(0.0, float(k), 0.0, ny / n))
        prm = Adjoint.params(steps=4, dt=2.0e-4, limiter_eps=1e-8, probe=(0.0, float(k), 0.0, 1.0), precision=precision)
        out.append(adj.forward(prm, *z))
        adj.close()
    # sums of 4e6 terms of one sign and magnitude
    assert abs(out[1] - out[0]) <= copies * n * ny * 2.0**-53 * abs(out[0])
