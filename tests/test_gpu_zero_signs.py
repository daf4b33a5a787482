"""Zeros keep their signs through the PARITY steps, byte for byte with the
oracle: velocities of -0.0 (a division whose numerator is a negative zero), as
the VTU writer would write them."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("acc,scheme,flux", [(1, 0, 3), (1, 0, 2), (2, 0, 3), (2, 0, 2), (2, 1, 3)])
@pytest.mark.parametrize("bounds", [(3, 3, 3, 3), (2, 2, 1, 2)])
def test_negative_zeros(gpu_lib, acc, scheme, flux, bounds):
    Z, nx, ny = gpu_lib, 40, 67
    box = (0.1, 1.3, -0.4, 0.5)
    gen = Z.Rectangle(*box)
    gen.set_boundaries(Z.Boundaries(*bounds))
    gen.set_sizes(nx, ny)
    mesh = Z.EuMesh(gen)
    eos = Z.IdealGas(1.4)
    solver = Z.SmFluid(eos)
    solver.set_accuracy(acc)
    solver.set_CFL(0.4)
    solver.set_limiter("MC")
    solver.set_method(Z.Fluxes(flux))
    solver.set_scheme(Z.Scheme(scheme))
    solver.add_types(mesh)
    osv = O.Solver(O.Mesh(nx, ny, *box, bounds=bounds), eos_kind=eos.kind, gamma=1.4, P0=0.0, e0=0.0, flux=flux,
                   limiter=3, accuracy=acc, scheme=scheme, CFL=0.4, threads=4)
    n = nx * ny
    rho = np.repeat(1.0 + 0.5 * np.random.default_rng(4).random(nx), ny)  # along x only
    u = np.where(np.arange(n) < n // 2, 0.25, -0.0)
    z = [rho, u, np.full(n, -0.0), np.where(np.arange(n) < n // 3, 2.0, 1.0), None]
    z[4] = eos.energy_rP(z[0], z[3])
    mesh.set_state(*z)
    osv.set_state(*z)
    for k in range(3):
        solver.update(mesh)
        osv.step()
        for q, (a, b) in enumerate(zip(mesh.get_state(), osv.state())):
            assert np.asarray(a).tobytes() == np.ascontiguousarray(b).tobytes(), (k, q)
    mesh.close()
