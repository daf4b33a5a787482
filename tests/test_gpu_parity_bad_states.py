"""PARITY second order with cells whose pressure is below the equation of
state's minimum (a sound speed that is not a number, from finite values), against
the oracle bit for bit: each side of a face sees such a neighbour in its own way."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

LIMS = {"unit": 1, "MC": 3, "van Albada": 5, "superbee": 12}


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("scheme,flux,lim", [(0, 3, "MC"), (1, 3, "MC"), (1, 3, "superbee"), (0, 2, "MC"),
                                             (1, 2, "van Albada"), (0, 3, "unit"), (1, 3, "unit"), (1, 2, "unit")])
def test_pressures_below_the_minimum(gpu_lib, scheme, flux, lim, seed):
    Z, nx, ny, bounds = gpu_lib, 29, 70, (3, 3, 1, 2)
    box = (0.1, 1.3, -0.4, 0.5)
    gen = Z.Rectangle(*box)
    gen.set_boundaries(Z.Boundaries(*bounds))
    gen.set_sizes(nx, ny)
    mesh = Z.EuMesh(gen)
    eos = Z.IdealGas(1.4)
    solver = Z.SmFluid(eos)
    solver.set_accuracy(2)
    solver.set_CFL(0.4)
    solver.set_limiter(lim)
    solver.set_method(Z.Fluxes(flux))
    solver.set_scheme(Z.Scheme(scheme))
    solver.add_types(mesh)
    osv = O.Solver(O.Mesh(nx, ny, *box, bounds=bounds), eos_kind=eos.kind, gamma=1.4, P0=0.0, e0=0.0, flux=flux,
                   limiter=LIMS[lim], accuracy=2, scheme=scheme, CFL=0.4, threads=4)
    rng = np.random.default_rng(seed)
    n = nx * ny
    rho, u, v = 1.0 + rng.random(n), 3.0 * rng.standard_normal(n), 3.0 * rng.standard_normal(n)
    p = 0.2 + rng.random(n)
    p[rng.choice(n, 120, replace=False)] = -0.05  # finite, and some face values of these cells are positive
    z = [rho, u, v, p, eos.energy_rP(rho, p)]
    mesh.set_state(*z)
    osv.set_state(*z)
    for k in range(2):
        solver.update(mesh)
        dt = osv.step()
        assert solver.dt() == dt, k
        for a, b in zip(mesh.get_state(), osv.state()):
            assert np.array_equal(a, b, equal_nan=True), k
        assert np.array_equal(mesh.get_wait(), osv.wait())
    mesh.close()
