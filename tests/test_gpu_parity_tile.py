"""The PARITY tile kernels of a rectangle (HLLC and HLL) against the oracle, bit
for bit: meshes around the tile's 30 columns and 12 rows and below its halo,
every kind of side, all stages, isolated cells, gas at rest (zero numerators),
and values that are not finite."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

LIMS = {"MC": 3, "van Albada": 5, "minmod": 2, "superbee": 12}


def _both(Z, nx, ny, bounds, acc, scheme, flux, lim, eos):
    box = (0.1, 1.3, -0.4, 0.5)
    gen = Z.Rectangle(*box)
    gen.set_boundaries(Z.Boundaries(*bounds))
    gen.set_sizes(nx, ny)
    mesh = Z.EuMesh(gen)
    solver = Z.SmFluid(eos)
    solver.set_accuracy(acc)
    solver.set_CFL(0.4)
    solver.set_limiter(lim)
    solver.set_method(Z.Fluxes(flux))
    solver.set_scheme(Z.Scheme(scheme))
    solver.add_types(mesh)
    osv = O.Solver(O.Mesh(nx, ny, *box, bounds=bounds), eos_kind=eos.kind, gamma=eos.gamma, P0=eos.P0, e0=eos.e0,
                   flux=flux, limiter=LIMS[lim], accuracy=acc, scheme=scheme, CFL=0.4, threads=4)
    return mesh, solver, osv


def _state(nx, ny, eos, seed, rest=False):
    rng = np.random.default_rng(seed)
    n = nx * ny
    rho = 1.0 + rng.random(n)
    u, v = (np.zeros(n), np.zeros(n)) if rest else rng.standard_normal((2, n))
    p = np.where(np.arange(n) % 7 < 4, 1.0, 1.0 if rest else 2.0)
    if rest:
        rho = np.where(np.arange(n) % ny < ny // 2, 1.0, 3.0)
        p[n // 2] = 5.0
    return [np.ascontiguousarray(a) for a in (rho, u, v, p, eos.energy_rP(rho, p))]


def _run(Z, mesh, solver, osv, z, wait, steps):
    mesh.set_state(*z)
    osv.set_state(*z)
    if wait is not None:
        mesh.set_wait(wait)
        osv.set_wait(wait)
    for k in range(steps):
        solver.update(mesh)
        dt = osv.step()
        assert solver.dt() == dt or (np.isnan(dt) and np.isnan(solver.dt())), k
        for a, b in zip(mesh.get_state(), osv.state()):
            assert np.array_equal(a, b, equal_nan=True), k
        assert np.array_equal(mesh.get_wait(), osv.wait())
    mesh.close()


@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 64), (64, 1), (2, 3), (11, 29), (12, 30), (13, 31), (24, 60), (25, 61),
                                   (16, 34), (37, 95)])
@pytest.mark.parametrize("bounds,acc,scheme,flux,lim", [
    ((1, 2, 2, 1), 1, 0, 3, "MC"), ((3, 3, 3, 3), 2, 0, 3, "MC"), ((3, 3, 1, 2), 2, 0, 2, "minmod"),
    ((2, 1, 3, 3), 2, 1, 3, "van Albada"), ((1, 1, 2, 2), 2, 0, 3, "superbee"), ((2, 2, 1, 1), 1, 0, 2, "MC")])
def test_tile_matches_oracle(gpu_lib, nx, ny, bounds, acc, scheme, flux, lim):
    Z = gpu_lib
    eos = Z.IdealGas(1.4)
    both = _both(Z, nx, ny, bounds, acc, scheme, flux, lim, eos)
    wait = None
    if acc == 2 and scheme == 0 and flux == 3:
        rng = np.random.default_rng(nx + ny)
        wait = np.where(rng.random(nx * ny) < 0.1, rng.integers(1, 4, nx * ny), 0).astype(np.int32)
    _run(Z, *both, _state(nx, ny, eos, nx * ny), wait, 3)


@pytest.mark.parametrize("acc,lim,stiff", [(1, "MC", False), (2, "MC", False), (2, "superbee", True)])
def test_gas_at_rest(gpu_lib, acc, lim, stiff):
    Z = gpu_lib
    eos = Z.StiffenedGas(4.4, 6.0) if stiff else Z.IdealGas(1.4)
    both = _both(Z, 40, 67, (1, 1, 2, 2), acc, 0, 3, lim, eos)
    _run(Z, *both, _state(40, 67, eos, 1, rest=True), None, 4)


@pytest.mark.parametrize("acc,flux", [(1, 3), (1, 2), (2, 3), (2, 2)])
@pytest.mark.parametrize("field,value", [(0, np.nan), (1, np.nan), (2, np.inf), (3, np.nan), (4, np.nan), (2, np.nan)])
def test_values_that_are_not_finite(gpu_lib, acc, flux, field, value):
    Z = gpu_lib
    eos = Z.IdealGas(1.4)
    both = _both(Z, 29, 70, (1, 2, 3, 3), acc, 0, flux, "MC", eos)
    z = _state(29, 70, eos, 5)
    z[field][[0, 1000, 1001, 29 * 70 - 1]] = value
    _run(Z, *both, z, None, 1)
