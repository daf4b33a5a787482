"""The next dt on a rectangle far from the origin, whose cells differ in size by
the rounding of their coordinates (1e-13 of x in steps of 1e-10: one part in a
thousand): the step kernels' dt is the minimum over all cells."""
import numpy as np
import pytest

from oracle import oracle as O
from zephyr_b200 import slabs as S

pytestmark = pytest.mark.gpu


H = 1e-10


def _box(nx, ny):
    return 1000.0, 1000.0 + nx * H, 0.0, 8.0 * ny * H  # (wide in y: the extent along x counts)


def _state(nx, ny, eos):
    """Gas at rest, its sound speed 8e-4 higher where a column is not one of the
    narrowest (which are 1.1e-3 narrower): the smallest term is a narrow cell's,
    although the fast cells' would be below it by a common size."""
    x0, x1 = _box(nx, ny)[:2]
    w = np.diff(x0 + ((x1 - x0) * np.arange(nx + 1)) / nx)
    assert w.max() > 1.001 * w.min()
    rho = np.repeat(np.where(w < 1.0005 * w.min(), 1.0, 1.0008**-2), ny)
    z = np.zeros(nx * ny)
    return [rho, z, z, z + 1.0, eos.energy_rP(rho, z + 1.0)]


@pytest.mark.parametrize("acc,scheme,flux", [(1, 0, 3), (2, 0, 3), (2, 1, 2)])
def test_parity(gpu_lib, acc, scheme, flux):
    Z, nx, ny = gpu_lib, 90, 70
    box, bounds = _box(nx, ny), (2, 2, 2, 2)
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
    z = _state(nx, ny, eos)
    mesh.set_state(*z)
    osv.set_state(*z)
    got, want = [], []
    for _ in range(4):  # (no read between the steps: their own next dt)
        solver.update(mesh)
        want.append(osv.step())
        got.append(solver.dt())
    assert got == want
    mesh.close()


@pytest.mark.parametrize("nx,ny,scheme", [(90, 70, 0), (400, 380, 0), (1100, 1040, 1)])
def test_fast(gpu_lib, nx, ny, scheme):
    Z = gpu_lib
    slab = S.Slab(nx, ny, _box(nx, ny), (2, 2, 2, 2), 1, 0)

    def configure(s):
        s.set_accuracy(2)
        s.set_CFL(0.4)
        s.set_limiter("van Albada")
        s.set_scheme(Z.Scheme(scheme))

    loc = S.GpuSlabSolver(slab, Z.IdealGas(1.4), configure)
    loc.set_state(*_state(nx, ny, Z.IdealGas(1.4)))
    loc.update()
    for _ in range(3):
        dmin = loc.cfl_min()  # k_cfl's own pass over the state
        loc.update()
        assert loc.dt() == 0.4 * dmin
    loc.close()
