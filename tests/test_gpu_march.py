"""The marching form of the structured second-order step (large meshes)
against the bit-exact PARITY kernels: sides of every kind, strips and segments
that end inside the mesh, isolated cells, both fluxes and a limiter that is
chosen at run time.  Tolerance: the FAST form's 1e-12 per step.  The MIXED form
against its own tile kernels: a large mesh of periodic copies of a small one.
Both do the same FP32 operations, and differ by FP64 rounding that may turn
an FP32 rounding of a stage value (2^-24 of it), which a step scales by less
than 8: 5e-7 of a field's magnitude."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(nx, ny, eos, seed):
    rng = np.random.default_rng(seed)
    x, y = (np.arange(nx) + 0.5)[:, None] / nx, (np.arange(ny) + 0.5)[None, :] / ny
    f = [sum(rng.uniform(0.02, 0.05) * np.sin(2 * np.pi * m * x + rng.uniform(0, 6)) *
             np.sin(2 * np.pi * m * y + rng.uniform(0, 6)) for m in range(1, 5)) for _ in range(4)]
    step = np.where((x > 0.4) & (y < 0.6), 0.3, 0.0)  # a jump, so that limiters and waves act
    rho, u, v, p = 1.0 + f[0] + step, 0.5 * f[1] + step, 0.5 * f[2], 1.0 + f[3] + step
    return tuple(np.ascontiguousarray(a.ravel()) for a in (rho, u, v, p, eos.energy_rP(rho, p)))


def _solver(Z, nx, ny, bounds, kernels, precision, flux, lim, scheme, eos):
    gen = Z.Rectangle(0.0, 1.0, 0.0, 1.0)
    gen.set_boundaries(Z.Boundaries(*bounds))
    gen.set_sizes(nx, ny)
    mesh = Z.EuMesh(gen)
    solver = Z.SmFluid(eos, precision=precision, kernels=kernels)
    solver.set_accuracy(2)
    solver.set_CFL(0.4)
    solver.set_limiter(lim)
    solver.set_method(flux)
    solver.set_scheme(scheme)
    solver.add_types(mesh)
    return mesh, solver


def _rel_cons(a, b):
    def cons(z):
        rho, u, v, p, e = z
        return [rho, rho * u, rho * v, rho * (e + 0.5 * (u * u + v * v))]
    return max(np.max(np.abs(x - y)) / np.max(np.abs(y)) for x, y in zip(cons(a), cons(b)))


@pytest.mark.parametrize("nx,ny,bounds,flux,lim,scheme,wait", [
    (1031, 1119, (1, 2, 2, 1), "HLLC", "van Albada", 0, False),
    (1400, 800, (2, 1, 1, 1), "HLL", "superbee", 0, False),
    (1120, 1037, (3, 3, 1, 2), "HLLC", "MC", 0, True),
    (1037, 1121, (2, 1, 3, 3), "HLLC", "minmod", 1, False),
    (2300, 57, (1, 1, 1, 1), "HLLC", "MC", 0, False),
    (30011, 57, (1, 2, 2, 2), "HLLC", "van Albada", 0, True),
])
def test_march_matches_parity(gpu_lib, nx, ny, bounds, flux, lim, scheme, wait):
    Z = gpu_lib
    eos = Z.IdealGas(1.4)
    z0 = _state(nx, ny, eos, nx + ny)
    w0 = np.zeros(nx * ny, np.int32)
    if wait:
        rng = np.random.default_rng(1)
        at = np.concatenate([rng.choice(nx * ny, 40, replace=False), [0, ny - 1, nx * ny - 1, (nx - 1) * ny]])
        w0[at] = rng.integers(1, 4, at.size)
    out = []
    for kernels in (Z.Kernels.PARITY, Z.Kernels.FAST):
        mesh, solver = _solver(Z, nx, ny, bounds, kernels, Z.Precision.FP64, Z.Fluxes[flux], lim, Z.Scheme(scheme),
                               eos)
        mesh.set_state(*z0)
        mesh.set_wait(w0)
        dts = []
        solver.update(mesh)
        dts.append(solver.dt())
        out.append((mesh.get_state(), mesh.get_wait(), dts))
        solver.update(mesh)  # the second step runs with the dt the first one found
        dts.append(solver.dt())
        mesh.close()
    (zp, wp, dp), (zf, wf, df) = out
    assert _rel_cons(zf, zp) <= 1e-12
    assert np.array_equal(wf, wp)
    assert np.allclose(df, dp, rtol=1e-12, atol=0.0)


@pytest.mark.parametrize("scheme,flux,wait", [(0, "HLLC", False), (0, "HLL", True), (1, "HLLC", False)])
def test_march_mixed_matches_tiles(gpu_lib, scheme, flux, wait):
    Z = gpu_lib
    eos = Z.IdealGas(1.4)
    n, kx, ky = 64, 31, 29  # 1984 x 1856 against 64 x 64; cells of 1/64, exact in both
    z0 = _state(n, n, eos, 5)
    w0 = np.zeros(n * n, np.int32)
    if wait:
        w0[[5, 700, 4095]] = (1, 2, 3)
    out = []
    for cx, cy in ((1, 1), (kx, ky)):
        gen = Z.Rectangle(0.0, float(cx), 0.0, float(cy))
        gen.set_boundaries(Z.Boundaries(3, 3, 3, 3))
        gen.set_sizes(cx * n, cy * n)
        mesh = Z.EuMesh(gen)
        solver = Z.SmFluid(eos, precision=Z.Precision.MIXED, kernels=Z.Kernels.FAST)
        solver.set_accuracy(2)
        solver.set_CFL(0.4)
        solver.set_limiter("van Albada")
        solver.set_method(Z.Fluxes[flux])
        solver.set_scheme(Z.Scheme(scheme))
        solver.add_types(mesh)
        mesh.set_state(*(np.tile(a.reshape(n, n), (cx, cy)).ravel() for a in z0))
        mesh.set_wait(np.tile(w0.reshape(n, n), (cx, cy)).ravel())
        solver.update(mesh)
        out.append(([a.reshape(cx * n, cy * n) for a in mesh.get_state()], mesh.get_wait().reshape(cx * n, cy * n),
                    solver.dt()))
        mesh.close()
    (zs, ws, ds), (zb, wb, db) = out
    assert db == ds
    assert np.array_equal(wb, np.tile(ws, (kx, ky)))
    for a, b in zip(zs, zb):
        assert np.max(np.abs(b - np.tile(a, (kx, ky)))) <= 5e-7 * np.max(np.abs(a))
