"""The PARITY predictor-corrector on meshes given cell by cell (four threads per
cell) against the same step on the rectangle they describe, bit for bit: sizes
around a block's 32 cells, walls and open sides, isolated cells, the run-time
limiters and fluxes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _arrays(nx, ny, box, bounds):
    """zephyr's AmrCells arrays of a rectangle, with the generator's formulas."""
    x0, x1, y0, y1 = box
    X, Y = x0 + ((x1 - x0) * np.arange(nx + 1)) / nx, y0 + ((y1 - y0) * np.arange(ny + 1)) / ny
    cx = 0.25 * (X[:-1] + X[1:] + X[:-1] + X[1:])
    cy = 0.25 * (Y[:-1] + Y[:-1] + Y[1:] + Y[1:])
    fxm, fym = 0.5 * (X[:-1] + X[1:]), 0.5 * (Y[:-1] + Y[1:])
    hx, hy = (x1 - x0) / nx, (y1 - y0) / ny
    n = nx * ny
    i, j = np.repeat(np.arange(nx), ny), np.tile(np.arange(ny), nx)
    ic = np.arange(n)
    dx2, dy2 = (X[1:] - X[:-1]) ** 2, (Y[1:] - Y[:-1]) ** 2
    g = {"cx": cx[i], "cy": cy[j], "vol": np.full(n, hx * hy), "inc": np.sqrt(np.minimum(dx2[i], dy2[j]))}
    for k in ("nx", "ny", "fx", "fy", "area"):
        g[k] = np.zeros((n, 8))
    g["boundary"], g["neib"] = np.full((n, 8), -1, np.int32), np.repeat(ic[:, None], 8, 1).astype(np.int32)
    for s, (inner, nb, nrm, fc, area) in enumerate((
            (i > 0, ic - ny, (-1.0, -0.0), (X[i], fym[j]), hy), (i < nx - 1, ic + ny, (1.0, 0.0), (X[i + 1], fym[j]), hy),
            (j > 0, ic - 1, (-0.0, -1.0), (fxm[i], Y[j]), hx), (j < ny - 1, ic + 1, (0.0, 1.0), (fxm[i], Y[j + 1]), hx))):
        g["boundary"][:, s] = np.where(inner, 0, bounds[s])
        g["neib"][:, s] = np.where(inner, nb, ic)
        g["nx"][:, s], g["ny"][:, s] = nrm
        g["fx"][:, s], g["fy"][:, s] = fc
        g["area"][:, s] = area
    return {k: np.ascontiguousarray(v.ravel()) for k, v in g.items()}


@pytest.mark.parametrize("nx,ny,bounds,flux,lim,wait", [
    (1, 1, (1, 2, 1, 2), "HLLC", "MC", False), (5, 7, (2, 2, 1, 1), "HLLC", "minmod", True),
    (8, 4, (1, 1, 1, 1), "HLL", "van Albada", True), (33, 31, (2, 1, 1, 2), "HLLC", "superbee", True),
    (40, 57, (1, 2, 2, 1), "RUSANOV", "MC", False), (64, 65, (2, 2, 2, 2), "HLLC", "van Leer", False)])
def test_slot_mesh_matches_rectangle(gpu_lib, nx, ny, bounds, flux, lim, wait):
    Z = gpu_lib
    eos = Z.StiffenedGas(4.4, 2.0)
    box = (-0.3, 0.9, 0.2, 1.0)
    gen = Z.Rectangle(*box)
    gen.set_boundaries(Z.Boundaries(*bounds))
    gen.set_sizes(nx, ny)
    rng = np.random.default_rng(nx * ny)
    n = nx * ny
    rho, p = 1.0 + rng.random(n), np.where(np.arange(n) % 5 < 3, 1.0, 2.0)
    u, v = np.where(np.arange(n) % 3 == 0, 0.0, rng.standard_normal(n)), rng.standard_normal(n)
    z = (rho, u, v, p, eos.energy_rP(rho, p))
    w = np.where(rng.random(n) < 0.1, rng.integers(1, 4, n), 0).astype(np.int32) if wait else np.zeros(n, np.int32)
    out = []
    for mesh in (Z.EuMesh(gen), Z.EuMesh.from_arrays(_arrays(nx, ny, box, bounds))):
        solver = Z.SmFluid(eos)
        solver.set_accuracy(2)
        solver.set_CFL(0.4)
        solver.set_limiter(lim)
        solver.set_method(Z.Fluxes[flux])
        solver.add_types(mesh)
        mesh.set_state(*z)
        mesh.set_wait(w)
        steps = []
        for _ in range(4):
            solver.update(mesh)
            steps.append((solver.dt(), mesh.get_state(), mesh.get_wait()))
        out.append(steps)
        mesh.close()
    for (da, za, wa), (db, zb, wb) in zip(*out):
        assert da == db
        assert all(np.array_equal(a, b) for a, b in zip(za, zb))
        assert np.array_equal(wa, wb)
