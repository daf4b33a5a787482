"""One rounding for the second-order steps of a rectangle: the FAST kernels
write out their roundings (smf_fused.cuh), so that a cell's result depends
neither on its place in the mesh (interior or border tile) nor on the kernel
that the mesh's size picks.

* Periodic data moved by any number of cells: the result moved, bit for bit.
* MIXED on a small mesh (tiles of 4 rows), on a middle one (14 rows) and on a
  large one (the march) made of copies of the small one: the same bits.
* MIXED results stay the ones they were: digests of states that the one tile
  kernel of 14 rows gave when it ran every mesh.
* Each face adds one flux to both of its cells, so the sum of the conserved
  density changes by the rounding of the sums alone: an update of a cell takes
  at most six FP64 roundings of about its density, 6 x 2^-53 of the total per
  step (Heun: twice that).  MIXED Heun is left out: its second stage starts
  from the stage value rounded to FP32.
"""
import hashlib
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def field(nx, ny):
    """Rough periodic data by exact arithmetic only: (rho, u, v, p)."""
    x, y = (np.arange(nx) + 0.5)[:, None] / nx, (np.arange(ny) + 0.5)[None, :] / ny
    b, c = 16.0 * x * x * (1.0 - x) * (1.0 - x), 16.0 * y * y * (1.0 - y) * (1.0 - y)
    i, j = np.arange(nx)[:, None], np.arange(ny)[None, :]
    n = ((i * 7 + j * 13) % 32) / 1024.0  # up and down from cell to cell
    step = np.where((x > 0.3) & (x < 0.7) & (y < 0.55), 0.375, 0.0)
    rho = 1.0 + 0.25 * b * c + n + step
    u = 1.25 * b * (1.0 - c) - 0.5 + n
    v = 0.75 * c - 0.375 + step
    p = 1.0 + 0.5 * (1.0 - b) * c + n + step
    return [np.broadcast_to(a, (nx, ny)).copy() for a in (rho, u, v, p)]


def advance(Z, z, precision, scheme, flux, lim, steps, bounds=(3, 3, 3, 3), eos="ideal", box=(1.0, 1.0), wait=None):
    E = Z.IdealGas(1.4) if eos == "ideal" else Z.StiffenedGas(4.4, 6.0e8, 1.0e4)
    rho, u, v, p = z
    if eos != "ideal":
        rho, u, v, p = 1000.0 * rho, 100.0 * u, 100.0 * v, 1.0e8 * p
    nx, ny = rho.shape
    gen = Z.Rectangle(0.0, box[0], 0.0, box[1])
    gen.set_boundaries(Z.Boundaries(*bounds))
    gen.set_sizes(nx, ny)
    mesh = Z.EuMesh(gen)
    solver = Z.SmFluid(E, precision=Z.Precision[precision], kernels=Z.Kernels.FAST)
    solver.set_accuracy(2)
    solver.set_CFL(0.4)
    solver.set_limiter(lim)
    solver.set_method(Z.Fluxes[flux])
    solver.set_scheme(Z.Scheme(scheme))
    solver.add_types(mesh)
    mesh.set_state(*(np.ascontiguousarray(a.ravel()) for a in (rho, u, v, p, E.energy_rP(rho, p))))
    if wait is not None:
        mesh.set_wait(np.ascontiguousarray(wait.ravel()))
    solver.update(mesh, steps=steps)
    out = np.array(mesh.get_state()).reshape(5, nx, ny)
    dt = solver.dt()
    mesh.close()
    return out, dt


@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
@pytest.mark.parametrize("scheme,flux,lim", [(0, "HLLC", "van Albada"), (0, "HLL", "van Albada"), (1, "HLL", "van Albada"),
                                             (1, "HLLC", "MC"), (0, "HLLC", "minmod"), (1, "HLL", "van Albada 2"),
                                             (0, "HLL", "Koren")])
@pytest.mark.parametrize("nx,ny", [(64, 50), (331, 290), (1500, 1402)])
def test_shifted_data_shift_the_result(gpu_lib, nx, ny, scheme, flux, lim, precision):
    z = field(nx, ny)
    steps = 3
    box = (nx / 64.0, ny / 64.0)  # cells of 1/64: the mesh's coordinates are exact
    a, da = advance(gpu_lib, z, precision, scheme, flux, lim, steps, box=box)
    for sh in ((17, 11), (1, 0), (0, 29)):
        b, db = advance(gpu_lib, [np.roll(q, sh, (0, 1)) for q in z], precision, scheme, flux, lim, steps,
                        box=box)
        assert db == da
        bad = np.roll(b, (-sh[0], -sh[1]), (1, 2)) != a
        assert not bad.any(), f"{int(bad.sum())} values differ after a shift by {sh}"
    if precision == "MIXED" and scheme == 1:
        return
    total = math.fsum(z[0].ravel())
    drift = abs(math.fsum(a[0].ravel()) - total) / total
    assert drift <= (1 + scheme) * steps * 6 * 2.0**-53


@pytest.mark.parametrize("scheme,flux,wait", [(0, "HLLC", False), (0, "HLL", False), (0, "HLLC", True),
                                              (1, "HLLC", False), (1, "HLL", False)])
def test_mixed_forms_give_the_same_bits(gpu_lib, scheme, flux, wait):
    n = 64  # cells of 1/64: exact in every mesh
    z = field(n, n)
    w = None
    if wait:
        w = np.zeros((n, n), np.int32)
        w.ravel()[[5, 700, 701, 4095]] = (1, 2, 3, 3)
    small, ds = advance(gpu_lib, z, "MIXED", scheme, flux, "van Albada", 4, wait=w)
    for kx, ky in ((8, 7), (34, 32)):
        big, db = advance(gpu_lib, [np.tile(q, (kx, ky)) for q in z], "MIXED", scheme, flux, "van Albada", 4,
                          box=(float(kx), float(ky)), wait=None if w is None else np.tile(w, (kx, ky)))
        assert db == ds
        bad = big != np.tile(small, (1, kx, ky))
        assert not bad.any(), f"{int(bad.sum())} values differ at {kx * n} x {ky * n}"


ZOE, WALL, PER = (2, 2, 2, 2), (1, 1, 1, 1), (3, 3, 3, 3)
CASES = [
    # nx, ny, scheme, flux, limiter, eos, bounds
    (57, 45, 0, "HLLC", "van Albada", "ideal", PER),
    (57, 45, 1, "HLLC", "van Albada", "ideal", PER),
    (57, 45, 1, "HLL", "MC", "ideal", (2, 1, 3, 3)),
    (57, 45, 0, "HLL", "minmod", "stiffened", WALL),
    (57, 45, 1, "HLLC", "van Albada 2", "ideal", ZOE),
    (57, 45, 0, "HLLC", "superbee", "ideal", PER),
    (401, 333, 0, "HLLC", "MC", "ideal", ZOE),
    (401, 333, 1, "HLLC", "van Albada", "stiffened", PER),
    (401, 333, 1, "HLL", "van Leer", "ideal", WALL),
    (401, 333, 0, "HLL", "van Albada", "ideal", PER),
    (1460, 1410, 0, "HLLC", "van Albada", "stiffened", PER),
    (1460, 1410, 1, "HLLC", "van Albada", "ideal", PER),
    (1460, 1410, 1, "HLL", "van Albada", "ideal", (1, 2, 2, 1)),
]
DIGESTS = [
    "fd00248acfa5dc05", "d16217221f54b380", "84e4d4ca662a2e84", "ed9f529c0222d4be", "def9871fe4d88d4a",
    "731a42ba02cf6cdf", "a20f556427aa6475", "0387343e4e26088d", "28d41c35a6352162", "532b3313a1aad0df",
    "eda40b3b78ff5682", "2e96de168d029152", "5a4dc3877fdbf958",
]


def digest(Z, case):
    nx, ny, scheme, flux, lim, eos, bounds = case
    out, dt = advance(Z, field(nx, ny), "MIXED", scheme, flux, lim, 12, bounds, eos)
    return hashlib.sha256((out + 0.0).tobytes() + np.float64(dt).tobytes()).hexdigest()[:16]


@pytest.mark.parametrize("k", range(len(CASES)), ids=["-".join(map(str, c[:6])) for c in CASES])
def test_mixed_results_are_the_ones_they_were(gpu_lib, k):
    assert digest(gpu_lib, CASES[k]) == DIGESTS[k]
