"""Slabs of a mesh that is large enough for the marching kernel, each of them
too small for it: the slabs' rows and dts are the single domain's, bit for bit
(cells of 1/1024: the local rectangles reproduce its coordinates)."""
import numpy as np
import pytest

from zephyr_b200 import slabs as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bounds,scheme,flux,lim", [((3, 3, 3, 3), 0, "HLLC", "van Albada"),
                                                    ((1, 2, 3, 3), 1, "HLLC", "van Albada"),
                                                    ((2, 1, 1, 2), 0, "HLL", "van Albada"),
                                                    ((3, 3, 1, 1), 1, "HLL", "MC")])
def test_slabs_of_a_marching_mesh(gpu_lib, bounds, scheme, flux, lim):
    Z, nx, ny, world, steps = gpu_lib, 1040, 1024, 4, 3
    box = (0.0, nx / 1024.0, 0.0, ny / 1024.0)
    rng = np.random.default_rng(2)
    rho, p = 1.0 + 0.5 * rng.random(nx * ny), 1.0 + 0.5 * rng.random(nx * ny)
    u, v = 0.3 * rng.standard_normal(nx * ny), 0.3 * rng.standard_normal(nx * ny)
    z = (rho, u, v, p, p / (0.4 * rho))

    def configure(s):
        s.set_accuracy(2)
        s.set_CFL(0.4)
        s.set_limiter(lim)
        s.set_method(Z.Fluxes[flux])
        s.set_scheme(Z.Scheme(scheme))

    whole = S.GpuSlabSolver(S.Slab(nx, ny, box, bounds, 1, 0), Z.IdealGas(1.4), configure)
    whole.set_state(*z)
    dts = []
    for _ in range(steps):
        whole.update()
        dts.append(whole.dt())
    want = np.array(whole.mesh.get_state())
    whole.close()

    comm = S.LocalComm()
    for r in range(world):
        slab = S.Slab(nx, ny, box, bounds, world, r, halo=S.halo_rows(2, scheme == 1))
        loc = S.GpuSlabSolver(slab, Z.IdealGas(1.4), configure)
        lo, hi = slab.rows
        gl, gh = slab.ghosts
        rows = np.arange(lo - gl, hi + gh) % nx
        loc.set_state(*(np.ascontiguousarray(a.reshape(nx, ny)[rows].ravel()) for a in z))
        comm.join(r, S.SlabStepper(slab, loc, comm, CFL=0.4))
    for k in range(steps):
        S.step_all(comm)
        assert {st.dt for st in comm.members.values()} == {dts[k]}
    got = np.concatenate([comm.members[r].owned_state()[0] for r in range(world)], axis=1)
    bad = got != want
    assert not bad.any(), f"{int(bad.sum())} values differ"
    for st in comm.members.values():
        st.local.close()
