"""The marching form of the second-order step (van Albada 1 on large meshes) at
shapes that reach it: every kind of side, both fluxes, both schemes, isolated
cells also beside a side and across a periodic seam.  Against the bit-exact
PARITY kernels to the FAST form's 1e-12 per step, after each of two steps; and
against the same mesh in slabs that are too short to march, bit for bit (cells of
1/64: their coordinates are exact)."""
import numpy as np
import pytest

from zephyr_b200 import slabs as S

pytestmark = pytest.mark.gpu


def segment_rows(nx, ny):
    """march_split of smf_march.cuh, FP64: rows per warp."""
    strips, cap, waves = (ny + 27) // 28, 148 * 4 * 4, 1
    while True:
        segs = max(waves * cap // strips, 1)
        rows = (nx + segs - 1) // segs
        if rows <= 96:
            return rows
        waves += 1


def state(nx, ny, seed):
    rng = np.random.default_rng(seed)
    x, y = (np.arange(nx) + 0.5)[:, None] / nx, (np.arange(ny) + 0.5)[None, :] / ny
    f = [sum(rng.uniform(0.02, 0.05) * np.sin(2 * np.pi * 300 * m * x + rng.uniform(0, 6)) *
             np.sin(2 * np.pi * m * y + rng.uniform(0, 6)) for m in range(1, 4)) for _ in range(4)]
    step = np.where((np.arange(nx)[:, None] % 100 > 40) & (y < 0.6), 0.3, 0.0)
    rho, u, v, p = 1.0 + f[0] + step, 0.5 * f[1] + step, 0.5 * f[2] - step, 1.0 + f[3] + step
    return [np.ascontiguousarray(a.ravel()) for a in (rho, u, v, p, p / (0.4 * rho))]


CASES = [
    # nx, ny, bounds, scheme, flux, waiting cells
    (40003, 57, (1, 2, 2, 1), 0, "HLLC", True),
    (40003, 57, (2, 1, 3, 3), 0, "HLL", True),
    (40003, 57, (3, 3, 1, 2), 0, "HLLC", True),
    (40003, 57, (3, 3, 3, 3), 0, "HLL", True),
    (20010, 61, (1, 1, 2, 1), 1, "HLLC", False),
    (20010, 61, (2, 2, 1, 1), 1, "HLL", False),
    (20010, 61, (3, 3, 2, 1), 1, "HLLC", False),
]


@pytest.mark.parametrize("nx,ny,bounds,scheme,flux,wait", CASES)
def test_march(gpu_lib, nx, ny, bounds, scheme, flux, wait):
    Z, world = gpu_lib, 3
    need = 16 if scheme else 48
    assert segment_rows(nx, ny) >= need > segment_rows(nx // world + 9, ny)
    box = (0.0, nx / 64.0, 0.0, ny / 64.0)
    z0 = state(nx, ny, 3)
    w0 = np.zeros(nx * ny, np.int32)
    if wait:
        rng = np.random.default_rng(1)
        at = np.concatenate([rng.choice(nx * ny, 300, replace=False), [0, 1, ny - 1, nx * ny - 1, (nx - 1) * ny],
                             np.arange(7, 12) * ny, np.arange(7, 12) * ny + ny - 1])
        w0[at] = rng.integers(1, 4, at.size)

    def configure(s):
        s.set_accuracy(2)
        s.set_CFL(0.4)
        s.set_limiter("van Albada")
        s.set_method(Z.Fluxes[flux])
        s.set_scheme(Z.Scheme(scheme))

    out = {}
    for kernels in ("PARITY", "FAST"):
        loc = S.GpuSlabSolver(S.Slab(nx, ny, box, bounds, 1, 0), Z.IdealGas(1.4), configure, kernels=Z.Kernels[kernels])
        loc.set_state(*z0, wait=w0)
        out[kernels] = []
        for _ in range(2):
            loc.update()
            out[kernels].append((np.array(loc.mesh.get_state()), loc.mesh.get_wait(), loc.dt()))
        loc.close()

    def cons(z):
        rho, u, v, p, e = z
        return [rho, rho * u, rho * v, rho * (e + 0.5 * (u * u + v * v))]
    for k, ((zp, wp, dp), (zf, wf, df)) in enumerate(zip(out["PARITY"], out["FAST"])):
        assert max(np.max(np.abs(a - b)) / np.max(np.abs(b)) for a, b in zip(cons(zf), cons(zp))) <= 1e-12 * (k + 1)
        assert np.array_equal(wf, wp)
        assert abs(df - dp) <= 1e-12 * dp

    comm = S.LocalComm()
    for r in range(world):
        slab = S.Slab(nx, ny, box, bounds, world, r, halo=S.halo_rows(2, scheme == 1))
        loc = S.GpuSlabSolver(slab, Z.IdealGas(1.4), configure)
        lo, hi = slab.rows
        gl, gh = slab.ghosts
        rows = np.arange(lo - gl, hi + gh) % nx
        loc.set_state(*(np.ascontiguousarray(a.reshape(nx, ny)[rows].ravel()) for a in z0),
                      wait=np.ascontiguousarray(w0.reshape(nx, ny)[rows].ravel()))
        comm.join(r, S.SlabStepper(slab, loc, comm, CFL=0.4))
    for k in range(2):
        S.step_all(comm)
        assert {st.dt for st in comm.members.values()} == {out["FAST"][k][2]}
    parts = [comm.members[r].owned_state() for r in range(world)]
    assert np.array_equal(np.concatenate([f for f, _ in parts], axis=1), out["FAST"][1][0])
    assert np.array_equal(np.concatenate([w for _, w in parts]), out["FAST"][1][1])
    for st in comm.members.values():
        st.local.close()
