"""Steps recorded into a CUDA graph, mixed with live ones: every order of
recording, replaying and live calls gives the states and the dts of live steps
alone, bit for bit (PARITY)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(Z, nx, ny, accuracy, scheme, flux, stream=None, amr=False):
    gen = Z.Rectangle(0.0, 1.0, 0.0, 1.0)
    gen.set_boundaries(Z.Boundaries(1, 2, 2, 1))
    gen.set_sizes(nx, ny)
    mesh = Z.EuMesh(gen, stream=stream)
    if amr:
        mesh.set_max_level(1)
    solver = Z.SmFluid(Z.IdealGas(1.4), kernels=Z.Kernels.PARITY)
    solver.set_accuracy(accuracy)
    solver.set_CFL(0.4)
    solver.set_limiter("MC")
    solver.set_method(Z.Fluxes[flux])
    solver.set_scheme(Z.Scheme(scheme))
    solver.add_types(mesh)
    return mesh, solver


def _state(nx, ny, seed):
    rng = np.random.default_rng(seed)
    rho, p = 1.0 + rng.random(nx * ny), 1.0 + rng.random(nx * ny)
    u, v = 0.5 * rng.standard_normal(nx * ny), 0.5 * rng.standard_normal(nx * ny)
    return rho, u, v, p, p / (0.4 * rho)


CASES = [(1, 0, "HLLC", False), (2, 0, "HLLC", False), (2, 1, "HLL", False), (2, 0, "RUSANOV", False),
         (2, 0, "HLLC", True)]


@pytest.mark.parametrize("accuracy,scheme,flux,amr", CASES)
def test_replays_between_live_steps(gpu_lib, accuracy, scheme, flux, amr):
    import torch
    Z, nx, ny = gpu_lib, 70, 45
    z0 = _state(nx, ny, 3)
    plain, ps = _solver(Z, nx, ny, accuracy, scheme, flux, amr=amr)
    plain.set_state(*z0)
    want, dts = [], []
    for _ in range(9):
        ps.update(plain)
        want.append(np.array(plain.get_state()))
        dts.append(ps.dt())
    plain.close()

    stream = torch.cuda.Stream()
    mesh, solver = _solver(Z, nx, ny, accuracy, scheme, flux, stream=stream.cuda_stream, amr=amr)
    mesh.set_state(*z0)
    solver.update(mesh, steps=1)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        solver.update(mesh, steps=2)  # an even number: the state returns to its buffers
    torch.cuda.synchronize()

    def replay():
        with torch.cuda.stream(stream):
            graph.replay()
        torch.cuda.synchronize()

    solver.update(mesh, steps=2)
    replay()
    assert solver.dt() == dts[4]
    solver.update(mesh)
    assert solver.dt() == dts[5]
    solver.update(mesh)
    replay()
    assert solver.dt() == dts[8]
    assert np.array_equal(np.array(mesh.get_state()), want[8])
    mesh.close()


def test_a_replayed_upload(gpu_lib):
    import torch
    Z, nx, ny = gpu_lib, 70, 45
    z0, z1 = _state(nx, ny, 3), _state(nx, ny, 4)
    plain, ps = _solver(Z, nx, ny, 2, 0, "HLLC")
    plain.set_state(*z1)
    ps.update(plain)
    want, dt = np.array(plain.get_state()), ps.dt()
    plain.close()

    stream = torch.cuda.Stream()
    mesh, solver = _solver(Z, nx, ny, 2, 0, "HLLC", stream=stream.cuda_stream)
    mesh.set_state(*z0)
    solver.update(mesh, steps=2)
    pinned = [torch.from_numpy(a).pin_memory().numpy() for a in z1]
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        # (set_state would wait for the stream)
        rc = mesh._lib.zg_state_upload(mesh.ctx, *(a.ctypes.data_as(C.POINTER(C.c_double)) for a in pinned))
    assert rc == 0
    torch.cuda.synchronize()
    solver.update(mesh, steps=2)
    with torch.cuda.stream(stream):
        graph.replay()
    torch.cuda.synchronize()
    solver.update(mesh)
    assert solver.dt() == dt
    assert np.array_equal(np.array(mesh.get_state()), want)
    mesh.close()
