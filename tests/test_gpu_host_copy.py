"""Downloads of device arrays into pageable host memory through the staged
copy: sizes around its lower limit and its chunks, several contexts at a time,
and the packed layouts, against the values that were uploaded."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(Z, nx, ny):
    gen = Z.Rectangle(0.0, 1.0, 0.0, 1.0)
    gen.set_sizes(nx, ny)
    mesh = Z.EuMesh(gen)
    Z.SmFluid(Z.IdealGas(1.4)).add_types(mesh)
    return mesh


# 5 fields of 8 bytes: 4 MB in all lies between 104857 and 104858 cells, a
# chunk of 2 MB holds 262144 values of one field
@pytest.mark.parametrize("nx,ny", [(1, 104857), (1, 104858), (1, 262143), (1, 262144), (1, 262145), (1031, 1021)])
def test_state_round_trip(gpu_lib, nx, ny):
    Z = gpu_lib
    mesh = _mesh(Z, nx, ny)
    z = [np.random.default_rng(k).random(nx * ny) for k in range(5)]
    mesh.set_state(*z)
    for a, b in zip(mesh.get_state(), z):
        assert np.array_equal(a, b)
    mesh.close()


def test_two_contexts_at_a_time(gpu_lib):
    Z = gpu_lib
    wrong = []

    def work(seed):
        mesh = _mesh(Z, 700, 800)
        z = [np.random.default_rng(seed + k).random(560000) for k in range(5)]
        mesh.set_state(*z)
        for _ in range(10):
            if not all(np.array_equal(a, b) for a, b in zip(mesh.get_state(), z)):
                wrong.append(seed)
        mesh.close()

    threads = [threading.Thread(target=work, args=(100 * k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("n", [7, 193, 401])
def test_mixture_states_round_trip(gpu_lib, n):
    Z = gpu_lib
    from zephyr_b200.mmf import Material, MixturePT, MmFluid
    gen = Z.Rectangle(0.0, 1.0, 0.0, 1.0)
    gen.set_sizes(n, n)
    mesh = Z.EuMesh(gen)
    solver = MmFluid(MixturePT([Material.stiffened("Water"), Material.ideal("Air")]))
    solver.add_types(mesh)
    rng = np.random.default_rng(n)
    cells = rng.random((n * n, 14))
    cells[:, 8:10] = 0.0  # materials 2 and 3 are absent
    solver.set_states(mesh, cells)
    got = solver.states(mesh)
    keep = [0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11]
    assert np.array_equal(got[:, keep], cells[:, keep])
    assert np.isnan(got[:, 12:]).all()
    mesh.close()
