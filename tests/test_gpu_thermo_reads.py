"""Energy, virial and kinetic sums are added up when they are read: reading them after every step,
after some or only at the end gives the same numbers, and a force without a kick or a kick without a
force leaves the other's sums standing."""
import numpy as np
import pytest

import tinymd
from helpers import make_sim

pytestmark = pytest.mark.gpu


def read(lib):
    t = np.zeros(4)
    assert lib.md_get_thermo(tinymd.ptr(t)) == 0
    return t


@pytest.fixture
def thermo_lib(product, cuda_device):
    product.md_set_thermo(1)
    yield product
    product.md_set_thermo(0)
    product.md_set_precision(0)


# sizes on both sides of the lanes-per-atom rules: the number of partial sums differs between the
# force and a separate kick below, and is the same above
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("cells", [(6, 6, 6), (22, 22, 22)])
def test_reads_at_any_cadence(thermo_lib, cells, precision):
    lib = thermo_lib
    lib.md_set_precision(precision)
    last = []
    for every in (1, 3, 12):
        sim = make_sim(lib, cells=cells, setup_lib=lib, reneigh=5)
        for k in range(12):
            sim.run(0.005, 1)
            if (k + 1) % every == 0:
                t = read(lib)
        sim.close()
        last.append(t)
    np.testing.assert_array_equal(last[0], last[1])
    np.testing.assert_array_equal(last[0], last[2])


@pytest.mark.parametrize("half", [False, True])
def test_parts_stand_until_replaced(thermo_lib, half):
    lib = thermo_lib
    sim = make_sim(lib, cells=(6, 6, 6), setup_lib=lib, half=half)
    sim.step(0.005, 3)
    a = read(lib)
    np.testing.assert_array_equal(read(lib), a)
    sim.force()  # the same positions: the same energy, and the kick's kinetic sum stands
    b = read(lib)
    np.testing.assert_allclose(b, a, rtol=1e-12)
    assert b[3] == a[3]
    sim.force()
    lib.md_final_integration(0.0)  # no change of velocity: every sum as before
    np.testing.assert_allclose(read(lib), a, rtol=1e-12)
    v = np.zeros((sim.n, 3))
    v[:, 0] = 2.0
    lib.md_set_velocities(tinymd.ptr(v))
    lib.md_final_integration(0.0)  # a kick alone: the force's sums stand
    c = read(lib)
    assert c[3] == 4.0 * sim.n
    np.testing.assert_allclose(c[:3], a[:3], rtol=1e-12)
    sim.close()
