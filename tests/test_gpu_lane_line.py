"""The mixed LJ kernels on both sides of the size from which an atom's list is no longer shared by four
lanes (31,000 atoms): forces and sums after 21 steps against the FP64 form of the same state."""
import numpy as np
import pytest

import tinymd
from helpers import make_sim, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(20, 20, 19), (19, 17, 24), (20, 19, 21), (20, 20, 20)])
def test_mixed_error(product, cuda_device, cells):
    """30,400 | 31,008, 31,920 and 32,000 atoms; the tolerance is the mixed form's stated error."""
    product.md_set_precision(1)
    product.md_set_thermo(1)
    try:
        sim = make_sim(product, cells=cells, setup_lib=product, reneigh=5)
        sim.step(0.005, 21)
        out = []
        for precision in (1, 0):
            product.md_set_precision(precision)
            sim.force()
            product.md_final_integration(0.0)
            sums = np.zeros(4)
            assert product.md_get_thermo(tinymd.ptr(sums)) == 0
            out.append((tinymd.full_state(product)[2], sums))
        sim.close()
    finally:
        product.md_set_precision(0)
        product.md_set_thermo(0)
    (f32, t32), (f64, t64) = out
    assert rel_err(f32, f64) <= 1e-5
    assert t32[2] == t64[2]
    np.testing.assert_allclose(t32[[0, 3]], t64[[0, 3]], rtol=1e-6)
