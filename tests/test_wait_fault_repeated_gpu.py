"""A wait that runs out always leaves a status, whichever role of the kernel gives up first.

Producer, issuer and epilogue wait with the same limit, so over many launches (see
test_wait_fault_gpu.py: every wait is bounded, no GPU fault is involved) each of them is the
first now and then.  Afterwards the plan still gives the same H psi.
"""
import os

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["centre_su2_real.npz", "centre_u1_cplx.npz"])
def test_every_aborted_launch_reports(name):
    import sadmrg
    from test_heff_gpu import build_problem
    h, z, m, psi = build_problem(os.path.join(GOLDEN, name))
    before = h.heff_apply(psi.data, sadmrg.PREC_TF32X3)
    for i in range(100):
        assert h.heff_wait_fault_test(2_000_000 + 10_000 * i) != 0, i
        assert h.device_status() == 0
    assert np.array_equal(h.heff_apply(psi.data, sadmrg.PREC_TF32X3), before)
