"""sadmrg_heff_launches_per_matvec against the launches that a context counts.

One handle has a chain (whose statistics hold the counter) and a plan; the counter's change
over one H_eff*psi is the figure of the entry point, with and without a penalty.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
def test_launches_of_a_matvec(cplx):
    import sadmrg
    h = sadmrg.Handle(sym=0, cplx=cplx)
    h.chain_create(1, 12, 16, 1, 0, True, 0.0)
    h.chain_idmrg()
    psi = h.chain_freeze(5)
    rng = np.random.default_rng(0)
    o = rng.standard_normal((2, psi.data.size)).astype(psi.data.dtype)

    def counted(prec):
        a = h.chain_stats()["launches"]
        h.heff_apply(psi.data, prec)
        return h.chain_stats()["launches"] - a

    for vecs, weights in (([], []), (o, [0.5, -0.25])):
        h.heff_set_penalty(vecs, weights)
        for prec in (sadmrg.PREC_FP64, sadmrg.PREC_TF32X3):
            assert counted(prec) == h.heff_launches_per_matvec(prec), (len(vecs), prec)
    h.close()
