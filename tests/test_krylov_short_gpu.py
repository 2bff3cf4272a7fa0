"""The Krylov vector kernels on vectors shorter than a warp's lanes, one problem and many.

As test_krylov_gpu.py, with Krylov sizes up to three below the vectors' length, so that
every shape runs: fewer vectors than a pass takes, as many, and remainders of 1 and 5.
"""
import numpy as np
import pytest

from test_krylov_gpu import _lanczos, _problem

pytestmark = pytest.mark.gpu

SHAPES = [(5, 3), (1, 17), (4, 5), (17, 1), (3, 9), (1, 31), (8, 4), (3, 5), (33, 1)]


@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("steps", [3, 4, 5, 8, 9, 12])
def test_short_vectors(steps, cplx):
    import sadmrg
    batch = sadmrg.Handle(sym=0, cplx=cplx)
    batch.set_lanczos_tol(1e-15)
    want, start = [], []
    for m, n in SHAPES:
        assert m * n >= steps + 3
        hl, hr, psi, tp, tl, tr = _problem(m, n, cplx, 11)
        h = sadmrg.Handle(sym=0, cplx=cplx)
        h.set_autotune(False)
        h.set_lanczos_tol(1e-15)
        h.heff_plan(tp, tl, tr, [], [])
        want.append(_lanczos(hl, hr, psi, steps))
        e, v, _ = h.heff_lanczos2(tp.data, steps)
        x = v.reshape((m, n), order="F")
        rq = np.vdot(x, hl.T @ x + x @ hr).real
        assert abs(e - want[-1]) <= 1e-12 * abs(want[-1]), (m, n)
        assert abs(rq - want[-1]) <= 1e-12 * abs(want[-1]) and abs(np.linalg.norm(x) - 1) < 1e-12, (m, n)
        batch.batch_add(h)
        start.append(tp.data)
        h.close()
    batch.batch_finalize()
    e, _, mv, _ = batch.batch_lanczos(np.concatenate(start), steps, sadmrg.PREC_FP64)
    assert len(e) == len(SHAPES)
    for s, (m, n) in enumerate(SHAPES):
        assert abs(e[s] - want[s]) <= 1e-12 * abs(want[s]), (m, n)
    batch.close()
