"""The Krylov vector kernels at the edges of their ranges, one problem and many at once.

Each problem has one U(1) sector: H psi = hl^T psi + psi hr with symmetric (Hermitian)
hl, hr, so a few Lanczos steps can be restated in numpy.  Vector lengths lie around
a thread block's 256 elements, below one warp and across several blocks; Krylov
sizes cross the groups of 8 vectors that one pass takes.  Energies after a fixed
number of steps agree with numpy's to 1e-12 relative (the sums differ only in
order; the spectra here are O(1)), and the Ritz vectors' Rayleigh quotients too.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(5, 3), (1, 31), (16, 16), (5, 51), (257, 1), (37, 90), (130, 41)]


def _problem(m, n, cplx, seed):
    import sadmrg
    rng = np.random.default_rng([m, n, seed])

    def rand(a, b):
        x = rng.standard_normal((a, b))
        return x + 1j * rng.standard_normal((a, b)) if cplx else x

    hl, hr, psi = rand(m, m), rand(n, n), rand(m, n)
    hl, hr = (hl + hl.conj().T) / np.sqrt(8 * m), (hr + hr.conj().T) / np.sqrt(8 * n)

    def bt(dirs, a):
        return sadmrg.BlockTensorData(dirs, [[0], [0]], [[a.shape[0]], [a.shape[1]]], 0, np.array([0], np.int64),
                                      np.ascontiguousarray(a.reshape(-1, order="F")))

    return hl, hr, psi, bt([1, -1], psi), bt([-1, 1], hl), bt([1, -1], hr)


def _lanczos(hl, hr, psi, steps):
    v = psi / np.linalg.norm(psi)
    basis, al, be = [v], [], []
    for k in range(steps):
        w = hl.T @ basis[-1] + basis[-1] @ hr
        al.append(np.vdot(basis[-1], w).real)
        for _ in range(2):
            for b in basis:
                w = w - np.vdot(b, w) * b
        be.append(np.linalg.norm(w))
        if be[-1] < 1e-10:
            break
        basis.append(w / be[-1])
    n = len(al)
    return np.linalg.eigvalsh(np.diag(al) + np.diag(be[:n - 1], 1) + np.diag(be[:n - 1], -1))[0]


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("steps", [7, 8, 13])
def test_lanczos_steps_match_numpy(cplx, steps):
    import sadmrg
    batch = sadmrg.Handle(sym=0, cplx=cplx)
    batch.set_lanczos_tol(1e-15)
    ref, start, probs = [], [], []
    for i, (m, n) in enumerate(SHAPES):
        hl, hr, psi, tp, tl, tr = _problem(m, n, cplx, 3)
        h = sadmrg.Handle(sym=0, cplx=cplx)
        h.set_autotune(False)
        h.set_lanczos_tol(1e-15)
        h.heff_plan(tp, tl, tr, [], [])
        if m * n > 4 * steps:       # no breakdown before the last step
            e, v, _ = h.heff_lanczos2(tp.data, steps)
            x = v.reshape((m, n), order="F")
            want = _lanczos(hl, hr, psi, steps)
            rq = np.vdot(x, hl.T @ x + x @ hr).real
            assert abs(e - want) <= 1e-12 * abs(want), (m, n)
            assert abs(rq - want) <= 1e-12 * abs(want) and abs(np.linalg.norm(x) - 1) < 1e-12, (m, n)
            batch.batch_add(h)
            ref.append(want)
            start.append(tp.data)
            probs.append((hl, hr, m, n))
        h.close()
    off = batch.batch_finalize()["offsets"]
    e, v, mv, _ = batch.batch_lanczos(np.concatenate(start), steps, sadmrg.PREC_FP64)
    for i, (hl, hr, m, n) in enumerate(probs):
        x = v[off[i]:off[i + 1]].reshape((m, n), order="F")
        rq = np.vdot(x, hl.T @ x + x @ hr).real
        assert abs(e[i] - ref[i]) <= 1e-12 * abs(ref[i]), (m, n)
        assert abs(rq - ref[i]) <= 1e-12 * abs(ref[i]), (m, n)
    batch.close()
