"""Block SVDs from two host threads with a handle each.

The kernels of the QR and of the Jacobi take the shared memory that the call's blocks need,
and have to be allowed their largest size once: allowed per call, one thread's small blocks
refused the other's launch.  Both threads' results are compared with the ones each gets
alone, bit for bit (a call's schedule does not depend on what else runs).
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(m, n, seed):
    from test_gemm_edges_gpu import _bt as _tensor
    rng = np.random.default_rng(seed)
    left, right, site = {0: m}, {0: n}, {-1: 1, 1: 1}
    fl = {q + s: k for q, k in left.items() for s in (-1, 1)}
    fr = {q + s: k for q, k in right.items() for s in (-1, 1)}
    psi = _tensor([1, -1], [fl, fr], {(q, q): rng.standard_normal((fl[q], fr[q])) for q in fl}, np.float64)

    def fuse(dirs, d):
        out = {}
        for a in d[0]:
            for b in d[1]:
                for c in d[2]:
                    if sum(s * q for s, q in zip(dirs, (a, b, c))) == 0:
                        out[(a, b, c)] = np.zeros((d[0][a], d[1][b], d[2][c]))
        return _tensor(dirs, d, out, np.float64)

    return psi, fuse([1, 1, -1], [left, site, fl]), fuse([1, -1, 1], [site, right, fr])


@pytest.mark.parametrize("precondition", [0, 2], ids=["plain", "qr"])
def test_two_threads_with_their_own_sizes(precondition):
    import sadmrg
    shapes = [(20, 18), (190, 180)]
    args = [_problem(m, n, m) for m, n in shapes]
    handles = []
    for _ in shapes:
        h = sadmrg.Handle(sym=0, cplx=False)
        h.set_svd_precondition(precondition)
        handles.append(h)
    alone = []
    for h, (m, n), a in zip(handles, shapes, args):
        u, v, kept, _ = h.svd_truncate(*a, 1.0, 0.0, 2 * min(m, n))
        alone.append((u.data.copy(), v.data.copy(), kept))
    bad = []

    def work(k, count):
        try:
            for _ in range(count):
                u, v, kept, _ = handles[k].svd_truncate(*args[k], 1.0, 0.0, 2 * min(shapes[k]))
                if kept != alone[k][2] or not np.array_equal(u.data, alone[k][0]) or not np.array_equal(v.data, alone[k][1]):
                    bad.append((k, "result"))
        except Exception as e:   # noqa: BLE001
            bad.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(0, 400)), threading.Thread(target=work, args=(1, 100))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]
    for h in handles:
        assert h.device_status() == 0
        h.close()
