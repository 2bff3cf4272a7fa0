"""sadmrg_svd_truncate with a sector of dimension zero among the others: it keeps nothing, and
the state is that of the other sectors."""
import numpy as np
import pytest

from test_gemm_edges_gpu import _bt as _tensor
from test_svd_random_gpu import _bt, _recompose

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precondition", [0, 2], ids=["plain", "qr"])
@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
def test_sector_of_dimension_zero(cplx, precondition):
    import sadmrg
    rng = np.random.default_rng(3)
    sizes = {0: (40, 37), 3: (0, 20), 6: (9, 12)}
    left, right, site = {q: s[0] for q, s in sizes.items()}, {q: s[1] for q, s in sizes.items()}, {-1: 1, 1: 1}
    fl = {q + s: n for q, n in left.items() for s in (-1, 1)}
    fr = {q + s: n for q, n in right.items() for s in (-1, 1)}
    dt = np.complex128 if cplx else np.float64

    def rand(*s):
        x = rng.standard_normal(s)
        return x + 1j * rng.standard_normal(s) if cplx else x

    def fuse(dirs, d):
        out = {}
        for a in d[0]:
            for b in d[1]:
                for c in d[2]:
                    if sum(s * q for s, q in zip(dirs, (a, b, c))) == 0:
                        out[(a, b, c)] = np.zeros((d[0][a], d[1][b], d[2][c]))
        return _tensor(dirs, d, out, dt)

    blocks = {(q, q): rand(fl[q], fr[q]) for q in fl}
    keep = sum(2 * min(n, m) for n, m in sizes.values())
    h = sadmrg.Handle(sym=0, cplx=cplx)
    h.set_svd_precondition(precondition)
    u, v, kept, _ = h.svd_truncate(_tensor([1, -1], [fl, fr], blocks, dt), fuse([1, 1, -1], [left, site, fl]),
                                   fuse([1, -1, 1], [site, right, fr]), 1.0, 0.0, keep)
    assert kept == keep and 0 not in u.ds[2]
    assert u.qs[2] == [q for q in sorted(fl) if fl[q]]
    got = _recompose(_bt(u, 0), _bt(v, 0))
    for (q, _), b in blocks.items():
        if b.size:
            x = [g for k, g in got.items() if k[0] + k[1] == q]
            assert len(x) == 1
            # u carries the singular values' power 1, so u v is the block itself
            np.testing.assert_allclose(x[0].reshape(b.shape, order="F"), b, rtol=0, atol=1e-12 * np.abs(b).max())
    assert h.device_status() == 0
    h.close()
