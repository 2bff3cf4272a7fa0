"""A block with NaNs among the blocks of an SVD: the call ends, and the other blocks are as
they are without it, bit for bit.

The Jacobi orders a block's columns by their norms, several of which are NaN here: the order
has to be a permutation all the same.
"""
import numpy as np
import pytest

from test_gemm_edges_gpu import _bt as _tensor
from test_svd_random_gpu import _bt, _recompose

pytestmark = pytest.mark.gpu

SIZES = {0: (40, 37), 3: (90, 70), 6: (12, 20)}


@pytest.mark.parametrize("precondition", [0, 2], ids=["plain", "qr"])
@pytest.mark.parametrize("block", [8, 16], ids=["b8", "b16"])
@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
def test_nan_stays_in_its_block(cplx, block, precondition):
    import sadmrg
    rng = np.random.default_rng(4)
    left, right, site = {q: n for q, (n, _) in SIZES.items()}, {q: m for q, (_, m) in SIZES.items()}, {-1: 1, 1: 1}
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

    tu, tv = fuse([1, 1, -1], [left, site, fl]), fuse([1, -1, 1], [site, right, fr])
    blocks = {(q, q): rand(fl[q], fr[q]) for q in fl}
    keep = sum(2 * min(n, m) for n, m in SIZES.values())
    bad = (2, 2)                      # of 90 x 70
    states = []
    for nan in (False, True):
        b = {k: x.copy() for k, x in blocks.items()}
        if nan:
            b[bad][5, ::7] = np.nan
            b[bad][:, 33] = np.nan
        h = sadmrg.Handle(sym=0, cplx=cplx)
        h.set_svd_block(block)
        h.set_svd_precondition(precondition)
        u, v, _, _ = h.svd_truncate(_tensor([1, -1], [fl, fr], b, dt), tu, tv, 1.0, 0.0, keep)
        assert h.device_status() == 0
        h.close()
        states.append(_recompose(_bt(u, 0), _bt(v, 0)))
    clean, got = states
    assert set(got) == set(clean) and len(clean) == len(fl)
    other = [k for k in clean if not np.array_equal(got[k], clean[k])]
    assert len(other) == 1 and np.isnan(got[other[0]]).any()   # one block per fused charge here
