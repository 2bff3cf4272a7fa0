"""The block Jacobi at the edges of its column blocks, rounds and shares of CTAs.

sadmrg_svd_truncate on random U(1) sector blocks whose column counts lie around the
widths of a column block (8, 16) and of a visit (16, 32), tall, wide and square, odd and
even, alone on a CTA or shared by several, with resident and streamed visits, against the
numpy oracle.  All singular values are kept; tolerance 1e-10 of the largest entry of the
recomposed state.
"""
import numpy as np
import pytest

from oracle.svd import svd_truncate
from test_gemm_edges_gpu import _bt as _tensor
from test_svd_random_gpu import _bt, _recompose

pytestmark = pytest.mark.gpu

EDGES = [(1, 1), (1, 5), (7, 2), (8, 8), (9, 7), (15, 40), (16, 16), (17, 17), (24, 23), (31, 31), (32, 33), (33, 32),
         (47, 200), (65, 64)]
FEW = [(150, 131), (3, 9), (20, 70)]


@pytest.mark.parametrize("precondition", [0, 2], ids=["plain", "qr"])
@pytest.mark.parametrize("block", [8, 16], ids=["b8", "b16"])
@pytest.mark.parametrize("stream", [0, 1], ids=["resident", "streamed"])
@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("sizes", [EDGES, FEW], ids=["edges", "few"])
def test_block_jacobi_at_edges(sizes, cplx, stream, block, precondition):
    import sadmrg
    rng = np.random.default_rng(len(sizes) + cplx)
    # bonds three charges apart: fused with a spin-1/2 site each gives two legs of its size
    left = {3 * i: n for i, (n, _) in enumerate(sizes)}
    right = {3 * i: m for i, (_, m) in enumerate(sizes)}
    fl = {q + s: n for q, n in left.items() for s in (-1, 1)}
    fr = {q + s: n for q, n in right.items() for s in (-1, 1)}
    dt = np.complex128 if cplx else np.float64

    def rand(*s):
        x = rng.standard_normal(s)
        return x + 1j * rng.standard_normal(s) if cplx else x

    site = {-1: 1, 1: 1}
    psi = _tensor([1, -1], [fl, fr], {(q, q): rand(fl[q], fr[q]) for q in fl}, dt)

    def fuse(dirs, d):
        out = {}
        for a in d[0]:
            for b in d[1]:
                for c in d[2]:
                    if sum(s * q for s, q in zip(dirs, (a, b, c))) == 0:
                        out[(a, b, c)] = np.zeros((d[0][a], d[1][b], d[2][c]))
        return _tensor(dirs, d, out, dt)

    tu, tv = fuse([1, 1, -1], [left, site, fl]), fuse([1, -1, 1], [site, right, fr])
    keep = sum(2 * min(n, m) for n, m in sizes)
    h = sadmrg.Handle(sym=0, cplx=cplx)
    h.set_svd_stream(stream)
    h.set_svd_block(block)
    h.set_svd_precondition(precondition)
    u, v, kept, _ = h.svd_truncate(psi, tu, tv, 1.0, 0.0, keep)
    assert kept == keep
    ou, ov, _ = svd_truncate(_bt(psi, 0), _bt(tu, 0), _bt(tv, 0), 1.0, 0.0, keep)
    assert u.qs[2] == list(ou.bonds[2][0]) and u.ds[2] == list(ou.bonds[2][1])
    ref, got = _recompose(ou, ov), _recompose(_bt(u, 0), _bt(v, 0))
    assert set(got) == set(ref)
    scale = max(np.abs(a).max() for a in ref.values())
    for k in ref:
        np.testing.assert_allclose(got[k], ref[k], rtol=0, atol=1e-10 * scale)
    assert h.device_status() == 0
    h.close()
