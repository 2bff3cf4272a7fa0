"""The FP64 grouped GEMM at the edges of its tiles, slabs and split reductions.

H_eff*psi of synthetic U(1) and SU(2) problems whose sector dimensions lie around the
8 x 8 strips, the 64-wide (complex: 64 x 32) tiles and the k slabs of 16 (8), with one
problem of few large sectors whose reductions are split into partial tiles, against plain
numpy products.  Tolerance 1e-12 of max |H psi|: sums of at most a few thousand O(1)
products in FP64, in another order.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33]
WIDE = [1, 63, 64, 65, 5, 127, 128, 129, 12]
LONG = [40, 700, 33]


def _dims(sym, sizes):
    return {(2 * i if sym else 2 * (i - len(sizes) // 2)): n for i, n in enumerate(sizes)}


def _bt(dirs, bonds, blocks, dtype):
    import sadmrg
    qs = [list(b) for b in bonds]
    ds = [list(b.values()) for b in bonds]

    def index(lab):
        i = 0
        for b in range(len(qs) - 1, -1, -1):
            i = i * len(qs[b]) + qs[b].index(lab[b])
        return i

    order = sorted(blocks, key=index)
    data = np.concatenate([blocks[k].reshape(-1, order="F") for k in order]).astype(dtype)
    return sadmrg.BlockTensorData(dirs, qs, ds, 0, np.array([index(k) for k in order], np.int64), data)


@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("sym", [0, 1], ids=["u1", "su2"])
@pytest.mark.parametrize("left,right", [(SMALL, SMALL[::-1]), (WIDE, SMALL[:9]), (WIDE, WIDE[::-1]), (LONG, LONG[::-1])],
                         ids=["small", "mixed", "wide", "long"])
def test_heff_fp64_matches_plain_products(sym, cplx, left, right):
    import sadmrg
    rng = np.random.default_rng(len(left) + 10 * sym + cplx)
    dt = np.complex128 if cplx else np.float64

    def rand(*s):
        x = rng.standard_normal(s)
        return x + 1j * rng.standard_normal(s) if cplx else x

    dl, dr = _dims(sym, left), _dims(sym, right)
    sr = 1 if sym else -1
    ch = {2: 1} if sym else {-2: 1, 0: 1, 2: 1}

    def op(d):
        out = {}
        for a in d:
            for b in d:
                for c in ch:
                    if (abs(a - b) <= 2 <= a + b) if sym else (b == a + c):
                        out[(a, c, b)] = rand(d[a], 1, d[b])
        return out

    psi = {(q, q): rand(dl[q], dr[q]) for q in dl}
    hl, hr = {(q, q): rand(n, n) for q, n in dl.items()}, {(q, q): rand(n, n) for q, n in dr.items()}
    ops = [(op(dl), op(dr)) for _ in range(2)]
    h = sadmrg.Handle(sym=sym, cplx=cplx)
    h.set_autotune(False)
    tens = []
    for a, b in ops:
        tens += [_bt([-1, -1, 1], [dl, ch, dl], a, dt), _bt([-sr, -sr, sr], [dr, ch, dr], b, dt)]
    p = _bt([1, sr], [dl, dr], psi, dt)
    h.heff_plan(p, _bt([-1, 1], [dl, dl], hl, dt), _bt([-sr, sr], [dr, dr], hr, dt), tens, [(0, 1), (2, 3)])
    ref = {k: hl[k].T @ b + b @ hr[k] for k, b in psi.items()}
    for a, b in ops:
        for (x, c, y), m in a.items():
            f = math.sqrt((y + 1) / (x + 1)) if sym else 1.0
            ref[(y, y)] = ref[(y, y)] + f * (m[:, 0].T @ psi[(x, x)] @ b[(x, c, y)][:, 0])
    want = np.concatenate([ref[k].reshape(-1, order="F") for k in psi])
    for _ in range(2):   # the second run finds the split tiles' counters as the first left them
        got = h.heff_apply(p.data, sadmrg.PREC_FP64)
        np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * np.abs(want).max())
    h.close()
