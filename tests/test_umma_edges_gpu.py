"""The tcgen05 matvec at the edges of its tiles, row groups, k steps and slabs.

H_eff*psi of synthetic U(1) problems whose operators and vector hold only -1, 0 and 1 (and
i times these), with sector dimensions around the row groups of 8, mma widths of 16, slabs
of 32 and tiles of 64 and 128, and one problem of few large sectors whose reductions are
split.  Every product and every sum is then an integer below 2^22, which the split-precision
path holds exactly (two TF32 parts, FP32 sums), so it has to equal the FP64 one to the last
bit: whatever a copy leaves out, adds or takes from another place shows.
"""
import numpy as np
import pytest

from test_gemm_edges_gpu import _bt, _dims

pytestmark = pytest.mark.gpu

SMALL = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33]
WIDE = [1, 63, 64, 65, 5, 127, 128, 129, 12]
LONG = [40, 600, 33]


@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("left,right", [(SMALL, SMALL[::-1]), (WIDE, SMALL[:9]), (SMALL[:9], WIDE), (WIDE, WIDE[::-1]),
                                        (LONG, LONG[::-1])], ids=["small", "mixed", "mixed2", "wide", "long"])
def test_split_precision_is_exact_on_integers(cplx, left, right):
    import sadmrg
    rng = np.random.default_rng(len(left) + cplx)
    dt = np.complex128 if cplx else np.float64

    def rand(*s):
        x = rng.integers(-1, 2, s).astype(np.float64)
        return x + 1j * rng.integers(-1, 2, s) if cplx else x

    dl, dr = _dims(0, left), _dims(0, right)
    ch = {-2: 1, 0: 1, 2: 1}

    def op(d):
        return {(a, c, b): rand(d[a], 1, d[b]) for a in d for b in d for c in ch if b == a + c}

    psi = {(q, q): rand(dl[q], dr[q]) for q in dl}
    hl, hr = {(q, q): rand(n, n) for q, n in dl.items()}, {(q, q): rand(n, n) for q, n in dr.items()}
    tens = []
    for a, b in [(op(dl), op(dr)) for _ in range(2)]:
        tens += [_bt([-1, -1, 1], [dl, ch, dl], a, dt), _bt([1, 1, -1], [dr, ch, dr], b, dt)]
    p = _bt([1, -1], [dl, dr], psi, dt)
    h = sadmrg.Handle(sym=0, cplx=cplx)
    h.set_autotune(False)
    h.heff_plan(p, _bt([-1, 1], [dl, dl], hl, dt), _bt([1, -1], [dr, dr], hr, dt), tens, [(0, 1), (2, 3)])
    ref = h.heff_apply(p.data, sadmrg.PREC_FP64)
    assert np.abs(ref).max() < 2 ** 22
    for _ in range(2):   # the second one on panels and counters that the first has left
        np.testing.assert_array_equal(h.heff_apply(p.data, sadmrg.PREC_TF32X3), ref)
    assert h.device_status() == 0
    h.close()
