"""Ritz pairs of a batch solved on the device against those of the host's solver.

A batch of eight instances or more diagonalises its tridiagonals on the device, one of
fewer on the host.  The same instances solved together and one at a time, for Krylov
sizes around 32 and 64 rows and above and beyond the device solver's limit of 128: equal
energies to 1e-12 relative and Ritz vectors to 1e-9 (a relative rounding of 1e-14 in the
Krylov coefficients over gaps of a thousandth of the spectrum and more).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[False, True], ids=["real", "complex"])
def instances(request):
    import sadmrg
    out = []
    for L, D, J2 in ((12, 8, 0.0), (16, 24, 0.0), (24, 32, 0.3)):
        h = sadmrg.Handle(sym=0, cplx=request.param)
        h.chain_create(1, L, D, 1, 0, True, J2)
        h.chain_idmrg()
        out.append((h, h.chain_freeze(L // 2 - 1)))
    return out


@pytest.mark.parametrize("mlanc", [3, 4, 6, 33, 34, 66, 100, 140])
def test_device_ritz_pairs_equal_host(instances, mlanc):
    import sadmrg
    rng = np.random.default_rng(mlanc)
    use = [instances[i % 3] for i in range(9)]
    xs = [rng.standard_normal(p.data.size) for _, p in use]
    cplx = np.iscomplexobj(use[0][1].data)
    if cplx:
        xs = [x + 1j * rng.standard_normal(x.size) for x in xs]
    many = sadmrg.Handle(sym=0, cplx=cplx)
    for h, _ in use:
        many.batch_add(h)
    off = many.batch_finalize()["offsets"]
    many.set_lanczos_tol(1e-15)
    e, v, _, _ = many.batch_lanczos(np.concatenate(xs), mlanc, sadmrg.PREC_FP64)
    for i, (h, _) in enumerate(use):
        one = sadmrg.Handle(sym=0, cplx=cplx)
        one.batch_add(h)
        one.batch_finalize()
        one.set_lanczos_tol(1e-15)
        e1, v1, _, _ = one.batch_lanczos(xs[i], mlanc, sadmrg.PREC_FP64)
        assert abs(e[i] - e1[0]) <= 1e-12 * abs(e1[0])
        w = v[off[i]:off[i + 1]]
        d = np.vdot(w, v1)
        w = w * (d / abs(d))
        assert np.linalg.norm(w - v1) <= 1e-9
        one.close()
    assert many.device_status() == 0
    many.close()
