"""Sector blocks without rows or columns beside others in one SVD call.

The Jacobi (with and without QRs before it) called directly: W V^H = op(A) to 1e-12 of the
largest entry, orthonormal V and numpy's singular values for the others.
"""
import numpy as np
import pytest

import native

pytestmark = pytest.mark.gpu

CASES = [[(0, 5), (20, 9), (7, 0), (33, 40), (0, 0)], [(64, 50), (0, 3)], [(0, 4)], [(3, 0), (0, 0)], [(1, 1), (0, 1)]]


@pytest.mark.parametrize("precondition", [0, 1, 2])
@pytest.mark.parametrize("block", [8, 16])
@pytest.mark.parametrize("stream", [0, 1], ids=["resident", "streamed"])
@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("sizes", CASES, ids=lambda s: "-".join(f"{m}x{n}" for m, n in s))
def test_empty_blocks(sizes, cplx, stream, block, precondition):
    import torch
    rng = np.random.default_rng(len(sizes))
    dt = np.complex128 if cplx else np.float64

    def rand(m, n):
        x = rng.standard_normal((m, n))
        return x + 1j * rng.standard_normal((m, n)) if cplx else x

    blocks = [rand(m, n) for m, n in sizes]
    flat = np.concatenate([b.ravel(order="F") for b in blocks] + [np.zeros(1)]).astype(dt)
    nw, nv, ns = (sum(f(m, n) for m, n in sizes) + 1 for f in (lambda m, n: m * n, lambda m, n: min(m, n) ** 2, min))
    a = torch.from_numpy(flat).cuda()
    w, v = torch.zeros(nw, dtype=a.dtype, device="cuda"), torch.zeros(nv, dtype=a.dtype, device="cuda")
    sv = torch.zeros(ns, dtype=torch.float64, device="cuda")
    m, n = (np.array([s[i] for s in sizes], np.int32) for i in (0, 1))
    torch.cuda.synchronize()
    sweeps = native.load().nc_jacobi(int(cplx), native.ptr(a), native.ptr(w), native.ptr(v), native.ptr(sv), len(sizes),
                                     native.ptr(m), native.ptr(n), precondition, stream, block)
    torch.cuda.synchronize()
    assert 1 <= sweeps < 60
    w, v, sv = w.cpu().numpy(), v.cpu().numpy(), sv.cpu().numpy()
    wo = vo = so = 0
    for b in blocks:
        op = b if b.shape[0] >= b.shape[1] else b.conj().T
        R, C = op.shape
        W, V = w[wo:wo + R * C].reshape((R, C), order="F"), v[vo:vo + C * C].reshape((C, C), order="F")
        if C:
            assert np.abs(W @ V.conj().T - op).max() <= 1e-12 * np.abs(op).max()
            assert np.abs(V.conj().T @ V - np.eye(C)).max() <= 1e-12
            want = np.linalg.svd(op, compute_uv=False)
            assert np.abs(np.sort(sv[so:so + C])[::-1] - want).max() <= 1e-12 * want[0]
        wo, vo, so = wo + R * C, vo + C * C, so + C
