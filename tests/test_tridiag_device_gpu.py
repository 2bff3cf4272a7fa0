"""The device tridiagonal solver against the host's, bit for bit.

Both run the same implicit QL; the sign of a Ritz vector depends on how often an almost
converged coupling is swept, so eigenvalue and vector have to agree to the last bit, sign
included.  Every size at which the kernel's layout changes, sizes mixed in one launch up to
the largest, and matrices of the kinds a Lanczos run makes and harder ones: random, close
eigenvalue pairs, zero couplings, graded over many decades, couplings near underflow, scaled
by 1e-150 and 1e+150.
"""
import ctypes

import numpy as np
import pytest

import native

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 7, 31, 32, 33, 40, 63, 64, 65, 77, 78, 100, 127, 128]
KINDS = ["lanczos", "pairs", "split", "graded", "tiny couplings", "small", "large"]


def _matrix(kind, n, rng):
    d, e = rng.standard_normal(n), np.abs(rng.standard_normal(max(n - 1, 0))) + 1e-3
    if kind == "lanczos":
        d, e = 0.1 * d - 1.0, 0.5 + 0.1 * e
    elif kind == "pairs":
        d, e = np.abs(np.arange(n) - (n - 1) / 2.0), np.ones(max(n - 1, 0))
    elif kind == "split":
        e[rng.random(e.size) < 0.2] = 0.0
    elif kind == "graded":
        d, e = d * 10.0 ** (-0.2 * np.arange(n)), e * 10.0 ** (-0.2 * np.arange(e.size))
    elif kind == "tiny couplings":
        e = e * 10.0 ** rng.integers(-320, 1, e.size).astype(float)
    elif kind == "small":
        d, e = d * 1e-150, e * 1e-150
    elif kind == "large":
        d, e = d * 1e150, e * 1e150
    return d, e


def _device(mats, nmax):
    import torch
    lib = native.load()
    ns = len(mats)
    nn = np.array([d.size for d, _ in mats], np.int32)
    a, b = np.zeros((nmax, ns)), np.zeros((nmax + 1, ns))
    for s, (d, e) in enumerate(mats):
        a[:d.size, s] = d
        b[1:d.size, s] = e
    dev = [torch.from_numpy(x).cuda() for x in (nn, a, b)]
    z0 = torch.full((ns, nmax + 1), 7.0, dtype=torch.float64, device="cuda")
    e0 = torch.full((ns,), 7.0, dtype=torch.float64, device="cuda")
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    s = torch.cuda.current_stream()
    s.synchronize()
    assert lib.nc_tridiag_device(ns, native.ptr(dev[0]), nmax, native.ptr(dev[1]), native.ptr(dev[2]), native.ptr(z0),
                                 nmax + 1, native.ptr(e0), native.ptr(st), ctypes.c_void_p(s.cuda_stream)) == 0
    torch.cuda.synchronize()
    return e0.cpu().numpy(), z0.cpu().numpy(), st.item()


def _host(d, e):
    e0, z0 = np.zeros(1), np.zeros(d.size)
    rc = native.load().nc_tridiag_host(d.size, native.ptr(d), native.ptr(e), native.ptr(e0), native.ptr(z0))
    return rc, e0[0], z0


def _compare(mats, nmax):
    e0, z0, st = _device(mats, nmax)
    assert st == 0
    for s, (d, e) in enumerate(mats):
        rc, we, wz = _host(d, e)
        assert rc == 0
        got = np.concatenate([e0[s:s + 1], z0[s, :d.size]])
        assert np.array_equal(got.view(np.int64), np.concatenate([[we], wz]).view(np.int64)), (s, d.size)
        assert np.all(z0[s, d.size:nmax] == 0.0) and z0[s, nmax] == 7.0


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", SIZES)
def test_equal_sizes(n, kind):
    rng = np.random.default_rng([n, KINDS.index(kind)])
    _compare([_matrix(kind, n, rng) for _ in range(40)], n)


@pytest.mark.parametrize("nmax", [32, 64, 128])
def test_mixed_sizes_in_one_launch(nmax):
    rng = np.random.default_rng(nmax)
    mats = [_matrix(KINDS[i % len(KINDS)], min(n, nmax), rng) for i, n in enumerate(SIZES * 6)]
    _compare(mats, nmax)


def test_segments_without_rows_are_left_alone():
    rng = np.random.default_rng(1)
    mats = [_matrix("lanczos", n, rng) for n in (9, 0, 5)]
    e0, z0, st = _device(mats, 9)
    assert st == 0 and e0[1] == 7.0 and np.all(z0[1] == 7.0)
    for s in (0, 2):
        _, we, wz = _host(*mats[s])
        assert e0[s] == we and np.array_equal(z0[s, :mats[s][0].size], wz)


def test_no_convergence_is_reported_by_both():
    d, e = np.array([1.0, np.nan, 2.0, 0.5]), np.ones(3)
    _, z0, st = _device([(d, e), _matrix("lanczos", 4, np.random.default_rng(2))], 4)
    assert st == 1 and np.all(z0[0, :4] == 0.0)
    assert _host(d, e)[0] == 1
