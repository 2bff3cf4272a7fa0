"""Linear combinations of more vectors than a block stages coefficients for.

Sizes around the staged 2,048 and beyond 48 KB of coefficients.  Entries and coefficients
are small integers, so that every sum is exact in any order: results have to be equal.
"""
import ctypes

import pytest

import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("nv", [1, 8, 2047, 2048, 2049, 3100, 6200])
def test_many_vectors(nv, cplx):
    import torch
    lib = native.load()
    n = 300
    g = torch.Generator(device="cuda").manual_seed(nv)

    def ints(*shape):
        x = torch.randint(-4, 5, shape, generator=g, device="cuda").double()
        return torch.complex(x, torch.randint(-4, 5, shape, generator=g, device="cuda").double()) if cplx else x

    V, c, x = ints(nv, n), ints(nv), ints(n)
    r = torch.randint(-4, 5, (nv,), generator=g, device="cuda").double()
    partial = torch.zeros(4 * 592, dtype=torch.float64, device="cuda")
    counter = torch.zeros(1, dtype=torch.int32, device="cuda")
    norm = torch.zeros(2, dtype=torch.float64, device="cuda")
    want_x = x - (c.unsqueeze(1) * V).sum(0)
    want_y = (r.unsqueeze(1) * V).sum(0)
    y = torch.full_like(x, -1)
    s = torch.cuda.current_stream()
    s.synchronize()
    st = ctypes.c_void_p(s.cuda_stream)
    assert lib.nc_axpy(int(cplx), ctypes.c_longlong(n), native.ptr(x), native.ptr(V), nv, native.ptr(c),
                       native.ptr(partial), native.ptr(counter), native.ptr(norm), st) == 0
    assert lib.nc_lincomb(int(cplx), ctypes.c_longlong(n), native.ptr(y), native.ptr(V), nv, native.ptr(r),
                          native.ptr(partial), native.ptr(counter), ctypes.c_void_p(norm.data_ptr() + 8), st) == 0
    torch.cuda.synchronize()
    assert torch.equal(x, want_x) and torch.equal(y, want_y)
    for k, w in enumerate((want_x, want_y)):
        s2 = (w.real ** 2 + (w.imag ** 2 if cplx else 0)).sum().item()   # whole numbers below 2^53
        assert abs(norm[k].item() - s2 ** 0.5) <= 1e-15 * s2 ** 0.5
    assert counter.item() == 0
