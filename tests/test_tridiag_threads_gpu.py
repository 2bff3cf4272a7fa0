"""The device tridiagonal solver from two host threads, each with its own stream and sizes.

Handles may be used from one host thread each, at the same time.  A launch of more than 77
rows takes more than 48 KB of shared memory, which the kernel has to be allowed once for
all sizes: allowed per call, one thread's smaller size refused the other's launch.
Couplings are zero, so the results are known: the smallest diagonal element and its unit
vector.
"""
import ctypes
import threading

import numpy as np
import pytest

import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(101, 65), (128, 66)])
def test_two_threads_with_their_own_sizes(sizes):
    import torch
    lib = native.load()
    bad = []

    def work(n):
        torch.cuda.set_device(0)
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            a = torch.arange(n, 0, -1, dtype=torch.float64, device="cuda")
            b = torch.zeros(n, dtype=torch.float64, device="cuda")
            nn = torch.tensor([n], dtype=torch.int32, device="cuda")
            z = torch.zeros(n, dtype=torch.float64, device="cuda")
            e0 = torch.zeros(1, dtype=torch.float64, device="cuda")
            st = torch.zeros(1, dtype=torch.int32, device="cuda")
            s.synchronize()
            for i in range(3000):
                rc = lib.nc_tridiag_device(1, native.ptr(nn), n, native.ptr(a), native.ptr(b), native.ptr(z), n,
                                           native.ptr(e0), native.ptr(st), ctypes.c_void_p(s.cuda_stream))
                if rc:
                    bad.append((n, i))
                if i % 100 == 99:
                    s.synchronize()
            want = np.zeros(n)
            want[n - 1] = 1.0
            if not np.array_equal(z.cpu().numpy(), want) or e0.item() != 1.0 or st.item():
                bad.append((n, "result"))

    torch.zeros(1, device="cuda")
    threads = [threading.Thread(target=work, args=(n,)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:5]
