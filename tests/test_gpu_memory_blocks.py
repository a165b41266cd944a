"""Large value arrays, kept one by one when their matrices go: reused in order across streams and threads,
and given up when another allocation needs the memory."""
import ctypes
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from conftest import ROOT, maxrel
from diaq_gb300 import hamiltonians as ham
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

GIVE_UP = """
import ctypes, torch
from diaq_gb300 import capi
L = capi.lib()
G = 1 << 30
N = 1 << 20
keep = capi.Matrix.create(N, N, [0])
big = capi.Matrix.create(N, N, list(range(150)))                 # 2 x 1.17 GiB
torch.cuda.synchronize()
fill = torch.empty(torch.cuda.mem_get_info()[0] - G, dtype=torch.uint8, device="cuda")   # 1 GiB is left
del big                                                          # kept by the library, not the driver's
E = ctypes.c_void_p()
capi.check(L.diaq_evolve_create(keep.h, 48, capi.EVOLVE_C128, ctypes.byref(E)))          # 2.25 GiB of vectors
L.diaq_evolve_destroy(E)
other = capi.Matrix.create(N, N, list(range(100)))               # 2 x 0.78 GiB, of no size kept
"""


def test_kept_arrays_make_room(native):
    r = subprocess.run([sys.executable, "-c", GIVE_UP], cwd=ROOT, capture_output=True, text=True,
                       env=dict(os.environ, PYTHONPATH=ROOT), timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_products_reuse_arrays_on_streams_of_their_own(native):
    """Third powers of 16-qubit chains (value arrays of 0.1-0.3 GB, the same sizes in every thread) on
    four threads and streams at a time, each against its first result and the oracle's product."""
    import torch

    capi, _ = native
    L = capi.lib()
    N = 1 << 16
    x = np.random.default_rng(5).standard_normal(N) + 1j * np.random.default_rng(6).standard_normal(N)
    errors = []

    def work(seed):
        try:
            s = torch.cuda.Stream()
            _, off, re, im = ham.xxz(16, seed=seed)
            A = orc.OMatrix(N, N, off, re, im)
            want = orc.spmv(A, orc.spmv(A, orc.spmv(A, x)))
            for _ in range(4):
                H = capi.Matrix.create(N, N, off, re, im, stream=s.cuda_stream)
                out = ctypes.c_void_p()
                capi.check(L.diaq_pow(H.h, 3, 0, s.cuda_stream, ctypes.byref(out)))
                C = capi.Matrix(out)
                xs = torch.from_numpy(np.stack([x.real, x.imag])).cuda()
                y = torch.empty_like(xs)
                torch.cuda.current_stream().synchronize()
                capi.check(L.diaq_spmv_z(C.h, xs[0].data_ptr(), xs[1].data_ptr(), y[0].data_ptr(), y[1].data_ptr(),
                                         s.cuda_stream))
                del C, H   # while the product may still be running
                s.synchronize()
                got = y.cpu().numpy()
                # three products of sums of at most a few hundred float64 terms
                assert maxrel(got[0] + 1j * got[1], want) < 1e-12
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i + 1,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("n", [6, 14, 18])
def test_destroying_a_matrix_waits_for_its_readers(native, n):
    """The arrays of a caller's matrix are reused only because freeing the matrix waits for the work queued
    on every stream: a product behind a sleeping stream has run when destroy returns."""
    import torch

    capi, _ = native
    N, off, re, im = ham.tfim(n)
    keep = capi.Matrix.create(64, 64, [0])
    A = capi.Matrix.create(N, N, off, re, im)
    x, y = torch.ones(2, N, device="cuda", dtype=torch.float64), torch.empty(2, N, device="cuda", dtype=torch.float64)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()

    def product():
        capi.check(capi.lib().diaq_spmv_z(A.h, x[0].data_ptr(), x[1].data_ptr(), y[0].data_ptr(), y[1].data_ptr(),
                                          s.cuda_stream))

    product()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        torch.cuda._sleep(100_000_000)
    product()
    assert not s.query()
    del A
    assert s.query()
    del keep


BOUND = """
import torch, numpy as np
from diaq_gb300 import capi
L = capi.lib()
N, rows, cols, k = 1 << 20, 64, 1 << 26, 3
keep = capi.Matrix.create(64, 64, [0])
F = capi.Matrix.create(rows, cols, [0], np.ones(rows), np.ones(rows), precision=capi.C128F2)
x, y = torch.ones(2, k, cols, device="cuda", dtype=torch.float64), torch.empty(2, k, rows, device="cuda", dtype=torch.float64)
def product():   # 3 GiB of scratch
    capi.check(L.diaq_spmm(F.h, k, x[0].data_ptr(), x[1].data_ptr(), cols, y[0].data_ptr(), y[1].data_ptr(), rows, None))
    torch.cuda.synchronize()
torch.cuda.synchronize()
free0 = torch.cuda.mem_get_info()[0]
kept = lambda: free0 - torch.cuda.mem_get_info()[0]
slack = 96 << 20
product()
assert 3 << 30 <= kept() <= (4 << 30) + slack, kept()
for _ in range(2):
    big = capi.Matrix.create(N, N, list(range(180)))              # 2 x 1.4 GiB
    del big
    product()
    assert kept() <= (4 << 30) + slack, kept()
"""


def test_kept_memory_is_bounded_together(native):
    """What the driver's pool keeps of scratch and the arrays kept beside it stay below 4 GiB in all."""
    r = subprocess.run([sys.executable, "-c", BOUND], cwd=ROOT, capture_output=True, text=True,
                       env=dict(os.environ, PYTHONPATH=ROOT), timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
