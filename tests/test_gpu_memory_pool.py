"""The library's memory pool: freed memory is kept only up to its bound and given back with the last
matrix, and threads on streams of their own can make and free matrices at the same time."""
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

GIVE_BACK = """
import ctypes, torch
from diaq_gb300 import capi, hamiltonians as ham
torch.cuda.init()
N, off, re, im = ham.xxz(10)
warm = capi.Matrix.create(N, N, off, re, im)
torch.cuda.synchronize()
free0 = torch.cuda.mem_get_info()[0]
big = capi.Matrix.create(1 << 20, 1 << 20, list(range(400)))       # 6.7 GB of zeros
assert free0 - torch.cuda.mem_get_info()[0] > 6 << 30
del big
torch.cuda.synchronize()
assert free0 - torch.cuda.mem_get_info()[0] <= (4 << 30) + (64 << 20)   # the pool's bound
small = capi.Matrix.create(1 << 20, 1 << 20, list(range(60)))      # 1 GB
del small, warm
assert free0 - torch.cuda.mem_get_info()[0] <= 64 << 20            # nothing of the library's left
"""


def test_freed_memory_is_bounded_and_given_back(native):
    r = subprocess.run([sys.executable, "-c", GIVE_BACK], cwd=ROOT, capture_output=True, text=True,
                       env=dict(os.environ, PYTHONPATH=ROOT), timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_threads_on_their_own_streams(native):
    import torch

    capi, _ = native
    L = capi.lib()
    errors = []

    def work(n, seed):
        try:
            s = torch.cuda.Stream()
            N, off, re, im = ham.xxz(n, seed=seed)
            want = orc.product(orc.OMatrix(N, N, off, re, im), orc.OMatrix(N, N, off, re, im), prune_result=False)
            for _ in range(6):
                H = capi.Matrix.create(N, N, off, re, im, stream=s.cuda_stream)
                out = ctypes.c_void_p()
                capi.check(L.diaq_spgemm(H.h, H.h, 0, s.cuda_stream, ctypes.byref(out)))
                C = capi.Matrix(out)
                o, cr, ci = C.download()
                assert np.array_equal(o, want.off)
                assert maxrel(cr + 1j * ci, want.re + 1j * want.im) < 1e-13
                out = ctypes.c_void_p()
                capi.check(L.diaq_pow(H.h, 3, 1, s.cuda_stream, ctypes.byref(out)))
                capi.Matrix(out)
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(8 + i, i + 1)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
