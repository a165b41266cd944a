"""Destroying a matrix while the driver refuses to free (a stream is being captured in global mode):
kernels that still read the matrix keep their data."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import ctypes, numpy as np, torch
from diaq_gb300 import capi, hamiltonians as ham
L = capi.lib()
N, off, re, im = ham.xxz(14)
keep = capi.Matrix.create(64, 64, [0])
A = capi.Matrix.create(N, N, off, re, im)
x = torch.from_numpy(np.ascontiguousarray(np.stack([ham.random_state(N, 1).real, ham.random_state(N, 1).imag]))).cuda()
want, got = torch.zeros_like(x), torch.zeros_like(x)
s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
torch.cuda.synchronize()
def product(y, s):
    capi.check(L.diaq_spmv_z(A.h, x[0].data_ptr(), x[1].data_ptr(), y[0].data_ptr(), y[1].data_ptr(), s.cuda_stream))
product(want, s1)                      # (builds the zero-tile mask)
torch.cuda.synchronize()
with torch.cuda.stream(s1):
    torch.cuda._sleep(400_000_000)     # some 0.2 s
product(got, s1)
g = torch.cuda.CUDAGraph()
refused = False
with torch.cuda.stream(s2):
    g.capture_begin(capture_error_mode="global")
    del A                              # the free is refused, which also ends the capture
    try:
        g.capture_end()
    except RuntimeError:
        refused = True
pending = not s1.query()
ones = np.ones_like(re)
B = [capi.Matrix.create(N, N, off, 7 * ones, ones, stream=s2.cuda_stream) for _ in range(3)]
torch.cuda.synchronize()
assert torch.equal(got, want)
print("refused", refused, "pending", pending)
"""


def test_planes_of_a_refused_free_are_not_reused(native):
    """The product is queued behind a sleeping stream when its matrix goes and others of the same size
    are made on another stream."""
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True,
                       env=dict(os.environ, PYTHONPATH=ROOT), timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert "refused True pending True" in r.stdout, r.stdout
