"""Products on both sides of the sizes at which one kernel takes over from another: several states
against one at a time, and recorded into a graph (where no zero-tile mask is taken) against run directly."""
import numpy as np
import pytest

from test_gpu_plane_mask import planes

pytestmark = pytest.mark.gpu

# rows x groups of states at which kernels change: c128 8,192 and 65,536 (one or two states a group), c64
# 32,768 and 262,144, float pairs 360,000 (no imaginary part; again from 622,592 to 747,110) and 900,000 rows x
# states
CASES = [("c128", 8192, 1), ("c128", 8193, 1), ("c128", 4096, 4), ("c128", 4097, 3), ("c128", 32768, 4), ("c128", 32769, 4), ("c128", 2730, 3), ("c128", 2731, 3), ("c128", 13107, 5), ("c128", 13108, 5),
         ("c128", 21845, 5), ("c128", 21846, 5), ("c128", 32769, 3),
         ("c64", 32768, 2), ("c64", 32769, 2), ("c64", 16384, 3), ("c64", 16385, 4), ("c64", 131072, 3), ("c64", 131073, 3),
         ("c128f2", 120000, 3), ("c128f2", 120001, 3), ("c128f2", 218000, 3), ("c128f2", 250000, 3), ("c128f2", 300000, 3), ("c128f2", 300001, 3)]
# sums of 9 complex products: 18 roundings of 2^-53 (2^-24, 2^-46) relative to sums of |a||x|
TOL = {"c128": 1e-14, "c64": 5e-6, "c128f2": 1e-12}


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("prec,rows,k", CASES)
def test_lines(native, prec, rows, k, real):
    import torch

    capi, _ = native
    L = capi.lib()
    off, re, im = planes(rows, rows, [0, 1, -1, 36, -37, 700, -701, 1501, 64], 3)
    if real:
        im[:] = 0
    code = {"c128": capi.C128, "c64": capi.C64, "c128f2": capi.C128F2}[prec]
    dt = torch.float32 if prec == "c64" else torch.float64
    A = capi.Matrix.create(rows, rows, off, re, im, precision=code)
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(2, k, rows, generator=g, device="cuda", dtype=torch.float64).to(dt)
    y, one, rec = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(x)

    def product(q, n, out, s):
        capi.check(L.diaq_spmm(A.h, n, x[0, q].data_ptr(), x[1, q].data_ptr(), rows, out[0, q].data_ptr(),
                               out[1, q].data_ptr(), rows, s))

    torch.cuda.synchronize()
    product(0, k, y, None)
    for q in range(k):
        product(q, 1, one, None)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        product(0, k, rec, torch.cuda.current_stream().cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    scale = float(y.abs().max())
    assert float((one - y).abs().max()) <= TOL[prec] * scale
    assert float((rec - y).abs().max()) <= TOL[prec] * scale
    assert scale > 0.5
