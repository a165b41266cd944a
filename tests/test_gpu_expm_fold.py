"""The exponential's Taylor terms folded into the series: terms that bring new diagonals (union of the
offsets) and terms that do not (in place), unsorted input offsets, diagonals that cancel, both
precisions, pruned and not; powers that start from the caller's matrix."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _matrix(capi, n, offs, seed, prec, kind):
    rng = np.random.default_rng(seed)
    L = [n - abs(d) for d in offs]
    re, im = rng.standard_normal(sum(L)) * 0.2, rng.standard_normal(sum(L)) * 0.2
    if kind == "real":
        im[:] = 0
    if kind == "nilpotent":   # one entry per diagonal: products vanish and are pruned
        keep = np.zeros(sum(L), dtype=bool)
        keep[np.cumsum(L) - 1] = True
        re[~keep] = im[~keep] = 0
    off = np.array(offs, dtype=np.int32)
    return capi.Matrix.create(n, n, off, re, im, precision=prec), orc.OMatrix(n, n, off, re, im).to_dense()


@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 2e-5)])
@pytest.mark.parametrize("n,offs", [(40, [3, 0, -2]), (33, [32, -1]), (7, list(range(-6, 7))), (300, [0, 100, -100])])
@pytest.mark.parametrize("kind", ["complex", "real", "nilpotent"])
@pytest.mark.parametrize("prune", [0, 1])
def test_exponential_and_power(native, prec, tol, n, offs, kind, prune):
    import torch

    capi, _ = native
    L = capi.lib()
    A, dense = _matrix(capi, n, offs, n, prec, kind)
    out = ctypes.c_void_p()
    # a float32 term's norm levels off near 1e-8: the tolerance is the precision's own
    capi.check(L.diaq_expm_negative(A.h, 0.7, 60, 1.0, 1e-12 if prec == 0 else 1e-7, prune, None, ctypes.byref(out), None, None))
    want = torch.linalg.matrix_exp(torch.from_numpy(-0.7j * dense)).numpy()
    got = capi.Matrix(out).to_dense()
    assert np.abs(got - want).max() / np.abs(want).max() < tol
    for p in (2, 3, 4, 5):
        out = ctypes.c_void_p()
        capi.check(L.diaq_pow(A.h, p, prune, None, ctypes.byref(out)))
        want = np.linalg.matrix_power(dense, p)
        got = capi.Matrix(out).to_dense()
        assert np.abs(got - want).max() <= tol * max(np.abs(want).max(), 1e-30)
    # the caller's matrix is what it was
    assert np.abs(A.to_dense() - dense).max() <= (0 if prec == 0 else 1e-7)
