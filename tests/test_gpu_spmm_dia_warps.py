"""spmm_dia_device where its warps' choice of diagonals can go wrong: rows that end inside a warp, one
row spread over warps and many rows in one, diagonals that reach some or none of a warp's rows, more
diagonals than a ballot holds, infinities outside the matrix."""
import numpy as np
import pytest

from oracle import oracle as orc
from test_spmm_dia import _device_spmm, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [True, False])
@pytest.mark.parametrize("M,K,R,nd", [(1, 1, 1, 1), (33, 31, 1, 5), (257, 300, 3, 33), (100, 40, 33, 70), (513, 512, 7, 64),
                                      (64, 1000, 2, 31)])
def test_warps_take_the_diagonals_that_reach_them(native, cplx, M, K, R, nd):
    capi, _ = native
    rng = np.random.default_rng(M + R)
    off = np.concatenate([[0], rng.integers(-M - 20, K + 20, nd - 1)]).astype(np.int64)   # some outside, some twice
    V = rng.standard_normal((nd, M)) + (1j * rng.standard_normal((nd, M)) if cplx else 0.0)
    B = rng.standard_normal((K, R)) + (1j * rng.standard_normal((K, R)) if cplx else 0.0)
    c = np.arange(M)[None, :] + off[:, None]
    V[(c < 0) | (c >= K)] = np.inf   # never looked at
    # sums of at most 70 float64 products of order 1
    assert _rel(_device_spmm(capi, off, V, K, B), orc.spmm_dia(off, V, K, B)) < 1e-13
