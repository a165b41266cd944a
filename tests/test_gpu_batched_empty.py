"""Batches small enough for chained launches with instances whose matrix holds no diagonal: their blocks
have no metadata to stage and still wait for the phase before them."""
import numpy as np
import pytest

from diaq_gb300 import hamiltonians as ham
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("horner", [False, True])
@pytest.mark.parametrize("prec", ["c64", "c128"])
def test_instances_without_diagonals(native, prec, horner):
    """A zero Hamiltonian leaves its states as they are, to the last bit, between instances that move
    (1-3 states: the planar kernel in both precisions)."""
    import torch

    capi, _ = native
    p = capi.C64 if prec == "c64" else capi.C128
    mats, oms, P0 = [], [], []
    for i, (n, k) in enumerate([(8, 1), (9, 3), (8, 2), (10, 1), (7, 3)]):
        if i % 2:
            N = 1 << n
            mats.append(capi.Matrix.create(N, N, [], precision=p))
            oms.append(None)
        else:
            N, off, re, im = ham.tfim(n)
            mats.append(capi.Matrix.create(N, N, off, re, im, precision=p))
            oms.append(orc.OMatrix(N, N, off, re, im))
        P0.append(ham.random_state(N, i, k=k).reshape(k, N))
    prs = [torch.from_numpy(np.ascontiguousarray(P.real)).cuda() for P in P0]
    pis = [torch.from_numpy(np.ascontiguousarray(P.imag)).cuda() for P in P0]
    B = capi.Batch(mats, prs, pis)
    B.set_horner(horner)
    B.set_config(2, 1)
    s, m = [0, 1, 0, 0, 2], [7, 3, 4, 9, 5]
    for _ in range(3):
        B.run(0.02, s, m, 4)
    torch.cuda.synchronize()
    for i, A in enumerate(oms):
        got = (prs[i] + 1j * pis[i]).cpu().numpy()
        for q, x in enumerate(P0[i]):
            if A is None:
                assert np.array_equal(got[q], x), (i, q)
            else:
                want = orc.ham_sim(A, x, 12 * 0.02, 12, m[i], substeps=1 << s[i])
                assert np.linalg.norm(got[q] - want) / np.linalg.norm(want) < (1e-6 if prec == "c64" else 1e-12), (i, q)
