"""Launch shapes that plans choose by themselves: what they are remembered under."""
import json

import numpy as np
import pytest

from diaq_gb300 import hamiltonians as ham
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _run(capi, H, P, mode, steps=1, m=4):
    import torch

    k, N = P.shape
    E = capi.Evolve(H, k, mode)
    pr, pi = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (P.real, P.imag))
    E.run(pr, pi, N, 0.05, steps, 0, m)
    torch.cuda.synchronize()
    return (pr + 1j * pi).cpu().numpy()


@pytest.mark.parametrize("mode", ["mixed", "horner"])
def test_real_and_complex_matrices_are_tuned_apart(native, mode, tmp_path, monkeypatch):
    """A chain and a complex matrix of the same size and offsets run different interleaved kernels: each
    is timed for itself, in either order."""
    capi, _ = native
    md = capi.EVOLVE_MIXED if mode == "mixed" else capi.EVOLVE_HORNER
    N, off, re, im = ham.xxz(9)
    real = capi.Matrix.create(N, N, off, re, im)
    cplx = capi.Matrix.create(N, N, off, re, 0.5 * re)
    P = ham.random_state(N, 3, k=4)
    seen = []
    for order in ((real, cplx), (cplx, real)):
        f = tmp_path / f"tune{len(seen)}.json"
        monkeypatch.setenv("DIAQ_AUTOTUNE_CACHE", str(f))
        _run(capi, order[0], P, md)
        first = set(json.loads(f.read_text()))
        _run(capi, order[1], P, md)
        both = set(json.loads(f.read_text()))
        assert len(first) == 1 and len(both) == 2
        _run(capi, order[0], P, md)
        assert set(json.loads(f.read_text())) == both
        seen.append(both)
    assert seen[0] == seen[1]


SHAPES = [(8, 1, 0), (8, 2, 0), (4, 2, 0), (2, 2, 0), (1, 2, 0), (2, 1, 0), (1, 1, 0)]


@pytest.mark.parametrize("n,k", [(6, 3), (10, 8), (12, 2), (12, 4), (13, 2), (12, 5), (13, 3), (14, 2), (12, 9)])
def test_complex128_results_do_not_depend_on_what_was_timed(native, n, k, tmp_path, monkeypatch):
    """Whatever shape another process's timing left in the file, the evolved states are the same bits: on
    both sides of the line up to which four warps share a row's diagonals (8,192 rows x state pairs)."""
    capi, _ = native
    N, off, re, im = ham.xxz(n)
    H = capi.Matrix.create(N, N, off, re, 0.3 * re)
    P = ham.random_state(N, n, k=k)
    f = tmp_path / "tune.json"
    monkeypatch.setenv("DIAQ_AUTOTUNE_CACHE", str(f))
    want = _run(capi, H, P, capi.EVOLVE_C128)
    keys = list(json.loads(f.read_text())) if f.exists() else []
    for shape in SHAPES:
        if keys:
            f.write_text(json.dumps({key: list(shape) for key in keys}))
        assert np.array_equal(_run(capi, H, P, capi.EVOLVE_C128), want), shape


@pytest.mark.parametrize("n", [6, 12, 15])
def test_one_complex128_state_is_not_tuned(native, n, tmp_path, monkeypatch):
    """A plan of one state has one shape: its first run copies no states (it works with every further
    allocation refused) and writes no file."""
    capi, _ = native
    import torch

    f = tmp_path / "tune.json"
    monkeypatch.setenv("DIAQ_AUTOTUNE_CACHE", str(f))
    N, off, re, im = ham.tfim(n)
    H = capi.Matrix.create(N, N, off, re, im)
    E = capi.Evolve(H, 1, capi.EVOLVE_C128)
    x = ham.random_state(N, 2)
    pr, pi = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (x.real, x.imag))
    monkeypatch.setenv("DIAQ_DEVICE_ALLOC_LIMIT", "1")
    E.run(pr, pi, N, 0.05, 2, 0, 8)
    torch.cuda.synchronize()
    assert not f.exists()
    want = orc.ham_sim(orc.OMatrix(N, N, off, re, im), x, 0.1, 2, 8)
    assert np.linalg.norm((pr + 1j * pi).cpu().numpy() - want) / np.linalg.norm(want) < 1e-12
