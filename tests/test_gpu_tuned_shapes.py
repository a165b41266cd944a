"""Launch shapes that plans choose by themselves: what they are remembered under."""
import json

import numpy as np
import pytest

from diaq_gb300 import hamiltonians as ham

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
