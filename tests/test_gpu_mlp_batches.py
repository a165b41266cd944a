"""The proposer's fused batch pass at the edges of its row groups: 8 rows per block and round, two
blocks per SM, then further rounds; a train step against the gradient it is made of."""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


def _batch(B, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal((B, 16)).astype(np.float32), rng.integers(0, 21, B).astype(np.int32),
            rng.integers(1, 31, B).astype(np.int32))


@pytest.mark.parametrize("B", [2, 8, 9, 63, 2431, 2433, 5001])
def test_batch_pass_matches_oracle(native, B):
    import torch

    capi, _ = native
    M = capi.Mlp(seed=B)
    X, ys, ym = _batch(B, B)
    Xd, ysd, ymd = (torch.from_numpy(a).cuda() for a in (X, ys, ym))
    grad = torch.empty(omlp.N_PARAMS, dtype=torch.float32, device="cuda")
    loss = torch.full((B + 8,), 7.0, dtype=torch.float32, device="cuda")
    logits = torch.full((B + 1, 51), 7.0, dtype=torch.float32, device="cuda")
    s = torch.full((B + 8,), -7, dtype=torch.int32, device="cuda")
    m = torch.full((B + 8,), -7, dtype=torch.int32, device="cuda")
    M.gradient(Xd, ysd, ymd, grad, loss)
    M.forward(Xd, logits)
    M.propose(Xd, s, m)
    p0 = M.params()
    wl, wg = omlp.loss_and_grad(p0, X, ys, ym)
    want, _ = omlp.forward(p0, X)
    # float32 sums of at most 64 products per layer and a mean over B rows: ~200 roundings of 6e-8
    # against the largest magnitudes, times the cancellation of a gradient's terms
    assert np.abs(logits.cpu().numpy()[:B] - want).max() <= 2e-5 * np.abs(want).max()
    assert np.abs(loss.cpu().numpy()[:B] - wl).max() <= 2e-5 * max(1.0, np.abs(wl).max())
    assert np.abs(grad.cpu().numpy() - wg).max() <= 1e-4 * np.abs(wg).max()
    # nothing past the batch is written
    assert (loss[B:] == 7.0).all() and (logits[B] == 7.0).all() and (s[B:] == -7).all() and (m[B:] == -7).all()
    lg = logits.cpu().numpy()[:B]
    assert np.array_equal(s.cpu().numpy()[:B], lg[:, :21].argmax(1))
    assert np.array_equal(m.cpu().numpy()[:B], lg[:, 21:].argmax(1) + 1)
    # first Adam step: p -= lr * g / (|g| + eps) up to float32 rounding
    M.train_step(Xd, ysd, ymd, 1e-3, None)
    g = grad.cpu().numpy().astype(np.float64)
    step = p0.astype(np.float64) - 1e-3 * g / (np.abs(g) + 1e-8)
    assert np.abs(M.params() - step).max() <= 1e-6
