"""Loss and gradients of a training batch against the FP64 oracle, at the batch
sizes where the row tiles (64), the parts of the gradient sums (whole steps of 16
rows, 32 rows at least, 128 parts at most) and the output layer's groups of 128
rows end, and as one model's batches grow and shrink."""
import numpy as np
import pytest

import cabi
from oracle import mlp_oracle
from test_gpu_learned import _unpack

pytestmark = pytest.mark.gpu

# A gradient is a sum over rows of products with up to 64 + 128 + 128 + 128 rounded
# terms behind each: random roundings give sqrt(450) 2^-24 = 1.3e-6 of a block's
# norm, 16 times that is allowed.
TOL = 2e-5


def _batch(n, seed):
    rng = np.random.default_rng(seed)
    feats = rng.normal(1.0, 2.0, (n, 64)).astype(np.float32)
    rows = np.zeros((n, 24), np.float32)
    rows[:, :21] = 0.1 * rng.standard_normal((n, 21))
    rows[:, 21:23] = rng.uniform(0.01, 0.05, (n, 2))
    return feats, rows


@pytest.mark.parametrize("sizes", [(1, 33), (130, 31, 64), (4095, 4130), (16 * 128 * 9 + 5, 700)])
def test_training_batch_matches_oracle(gpu, sizes):
    model = cabi.Mlp(seed=5)
    rng = np.random.default_rng(1)
    mean = rng.normal(1.0, 0.2, 64).astype(np.float32)
    inv = rng.uniform(0.3, 0.7, 64).astype(np.float32)
    inv[7] = 0.0
    model.set_normalization(mean, inv)
    p = model.params
    p[-516:] += rng.normal(0, 0.1, 516).astype(np.float32)
    model.params = p
    ref = _unpack(p.astype(np.float64))
    for k, n in enumerate(sizes):
        feats, rows = _batch(n, 10 + k)
        X = (feats.astype(np.float64) - mean) * inv
        loss, g = model.loss_grad(feats, rows, lam=0.7)
        want, gr = mlp_oracle.loss_and_grads(ref, X, rows.astype(np.float64), lam=0.7)
        assert abs(loss - want) < TOL * abs(want)
        at = 0
        for block in gr:
            b = np.asarray(block).ravel()
            err = np.linalg.norm(g[at:at + b.size] - b)
            assert err < TOL * np.linalg.norm(b)
            at += b.size
        assert at == g.size
