"""The estimator's one-kernel prediction: against the numpy oracle's layers at
the sizes around a tile (128 samples), the small-call limit (512), one round of
a CTA's two tiles (2 x 128 per SM) and several chunks; and the same samples
in pieces give the same bits."""
import numpy as np
import pytest

import wukonggpu_gb300 as W
from oracle import mlp_ref

pytestmark = pytest.mark.gpu

N_IDS = 26


def _estimator(gpu_small, seed):
    est = W.Estimator(gpu_small, N_IDS, max_batch=256, seed=seed)
    rng = np.random.default_rng(seed)
    p = est.get_params() + rng.normal(0, 0.02, est.num_params()).astype(np.float32)   # non-zero biases
    est.set_params(p)
    return est, p


def _samples(n, seed):
    rng = np.random.default_rng(seed)
    f = rng.normal(0, 1, size=(n, 48)).astype(np.float32)
    f[:, 7:13] = rng.uniform(0, 16, size=(n, 6))
    return f, rng.integers(-2, N_IDS + 3, size=n).astype(np.int32)   # ids outside 0..N_IDS are clamped


def _reference(p, f, pids):
    """Predictions and, per sample, a bound on what bf16 roundings that fall the
    other way can change: an fp32 sum in another order moves an activation by
    at most one bf16 step (2^-8 of it); each of the three layers contributes at
    most that share of the sum of the output's absolute terms."""
    Ws, b, emb = mlp_ref.unpack(p, N_IDS)
    h = mlp_ref.bf16(np.concatenate([f, emb[np.clip(pids, 0, N_IDS)]], axis=1))
    for layer in range(3):
        h = mlp_ref.bf16(mlp_ref.gelu((h @ mlp_ref.bf16(Ws[layer]).T + b[layer]).astype(np.float32)))
    w4 = mlp_ref.bf16(Ws[3])
    return (h @ w4.T)[:, 0] + b[3][0], 3 * 2.0 ** -8 * (np.abs(h) @ np.abs(w4).T)[:, 0]


@pytest.mark.parametrize("n", [1, 127, 128, 129, 511, 512, 513, 4097, 20_001, 40_003])
def test_predictions_match_the_oracle(gpu_small, n):
    est, p = _estimator(gpu_small, 3)
    f, pids = _samples(n, n)
    got = est.predict(f, pids)
    ref, bound = _reference(p, f, pids)
    assert np.all(np.abs(got - ref) <= bound), float(np.max(np.abs(got - ref) / bound))
    est.close()


def test_pieces_give_the_same_bits(gpu_small):
    est, _ = _estimator(gpu_small, 4)
    f, pids = _samples(130_000, 9)      # four chunks on 152 SMs
    whole = est.predict(f, pids)
    assert np.array_equal(whole, est.predict(f, pids))
    for a, b in ((0, 1), (100, 612), (5_000, 5_513), (77_777, 130_000)):
        assert np.array_equal(whole[a:b], est.predict(f[a:b], pids[a:b]))
    assert est.predict(f[:0], pids[:0]).size == 0
    est.close()
