"""The estimator's gradients where the step's tiles meet the batch: 16 rows a
CTA of the output layer, 128 rows a tile, 64 rows of padding, and batches large
enough for each tile width; each batch after a larger one, whose rows must not
be seen."""
import numpy as np
import pytest

import wukonggpu_gb300 as W
from oracle import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 15, 16, 17, 63, 65, 127, 128, 129, 1000, 1024, 5000, 10_000, 20_000])
def test_gradients_after_a_larger_batch(gpu_small, M):
    n_ids = 26
    est = W.Estimator(gpu_small, n_ids, max_batch=M + 200, seed=5)
    rng = np.random.default_rng(M)
    params = est.get_params()
    params += rng.normal(0, 0.01, size=params.shape).astype(np.float32)
    est.set_params(params)
    for m in (M + 150, M):
        feats = rng.normal(0, 1, size=(m, 48)).astype(np.float32)
        pids = rng.integers(0, n_ids + 1, size=m).astype(np.int32)
        tgt = rng.normal(2, 1, size=m).astype(np.float32)
        g_gpu, loss_gpu = est.gradients(feats, pids, tgt)
    loss_ref, g_ref = mlp_ref.forward_backward(params, n_ids, feats, pids, tgt)
    # the same BF16 roundings as the oracle with FP32 sums in another order: a
    # rounding that falls the other way is 2^-9 of one product
    assert abs(loss_gpu - loss_ref) <= 1e-2 * max(1.0, abs(loss_ref))
    ends = np.cumsum([256 * 80, 65536, 65536, 256, 832, (n_ids + 1) * 32])
    assert ends[-1] == len(g_ref)
    for a, b in zip(np.r_[0, ends[:-1]], ends):
        x, y = g_gpu[a:b].astype(np.float64), g_ref[a:b].astype(np.float64)
        assert np.linalg.norm(x - y) <= 0.005 * np.linalg.norm(y) + 1e-6, (a, b)


@pytest.mark.parametrize("n", [1023, 1024, 1025, 16383, 16384, 16385])
def test_predictions_at_the_copy_limits(gpu_small, n):
    """features through the pinned block up to 1024 samples, ids and outputs up to 16,384: the same bits in pieces"""
    est = W.Estimator(gpu_small, 26, max_batch=64, seed=5)
    rng = np.random.default_rng(n)
    feats = rng.normal(0, 1, size=(n, 48)).astype(np.float32)
    pids = rng.integers(-1, 28, size=n).astype(np.int32)
    whole = est.predict(feats, pids)
    cut = [0, 100, n // 2, n - 7, n]
    parts = [est.predict(feats[a:b], pids[a:b]) for a, b in zip(cut, cut[1:])]
    assert np.array_equal(whole, np.concatenate(parts))
