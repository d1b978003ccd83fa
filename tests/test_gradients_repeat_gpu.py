"""The estimator's weight gradients are products with a fixed order of addition:
the same batch gives the same bits.  (The hidden layers' biases and the embedding
are added up by atomics and are not asked for bits.)"""
import numpy as np
import pytest

import wukonggpu_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 65, 1024, 5000])
def test_same_bits(gpu_small, M):
    est = W.Estimator(gpu_small, 26, max_batch=M, seed=5)
    rng = np.random.default_rng(M)
    feats = rng.normal(0, 1, size=(M, 48)).astype(np.float32)
    pids = rng.integers(0, 27, size=M).astype(np.int32)
    tgt = rng.normal(2, 1, size=M).astype(np.float32)
    weights = 256 * 80 + 2 * 65536 + 256
    first, loss = est.gradients(feats, pids, tgt)
    assert np.any(first[weights - 256:weights] != 0.0)
    for _ in range(8):
        again, l2 = est.gradients(feats, pids, tgt)
        assert l2 == loss and np.array_equal(again[:weights], first[:weights])
