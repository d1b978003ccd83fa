"""Batches of more queries than their tables hold values, against the oracle."""
import numpy as np
import pytest

import oracle
import wukonggpu_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def store(lib_built):
    s = (W.VID_BASE + np.arange(64)).astype(np.int32)
    p = np.full(64, 2, np.int32)
    rc = W.RCache(device=0)
    rc.build_store(s, p, s + 100, 2)
    yield rc, oracle.Oracle(s, p, s + 100, 2)
    rc.close()


# 64 entities have the one neighbour, the others none
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("nq", [33, 1000, 4096])
def test_fewer_values_than_queries(store, nq, fused):
    rc, orc = store
    b = W.Batch(rc, max_queries=nq, max_steps=2, capacity_ints=24)
    b.set_fused(fused)
    full = [[W.VID_BASE + i % 64, 2, W.OUT, -1] for i in range(nq)]
    with pytest.raises(W.WkError) as e:
        b.run(full)
    assert e.value.status == W.WK_EOVERFLOW
    few = [[W.VID_BASE + (i // (nq // 16) if i % (nq // 16) == 0 else 100_000 + i), 2, W.OUT, -1] for i in range(nq)]
    got = b.download(b.run(few))
    for q, t in zip(few, got):
        exp, _ = orc.execute(q)
        assert np.array_equal(t.reshape(exp.shape), exp)
    b.close()
