"""Batches around the step kernels' tile rule (a tile is total rows / warps of
the grid, a power of two below 32 rows, then a multiple of 32): one query, few
and many queries whose steps hold empty queries in runs of more than 32, lists
that are written by a thread and by a warp, the widest and narrowest grids,
and queries beyond one pass of the layout scan -- each query's rows equal to
the oracle's, in the three-kernel and the one-kernel form."""
import numpy as np
import pytest

import oracle
import wukonggpu_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph(lib_built):
    """Subjects with 0 .. 300 neighbours: many empty, some long lists."""
    rng = np.random.default_rng(3)
    n = 600
    deg = np.where(rng.random(n) < 0.5, 0, rng.integers(1, 12, size=n))
    deg[::37] = 300
    s = np.repeat(W.VID_BASE + np.arange(n), deg).astype(np.int32)
    o = np.concatenate([W.VID_BASE + rng.choice(n, size=d, replace=False) for d in deg if d]).astype(np.int32)
    p = np.full(len(s), 2, np.int32)
    rc = W.RCache(device=0)
    rc.build_store(s, p, o, 2)
    yield rc, oracle.Oracle(s, p, o, 2)
    rc.close()


def _queries(nq, seed):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(nq):
        # runs of starts without a neighbour, then a few with long lists
        v = W.VID_BASE + (int(rng.integers(0, 600)) if (i // 50) % 3 else 600 + i % 7)
        if i % 97 == 5:
            v = W.VID_BASE + 37 * int(rng.integers(0, 17))
        q = [v, 2, W.OUT, -1]
        if i % 4 == 1:
            q += [-1, 2, W.OUT, -2]
        if i % 4 == 2:
            q += [-1, 2, W.OUT, W.VID_BASE + 37]
        if i % 4 == 3:
            q += [-1, 2, W.IN, -2, -2, 2, W.OUT, -1]
        out.append(q)
    return out


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("nq,tuning", [(1, (4, 128, 64)), (33, (1, 32, 1)), (700, (16, 256, 256)), (1500, (1, 32, 16)),
                                       (4096, (4, 128, 64))])
def test_tiles_and_layouts(graph, nq, tuning, fused):
    rc, orc = graph
    qs = _queries(nq, nq)
    b = W.Batch(rc, max_queries=nq, max_steps=3, capacity_ints=1 << 24)
    b.set_tuning(*tuning)
    b.set_fused(fused)
    b.run(qs)
    tables = b.download(nq)
    memo = {}
    for q, t in zip(qs, tables):
        key = tuple(q)
        if key not in memo:
            memo[key] = orc.execute(q)[0]
        exp = memo[key]
        assert np.array_equal(t.reshape(exp.shape) if t.size == exp.size else t, exp), q
    b.close()
