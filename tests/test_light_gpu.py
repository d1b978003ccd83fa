"""Requests from a short list in one launch: chains of k2u, k2k and k2c over
functional, list and hashed directions against the oracle, at the edges of the
launch's table (2048 rows, 1024 threads a round), where a step outgrows it and
the steps' own kernels go on, where every row is lost, and past the row limit."""
import numpy as np
import pytest

import oracle
import wukonggpu_gb300 as W

pytestmark = pytest.mark.gpu

V = W.VID_BASE
FAN = [1, 1023, 1024, 1025, 2047, 2048, 2049, 7]      # object lists of vertices V .. V + 7
FUNC, LIST, SPARSE = 3, 4, 5


@pytest.fixture(scope="module")
def graph(lib_built):
    rng = np.random.default_rng(3)
    n = 2200
    obj = V + 100 + np.arange(n)
    t = [(V + i, 2, x) for i, k in enumerate(FAN) for x in obj[rng.permutation(n)[:k]]]
    t += [(x, FUNC, V + 5000 + int(rng.integers(0, 30))) for x in obj if rng.random() < 0.9]
    t += [(x, LIST, V + 6000 + int(y)) for x in obj[::3] for y in rng.permutation(40)[:rng.integers(1, 4)]]
    t += [(x, SPARSE, V + 7000 + int(y)) for x in obj[::211] for y in rng.permutation(40)[:2]]
    s, p, o = (np.array(a, np.int32) for a in zip(*t))
    rc = W.RCache(device=0)
    rc.build_store(s, p, o, SPARSE)
    yield rc, oracle.Oracle(s, p, o, SPARSE)
    rc.close()


def _run(graph, start, steps):
    rc, orc = graph
    cmd = [start, 2, W.OUT, -1] + [x for st in steps for x in st]
    before = rc.kernel_launches()
    req, rows = rc.execute(cmd)
    launches = rc.kernel_launches() - before
    table, want = None, []
    for i in range(0, len(cmd), 4):
        table, _ = orc.step(table, i == 0, cmd[i], cmd[i + 1], cmd[i + 2], cmd[i + 3])
        want.append(len(table))
    assert list(rows) == want
    got = np.asarray(req.result_table)
    assert got.size == table.size and np.array_equal(got.reshape(table.shape), table)
    return launches, want


@pytest.mark.parametrize("k", range(len(FAN)))
@pytest.mark.parametrize("steps", [
    [(-1, FUNC, W.OUT, -2)],
    [(-1, LIST, W.OUT, -2), (-1, FUNC, W.OUT, -3), (-1, LIST, W.OUT, -2)],
    [(-1, SPARSE, W.OUT, -2), (-2, SPARSE, W.IN, -3), (-3, FUNC, W.OUT, V + 5004)],
    [(-1, FUNC, W.OUT, -2), (-2, FUNC, W.IN, -3), (-3, LIST, W.OUT, -4)],     # a large fan-out: outgrows the launch
    [(-1, LIST, W.OUT, V + 6003), (-1, FUNC, W.OUT, V + 4999), (-1, LIST, W.OUT, -2)],   # every row lost
], ids=["func", "lists", "hashed", "outgrows", "empty"])
def test_chain(graph, k, steps):
    launches, rows = _run(graph, V + k, steps)
    if max(rows) <= 2048:
        assert launches == 1


def test_row_limit(graph):
    rc, _ = graph
    rc.set_row_limit(1000)
    try:
        with pytest.raises(W.WkError):
            rc.execute([V + 4, 2, W.OUT, -1, -1, FUNC, W.OUT, -2])
    finally:
        rc.set_row_limit(0)
    assert _run(graph, V + 4, [(-1, FUNC, W.OUT, -2)])[0] == 1
