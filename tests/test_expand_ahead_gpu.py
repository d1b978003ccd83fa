"""The expansion that a k2u op sends in behind its count when the output buffer
may already be large enough: steps that fit it, outgrow it, have no rows, or
pass the context's row limit, each against the oracle."""
import numpy as np
import pytest

import oracle
import wukonggpu_gb300 as W

pytestmark = pytest.mark.gpu

DEGREES = [700, 1, 33, 7, 64]


@pytest.fixture(scope="module")
def graph(lib_built):
    subj = W.VID_BASE + np.arange(len(DEGREES), dtype=np.int32)
    s = np.repeat(subj, DEGREES).astype(np.int32)
    o = np.concatenate([W.VID_BASE + 100 + 3 * np.arange(d) for d in DEGREES]).astype(np.int32)
    return s, np.full(len(s), 2, np.int32), o


def _table(seed, R, C, top):
    rng = np.random.default_rng(seed)
    h = rng.integers(W.VID_BASE, W.VID_BASE + 64, size=(R, C)).astype(np.int32)
    h[:, 0] = W.VID_BASE + rng.integers(top, 8, size=R)   # 5..7 have no list
    return h


def _step(rc, orc, h):
    req = W.Request([])
    rc.upload_history(req, h)
    rc.known_to_unknown(req, -1, W.OUT, 2)
    got = rc.download(req)
    exp, _ = orc.step(h, False, -1, 2, W.OUT, -h.shape[1] - 1)
    assert got.shape == exp.shape and np.array_equal(got, exp)
    return req


@pytest.mark.parametrize("C", [1, 3, 9])
def test_buffer_grown_by_an_earlier_step(graph, C):
    s, p, o = graph
    orc = oracle.Oracle(s, p, o, 2)
    rc = W.RCache(device=0)
    rc.build_store(s, p, o, 2)
    # (rows, lowest vertex): the first steps grow the buffer, later ones fit it,
    # one just outgrows it again, one has no output at all
    for i, (R, top) in enumerate([(2000, 0), (2000, 0), (5, 1), (1025, 3), (3000, 5), (2600, 0), (30_000, 3), (1, 0)]):
        _step(rc, orc, _table(10 * C + i, R, C, top))
    rc.close()


def test_row_limit_leaves_the_other_table(graph):
    s, p, o = graph
    orc = oracle.Oracle(s, p, o, 2)
    rc = W.RCache(device=0)
    rc.build_store(s, p, o, 2)
    _step(rc, orc, _table(1, 3000, 2, 0))
    h = _table(2, 3000, 2, 0)
    rows = len(orc.step(h, False, -1, 2, W.OUT, -3)[0])
    first = W.Request([])
    rc.upload_history(first, h)
    rc.known_to_unknown(first, -1, W.OUT, 2)
    want = rc.download(first)
    rc.set_row_limit(rows * 32)
    with pytest.raises(W.WkError):       # one step further: past the limit, input untouched
        rc.known_to_unknown(first, -1, W.OUT, 2)
    assert np.array_equal(rc.download(first), want)
    rc.close()
