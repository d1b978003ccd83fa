"""The output of a k2u op over a dense functional direction: sized by its rows
and not by the input's, refused past the row limit before anything is written,
and the same rows, against the oracle's step, whether the buffer is there before
they are counted (one launch) or not (two)."""
import numpy as np
import pytest

import oracle
import wukonggpu_gb300 as W

pytestmark = pytest.mark.gpu

N = 3000   # subjects VID_BASE .. VID_BASE + N - 1, one in eight without a neighbour


@pytest.fixture(scope="module")
def graph(lib_built):
    rng = np.random.default_rng(11)
    s = W.VID_BASE + np.flatnonzero(np.arange(N) % 8 != 3).astype(np.int32)
    o = (W.VID_BASE + rng.integers(0, 40, size=len(s))).astype(np.int32)
    return s, np.full(len(s), 2, np.int32), o


def _context(graph, capacity):
    rc = W.RCache(device=0, history_capacity=capacity)
    rc.build_store(*graph, 2)
    lay = rc.seg_layout(2)
    assert lay["dense"][W.OUT] and lay["functional"][W.OUT]
    return rc


def _table(R, C, seed, share):
    """About `share` of the rows start at an id of the direction."""
    rng = np.random.default_rng(seed)
    h = (W.VID_BASE + rng.integers(0, N, size=(R, C))).astype(np.int32)
    h[rng.random(R) >= share, 0] += 10 * N
    return h


def _step(rc, orc, h):
    req = W.Request([])
    rc.upload_history(req, h)
    rc.known_to_unknown(req, -1, W.OUT, 2)
    exp, _ = orc.step(h, False, -1, 2, W.OUT, -h.shape[1] - 1)
    got = rc.download(req)
    assert np.array_equal(got.reshape(exp.shape), exp)


@pytest.mark.parametrize("C", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10])
def test_rows_with_and_without_the_buffer(graph, C):
    orc = oracle.Oracle(*graph, 2)
    # block edges, one block, more blocks than the writing trails by; blocks that
    # keep everything, little (their rows are read after they are counted), nothing
    for i, (R, share) in enumerate([(1, 1.0), (1023, 0.1), (1024, 1.0), (1025, 0.0), (5000, 0.1), (400_003, 1.0),
                                    (300_001, 0.02), (300_001, 0.0)]):
        rc = _context(graph, 1)
        h = _table(R, C, 100 * C + i, share)
        _step(rc, orc, h)                  # nothing there yet
        _step(rc, orc, h)                  # as many bytes as there were rows
        rc.known_to_unknown(_uploaded(rc, _table(R + 2000, C, i, 1.0)), -1, W.OUT, 2)
        rc.known_to_unknown(_uploaded(rc, _table(2 * R + 4000, C, i, 1.0)), -1, W.OUT, 2)
        _step(rc, orc, h)                  # room for a row per row
        rc.close()


def _uploaded(rc, h):
    req = W.Request([])
    rc.upload_history(req, h)
    return req


def test_row_limit_leaves_the_other_table(graph):
    orc = oracle.Oracle(*graph, 2)
    rc = _context(graph, 1 << 20)          # both tables have room for every row
    h = _table(3000, 2, 3, 1.0)
    first = _uploaded(rc, h)
    kept = W.wk_history(first.hist.data, first.hist.size, first.hist.col_num, 0)
    rc.known_to_unknown(first, -1, W.OUT, 2)
    want = rc.download(first)
    rows = len(orc.step(want, False, -1, 2, W.OUT, -4)[0])
    rc.set_row_limit(rows - 1)
    with pytest.raises(W.WkError) as e:    # would go where the uploaded table is
        rc.known_to_unknown(first, -1, W.OUT, 2)
    assert e.value.status == W.WK_EOVERFLOW
    rc.sync()
    assert np.array_equal(rc.download(first), want)
    old = W.Request([])
    old.hist = kept
    assert np.array_equal(rc.download(old), h)
    rc.set_row_limit(rows)                 # below the input's rows, not below the output's
    rc.known_to_unknown(first, -1, W.OUT, 2)
    assert np.array_equal(rc.download(first), orc.step(want, False, -1, 2, W.OUT, -4)[0])
    rc.close()


def test_memory_follows_the_rows(graph):
    """4M rows of 3 columns of which about 80,000 match: the op's scratch is 4 B a
    row (16 MB), its output 1.3 MB, a row per row would be 64 MB."""
    torch = pytest.importorskip("torch")
    rc = _context(graph, 1)
    req = _uploaded(rc, _table(4_000_000, 3, 5, 0.02))
    rc.sync()
    free = torch.cuda.mem_get_info(0)[0]
    rc.known_to_unknown(req, -1, W.OUT, 2)
    rc.sync()
    assert 0 < req.get_row_num() < 100_000
    assert free - torch.cuda.mem_get_info(0)[0] < 32 << 20
    rc.close()
