"""The one-launch ops over a dense functional direction: k2u, k2k and k2c
against the oracle's step on tables around the block size (1024 rows), with
more blocks than the writing trails by, of every width that the launch takes
and above, from a table that does not start on a 16 B boundary, and with
starts that are index keys or no vertices."""
import numpy as np
import pytest

import oracle
import wukonggpu_gb300 as W

pytestmark = pytest.mark.gpu

N = 3000   # subjects VID_BASE .. VID_BASE + N - 1, seven in eight with a neighbour


@pytest.fixture(scope="module")
def graph(lib_built):
    rng = np.random.default_rng(5)
    s = W.VID_BASE + np.flatnonzero(np.arange(N) % 8 != 3).astype(np.int32)
    o = (W.VID_BASE + rng.integers(0, 40, size=len(s))).astype(np.int32)
    p = np.full(len(s), 2, np.int32)
    rc = W.RCache(device=0)
    rc.build_store(s, p, o, 2)
    lay = rc.seg_layout(2)
    assert lay["dense"][W.OUT] and lay["functional"][W.OUT]
    yield rc, oracle.Oracle(s, p, o, 2)
    rc.close()


def _table(R, C, seed, zeros):
    rng = np.random.default_rng(seed)
    h = (W.VID_BASE + rng.integers(-20, N + 20, size=(R, C))).astype(np.int32)
    h[:, C - 1] = W.VID_BASE + rng.integers(0, 40, size=R)          # the filters' end column
    h[rng.random(R) < 0.02, 0] = -5                                  # no vertex
    if zeros:
        h[rng.random(R) < 0.01, 0] = 0                               # index keys
        h[R // 2, 0] = 0
    return h


def _ops(rc, orc, req_of, h, C):
    """k2u and, from two columns up, k2k and k2c of table h."""
    req = req_of(h)
    rc.known_to_unknown(req, -1, W.OUT, 2)
    exp, _ = orc.step(h, False, -1, 2, W.OUT, -C - 1)
    st = rc.last_op_stats()
    assert st["rows_out"] == len(exp) and st["rows_in"] == len(h)
    got = rc.download(req)
    assert np.array_equal(got.reshape(exp.shape), exp)
    ends = [W.VID_BASE + 7] + ([-C] if C > 1 else [])
    for end in ends:
        req = req_of(h)
        if end < 0:
            rc.known_to_known(req, -1, W.OUT, 2, end)
        else:
            rc.known_to_const(req, -1, W.OUT, 2, end)
        exp, scanned = orc.step(h, False, -1, 2, W.OUT, end)
        got = rc.download(req)
        assert np.array_equal(got.reshape(exp.shape), exp), end


@pytest.mark.parametrize("zeros", [False, True])
@pytest.mark.parametrize("C", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13])
@pytest.mark.parametrize("R", [1, 511, 1024, 1025, 4097])
def test_tile_edges(graph, R, C, zeros):
    rc, orc = graph

    def req_of(h):
        req = W.Request([])
        rc.upload_history(req, h)
        return req
    _ops(rc, orc, req_of, _table(R, C, 31 * R + C, zeros), C)


@pytest.mark.parametrize("R,C", [(400_003, 3), (1_500_007, 8), (5_000_011, 2)])
def test_more_blocks_than_the_lag(graph, R, C):
    rc, orc = graph

    def req_of(h):
        req = W.Request([])
        rc.upload_history(req, h)
        return req
    _ops(rc, orc, req_of, _table(R, C, R, False), C)


@pytest.mark.parametrize("R,C", [(1, 3), (2049, 1), (3000, 4), (5000, 5)])
def test_table_off_a_16_byte_boundary(graph, R, C):
    """A caller's table one word past its buffer's start."""
    rc, orc = graph
    owner = W.RCache(device=0)

    def req_of(h):
        whole = W.Request([])
        owner.upload_history(whole, np.concatenate([[0], h.reshape(-1)]).astype(np.int32))
        owner.sync()
        req = W.Request([])
        req.hist = W.wk_history(whole.hist.data + 4, h.size, C, 0)
        return req
    _ops(rc, orc, req_of, _table(R, C, 7 * R + C, False), C)
    owner.close()
