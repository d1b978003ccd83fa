"""What follows when the device waits of a one-launch op run out: the kernel gives
up and returns, and the op runs as separate kernels, with the oracle's rows; so
does the next op, with and without waits that run out."""
import numpy as np
import pytest

import oracle
import wukonggpu_gb300 as W

pytestmark = pytest.mark.gpu

N = 3000   # subjects VID_BASE .. VID_BASE + N - 1, one in eight without a neighbour


@pytest.fixture(scope="module")
def graph(lib_built):
    rng = np.random.default_rng(13)
    s = W.VID_BASE + np.flatnonzero(np.arange(N) % 8 != 3).astype(np.int32)
    o = (W.VID_BASE + rng.integers(0, 40, size=len(s))).astype(np.int32)
    p = np.full(len(s), 2, np.int32)
    rc = W.RCache(device=0)
    rc.build_store(s, p, o, 2)
    yield rc, oracle.Oracle(s, p, o, 2)
    rc.close()


@pytest.mark.parametrize("C", [1, 3, 8])
@pytest.mark.parametrize("R", [1, 2049, 700_001, 3_000_001])
def test_waits_that_run_out(graph, R, C):
    rc, orc = graph
    rng = np.random.default_rng(R + C)
    h = (W.VID_BASE + rng.integers(0, N + 20, size=(R, C))).astype(np.int32)
    h[:, C - 1] = W.VID_BASE + rng.integers(0, 40 if C > 1 else N, size=R)
    ends = [None, W.VID_BASE + 7] + ([-C] if C > 1 else [])
    exp = [orc.step(h, False, -1, 2, W.OUT, -C - 1 if e is None else e)[0] for e in ends]
    reruns = 0
    for polls in (0, 0, 1, -1, 0):
        rc.set_wait_polls(polls)
        for e, want in zip(ends, exp):
            req = W.Request([])
            rc.upload_history(req, h)
            if e is None:
                rc.known_to_unknown(req, -1, W.OUT, 2)
            elif e < 0:
                rc.known_to_known(req, -1, W.OUT, 2, e)
            else:
                rc.known_to_const(req, -1, W.OUT, 2, e)
            k = rc.last_op_stats()["kernels"]
            assert np.array_equal(rc.download(req).reshape(want.shape), want), (polls, e)
            # (a launch that had to grow its buffer has a second one)
            reruns += k > 2
            assert polls != -1 or k <= 2, (polls, e, k)
    rc.set_wait_polls(-1)
    assert reruns > 0
