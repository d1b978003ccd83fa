"""The general k2u expansion where its windows of 32 output rows meet list
boundaries: lists of 1, 31, 32, 33, 63, 64, 65 and 9000 entries (the last
spans slices), tables whose blocks start at every 16 B phase, every
specialised width and widths above."""
import numpy as np
import pytest

import oracle
import wukonggpu_gb300 as W

pytestmark = pytest.mark.gpu

DEGREES = [1, 31, 32, 33, 63, 64, 65, 2, 95, 96, 97, 3, 9000]


@pytest.fixture(scope="module")
def graph(lib_built):
    subj = W.VID_BASE + np.arange(len(DEGREES), dtype=np.int32)
    s = np.repeat(subj, DEGREES).astype(np.int32)
    o = np.concatenate([W.VID_BASE + 100 + 3 * np.arange(d) for d in DEGREES]).astype(np.int32)
    p = np.full(len(s), 2, np.int32)
    rc = W.RCache(device=0)
    rc.build_store(s, p, o, 2)
    yield rc, oracle.Oracle(s, p, o, 2)
    rc.close()


@pytest.mark.parametrize("C", [1, 2, 3, 4, 5, 6, 7, 8, 11, 31, 40])
@pytest.mark.parametrize("R", [1, 5, 1024, 2051])
def test_lists_across_windows(graph, R, C):
    rc, orc = graph
    rng = np.random.default_rng(100 * R + C)
    h = rng.integers(W.VID_BASE, W.VID_BASE + 64, size=(R, C)).astype(np.int32)
    # short lists mostly, a few of the long one, and vertices without a list
    pick = np.where(rng.random(R) < 0.003, 12, rng.integers(0, 16, size=R))
    pick[0] = 12
    h[:, C // 2] = W.VID_BASE + np.where(pick == 12, 12, np.where(pick > 12, pick + 50, pick))
    req = W.Request([])
    rc.upload_history(req, h)
    rc.known_to_unknown(req, -(C // 2) - 1, W.OUT, 2)
    got = rc.download(req)
    exp, _ = orc.step(h, False, -(C // 2) - 1, 2, W.OUT, -C - 1)
    assert got.shape == exp.shape and np.array_equal(got, exp)
