"""k2k and k2c where a filter's copy changes hands: a CTA per block of 1024 rows
up to 16 blocks an SM, a warp per block above, over a functional direction (one
launch) and one with lists (three), every share of kept rows a block can have."""
import numpy as np
import pytest

import wukonggpu_gb300 as W

pytestmark = pytest.mark.gpu

N = 500      # subjects
SMS = 152


@pytest.fixture(scope="module", params=["functional", "lists"])
def graph(request, lib_built):
    rng = np.random.default_rng(11)
    deg = np.ones(N, np.int64) if request.param == "functional" else rng.integers(0, 70, N)
    s = np.repeat(np.arange(N), deg)
    o = np.concatenate([rng.permutation(300)[:d] for d in deg])
    rc = W.RCache(device=0)
    rc.build_store((W.VID_BASE + s).astype(np.int32), np.full(len(s), 2, np.int32),
                   (W.VID_BASE + 1000 + o).astype(np.int32), 2)
    assert bool(rc.seg_layout(2)["functional"][W.OUT]) == (request.param == "functional")
    holds = np.zeros((N + 10, 300), bool)
    holds[s, o] = True
    yield rc, holds
    rc.close()


@pytest.mark.parametrize("blocks", [1, 2, 9, 1300, 16 * SMS, 16 * SMS + 1])
@pytest.mark.parametrize("C", [2, 5, 9])
def test_copy_of_kept_rows(graph, blocks, C):
    rc, holds = graph
    if blocks >= 1300 and C == 9:
        C = 3
    rng = np.random.default_rng(blocks + C)
    R = blocks * 1024 - (blocks % 7) * 3
    h = np.empty((R, C), np.int32)
    h[:, 2:] = np.arange(R, dtype=np.int32)[:, None]
    start = rng.integers(0, N + 10, R)
    end = rng.integers(0, 300, R)
    # per block: nothing kept, everything a functional row can keep, or a mix
    first = holds.argmax(axis=1)
    kind = (np.arange(R) // 1024) % 3
    end = np.where(kind == 1, first[start], end)
    end = np.where(kind == 0, 299, np.where((kind == 2) & (rng.random(R) < 0.5), first[start], end))
    h[:, 0] = W.VID_BASE + start
    h[:, 1] = W.VID_BASE + 1000 + end
    for k2c in (False, True):
        const = 7
        keep = holds[start, const if k2c else end]
        req = W.Request([])
        rc.upload_history(req, h)
        if k2c:
            rc.known_to_const(req, -1, W.OUT, 2, W.VID_BASE + 1000 + const)
        else:
            rc.known_to_known(req, -1, W.OUT, 2, -2)
        got = rc.download(req)
        assert np.array_equal(got.reshape(-1, C), h[keep])
