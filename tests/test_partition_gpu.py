"""The device split around its rules: up to 8 owners (counted in bytes of a
word) and above, tiles of 2048 rows down to 256 as the width grows, rows too
wide for a staged tile (25 columns up), vectors of one, two and four words,
tables that start off a 16 B or 8 B boundary, counts scanned by one block and
by three launches, and values that are negative as int32 (owner = value as
unsigned modulo the parts) -- against a numpy stable split."""
import numpy as np
import pytest

import wukonggpu_gb300 as W

pytestmark = pytest.mark.gpu


def _check(rc, req, table, col, nparts):
    counts = rc.partition(req, -col - 1, nparts)
    owner = table[:, col].view(np.uint32) % np.uint32(nparts)
    order = np.argsort(owner, kind="stable")
    assert np.array_equal(counts, np.bincount(owner, minlength=nparts))
    got = rc.download(req)
    assert np.array_equal(got, table[order])


def _table(R, C, seed):
    rng = np.random.default_rng(seed)
    t = rng.integers(-(1 << 31), 1 << 31, size=(R, C)).astype(np.int32)
    t[: R // 3, C // 2] = 7                         # a run of one owner
    return t


@pytest.mark.parametrize("nparts", [1, 2, 7, 8, 9, 255, 256])
@pytest.mark.parametrize("C", [1, 2, 3, 4, 5, 6, 7, 8, 12, 24, 25, 28, 40])
def test_widths_and_parts(gpu_small, C, nparts):
    for R in (1, 255, 2048, 6145):
        t = _table(R, C, R + C)
        req = W.Request([])
        gpu_small.upload_history(req, t)
        _check(gpu_small, req, t, C // 2, nparts)


@pytest.mark.parametrize("off", [1, 2, 4])
@pytest.mark.parametrize("C", [1, 2, 3, 4, 6, 26])
def test_tables_off_their_vectors_alignment(gpu_small, C, off):
    owner = W.RCache(device=0)
    t = _table(5000, C, C + off)
    whole = W.Request([])
    owner.upload_history(whole, np.concatenate([np.zeros(off, np.int32), t.reshape(-1)]))
    owner.sync()
    req = W.Request([])
    req.hist = W.wk_history(whole.hist.data + 4 * off, t.size, C, 0)
    _check(gpu_small, req, t, 0, 8)
    owner.close()


@pytest.mark.parametrize("R", [2048 * 511, 2048 * 512 + 1, 2048 * 700 + 5])   # 256 parts: 131072 counts and more
def test_counts_of_one_block_and_more(gpu_small, R):
    t = _table(R, 2, R)
    req = W.Request([])
    gpu_small.upload_history(req, t)
    _check(gpu_small, req, t, 1, 256)
