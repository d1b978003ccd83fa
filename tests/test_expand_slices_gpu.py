"""The general k2u expansion over many slices of one block: more full slices
than the GPU holds at once (CTAs of 128 threads), for the specialised widths
and the staged ones, and more slices than the op keeps records for (the
expansion in rounds), with the context's buffers and with the caller's own."""
import ctypes

import numpy as np
import pytest

import oracle
import wukonggpu_gb300 as W

pytestmark = pytest.mark.gpu

BIG = 20_000                        # entries of vertex 0's list
DEGREES = [BIG, 1, 33, 7]


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


def _list(orc):
    """vertex 0's list in the store's order"""
    out, _ = orc.step(np.array([[W.VID_BASE]], np.int32), False, -1, 2, W.OUT, -2)
    return out[:, 1]


@pytest.mark.parametrize("C", [1, 2, 3, 5, 7, 8, 11])
def test_many_full_slices(graph, C):
    rc, orc = graph
    rng = np.random.default_rng(C)
    R = 640
    h = rng.integers(W.VID_BASE, W.VID_BASE + 64, size=(R, C)).astype(np.int32)
    v = np.zeros(R, np.int32)
    v[[0, 3, 17, 320, R - 1]] = [1, 2, 3, 50, 2]    # short lists and none among the long ones
    h[:, C - 1] = W.VID_BASE + v
    req = W.Request([])
    rc.upload_history(req, h)
    rc.known_to_unknown(req, -C, W.OUT, 2)
    got = rc.download(req)
    lists = {0: _list(orc)}
    for k in (1, 2, 3):
        lists[k], _ = orc.step(np.array([[W.VID_BASE + k]], np.int32), False, -1, 2, W.OUT, -2)
        lists[k] = lists[k][:, 1]
    lists[50] = np.zeros(0, np.int32)
    deg = np.array([len(lists[int(k)]) for k in v])
    assert got.shape == (deg.sum(), C + 1)
    assert got.shape[0] > 8 * 160 * 8192            # slices of 8192 rows for 8 CTAs on 160 SMs
    at = 0
    for r in range(R):
        part = got[at:at + deg[r]]
        assert (part[:, :C] == h[r]).all() and np.array_equal(part[:, C], lists[int(v[r])])
        at += deg[r]


def _check_on_device(out, rows, lst, torch):
    """out: (rows * BIG, 2) on the device, rows of vertex 0 with a running second column"""
    want = torch.from_numpy(lst).cuda()
    o = out.view(rows, BIG, 2)
    for r0 in range(0, rows, 4096):
        part = o[r0:r0 + 4096]
        assert bool((part[:, :, 0] == W.VID_BASE).all())
        assert bool((part[:, :, 1] == want).all())


def test_records_in_rounds(graph):
    """4,000 rows x 20,000 entries: 9,768 slices at most, records for 4,160"""
    torch = pytest.importorskip("torch")
    rc, orc = graph
    rows = 4_000
    req = W.Request([])
    rc.upload_history(req, np.full((rows, 1), W.VID_BASE, np.int32))
    rc.known_to_unknown(req, -1, W.OUT, 2)
    assert rc.last_op_stats()["kernels"] == 7       # count, and records and expansion three times

    class View:
        __cuda_array_interface__ = {
            "shape": (rows * BIG, 2), "typestr": "<i4", "version": 3,
            "data": (req.hist.data, False)}
    assert req.hist.size == rows * BIG * 2
    rc.sync()
    _check_on_device(torch.as_tensor(View(), device="cuda"), rows, _list(orc), torch)
    torch.cuda.synchronize()


def test_records_in_rounds_noalloc(graph):
    """7,000 rows x 20,000 entries: over 17,000 slices, records for 16,384"""
    torch = pytest.importorskip("torch")
    rc, orc = graph
    rows = 7_000
    h = torch.full((rows, 1), W.VID_BASE, dtype=torch.int32, device="cuda")
    out = torch.zeros(rows * BIG * 2 + 4, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    n = ctypes.c_int64(0)
    as_i32p = lambda t: ctypes.cast(ctypes.c_void_p(t.data_ptr()), W._I32P)
    st = W.load_library().wk_known_to_unknown_noalloc(rc._h, as_i32p(h), rows, 1, -1, W.OUT, 2, as_i32p(out),
                                                      rows * BIG * 2, ctypes.byref(n))
    assert st == W.WK_OK and n.value == rows * BIG
    _check_on_device(out[:rows * BIG * 2], rows, _list(orc), torch)
    assert bool((out[rows * BIG * 2:] == 0).all())
