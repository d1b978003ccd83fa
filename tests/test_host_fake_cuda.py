"""Host code around the kernels, run without a GPU: the library's objects linked
against a CUDA runtime with two devices whose kernels do nothing
(fake_cuda/fake_cudart.cpp).  Each test is a program of its own."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PRELUDE = """
import ctypes as C, sys, threading
from pathlib import Path
import numpy as np
sys.path.insert(0, {root!r})
import wukonggpu_gb300 as W
W._LIB_PATH = Path({lib!r})
lib = W.load_library()
fake = C.CDLL({lib!r})
for f in ("fake_wrong_device", "fake_launches", "fake_bytes_on", "fake_pending"):
    getattr(fake, f).restype = C.c_long

# vertex VID_BASE + i has the one neighbour VID_BASE + 100 + i in predicate 2
def context(device, **kw):
    s = (W.VID_BASE + np.arange(64)).astype(np.int32)
    rc = W.RCache(device=device, **kw)
    rc.build_store(s, np.full(64, 2, np.int32), s + 100, 2)
    return rc
"""


@pytest.fixture(scope="session")
def fake_lib(lib_built, tmp_path_factory):
    from wukonggpu_gb300 import build as wb
    out = tmp_path_factory.mktemp("fake") / "libwkgpu_fake.so"
    objs = [wb.BUILD / (p.name + ".o") for pat in ("*.cpp", "*.cu") for p in sorted(wb.CSRC.glob(pat))]
    cmd = ["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", str(wb._cuda_home() / "include"), "-o", str(out),
           str(ROOT / "tests" / "fake_cuda" / "fake_cudart.cpp"), *map(str, objs), "-lpthread", "-Wl,--no-undefined"]
    subprocess.run(cmd, check=True, capture_output=True, text=True)
    return out


def _run(fake_lib, body):
    code = PRELUDE.format(root=str(ROOT), lib=str(fake_lib)) + body + "\nprint('ok', flush=True)\nimport os; os._exit(0)\n"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120,
                       env={**os.environ, "OPENBLAS_NUM_THREADS": "1"})
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr


def test_light_request_runs_on_its_contexts_device(fake_lib):
    """Two contexts on two devices in one thread, and a context used from a new
    thread: every launch and allocation of a short request is its device's."""
    _run(fake_lib, """
q = [W.VID_BASE + 1, 2, W.OUT, -1, -1, 2, W.OUT, -2]
def short(rc):
    try:
        rc.execute(q)
    except W.WkError as e:      # the kernels publish nothing here
        assert "without publishing" in str(e), e
a, b = context(0, history_capacity=64), context(1, history_capacity=64)
on1 = fake.fake_bytes_on(1)
n = fake.fake_launches()
short(a)                        # device 1 is current
assert fake.fake_launches() > n
assert fake.fake_wrong_device() == 0 and fake.fake_bytes_on(1) == on1
t = threading.Thread(target=short, args=(b,))    # a new thread: device 0 is current
on0 = fake.fake_bytes_on(0)
t.start(); t.join()
assert fake.fake_wrong_device() == 0 and fake.fake_bytes_on(0) == on0
""")


def test_group_sums_after_a_failed_allocation(fake_lib):
    """An op after one whose group sums could not be allocated allocates them
    again: the buffer that was given back for the larger one is gone."""
    _run(fake_lib, """
rc = context(0)
h = np.full((300, 1), W.VID_BASE + 1, np.int32)
def step():
    req = W.Request([])
    rc.upload_history(req, h)
    try:
        rc.known_to_unknown(req, -1, W.OUT, 2)
    except W.WkError as e:
        assert "without publishing" in str(e), e
    return req
step()
fake.fake_fail_mallocs(2)       # the reservation and its retry
req = W.Request([])
rc.upload_history(req, h)
try:
    rc.partition(req, -1, 2)
    raise SystemExit("no error")
except W.WkError as e:
    assert e.status == W.WK_ENOMEM, e
fake.fake_fail_mallocs(0)
before = fake.fake_bytes_on(0)
step()
assert fake.fake_bytes_on(0) > before
""")


def test_batch_holds_a_row_for_each_query(fake_lib):
    """The rows' counts and list offsets of a batch have room for step 0's one
    row per query however small the capacity is: all that a capacity below the
    number of queries saves is the two tables."""
    _run(fake_lib, """
rc = context(0)
def size(cap):
    before = fake.fake_bytes_on(0)
    b = W.Batch(rc, max_queries=4096, max_steps=2, capacity_ints=cap)
    n = fake.fake_bytes_on(0) - before
    b.close()
    assert fake.fake_bytes_on(0) == before
    return n
assert size(4096) - size(1) == 2 * 4 * 4095
""")


def test_new_context_holds_a_small_piece(fake_lib):
    """Beside its two tables, a context allocates something small when it is made,
    so that its first step finds the piece of device memory that small
    allocations come from."""
    _run(fake_lib, """
rc = W.RCache(device=0, history_capacity=1 << 20)
assert 0 < fake.fake_bytes_on(0) - 2 * (4 << 20) <= 1 << 16
""")


@pytest.mark.parametrize("cols", [1 << 23, 1 << 24])
def test_partition_of_very_wide_rows(fake_lib, cols):
    """Widths whose words per tile pass 32 bits are copied row by row, as every
    width above a tile's is."""
    _run(fake_lib, f"""
rc = context(0)
req = W.Request([])
rc.upload_history(req, np.zeros((1, {cols}), np.int32))
n = fake.fake_launches()
rc.partition(req, -1, 2)        # the kernels do nothing: only the launches count
assert fake.fake_launches() - n == 3
""")


def test_estimator_errors_leave_nothing_in_flight(fake_lib):
    """A call that fails on the host once copies are queued returns when they are
    done: the caller's arrays are the caller's again."""
    _run(fake_lib, """
est = W.Estimator(context(0), 4, max_batch=4096, seed=1)
def samples(n):
    return np.zeros((n, 48), np.float32), np.ones(n, np.int32), np.zeros(n, np.float32)
fake.fake_no_driver_entry(1)    # no tensor map can be made
calls = [lambda n=n: est.predict(*samples(n)[:2]) for n in (16, 2000, 20_000, 100_000)]
calls += [lambda n=n: est.gradients(*samples(n)) for n in (16, 2000)]
for call in calls:
    try:
        call()
        raise SystemExit("no error")
    except W.WkError as e:
        assert e.status == W.WK_EDEVICE, e
    assert fake.fake_pending() == 0
fake.fake_no_driver_entry(0)
calls[0]()                      # and the next call is its own
""")
