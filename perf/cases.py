"""What is measured: the calls a user of the framework makes, through its public entry points.

The dataset is the single-query-scale graph of ``workloads`` (about 100M triples over 2M
entities: 8 functional, 16 Zipf and 8 many-to-one predicates, 15 classes), built once per
process, as a user's process loads its dataset once.  What changes from call to call -- the
queries, the history tables, the samples -- comes from the seed.

Kinds of case:

* ``query``: one whole query through ``RCache.execute``; a light one (constant start) brings its
  rows to the host, a heavy one (type index start) leaves its table on the device;
* ``k2u`` / ``k2k`` / ``k2c``: one pattern applied to a history table on the device, the ops a
  caller of the reference's ``RCache`` makes; the new table stays on the device for the next op;
* ``batch``: light queries run together by ``Batch`` with every result brought to the host;
* ``partition``: the fork-join split of a table by owner;
* ``predict`` / ``gradients``: the learned estimator's forward pass over host samples, and one
  forward + backward pass over a training batch.
"""
import math

import numpy as np
import torch

import wukonggpu_gb300 as W
from wukonggpu_gb300 import mix, workloads

LAYOUT = workloads.SQ
N_ENTITIES = 2_000_000
# list entries per start vertex: one neighbour in a functional or many-to-one predicate's OUT
# direction; a Zipf predicate's ~4.1M triples over all entities (OUT: 0.65% of them hold long
# lists); a many-to-one predicate's hubs hold 100 subjects each
FAN = {"func": 1.0, "m2o": 1.0, "zipf": 2.07, "hub": 100.0, "type": 1.0}
N_IDS = 48                  # predicates and classes of the graph: embedding rows of the estimator
N_PARAMS_W = [(256, 80), (256, 256), (256, 256), (1, 256)]
N_PARAMS_B = [256, 256, 256, 64]


def listed():
    return [
        # a light request alone: attribute, hub, co-members and their attribute of one entity
        # (about 100 rows), the latency a user sees between submitting it and holding its rows
        {"name": "light query", "kind": "query", "shape": "light"},
        # a six-pattern chain and star of the benchmark mix, the largest of its three shapes
        # (5 * 10^7 rows of 6 columns)
        {"name": "heavy query", "kind": "query", "shape": "chain_zipf_hub"},
        # fan-out through hubs: few input rows, a hundred output rows each
        {"name": "k2u hub fan-out", "kind": "k2u", "pred": "hub", "dir": W.IN, "rows": 120_011, "cols": 3, "run": 1},
        # a sparse predicate with long lists on a large table (hashed keys; most rows find nothing)
        {"name": "k2u sparse", "kind": "k2u", "pred": "zipf", "dir": W.OUT, "rows": 9_000_001, "cols": 5, "run": 3},
        # a functional predicate on a large table: one attribute per row
        {"name": "k2u functional", "kind": "k2u", "pred": "func", "dir": W.OUT, "rows": 12_000_003, "cols": 4, "run": 1},
        # a query with many variables: a wide table
        {"name": "k2u wide", "kind": "k2u", "pred": "zipf", "dir": W.IN, "rows": 800_003, "cols": 10, "run": 1},
        # closing a cycle on a large table, two rows in five kept
        {"name": "k2k cycle", "kind": "k2k", "pred": "func", "dir": W.OUT, "rows": 10_000_003, "cols": 3, "run": 1,
         "keep": 0.4},
        # checking a class, one row in fifteen kept
        {"name": "k2c class", "kind": "k2c", "pred": "type", "dir": W.OUT, "rows": 3_000_017, "cols": 6, "run": 2},
        # a full batch of light requests of the serving mix
        {"name": "batch of light queries", "kind": "batch", "queries": 4096},
        # the fork-join split of a table over 8 ranks
        {"name": "partition", "kind": "partition", "rows": 6_000_001, "cols": 3, "parts": 8},
        # the estimator over an evaluation set
        {"name": "estimator predict", "kind": "predict", "samples": 100_003},
        # one training batch of the estimator: loss and every gradient
        {"name": "estimator gradients", "kind": "gradients", "samples": 1024},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["k2u", "k2u", "k2u", "k2u", "k2k", "k2k", "k2c", "query", "batch", "partition", "predict",
                       "gradients"])
    if kind == "query":
        return {"kind": kind, "shape": rng.choice(["light", "star_chain_hub", "star_fan_in"]),
                "variant": rng.randrange(1, 1000)}
    if kind == "batch":
        return {"kind": kind, "queries": _log_uniform(rng, 4, 4096)}
    if kind == "predict":
        return {"kind": kind, "samples": _log_uniform(rng, 16, 100_000)}
    if kind == "gradients":
        return {"kind": kind, "samples": _log_uniform(rng, 16, 4096)}
    cols = rng.randint(1, 12) if kind == "k2u" else rng.randint(2, 12)
    if kind == "partition":
        cols = rng.randint(1, 8)
    # tables of up to 48M values, in and out
    if kind == "k2u":
        pred, d = rng.choice([("func", W.OUT), ("func", W.IN), ("m2o", W.OUT), ("zipf", W.OUT), ("zipf", W.IN),
                              ("hub", W.IN)])
        most = int(min(48e6 / cols, 48e6 / (FAN[pred] * (cols + 1))))
    elif kind == "k2k":
        pred, d = rng.choice([("func", W.OUT), ("m2o", W.OUT), ("zipf", W.OUT)])
        most = int(30e6 / cols)
    elif kind == "k2c":
        pred, d = "type", W.OUT
        most = int(30e6 / cols)
    else:
        return {"kind": kind, "rows": _log_uniform(rng, 1000, 24e6 / cols), "cols": cols,
                "parts": rng.choice([2, 3, 4, 8, 16, 72])}
    case = {"kind": kind, "pred": pred, "dir": d, "rows": _log_uniform(rng, 300, most), "cols": cols,
            "run": rng.choice([1, 1, 3, 40])}
    if kind == "k2k":
        case["keep"] = round(rng.uniform(0.0, 1.0), 3)
    return case


# ------------------------------------------------------------------ the dataset
_dataset = {}


def _data():
    if not _dataset:
        g = W.Graph(W.spec_single_query())
        s, p, o = g.arrays()
        rc = W.RCache(device=0)
        rc.build_store(s, p, o, g.num_ids, on_device=True)
        _dataset["rc"], _dataset["graph"] = rc, g
        m = mix.Mix(mix.MIX_DIR / "serving" / "mix_config", LAYOUT)
        m.fill_candidates(rc)
        _dataset["mix"] = m
    return _dataset


def _context():
    """A context of its own on the shared store, as each worker thread of a program keeps one."""
    rc = W.RCache(device=0)
    rc.share_store(_data()["rc"])
    return rc


def _predicate(case):
    pred, k = case["pred"], case["rows"] % 8   # another of the eight alike predicates for another size
    return {"func": LAYOUT.func[k], "zipf": LAYOUT.zipf[k], "m2o": LAYOUT.m2o[k], "hub": LAYOUT.m2o[k],
            "type": W.TYPE_ID}[pred]


def _neighbour_of(pid):
    """Entity -> its one neighbour in a functional or many-to-one predicate, on the GPU."""
    key = ("nb", pid)
    if key not in _dataset:
        s, p, o = _data()["graph"].arrays()
        m = np.flatnonzero(p == pid)
        nb = np.full(N_ENTITIES, W.VID_BASE, np.int32)
        nb[s[m] - W.VID_BASE] = o[m]
        _dataset[key] = torch.from_numpy(nb).cuda()
    return _dataset[key]


def _triples_of(pid):
    """The subjects and objects of a predicate's triples, on the GPU."""
    key = ("so", pid)
    if key not in _dataset:
        s, p, o = _data()["graph"].arrays()
        m = np.flatnonzero(p == pid)
        _dataset[key] = (torch.from_numpy(s[m]).cuda(), torch.from_numpy(o[m]).cuda())
    return _dataset[key]


def _runs(gen, rows, run):
    """Row -> run index: runs of `run` rows on average, as an expansion repeats its input rows."""
    if run == 1:
        return torch.arange(rows, device="cuda")
    heads = torch.rand(rows, generator=gen, device="cuda") < 1.0 / run
    return torch.cumsum(heads, 0)


def _pattern_columns(case, gen):
    """The columns the pattern asks about: the start vertices, in runs, and for k2k the ends, which
    are the start's neighbour in about `keep` of the rows."""
    rows, pid = case["rows"], _predicate(case)
    idx = _runs(gen, rows, case["run"])
    n = int(idx[-1]) + 1
    pick = torch.randint(0, N_ENTITIES, (n,), generator=gen, device="cuda")
    start = pick.to(torch.int32) + W.VID_BASE
    if case["pred"] == "hub":
        hubs = torch.from_numpy(_data()["rc"].get_edges(0, pid, W.OUT)).cuda()
        start = hubs[pick % hubs.numel()]
    if case["kind"] != "k2k":
        return start[idx], None
    end = torch.randint(W.VID_BASE, W.VID_BASE + N_ENTITIES, (rows,), generator=gen, device="cuda", dtype=torch.int32)
    if case["pred"] == "zipf":
        subj, obj = _triples_of(pid)
        e = torch.randint(0, subj.numel(), (n,), generator=gen, device="cuda")
        hit = torch.rand(n, generator=gen, device="cuda") < case["keep"]
        start, end = torch.where(hit, subj[e], start), torch.where(hit[idx], obj[e][idx], end)
        return start[idx], end
    start = start[idx]
    hit = torch.rand(rows, generator=gen, device="cuda") < case["keep"]
    return start, torch.where(hit, _neighbour_of(pid)[start.long() - W.VID_BASE], end)


def _table(case, seed):
    """A history table.  The other columns hold entities drawn by the seed; the pattern's columns
    are the case's own, shifted cyclically by the seed, so that every seed gives as many rows."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 1_000_003 + 17)
    rows, cols = case["rows"], case["cols"]
    t = torch.randint(W.VID_BASE, W.VID_BASE + N_ENTITIES, (rows, cols), generator=gen, device="cuda",
                      dtype=torch.int32)
    col = rows % (cols - 1 if case["kind"] == "k2k" else cols)
    if case["kind"] == "partition":
        return t, col
    fixed = torch.Generator(device="cuda")
    fixed.manual_seed(rows * 16 + cols)
    shift = (seed * 7919 + 1) % rows
    start, end = _pattern_columns(case, fixed)
    t[:, col] = torch.roll(start, shift)
    if end is not None:
        t[:, cols - 1] = torch.roll(end, shift)
    return t, col


class _DeviceTable:
    """A context's history table as an array: it keeps the context, whose buffer it is, alive."""

    def __init__(self, rc, ptr, rows, cols):
        self.owner = rc
        self.__cuda_array_interface__ = {"shape": (rows, cols), "typestr": "<i4", "data": (ptr, False), "version": 2}


def _on_device(rc, req):
    """The request's table where the op left it, for the next consumer on the device."""
    rows, cols = req.get_row_num(), req.col_num
    if rows == 0:
        return torch.empty((0, cols), dtype=torch.int32, device="cuda")
    return torch.as_tensor(_DeviceTable(rc, req.hist.data, rows, cols), device="cuda")


def _params(seed):
    rng = np.random.default_rng(seed)
    parts = [rng.uniform(-1.0, 1.0, r * c) * math.sqrt(6.0 / c) * (0.5 if r == 1 else 1.0) for r, c in N_PARAMS_W]
    parts += [rng.normal(0.0, 0.05, n) for n in N_PARAMS_B]
    parts.append(rng.normal(0.0, 0.1, (N_IDS + 1) * 32))
    return np.concatenate(parts).astype(np.float32)


def _samples(n, seed):
    """Plan-step features as the planner makes them: one-hots of the step's kind, direction and end,
    log counts and degrees, the rest zero; targets are log(1 + rows)."""
    rng = np.random.default_rng(seed + 5)
    f = np.zeros((n, 48), np.float32)
    rows = np.arange(n)
    f[rows, rng.integers(0, 5, n)] = 1.0
    f[rows, 5 + rng.integers(0, 2, n)] = 1.0
    f[:, 7:10] = rng.uniform(9.0, 15.5, (n, 3))
    f[:, 10:12] = rng.uniform(0.7, 6.0, (n, 2))
    f[:, 12] = rng.uniform(0.0, 17.0, n)
    f[:, 13] = rng.integers(0, 6, n) / 6.0
    f[:, 14] = rng.integers(0, 7, n) / 8.0
    f[rows, 15 + rng.integers(0, 3, n)] = 1.0
    f[:, 19:24] = rng.uniform(0.0, 16.0, (n, 5))
    f[:, 25] = rng.integers(0, 2, n)
    return f, rng.integers(1, N_IDS + 1, n).astype(np.int32), rng.uniform(0.0, 17.0, n).astype(np.float32)


# the pattern of each heavy shape whose functional predicate adds an attribute and leaves the row
# counts as they are: the seed chooses which of the eight
_ATTRIBUTE = {"star_chain_hub": 3, "chain_zipf_hub": 4, "star_fan_in": 4}


def _light_query(seed):
    """Attribute, hub, co-members and their attribute (a template of the serving mix) of an entity
    whose hub has exactly 100 members, so that every seed gives as many rows."""
    m, rc = _data()["mix"], _data()["rc"]
    rng = np.random.default_rng(seed)
    while True:
        q = m.instantiate(m.types[3], int(rng.integers(0, 1 << 31)))
        attribute = int(rc.get_edges(q[0], q[1], q[2])[0])
        hub = int(rc.get_edges(attribute, q[5], q[6])[0])
        if len(rc.get_edges(hub, q[9], q[10])) == 100:
            return q


# ------------------------------------------------------------------ one case
def prepare(case, seed):
    kind, data = case["kind"], _data()
    if kind == "query":
        rc, variant = _context(), case.get("variant", 0)
        if case["shape"] == "light":
            return {"kind": "light", "rc": rc, "query": _light_query(seed + variant)}
        q = next(list(q) for name, q in workloads.scale_queries(1) if name.startswith(case["shape"]))
        q[0] = LAYOUT.first_class + variant % LAYOUT.n_classes
        q[4 * _ATTRIBUTE[case["shape"]] + 1] = LAYOUT.func[seed % 8]
        return {"kind": "heavy", "rc": rc, "query": q}
    if kind == "batch":
        # the case's own requests in an order of the seed's
        m = data["mix"]
        light = np.asarray(m.weights[:m.n_light], np.float64)
        fixed = np.random.default_rng(case["queries"])
        types = fixed.choice(m.n_light, case["queries"], p=light / light.sum())
        queries = [m.instantiate(m.types[k], int(fixed.integers(0, 1 << 31))) for k in types]
        queries = [queries[i] for i in np.random.default_rng(seed).permutation(len(queries))]
        rc = _context()
        pinned = W.PinnedBuffer(1 << 22)   # kept by the process: the results are views into it
        data.setdefault("pinned", []).append(pinned)
        # the requests as the C ABI takes them, as a front end that received them in arrays holds them
        return {"kind": kind, "queries": queries, "packed": W.Batch.pack(queries), "pinned": pinned,
                "batch": W.Batch(rc, max_queries=case["queries"], max_steps=4, capacity_ints=1 << 24)}
    if kind in ("predict", "gradients"):
        f, p, t = _samples(case["samples"], seed)
        est = W.Estimator(_context(), N_IDS, max_batch=4096, seed=1)
        est.set_params(_params(seed))
        return {"kind": kind, "est": est, "feats": f, "pids": p, "target": t}
    table, col = _table(case, seed)
    torch.cuda.synchronize()
    rc, req = _context(), W.Request([])
    rc.from_device(req, table.data_ptr(), table.numel(), case["cols"])
    state = {"kind": kind, "rc": rc, "table": req.hist, "var": -col - 1}
    if kind == "partition":
        return dict(state, parts=case["parts"])
    state.update(pid=_predicate(case), dir=case["dir"])
    if kind == "k2k":
        state["end"] = -case["cols"]
    if kind == "k2c":
        state["end"] = LAYOUT.first_class + case["rows"] % LAYOUT.n_classes
    return state


def run(state):
    kind = state["kind"]
    if kind == "light":
        req, rows = state["rc"].execute(state["query"])
        return req.result_table, rows
    if kind == "heavy":
        req, rows = state["rc"].execute(state["query"], download=False)
        return _on_device(state["rc"], req), rows
    if kind == "batch":
        b = state["batch"]
        n = b.run(state["queries"], packed=state["packed"])
        host = state["pinned"]
        tables = b.download(n, into=host)   # the queries' tables, packed in order
        last = tables[n - 1]
        total = (last.ctypes.data - host.array.ctypes.data) // 4 + last.size
        return host.array[:total]
    if kind == "predict":
        return state["est"].predict(state["feats"], state["pids"])
    if kind == "gradients":
        return state["est"].gradients(state["feats"], state["pids"], state["target"])
    rc, h = state["rc"], state["table"]
    req = W.Request([])
    req.hist = W.wk_history(h.data, h.size, h.col_num, h.step)
    if kind == "partition":
        counts = rc.partition(req, state["var"], state["parts"])
        return _on_device(rc, req), counts
    if kind == "k2u":
        rc.known_to_unknown(req, state["var"], state["dir"], state["pid"])
    elif kind == "k2k":
        rc.known_to_known(req, state["var"], state["dir"], state["pid"], state["end"])
    else:
        rc.known_to_const(req, state["var"], state["dir"], state["pid"], state["end"])
    return _on_device(rc, req)


# rows after every step of the heavy shapes on this graph, per start row of a class (2M / 15 members)
_HEAVY = {"star_chain_hub": [1, 1, 100, 100, 100, 100], "chain_zipf_hub": [1, 2.07, 2.07, 207, 207, 428],
          "star_fan_in": [1, 1, 1, 100, 100, 207]}


def work(case):
    """Bytes: the input table read once, 4 B per looked-up neighbour or list entry, the output table
    written once (a query: its final table, and 4 B per looked-up value of every step)."""
    kind = case["kind"]
    if kind == "query":
        if case["shape"] == "light":
            return {"bytes": 4.0 * (1 + 1 + 100 + 100) + 1600.0, "flops": 0}
        rows = [N_ENTITIES / 15 * x for x in _HEAVY[case["shape"]]]
        return {"bytes": 4.0 * sum(rows) + 24.0 * rows[-1], "flops": 0}
    if kind == "batch":
        return {"bytes": case["queries"] * 4.0 * 200, "flops": 0}
    if kind in ("predict", "gradients"):
        macs = sum(r * c for r, c in N_PARAMS_W)
        n = case["samples"]
        out = 4.0 * n if kind == "predict" else 4.0 * len(_params(0))
        return {"bytes": n * (4.0 * 48 + 8) + 4.0 * macs + out,
                "flops": (2.0 if kind == "predict" else 6.0) * macs * n}
    rows, cols = case["rows"], case["cols"]
    if kind == "partition":
        return {"bytes": 8.0 * rows * cols, "flops": 0}
    if kind == "k2u":
        out = rows * FAN[case["pred"]]
        return {"bytes": 4.0 * (rows * cols + rows + out * (cols + 1)) + (4.0 * out if out > rows else 0), "flops": 0}
    keep = case.get("keep", 1 / 15)
    return {"bytes": 4.0 * (rows * cols + rows + keep * rows * cols), "flops": 0}


def exact(case, seed):
    """The estimator's outputs in 64 bits; every other output is whole numbers."""
    if case["kind"] not in ("predict", "gradients"):
        return None
    f, pid, t = _samples(case["samples"], seed)
    w = torch.from_numpy(_params(seed).astype(np.float64)).requires_grad_(case["kind"] == "gradients")
    at, mats, bias = 0, [], []
    for r, c in N_PARAMS_W:
        mats.append(w[at:at + r * c].view(r, c))
        at += r * c
    for n in N_PARAMS_B:
        bias.append(w[at:at + n])
        at += n
    emb = w[at:].view(N_IDS + 1, 32)
    x = torch.cat([torch.from_numpy(f.astype(np.float64)), emb[torch.from_numpy(pid.astype(np.int64))]], 1)
    for m, b in zip(mats[:3], bias[:3]):
        x = torch.nn.functional.gelu(x @ m.t() + b)
    y = (x @ mats[3].t())[:, 0] + bias[3][0]
    if case["kind"] == "predict":
        return y.numpy()
    loss = ((y - torch.from_numpy(t.astype(np.float64))) ** 2).mean()
    loss.backward()
    return w.grad.numpy(), float(loss.item())
