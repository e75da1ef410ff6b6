"""The work this framework does for its users, as cases that can be timed.

listed() names the cases, draw() gives more of the same ranges, prepare()
makes what a program holds before the call (index, graph or codes, and the
inputs), run() is one pass through the public entry points, work() the bytes
and operations that pass cannot do without, exact() its distances in 64 bits.

Data are the generators' of fknn/datagen.py restated on the GPU (so that
making them is quick): rows from a mixture of 256 Gaussian clusters, Zipf
categories, timestamps U[0, 1]; queries from the same mixture with a
predicate of type 0 none, 1 category, 2 window, 3 both.  "uniform" windows
are U[0.05, 0.5] wide (the plain and precision workloads), "loguniform" ones
log-U[1e-4, 1] (uneven selectivity, serving), "bucket" ones U[0.2, 0.95] (the
windows a time bucket's graph is searched under).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sigmod-2024-contest_b200"))

import fknn  # noqa: E402

DIM = 100
CODE = 112

# (Zipf exponent, number of categories, window widths)
PLAIN = {"zipf": 1.1, "labels": 1000, "window": "uniform"}
UNEVEN = {"zipf": 1.5, "labels": 10000, "window": "loguniform"}
BUCKET = {"zipf": 1.5, "labels": 10000, "window": "bucket"}


def listed():
    return [
        # An interactive request: a handful of mixed queries from host memory
        # against a resident index, exact.  Latency and launches count.
        {"name": "exact_online", "op": "search", "mode": "exact", "n": 1_000_000, "nq": 16, "k": 100, "host": True,
         **PLAIN},
        # The plain exact workload (N = 1e5, Q = 1e4), queries and results in host memory.
        {"name": "exact_plain", "op": "search", "mode": "exact", "n": 100_000, "nq": 10_000, "k": 100, "host": True,
         **PLAIN},
        # The exact path at scale (N = 1e6, Q = 1e5): ground truth for a whole batch.
        {"name": "exact_batch", "op": "search", "mode": "exact", "n": 1_000_000, "nq": 100_000, "k": 100,
         "host": False, **PLAIN},
        # A small serving batch of the reduced-precision form: what the request
        # loop dispatches at low load, another size each time (host-planned).
        {"name": "bf16_online", "op": "search", "mode": "bf16", "kprime": 112, "graph": False, "n": 1_000_000,
         "nq": 50, "k": 100, "host": False, **UNEVEN},
        # The request loop's largest batch (4,096) on the uneven-selectivity workload.
        {"name": "bf16_serving", "op": "search", "mode": "bf16", "kprime": 200, "graph": False, "n": 2_000_000,
         "nq": 4096, "k": 100, "host": False, **UNEVEN},
        # The precision workload: a large offline batch, planned on the device,
        # one captured graph, the tuning table's k'.
        {"name": "bf16_batch", "op": "search", "mode": "bf16", "kprime": 112, "graph": True, "n": 4_000_000,
         "nq": 100_000, "k": 100, "host": False, **PLAIN},
        # Predicate evaluation + row compaction over whole columns, eight predicates a call.
        {"name": "filter_preds", "op": "filter", "n": 4_000_000, "np": 8, **PLAIN},
        # The SQ8 slab brute force over the largest slab the reference's router
        # sends there (4.5 % of 1e7 rows), a batch and the reference's own
        # one-query call.
        {"name": "sq8_batch", "op": "sq8", "n": 450_000, "nq": 2048, "k": 140, **PLAIN},
        {"name": "sq8_single", "op": "sq8", "n": 450_000, "nq": 1, "k": 140, **PLAIN},
        # A category graph searched with the reference's SearchFilter, its
        # candidates re-ranked in FP32 (the category route of BatchSearch).
        {"name": "graph_rerank", "op": "graph", "form": "filter", "n": 100_000, "nq": 10_000, "pool": 256,
         "refine": 150, **PLAIN},
        # A time-bucket graph under windows of the widths the router sends to
        # SearchRangeFilterSubTime (a fifth of the bucket's rows and more).
        {"name": "graph_window", "op": "graph", "form": "range", "n": 100_000, "nq": 3000, "pool": 680,
         "refine": 150, **BUCKET},
        # HybridGraph::BatchSearch: every route, host arrays in and out.
        {"name": "batch_search", "op": "router", "n": 200_000, "nq": 2000, **UNEVEN},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["exact", "exact", "bf16", "bf16", "filter", "sq8", "sq8", "graph", "graph", "router"])
    data = dict(rng.choice([PLAIN, UNEVEN]))
    if op in ("exact", "bf16"):
        top = 1_000_000 if op == "exact" else 4_000_000
        n = _log_int(rng, 100_000, top)
        nq = _log_int(rng, 1, 100_000)
        c = {"op": "search", "mode": op, "n": n, "nq": nq, "k": rng.choice([10, 100, 100, 100, 128]),
             "host": rng.random() < 0.3, **data}
        if op == "bf16":
            c.update(kprime=rng.choice([130, 200, 400]), graph=rng.random() < 0.5, host=False)
        return c
    if op == "filter":
        return {"op": "filter", "n": _log_int(rng, 50_000, 4_000_000), "np": rng.randint(1, 24), **data}
    if op == "sq8":
        return {"op": "sq8", "n": _log_int(rng, 2_000, 450_000), "nq": _log_int(rng, 1, 4096),
                "k": rng.randint(100, 200), **data}
    if op == "graph":
        pool = _log_int(rng, 64, 1024)
        form = rng.choice(["filter", "range"])
        if form == "range":
            data = BUCKET
        return {"op": "graph", "form": form, "n": _log_int(rng, 10_000, 100_000), "nq": _log_int(rng, 50, 10_000),
                "pool": pool, "refine": min(150, pool), **data}
    return {"op": "router", "n": _log_int(rng, 100_000, 200_000), "nq": _log_int(rng, 100, 2000), **UNEVEN}


# ------------------------------------------------------------------ data --


def _category_p(case):
    p = np.arange(1, case["labels"] + 1, dtype=np.float64) ** -case["zipf"]
    return p / p.sum()


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 7919 + 17)
    return g


def _mixture(centres, m, g):
    c = torch.randint(0, centres.shape[0], (m,), generator=g, device="cuda")
    x = torch.randn((m, DIM), generator=g, device="cuda")
    return x.mul_(0.3).add_(centres[c])


def _base(case, g):
    """centres, rows (n, 100), categories (n,), timestamps (n,) on the GPU."""
    n = case["n"]
    centres = torch.randn((256, DIM), generator=g, device="cuda")
    vecs = torch.empty((n, DIM), device="cuda")
    for s in range(0, n, 1 << 20):
        e = min(n, s + (1 << 20))
        vecs[s:e] = _mixture(centres, e - s, g)
    cum = torch.from_numpy(np.cumsum(_category_p(case))).cuda()
    u = torch.rand((n,), generator=g, device="cuda", dtype=torch.float64)
    labels = torch.searchsorted(cum, u).clamp_(max=case["labels"] - 1).float()
    ts = torch.rand((n,), generator=g, device="cuda")
    return centres, vecs, labels, ts


def _windows(case, m, g):
    u = torch.rand((m,), generator=g, device="cuda", dtype=torch.float64)
    if case["window"] == "uniform":
        w = 0.05 + 0.45 * u
    elif case["window"] == "bucket":
        w = 0.2 + 0.75 * u
    else:
        w = torch.exp(math.log(1e-4) * u)
    lo = torch.rand((m,), generator=g, device="cuda", dtype=torch.float64) * (1.0 - w)
    return lo, lo + w


def _metas(case, m, g):
    """(m, 4) predicates (type, v, l, r); types a shuffled 0..3 cycle."""
    types = (torch.randperm(m, generator=g, device="cuda") % 4).float()
    cum = torch.from_numpy(np.cumsum(_category_p(case))).cuda()
    u = torch.rand((m,), generator=g, device="cuda", dtype=torch.float64)
    v = torch.searchsorted(cum, u).clamp_(max=case["labels"] - 1).float()
    lo, hi = _windows(case, m, g)
    none = torch.full((m,), -1.0, device="cuda")
    by_cat = (types == 1) | (types == 3)
    by_ts = types >= 2
    return torch.stack([types, torch.where(by_cat, v, none), torch.where(by_ts, lo.float(), none),
                        torch.where(by_ts, hi.float(), none)], 1).contiguous()


def _inputs(case, seed):
    """The base and the queries of a case, on the GPU."""
    g = _gen(seed)
    centres, vecs, labels, ts = _base(case, g)
    nq = case.get("nq", 0)
    q = _mixture(centres, nq, g) if nq else None
    metas = _metas(case, case.get("np", nq), g)
    return vecs, labels, ts, q, metas, g


def _host(*xs):
    return [x.cpu().numpy() for x in xs]


# ---------------------------------------------------------------- graphs --


def _near(x, idx, near, far, g):
    """For the rows idx of x: their `near` nearest rows of idx and `far` random
    ones (positions in x), the links of a navigable graph."""
    sub = x[idx]
    m = idx.shape[0]
    near = min(near, max(1, m - 1))
    norm = (sub * sub).sum(1)
    out = torch.empty((m, near + far), dtype=torch.int64, device="cuda")
    step = max(1, min(m, (1 << 28) // max(1, m)))
    for s in range(0, m, step):
        e = min(m, s + step)
        d = torch.addmm(norm[None, :], sub[s:e], sub.T, alpha=-2.0)
        d[torch.arange(e - s, device="cuda"), torch.arange(s, e, device="cuda")] = math.inf
        out[s:e, :near] = d.topk(near, dim=1, largest=False).indices
    out[:, near:] = torch.randint(0, m, (m, far), generator=g, device="cuda")
    return idx[out]


def _graph_bytes(x, ts, g, degree=32):
    """A saved graph (Graph::save layout) over the rows of x: out-degree 32 at
    level 0, edge timestamps those of the neighbours, and the sparser upper
    layers (one row in 16 a level) the search descends through."""
    n = x.shape[0]
    every = torch.arange(n, device="cuda")
    adj = _near(x, every, degree - 8, 8, g)
    if adj.shape[1] < degree:
        adj = torch.nn.functional.pad(adj, (0, degree - adj.shape[1]), value=-1)
    ets = ts[adj.clamp(min=0)]
    up = 16
    level = torch.zeros(n, dtype=torch.int64, device="cuda")
    idx, lists = every, []
    while idx.shape[0] >= 512 and len(lists) < 4:
        idx = idx[torch.rand((idx.shape[0],), generator=g, device="cuda") < 1 / 16]
        if idx.shape[0] < 2 * up:
            break
        level[idx] += 1
        lists.append((idx, _near(x, idx, 12, 4, g)))
    ep = int(torch.argmax(level))
    cnt = (level * up).cpu().numpy()
    off = np.concatenate([[0], np.cumsum(cnt + 1)])
    words = np.full(off[-1], -1, np.int32)
    words[off[:-1]] = cnt
    for lv, (rows, nb) in enumerate(lists):
        at = off[rows.cpu().numpy()] + 1 + lv * up
        words[at[:, None] + np.arange(up)[None, :]] = nb.cpu().numpy()
    head = np.array([0, n, degree], np.int32)
    return b"".join([head.tobytes(), adj.to(torch.int32).cpu().numpy().tobytes(),
                     ets.float().contiguous().cpu().numpy().tobytes(), np.array([n, up, ep], np.int32).tobytes(),
                     words.tobytes()])


# --------------------------------------------------------------- prepare --


def prepare(case, seed):
    vecs, labels, ts, q, metas, g = _inputs(case, seed)
    op = case["op"]
    if op == "search":
        mode = fknn.MODE_EXACT_FP32 if case["mode"] == "exact" else fknn.MODE_BF16_RERANK
        hv, hl, ht = _host(vecs, labels, ts)
        del vecs
        idx = fknn.Index(hv, hl, ht, device=0, build_bf16=case["mode"] == "bf16")
        idx.apply_tuning(mode)
        if case["host"]:
            q, metas = _host(q, metas)
        st = {"case": case, "index": idx, "q": q, "metas": metas, "mode": mode}
        if case.get("graph"):  # a captured search is replayed into buffers that the program keeps
            st["ids"] = torch.empty((case["nq"], case["k"]), dtype=torch.int32, device="cuda")
            st["dists"] = torch.empty((case["nq"], case["k"]), dtype=torch.float32, device="cuda")
        return st
    if op == "filter":
        hv, hl, ht = _host(vecs, labels, ts)
        del vecs
        idx = fknn.Index(hv, hl, ht, device=0)
        np_ = case["np"]
        return {"case": case, "index": idx, "metas": metas.cpu().numpy(),
                "out": torch.zeros((np_, case["n"]), dtype=torch.int32, device="cuda"),
                "counts": torch.zeros(np_, dtype=torch.int64, device="cuda")}
    if op == "sq8":
        quant = fknn.SQ8SymmetricQuantizer(DIM)
        quant.train(vecs.cpu().numpy())
        qc = quant.encode(q.cpu().numpy())
        nq, k = case["nq"], case["k"]
        return {"case": case, "alpha": float(quant.alpha), "codes": torch.from_numpy(quant.codes).cuda(),
                "q": torch.from_numpy(qc).cuda(), "out": torch.empty((nq, k), dtype=torch.int32, device="cuda"),
                "dists": torch.empty((nq, k), dtype=torch.float32, device="cuda")}
    if op == "graph":
        order = torch.argsort(ts)
        vecs, labels, ts = vecs[order].contiguous(), labels[order], ts[order]
        gs = fknn.GraphSearcher(_graph_bytes(vecs, ts, g), vecs)
        st = {"case": case, "graph": gs, "q": q}
        if case["form"] == "filter":
            st["index"] = fknn.Index(*_host(vecs, labels, ts), device=0)
        else:
            lo, hi = _windows(case, case["nq"], g)
            b = torch.stack([lo.float(), hi.float()], 1).contiguous()
            s = torch.searchsorted(ts, b[:, 0].contiguous()).clamp_(max=case["n"] - 1)
            e = torch.searchsorted(ts, b[:, 1].contiguous(), right=True)
            st["bounds"] = b
            st["id_bounds"] = torch.stack([s, torch.maximum(e - 1, s)], 1).to(torch.int32).contiguous()
        return st
    # router: the reference's sub-indexes -- a graph for the largest
    # categories and one per tenth of the time range
    hv, hl, ht = _host(vecs, labels, ts)
    by_cat = np.lexsort((ht, hl)).astype(np.uint32)
    by_time = np.argsort(ht, kind="stable").astype(np.uint32)
    vals, start, count = np.unique(hl[by_cat], return_index=True, return_counts=True)
    cats, buckets = [], []
    for v, s, c in zip(vals, start, count):
        if c >= 0.045 * case["n"]:
            rows = torch.from_numpy(by_cat[s:s + c].astype(np.int64)).cuda()
            cats.append((int(v), int(s), int(c), _graph_bytes(vecs[rows], ts[rows], g)))
    tt = ht[by_time]
    for b in range(10):
        s = int(np.searchsorted(tt, np.float32(b / 10), "left"))
        e = case["n"] if b == 9 else int(np.searchsorted(tt, np.float32((b + 1) / 10), "left"))
        rows = torch.from_numpy(by_time[s:e].astype(np.int64)).cuda()
        buckets.append((b, s, e - s, _graph_bytes(vecs[rows], ts[rows], g)))
    r = fknn.Router(hv, hl, ht, by_cat, by_time, cats, buckets, int(count.max()), int(count.min()))
    p = fknn.Router.default_params()
    p.sel_rows = case["n"]
    return {"case": case, "router": r, "params": p, "q": q.cpu().numpy(), "metas": metas.cpu().numpy()}


# ------------------------------------------------------------------- run --


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "search":
        return state["index"].search(state["q"], state["metas"], k=case["k"], mode=state["mode"],
                                     kprime=case.get("kprime", 0), graph=case.get("graph", False),
                                     ids=state.get("ids"), dists=state.get("dists"))
    if op == "filter":
        return state["index"].filter_rows_batch(state["metas"], out=state["out"], counts=state["counts"])
    if op == "sq8":
        fknn.bruteforce_subgraph(DIM, case["k"], state["out"], state["dists"], case["n"], state["codes"],
                                 state["alpha"], case["nq"], state["q"])
        return state["out"], state["dists"]
    if op == "graph":
        if case["form"] == "filter":
            cand = state["graph"].SearchFilter(state["q"], case["pool"], case["refine"])
            return (cand,) + tuple(state["index"].rerank(state["q"], cand, k=min(100, case["refine"])))
        return state["graph"].SearchRangeFilterSubTime(state["q"], case["pool"], case["refine"], state["bounds"],
                                                       state["id_bounds"])
    return state["router"].search(state["q"], state["metas"], state["params"])[0]


# ------------------------------------------------------------------ work --


def _selectivity(case):
    """Mean share of the rows that pass a predicate, by type."""
    p = _category_p(case)
    cat = float((p * p).sum())
    win = 0.275 if case["window"] == "uniform" else (1 - 1e-4) / math.log(1e4)
    return [1.0, cat, win, cat * win]


def work(case):
    op = case["op"]
    n, nq = case["n"], case.get("nq", 0)
    if op == "search":
        # 200 operations per (query, passing row) pair; rows, attributes and
        # queries read once, ids and distances written once
        pairs = nq * n * sum(_selectivity(case)) / 4
        row = 2 * DIM if case["mode"] == "bf16" else 4 * DIM
        return {"bytes": n * (row + 8) + nq * (4 * DIM + 16) + nq * case["k"] * 8, "flops": 2 * DIM * pairs}
    if op == "filter":
        passing = n * case["np"] * sum(_selectivity(case)) / 4
        return {"bytes": 8 * n + 4 * passing, "flops": 4 * n * case["np"]}
    if op == "sq8":
        return {"bytes": (n + nq) * CODE + nq * case["k"] * 8, "flops": 2 * DIM * n * nq}
    if op == "graph":
        # every pool slot was scored once and expanded once: a code per slot,
        # its neighbour list (and their timestamps under a window)
        per = case["pool"] * (CODE + 4 * 32 * (1 if case["form"] == "filter" else 2))
        rr = case["refine"] * 4 * DIM if case["form"] == "filter" else 0
        return {"bytes": nq * (4 * DIM + per + rr + case["refine"] * 8),
                "flops": nq * 2 * DIM * (case["pool"] + (case["refine"] if rr else 0))}
    # router: at least the pool of one graph search or of one slab per query,
    # and its re-rank
    return {"bytes": n * CODE + nq * (4 * DIM + 16 + 150 * 4 * DIM + 400), "flops": nq * 2 * DIM * (2000 + 150)}


# ----------------------------------------------------------------- exact --


def exact(case, seed):
    """The k smallest distances of each query over its passing rows, in 64
    bits (the ids have no such value).  Only the searches return distances
    that plain arithmetic can give; the pass is left out where it is long."""
    if case["op"] != "search" or case["n"] * case["nq"] > 120_000_000_000:
        return None
    vecs, labels, ts, q, metas, _ = _inputs(case, seed)
    x = vecs.double()
    xn = (x * x).sum(1)
    n, nq, k = case["n"], case["nq"], case["k"]
    out = torch.empty((nq, k), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 28) // n)
    for s in range(0, nq, step):
        e = min(nq, s + step)
        y, m = q[s:e].double(), metas[s:e]
        d = torch.addmm(xn[None, :], y, x.T, alpha=-2.0).add_((y * y).sum(1)[:, None])
        t = m[:, :1]
        fail = ((t == 1) | (t == 3)) & (labels[None, :] != m[:, 1:2])
        fail |= (t >= 2) & ((ts[None, :] < m[:, 2:3]) | (ts[None, :] > m[:, 3:4]))
        d.masked_fill_(fail, math.inf)
        out[s:e] = d.topk(k, dim=1, largest=False).values
    return None, (out.cpu().numpy() if case["host"] else out)
