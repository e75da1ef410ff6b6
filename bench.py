"""Benchmark of the filtered-kNN hot path on B200.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Workload (default): the precision configuration the recall-gated metric is
quoted on -- N=10,000,000 base rows, d=100 float32 (256-cluster Gaussian
mixture), category ~ Zipf(1.1) over 1,000 values, timestamp ~ U[0,1];
Q=1,000,000 queries of uniform type 0..3 per step, k=100 (--config 2 gives
N=1e6, Q=1e5).  One step = one fknn_search over the whole query batch.  The
row orders (2 x 4.04 GB FP32, 2 x 2.29 GB BF16) are far larger than the
126 MB L2, so steps are not served from cache.

Both forms run on the same queries: the exact FP32 path (ids bit-identical
to the reference brute force) and the BF16 tensor-core screen + FP32
re-rank (k' from the autotuner's table, or --kprime).  The headline is the
BF16 form when its recall@100 against the exact path's ids over all queries
is >= 0.99, else the exact path.  The exact leg, ~16 s per step at the
default size, is timed over --exact-steps steps after one warm-up step.
Recall of both forms against an FP64 oracle sample is in the line too.

Printed: one JSON line (rank 0).  value = queries/s with inputs resident in
HBM; e2e = the same through the C ABI with pinned host buffers (H2D of the
queries and predicates, D2H of the ids -- the result the reference's batch
interface returns -- inside the timed region).  Multi-GPU runs
replicate the base and give every rank its own query batch (weak scaling,
no data-path collective).
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "sigmod-2024-contest_b200"))
sys.path.insert(0, os.path.join(ROOT, "oracle"))

import numpy as np  # noqa: E402

METRIC = "filtered queries/s at recall@100≥0.99 vs exact-FP32 GPU; p50/p99 latency, 1×B200"
UNIT = "queries/s"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--config", type=int, default=3)
    ap.add_argument("--n", type=int, default=None, help="override base rows (smaller runs)")
    ap.add_argument("--nq", type=int, default=None, help="override queries per step")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--cpu-sample", type=int, default=0,
                    help="queries in the CPU-baseline sample (default: about 10 s of reference work)")
    ap.add_argument("--exact-steps", type=int, default=0,
                    help="timed steps of the exact leg (default: --steps when a step is short, else 2)")
    ap.add_argument("--kprime", type=int, default=None,
                    help="candidate width of the BF16 form (default: the autotuned one, else 200)")
    ap.add_argument("--sweep", action="store_true",
                    help="precision sweep instead of the headline: exact, BF16 and FP8 forms at k' in "
                         "--kprimes, recall and distance error against an FP64 oracle sample; one JSON line each")
    ap.add_argument("--kprimes", default="200,400,800")
    ap.add_argument("--f64-sample", type=int, default=128, help="queries checked against the FP64 oracle")
    ap.add_argument("--serve", action="store_true",
                    help="request-loop run instead of the headline: Poisson arrivals at --rates per form; "
                         "one JSON line per (form, rate)")
    ap.add_argument("--rates", default="10000,50000,200000")
    ap.add_argument("--serve-seconds", type=float, default=2.0)
    ap.add_argument("--serve-forms", default="bf16,exact")
    ap.add_argument("--filter", action="store_true",
                    help="predicate-compaction run instead of the headline: fknn_filter_rows over the base for a "
                         "sample of the workload's predicates; HBM GB/s of algorithmic bytes")
    ap.add_argument("--sq8", action="store_true",
                    help="SQ8 slab brute force instead of the headline (bruteforce.h:244 with K'=140): codes/s and "
                         "GB/s over a slab of 4.5 %% of N=1e7 codes, batched queries")
    ap.add_argument("--sq8-callers", type=int, default=0,
                    help="with --sq8: this many host threads each calling with one query at a time, as the "
                         "reference's OpenMP workers do (hybrid_graph.cpp:211)")
    ap.add_argument("--graph", action="store_true",
                    help="graph-path run instead of the headline: per-category HNSW graphs (reference build), "
                         "batched beam search + FP32 re-rank, recall against the exact path; one JSON line per beam")
    ap.add_argument("--plan", choices=["graph", "host"], default="graph",
                    help="BF16 leg: plan on the device and replay a captured CUDA graph, or plan on the host")
    ap.add_argument("--router", action="store_true",
                    help="reference-routing run instead of the headline: fknn_router beside the reference pipeline's "
                         "BatchSearch over the same subgraphs; q/s and recall per query type")
    ap.add_argument("--graph-beams", default="64,128,256,512")
    ap.add_argument("--graph-cats", type=int, default=8, help="largest categories that get a graph")
    a = ap.parse_args()
    a.kprime_set = a.kprime is not None
    if a.kprime is None:
        a.kprime = 200
    return a


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled every 200 ms."""
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index: int):
        self.dev = device_index
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.p = None

    def start(self):
        try:
            self.p = subprocess.Popen(["nvidia-smi", "-i", str(self.dev), f"--query-gpu={self.FIELDS}",
                                       "--format=csv,noheader,nounits", "-lms", "200"], stdout=self.f,
                                      stderr=subprocess.DEVNULL)
        except OSError:
            self.p = None

    def stop(self) -> dict:
        if self.p is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.p.terminate()
        try:
            self.p.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.p.kill()
        self.f.flush()
        self.f.seek(0)
        rows = [r.split(",") for r in self.f.read().strip().splitlines() if r.strip()]
        os.unlink(self.f.name)
        sm, smax, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            try:
                sm.append(float(r[1]))
                smax = float(r[2])
                for nm, v in zip(names, r[5:9]):
                    if v.strip().lower() == "active":
                        reasons.add(nm)
            except (ValueError, IndexError):
                continue
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": smax, "reasons": sorted(reasons),
                "samples": len(sm)}


def measured_peaks() -> dict:
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return json.load(f)
    except OSError:
        return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "fallback": True}


def fp32_gemm_peak_tflops(torch) -> float:
    """Measured FP32 CUDA-core throughput: cuBLAS SGEMM with TF32 off, 8192^3."""
    prev = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    a = torch.randn(8192, 8192, device="cuda")
    b = torch.randn(8192, 8192, device="cuda")
    for _ in range(2):
        torch.matmul(a, b)
    best = 1e9
    for _ in range(5):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        torch.matmul(a, b)
        e.record()
        e.synchronize()
        best = min(best, s.elapsed_time(e))
    torch.backends.cuda.matmul.allow_tf32 = prev
    del a, b
    return 2 * 8192 ** 3 / (best * 1e-3) / 1e12


def traffic_per_pair(name: str = "k_exact_screen_traffic.json"):
    """DRAM bytes per screened (query, row) pair of a screening kernel,
    from the committed ncu summary (None if not measured yet)."""
    p = os.path.join(ROOT, "profiles", name)
    try:
        with open(p) as f:
            return json.load(f).get("dram_bytes_per_screened_pair")
    except OSError:
        return None


def default_cpu_sample(n: int) -> int:
    """Queries in the CPU-baseline sample: about 10 s of the reference's
    Bruteforce on 16 host cores (2.2 ms per query per 1e6 rows measured)."""
    return int(min(4096, max(64, 4.5e9 / max(n, 1))))


def cpu_baseline(vecs, labels, ts, q, metas, sample: int, kind_pref: str = "reference") -> dict:
    """The reference Bruteforce (utils.h:80) compiled from its sources
    (oracle/_ref) on all host cores, on a bounded sample of the workload's
    queries (those with >= 100 passing rows: the reference throws on the
    others).  Falls back to the oracle restatement if _ref is absent."""
    import ctypes

    import oracle
    from fknn import datagen
    counts = oracle.count_matches_sorted(labels, ts, metas)
    ok = np.nonzero(counts >= 100)[0]
    rng = np.random.default_rng(99)
    sel = np.sort(rng.choice(ok, size=min(sample, len(ok)), replace=False))
    R = oracle.ref_exact() if kind_pref == "reference" else None
    cores = os.cpu_count() or 1
    if R is not None:
        rows = datagen.to_rows(vecs, labels, ts)
        qrows = datagen.to_query_rows(q[sel], metas[sel])
        gt = np.empty((len(sel), 100), dtype=np.uint32)
        secs = ctypes.c_double()
        rc = R.ref_exact_bruteforce(rows.ctypes.data, rows.shape[0], qrows.ctypes.data, len(sel), gt.ctypes.data,
                                    ctypes.byref(secs))
        if rc != 0:
            raise RuntimeError("reference Bruteforce failed")
        t = secs.value
        kind = "reference"
    else:
        t0 = time.perf_counter()
        oracle.exact_knn(vecs, labels, ts, q[sel], metas[sel], nthreads=cores)
        t = time.perf_counter() - t0
        kind = "port"
    return {"value": len(sel) / t, "unit": UNIT, "cores": cores, "kind": kind,
            "sample": f"{len(sel)} seeded-random queries of the workload with >=100 passing rows, "
                      f"full N={vecs.shape[0]} scan each; {t:.2f} s"}


def run_reference(args, rank: int, world: int):
    """--impl reference: the reference's own CPU Bruteforce (utils.h:80) on
    the host cores, rank 0 only, bounded samples per step."""
    if rank != 0:
        return
    import ctypes

    import oracle
    from fknn import datagen
    vecs, labels, ts, q, metas = datagen.make_workload(args.config, n=args.n, nq=args.nq)
    cfg = {"workload": datagen.WORKLOADS[args.config].name, "n": int(vecs.shape[0]), "nq": int(q.shape[0]), "k": 100}
    counts = oracle.count_matches_sorted(labels, ts, metas)
    ok = np.nonzero(counts >= 100)[0]
    R = oracle.ref_exact()
    kind = "reference" if R is not None else "port"
    cores = os.cpu_count() or 1
    # about a second of reference work per step (256 queries at N=1e6, 45 at N=1e7)
    per_step = int(min(256, max(16, 4.5e8 / vecs.shape[0])))
    rng = np.random.default_rng(5)
    rows = datagen.to_rows(vecs, labels, ts)
    times = []
    for step in range(args.warmup + args.steps):
        sel = np.sort(rng.choice(ok, size=min(per_step, len(ok)), replace=False))
        if R is not None:
            qrows = datagen.to_query_rows(q[sel], metas[sel])
            gt = np.empty((len(sel), 100), dtype=np.uint32)
            secs = ctypes.c_double()
            if R.ref_exact_bruteforce(rows.ctypes.data, rows.shape[0], qrows.ctypes.data, len(sel), gt.ctypes.data,
                                      ctypes.byref(secs)) != 0:
                raise RuntimeError("reference Bruteforce failed")
            t = secs.value
        else:
            t0 = time.perf_counter()
            oracle.exact_knn(vecs, labels, ts, q[sel], metas[sel], nthreads=cores)
            t = time.perf_counter() - t0
        if step >= args.warmup:
            times.append(t)
    per_step = int(min(per_step, len(ok)))
    mean_t = sum(times) / len(times)
    value = per_step / mean_t
    sample = f"{per_step} seeded-random queries with >=100 passing rows per step, full N={vecs.shape[0]} scan each"
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": mean_t * 1e3, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic", "config": cfg,
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": kind, "sample": sample},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "latency_ms": {"p50": statistics.median(times) * 1e3,
                           "p99": float(np.percentile(np.array(times) * 1e3, 99))}}
    print(json.dumps(line), flush=True)


def run_sweep(args):
    """Per form and k': queries/s (inputs resident), recall@100 against the
    exact GPU path over all queries and against the FP64 oracle on a seeded
    sample, and the distance error against FP64: max relative error of the
    returned distances (FP64 recomputed for the same ids) and of the k-th
    distance (against the FP64 oracle's k-th)."""
    import torch

    import fknn
    import oracle
    from fknn import datagen
    torch.cuda.set_device(0)
    w = datagen.WORKLOADS[args.config]
    n, nq = args.n or w.n, args.nq or w.nq
    vecs, labels, ts, q, metas = datagen.make_workload(args.config, n=n, nq=nq)
    idx = fknn.Index(vecs, labels, ts, build_bf16=True, build_fp8=True)
    for md in (fknn.MODE_EXACT_FP32, fknn.MODE_BF16_RERANK, fknn.MODE_FP8_RERANK):
        idx.apply_tuning(md)  # plan / kernel parameters only; k' is swept here
    stream = torch.cuda.current_stream()
    dq, dm = torch.from_numpy(q).cuda(), torch.from_numpy(metas).cuda()
    rng = np.random.default_rng(17)
    sel = np.sort(rng.choice(nq, size=min(args.f64_sample, nq), replace=False))
    t0 = time.perf_counter()
    o_ids, o_d = oracle.exact_knn(vecs, labels, ts, q[sel], metas[sel], f64=True)
    t_oracle = time.perf_counter() - t0

    def run(mode, kprime):
        ids = torch.empty((nq, 100), dtype=torch.int32, device="cuda")
        dd = torch.empty((nq, 100), dtype=torch.float32, device="cuda")
        graph = args.plan == "graph" and mode != fknn.MODE_EXACT_FP32
        for _ in range(args.warmup):
            idx.search(dq, dm, k=100, mode=mode, kprime=kprime, ids=ids, dists=dd, stream=stream.cuda_stream,
                       graph=graph)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(args.steps):
            idx.search(dq, dm, k=100, mode=mode, kprime=kprime, ids=ids, dists=dd, stream=stream.cuda_stream,
                       graph=graph)
        e1.record(stream)
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / args.steps, ids.cpu().numpy().view(np.uint32).copy(), dd.cpu().numpy()

    def errors(ids, dd):
        s_ids, s_d = ids[sel], dd[sel]
        valid = s_ids != 0xFFFFFFFF
        x = vecs[np.where(valid, s_ids, 0)].astype(np.float64)
        d64 = ((x - q[sel][:, None, :].astype(np.float64)) ** 2).sum(-1)
        rel = np.abs(s_d.astype(np.float64) - d64) / np.maximum(d64, 1e-30)
        o_valid = o_ids != 0xFFFFFFFF
        kth = []
        for i in range(len(sel)):
            m = int(min(valid[i].sum(), o_valid[i].sum()))
            if m:
                kth.append(abs(float(s_d[i, m - 1]) - float(o_d[i, m - 1])) / max(float(o_d[i, m - 1]), 1e-30))
        return {"recall_at_100_vs_f64_oracle": datagen.recall_matrix(s_ids, o_ids),
                "max_rel_dist_error_returned": float(rel[valid].max()) if valid.any() else 0.0,
                "max_rel_kth_dist_error": max(kth) if kth else 0.0}

    ms_e, ids_e, d_e = run(fknn.MODE_EXACT_FP32, 0)
    base = {"config": {"workload": w.name, "n": n, "nq": nq, "k": 100, "d": 100},
            "f64_sample": {"queries": int(len(sel)), "oracle_seconds": t_oracle}}
    print(json.dumps({**base, "form": "exact_fp32", "kprime": None, "value": nq / (ms_e * 1e-3), "unit": UNIT,
                      "ms_per_step": ms_e, "recall_at_100_vs_exact_gpu": 1.0, **errors(ids_e, d_e)}), flush=True)
    for mode, name in ((fknn.MODE_BF16_RERANK, "bf16_rerank"), (fknn.MODE_FP8_RERANK, "fp8_rerank")):
        for kp in [int(x) for x in args.kprimes.split(",")]:
            ms, ids, dd = run(mode, kp)
            print(json.dumps({**base, "form": name, "kprime": kp, "value": nq / (ms * 1e-3), "unit": UNIT,
                              "ms_per_step": ms, "speedup_vs_exact": ms_e / ms,
                              "recall_at_100_vs_exact_gpu": datagen.recall_matrix(ids, ids_e),
                              **errors(ids, dd)}), flush=True)
    idx.close()


def run_serve(args):
    """The request loop (fknn.Server) under Poisson arrivals: for each form
    and rate, requests (one query each, config-4/5 generator) arrive for
    --serve-seconds; a client thread submits each due request with its
    arrival stamp, so queueing before submission counts as latency.  Reports
    p50/p99 latency (arrival -> result), sustained queries/s (results / first
    arrival to last result) and recall@100 of the served ids against the
    exact path's ids for the same queries."""
    import torch

    import fknn
    from fknn import datagen
    torch.cuda.set_device(0)
    cfg = 5 if args.config == 2 else args.config
    w = datagen.WORKLOADS[cfg]
    n = args.n or w.n
    rates = [int(x) for x in args.rates.split(",")]
    nreq = int(max(rates) * args.serve_seconds) + 1
    vecs, labels, ts, q, metas = datagen.make_workload(cfg, n=n, nq=nreq)
    idx = fknn.Index(vecs, labels, ts, build_bf16=True)
    idx.apply_tuning(fknn.MODE_EXACT_FP32)
    kp_tuned = idx.apply_tuning(fknn.MODE_BF16_RERANK)
    exact_ids, _ = idx.search(q, metas, k=100, mode=fknn.MODE_EXACT_FP32)
    kp = args.kprime if args.kprime_set or not kp_tuned else kp_tuned
    forms = {"bf16": (fknn.MODE_BF16_RERANK, kp), "exact": (fknn.MODE_EXACT_FP32, 0)}
    for fname in args.serve_forms.split(","):
        mode, kp = forms[fname]
        with fknn.Server(idx, mode=mode, kprime=kp, max_batch=4096, slots=3) as srv:
            # size every slot's scratch for a full batch of each query type first
            for t in range(4):
                sel = np.nonzero(metas[:, 0] == t)[0][:4096]
                for _ in range(3):
                    srv.submit(q[sel], metas[sel], with_dists=False)
            srv.drain()
            srv.stats(reset=True)
            for rate in rates:
                m = int(rate * args.serve_seconds)
                rng = np.random.default_rng(rate)
                arr = np.cumsum(rng.exponential(1e9 / rate, m)).astype(np.int64)
                ids = np.empty((m, 100), dtype=np.uint32)
                t0 = srv.now_ns() + 1_000_000
                arr += t0
                i = 0
                while i < m:
                    now = srv.now_ns()
                    j = int(np.searchsorted(arr, now, side="right"))
                    if j > i:
                        srv.submit(q[i:j], metas[i:j], arrival_ns=arr[i:j], with_dists=False, ids=ids[i:j])
                        i = j
                    else:
                        time.sleep(max(0.0, min(2e-4, (arr[i] - now) * 1e-9)))
                srv.drain()
                st = srv.stats(reset=True)
                rec = datagen.recall_matrix(ids, exact_ids[:m].view(np.uint32))
                print(json.dumps({
                    "mode": "serve", "form": fname, "kprime": kp or None,
                    "config": {"workload": w.name, "n": n, "k": 100, "d": 100, "arrivals": "poisson",
                               "offered_qps": rate, "seconds": args.serve_seconds, "requests": m,
                               "max_batch": 4096, "slots": 3},
                    "sustained_qps": st["qps"], "p50_ms": st["p50_ms"], "p99_ms": st["p99_ms"],
                    "max_ms": st["max_ms"], "mean_batch": st["mean_batch"], "batches": st["batches"],
                    "admission_waits": st["admission_waits"], "budget_trims": st["budget_trims"],
                    "scratch_bytes": st["scratch_bytes"], "recall_at_100_vs_exact": rec}), flush=True)
    idx.close()


def run_graph(args):
    """Per-category graph search (config-4 generator, Zipf 1.5 over 10,000
    categories): one graph of out-degree 32 per large category, built by the
    reference's HNSW::Build (oracle/_ref) over that category's rows in
    timestamp order (the order the reference's category searchers hold,
    utils.h:395-425).  Type-1 queries of those categories search their
    category's graph with SearchFilter and type-3 queries with
    SearchCategoryRange (the window and its row range seed the pool,
    searcher.hpp:301-374), pool = beam; their refine = min(150, beam)
    candidates are re-ranked in FP32 on the GPU (fknn_rerank), and recall@100
    is taken per type against the exact path's ids, over all of them and
    over those the reference's BatchSearch routes to a category graph
    (selectivity >= 0.045 for type 1, >= 0.08 for type 3; the narrower
    windows go to its slab brute force).  queries/s counts the
    graph searches plus the re-ranks, inputs resident.  The reference
    Searcher is timed on a sample of the largest category's type-1 queries
    on one host thread."""
    import torch

    import fknn
    import oracle
    from fknn import datagen
    torch.cuda.set_device(0)
    R = oracle.ref_graph()
    if R is None:
        print(json.dumps({"mode": "graph", "unavailable": "reference graph build (oracle/_ref/libref_graph.so) not built"}))
        return
    n = args.n or 1_000_000
    nq_all = args.nq or 200_000
    vecs, labels, ts, q, metas = datagen.make_workload(4, n=n, nq=nq_all)
    lab = labels.astype(np.int64)
    counts = np.bincount(lab)
    cats = np.argsort(-counts, kind="stable")[:args.graph_cats]
    idx = fknn.Index(vecs, labels, ts)
    graphs, t_build = {}, 0.0
    tmp = tempfile.mkdtemp()
    for c in cats:
        rows = np.nonzero(lab == c)[0]
        rows = rows[np.argsort(ts[rows], kind="stable")]
        t0 = time.perf_counter()
        gb = oracle.ref_hnsw_graph(vecs[rows], ts[rows], 32, 100, os.path.join(tmp, f"g{c}.bin"))
        t_build += time.perf_counter() - t0
        graphs[int(c)] = (rows, fknn.GraphSearcher(gb, vecs[rows]), os.path.join(tmp, f"g{c}.bin"))
    catq = np.isin(metas[:, 1].astype(np.int64), cats)
    sel = np.nonzero(((metas[:, 0] == 1) | (metas[:, 0] == 3)) & catq)[0]
    qs, ms = q[sel], metas[sel]
    exact_ids, _ = idx.search(qs, ms, k=100, mode=fknn.MODE_EXACT_FP32)
    passing = idx.count_matches(ms).astype(np.int64)
    groups = {}
    for c in cats:
        for t in (1, 3):
            ix = np.nonzero((ms[:, 1].astype(np.int64) == c) & (ms[:, 0] == t))[0]
            if len(ix) == 0:
                continue
            rows = graphs[int(c)][0]
            tr = ts[rows]
            g = {"ix": ix, "q": torch.from_numpy(np.ascontiguousarray(qs[ix])).cuda(),
                 "rows": torch.from_numpy(rows.astype(np.int64)).cuda()}
            if t == 3:
                l, r = ms[ix, 2], ms[ix, 3]
                g["bounds"] = np.ascontiguousarray(np.stack([l, r], 1), np.float32)
                g["id_bounds"] = np.ascontiguousarray(np.stack([np.searchsorted(tr, l, "left"),
                                                                np.searchsorted(tr, r, "right")], 1), np.int32)
            groups[(int(c), t)] = g
    for beam in [int(b) for b in args.graph_beams.split(",")]:
        refine = min(150, beam)
        out = np.full((len(sel), 100), 0xFFFFFFFF, np.uint32)  # beams under 100 return fewer ids
        for rep in range(2):  # first pass warms up
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            res = {}
            for (c, t), g in groups.items():
                gs = graphs[c][1]
                if t == 1:
                    loc = gs.SearchFilter(g["q"], beam, refine)
                else:
                    loc = gs.SearchCategoryRange(g["q"], beam, refine, g["bounds"], g["id_bounds"])
                cand = g["rows"][loc.long().clamp(min=0)].to(torch.int32).contiguous()
                res[(c, t)] = idx.rerank(g["q"], cand, k=min(100, refine), with_dists=False)[0]
            e1.record()
            torch.cuda.synchronize()
        ms_gpu = e0.elapsed_time(e1)
        for key, g in groups.items():
            out[g["ix"], :res[key].shape[1]] = res[key].cpu().numpy().view(np.uint32)
        rec = {str(t): datagen.recall_matrix(out[ms[:, 0] == t], exact_ids[ms[:, 0] == t]) for t in (1, 3)}
        # the queries the reference's BatchSearch sends to a category graph
        # (hybrid_graph.cpp:201,249-254): selectivity >= bf_thr (type 1) or
        # >= bf_thr3 (type 3), selectivity = passing rows / 1e7
        rec_routed = {}
        for t, thr in ((1, 0.045), (3, 0.08)):
            m = (ms[:, 0] == t) & (passing >= thr * 1e7)
            rec_routed[str(t)] = {"queries": int(m.sum()),
                                  "recall": datagen.recall_matrix(out[m], exact_ids[m]) if m.any() else None}
        c0 = int(cats[0])
        smp = groups[(c0, 1)]["ix"][:300]
        rows0 = graphs[c0][0]
        v0, l0, t0_ = vecs[rows0], labels[rows0], ts[rows0]
        tl = []  # the reference's query loop alone (graph load and SetData excluded)
        oracle.ref_graph_search(graphs[c0][2], v0, l0, t0_, qs[smp], 1, beam, refine, timing=tl)
        t_ref = max(1e-9, tl[0])
        print(json.dumps({
            "mode": "graph", "metric": "filtered queries/s, graph beam search + FP32 re-rank", "unit": UNIT,
            "value": len(sel) / (ms_gpu * 1e-3), "ms": ms_gpu, "beam": beam, "refine": refine,
            "recall_at_100_vs_exact": datagen.recall_matrix(out, exact_ids), "recall_at_100_by_type": rec,
            "recall_at_100_routed_by_type": rec_routed,
            "config": {"workload": "uneven-selectivity (config-4 generator)", "n": n, "queries": int(len(sel)),
                       "query_types": {"1": int((ms[:, 0] == 1).sum()), "3": int((ms[:, 0] == 3).sum())},
                       "categories_with_graphs": [int(c) for c in cats],
                       "category_rows": [int(counts[c]) for c in cats], "out_degree": 32, "ef_construction": 100},
            "graph_build_s_reference_cpu": t_build,
            "reference_cpu": {"value": len(smp) / t_ref, "unit": UNIT, "cores": 1, "kind": "reference",
                              "sample": f"{len(smp)} type-1 queries of category {c0} (largest graph), SearchFilter, "
                                        f"one thread"},
        }), flush=True)
    idx.close()


def run_router(args):
    """HybridGraph::BatchSearch's routing on the GPU (fknn_router) beside the
    reference pipeline itself (oracle/_ref, its BatchSearch on the host
    cores), over the same subgraphs and base orders the reference built
    (HNSW M=16, efConstruction 100) on the uneven-selectivity generator;
    queries/s of each (the router's wall time per call, host arrays in and
    out, as the reference's BatchSearch is timed) and recall@100 per query
    type against the exact ids."""
    import torch

    import fknn
    import oracle
    from fknn import datagen
    torch.cuda.set_device(0)
    if oracle.ref_hybrid() is None:
        print(json.dumps({"mode": "router", "unavailable": "reference pipeline (oracle/_ref/libref_hybrid.so) not built"}))
        return
    n = args.n or 1_200_000
    nq = args.nq or 20_000
    vecs, labels, ts, q, metas = datagen.make_workload(4, n=n, nq=nq)
    d = tempfile.mkdtemp()
    datagen.write_base(d + "/base.bin", vecs, labels, ts)
    datagen.write_queries(d + "/queries.bin", q, metas)
    t0 = time.perf_counter()
    ref_ids, ref_s = oracle.ref_hybrid_run(d + "/base.bin", d + "/queries.bin", d, nq)
    ref_total = time.perf_counter() - t0
    h = oracle.read_hybrid_dir(d, n)
    with fknn.Index(vecs, labels, ts) as idx:
        gt, _ = idx.search(q, metas)
    with fknn.Router(vecs, labels, ts, h["sorted_base_ids"], h["sorted_base_ids_by_full_time"], h["categories"],
                     h["buckets"], h["maxc_size"], h["minc_size"]) as router:
        for _ in range(args.warmup):
            ids, st = router.search(q, metas)
        ms = []
        for _ in range(args.steps):
            t1 = time.perf_counter()
            ids, st = router.search(q, metas)
            ms.append((time.perf_counter() - t1) * 1e3)
    rec = {}
    for t in range(4):
        sm = metas[:, 0] == t
        rec[str(t)] = {"queries": int(sm.sum()), "router": datagen.recall_matrix(ids[sm], gt[sm]),
                       "reference": datagen.recall_matrix(ref_ids[sm], gt[sm])}
    print(json.dumps({"mode": "router", "metric": "filtered queries/s, reference routing (BatchSearch)", "unit": UNIT,
                      "value": nq / (statistics.median(ms) * 1e-3), "ms_per_batch_median": statistics.median(ms),
                      "recall_at_100_by_type": rec,
                      "recall_at_100_all": {"router": datagen.recall_matrix(ids, gt),
                                            "reference": datagen.recall_matrix(ref_ids, gt)},
                      "routes": st,
                      "reference_cpu": {"value": nq / ref_s, "unit": UNIT, "cores": os.cpu_count(),
                                        "kind": "reference", "batchsearch_s": ref_s,
                                        "build_and_search_s": ref_total},
                      "config": {"workload": "uneven-selectivity (config-4 generator)", "n": n, "nq": nq,
                                 "graphs": "reference HNSW, M=16, efConstruction=100",
                                 "categories_with_graphs": len(h["categories"]), "time_buckets": len(h["buckets"])}}),
          flush=True)


def filter_measure(idx, metas, labels, ts, warmup: int, reps: int, batches=(1, 8)) -> dict:
    """fknn_filter_rows_batch (predicate + compaction, device-side counts)
    over the resident columns, the workload's predicates taken P at a time
    for each P in batches.  Every timed call is preceded by a 256 MB write
    that flushes L2 (the columns, 8 B per row, fit in it at N = 1e7) and is
    timed alone by CUDA events on its stream.  Algorithmic bytes per call:
    8 B per row (int32 label + float32 timestamp, read once for the P
    predicates) plus 4 B per passing row written.  The counts are checked
    against the oracle's sorted-column count."""
    import torch

    import oracle
    n = int(labels.shape[0])
    stream = torch.cuda.current_stream()
    flush = torch.empty(64 << 20, dtype=torch.int32, device="cuda")
    want = oracle.count_matches_sorted(labels, ts, metas)
    peaks = measured_peaks()
    pk = peaks.get("hbm_gbs", 6650.0)
    res = {"kernels": ["k_filter_coop"], "unit": "GB/s", "peak": pk,
           "peak_source": "MEASURED_PEAKS.json hbm_gbs" + (" [fallback]" if peaks.get("fallback") else ""),
           "algorithmic": "8 B per row (label + timestamp, once per call) + 4 B per passing row",
           "l2": "flushed (256 MB write) before every timed call", "counts_equal_oracle": True}
    for P in batches:
        out = torch.empty((P, n), dtype=torch.int32, device="cuda")
        counts = torch.empty(P, dtype=torch.int64, device="cuda")
        ms, byts = [], []
        for g0 in range(0, metas.shape[0] - P + 1, P):
            g = np.ascontiguousarray(metas[g0:g0 + P])
            for rep in range(warmup + reps):
                flush.zero_()
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                idx.filter_rows_batch(g, out, counts, stream.cuda_stream)
                e1.record(stream)
                e1.synchronize()
                c = counts.cpu().numpy()
                if not np.array_equal(c, want[g0:g0 + P].astype(np.int64)):
                    res["counts_equal_oracle"] = False
                if rep >= warmup:
                    ms.append(e0.elapsed_time(e1))
                    byts.append(8.0 * n + 4.0 * float(c.sum()))
        gbs = float(np.sum(byts) / (np.sum(ms) * 1e-3) / 1e9)
        res[f"p{P}"] = {"value": gbs, "frac": gbs / pk, "calls": len(ms), "ms_per_call_mean": float(np.mean(ms)),
                        "passing_rows_mean_per_predicate": float(np.mean(byts) - 8.0 * n) / 4.0 / P}
        del out, counts
    res["value"] = res["p1"]["value"]
    res["frac"] = res["p1"]["frac"]
    # context: a device-to-device copy (torch) moving the same bytes as a
    # one-predicate call (half read, half written), timed the same way
    nbytes = int(np.mean([8.0 * n + 4.0 * float(c) for c in want[:64]]))
    src = torch.empty(nbytes // 8, dtype=torch.float32, device="cuda")
    dst = torch.empty_like(src)
    cms = []
    for rep in range(3 + 20):
        flush.zero_()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        dst.copy_(src)
        e1.record(stream)
        e1.synchronize()
        if rep >= 3:
            cms.append(e0.elapsed_time(e1))
    cgbs = 2.0 * src.numel() * 4 / (float(np.median(cms)) * 1e-3) / 1e9
    res["same_bytes_copy"] = {"value": cgbs, "frac": cgbs / pk, "bytes": int(2 * src.numel() * 4),
                              "what": "torch device-to-device copy of the same total bytes, L2 flushed, median"}
    del flush, src, dst
    return res


def run_filter(args):
    """fknn_filter_rows (the predicate + compaction kernels) on the resident
    columns for 64 predicates of the workload (filter_measure)."""
    import torch

    import fknn
    from fknn import datagen
    torch.cuda.set_device(0)
    w = datagen.WORKLOADS[args.config]
    n = args.n or w.n
    vecs, labels, ts, q, metas = datagen.make_workload(args.config, n=n, nq=64)
    idx = fknn.Index(vecs, labels, ts)
    r = filter_measure(idx, metas, labels, ts, args.warmup, args.steps)
    print(json.dumps({"mode": "filter", "metric": "predicate compaction HBM GB/s (algorithmic bytes)",
                      "config": {"workload": w.name, "n": n}, **r}), flush=True)
    idx.close()


def run_sq8(args):
    """fknn_sq8_bruteforce_subgraph over one slab of symmetric SQ8 codes (the
    reference's brute-force leg for selective queries, hybrid_graph.cpp:206-211
    and :406-410, K' = 140 in heap-array order), device-resident codes and
    queries, nq queries per call.  Algorithmic bytes: 112 B per (query, code)
    pair read; the slab (50 MB) stays in L2 across the queries of a call."""
    import torch

    import fknn
    from fknn import _lib, datagen
    torch.cuda.set_device(0)
    w = datagen.WORKLOADS[3]
    npoints = args.n or 450_000
    nq = args.nq or 2048
    vecs, labels, ts = datagen.make_base(npoints, w.zipf_s, w.n_labels, 1237)
    q, _ = datagen.make_queries(nq, w.zipf_s, w.n_labels, w.window, w.balanced_types, 1237, 1238)
    quant = fknn.SQ8SymmetricQuantizer(100)
    quant.train(vecs)
    codes = torch.from_numpy(quant.codes).cuda()
    qc = torch.from_numpy(quant.encode(q)).cuda()
    k = 140
    ids = torch.empty((nq, k), dtype=torch.int32, device="cuda")
    dd = torch.empty((nq, k), dtype=torch.float32, device="cuda")
    lib = _lib.load()
    import ctypes

    def call():
        _lib.check(lib.fknn_sq8_bruteforce_subgraph(100, k, ids.data_ptr(), dd.data_ptr(), npoints, codes.data_ptr(),
                                                    ctypes.c_float(quant.alpha), nq, qc.data_ptr()))
    if args.sq8_callers:
        # T host threads, each answering its share of the queries one call
        # per query; wall time over all of them (each call is synchronous)
        import concurrent.futures as cf
        nthreads = args.sq8_callers
        qrows = [qc[i:i + 1] for i in range(nq)]

        def worker(t):
            for i in range(t, nq, nthreads):
                _lib.check(lib.fknn_sq8_bruteforce_subgraph(100, k, ids[i].data_ptr(), dd[i].data_ptr(), npoints,
                                                            codes.data_ptr(), ctypes.c_float(quant.alpha), 1,
                                                            qrows[i].data_ptr()))
        with cf.ThreadPoolExecutor(nthreads) as ex:
            for _ in range(args.warmup):
                list(ex.map(worker, range(nthreads)))
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for _ in range(args.steps):
                list(ex.map(worker, range(nthreads)))
            torch.cuda.synchronize()
    else:
        for _ in range(args.warmup):
            call()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(args.steps):
            call()
        torch.cuda.synchronize()
    sec = (time.perf_counter() - t0) / args.steps
    pairs = nq * npoints
    line = {"mode": "sq8", "metric": "SQ8 slab brute force, codes scanned per second",
            "value": pairs / sec, "unit": "codes/s", "gbs_algorithmic": pairs * 112 / sec / 1e9,
            "ms_per_call": sec * 1e3, "queries_per_s": nq / sec,
            "config": {"slab_codes": npoints, "queries_per_call": 1 if args.sq8_callers else nq,
                       "queries_per_step": nq, "host_threads": args.sq8_callers or 1, "k": k, "code_bytes": 112}}
    # The reference's own bruteforce() (compiled from its sources) on the
    # host cores, one query per call as hybrid_graph.cpp:211 calls it, over a
    # sample of the same queries; its heap-array ids must equal ours.
    if not args.no_cpu_baseline:
        import concurrent.futures as cf

        import oracle as orc
        ref = orc.ref_sq8()
        kind = "reference" if ref is not None else "port"
        codes_h = np.ascontiguousarray(quant.codes)
        qc_h = np.ascontiguousarray(quant.encode(q))
        sample = min(nq, args.cpu_sample)
        out = np.empty((sample, k), dtype=np.int32)

        def one(i):
            if ref is not None:
                ref.ref_sq8_bruteforce(k, out[i].ctypes.data, npoints, codes_h.ctypes.data, quant.alpha,
                                       qc_h[i].ctypes.data)
            else:
                out[i] = orc.sq8_bruteforce(k, codes_h, quant.alpha, qc_h[i])
        cores = os.cpu_count() or 1
        t0 = time.perf_counter()
        with cf.ThreadPoolExecutor(cores) as ex:
            list(ex.map(one, range(sample)))
        cs = time.perf_counter() - t0
        got = ids[:sample].cpu().numpy()
        line["cpu_baseline"] = {"value": sample * npoints / cs, "unit": "codes/s", "cores": cores, "kind": kind,
                                "sample": f"{sample} queries x {npoints} codes"}
        line["ids_equal_reference"] = bool((got == out).all())
    print(json.dumps(line), flush=True)


def main():
    args = parse()
    if args.sq8:
        return run_sq8(args)
    if args.filter:
        return run_filter(args)
    if args.graph:
        return run_graph(args)
    if args.router:
        return run_router(args)
    if args.sweep:
        return run_sweep(args)
    if args.serve:
        return run_serve(args)
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        return run_reference(args, rank, world)

    import torch
    import torch.distributed as dist

    import fknn
    from fknn import datagen
    torch.cuda.set_device(local)
    if world > 1:
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))

    w = datagen.WORKLOADS[args.config]
    n = args.n or w.n
    nq = args.nq or w.nq
    vecs, labels, ts = datagen.make_base(n, w.zipf_s, w.n_labels, 1234 + args.config)
    # every rank its own query batch (weak scaling); rank 0 = the workload's queries
    from fknn import replicas
    q, metas = replicas.rank_queries(args.config, nq, rank)
    idx = fknn.Index(vecs, labels, ts, device=local, build_bf16=True)
    # autotuned plan / kernel parameters and k' for this device and base size, if recorded
    idx.apply_tuning(fknn.MODE_EXACT_FP32)
    tuned_kp = idx.apply_tuning(fknn.MODE_BF16_RERANK)
    if tuned_kp and not args.kprime_set:
        args.kprime = tuned_kp
    stream = torch.cuda.current_stream()
    dq = torch.from_numpy(q).cuda()
    dm = torch.from_numpy(metas).cuda()
    ids = torch.empty((nq, 100), dtype=torch.int32, device="cuda")
    dd = torch.empty((nq, 100), dtype=torch.float32, device="cuda")

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    def max_over_ranks(x):
        return replicas.max_over_ranks(x, "cuda")

    def timed(mode, kprime, out_ids, steps, warmup, graph=False):
        """warmup untimed steps, then `steps` steps between barriers, CUDA
        events on the launching stream; returns (ms per step, per-step stats).
        graph: the search planned on the device and replayed as a captured
        CUDA graph (FKNN_SEARCH_GRAPH)."""
        def step():
            return idx.search(dq, dm, k=100, mode=mode, kprime=kprime, ids=out_ids, dists=dd,
                              stream=stream.cuda_stream, return_stats=True, graph=graph)[2]
        for _ in range(warmup):
            step()
        barrier()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        st = []
        e0.record(stream)
        for _ in range(steps):
            st.append(step())
        e1.record(stream)
        barrier()
        return max_over_ranks(e0.elapsed_time(e1) / steps), st

    clocks = ClockSampler(local)
    clocks.start()
    # The exact leg: one warm-up step first; when a step is long (~16 s at
    # N=1e7, Q=1e6) it is timed over --exact-steps (default 2) steps only.
    ms_first, _ = timed(fknn.MODE_EXACT_FP32, 0, ids, 1, 0)
    if args.exact_steps:
        ex_steps, ex_warm = args.exact_steps, 0
    elif ms_first < 1000.0:
        ex_steps, ex_warm = args.steps, max(0, args.warmup - 1)
    else:
        ex_steps, ex_warm = min(args.steps, 2), 0
    ms_exact, st_exact = timed(fknn.MODE_EXACT_FP32, 0, ids, ex_steps, ex_warm)
    exact_ids = ids.cpu().numpy().view(np.uint32).copy()
    exact_d = dd.cpu().numpy().copy()
    ids_b = torch.empty_like(ids)
    use_graph = args.plan == "graph"
    ms_bf16, st_bf16 = timed(fknn.MODE_BF16_RERANK, args.kprime, ids_b, args.steps, args.warmup, graph=use_graph)
    # the other planning form of the same search, for comparison (a few steps)
    ms_bf16_other, _ = timed(fknn.MODE_BF16_RERANK, args.kprime, torch.empty_like(ids), min(args.steps, 5), 1,
                             graph=not use_graph)
    clk = clocks.stop()
    bf16_ids = ids_b.cpu().numpy().view(np.uint32)
    recall_bf16 = datagen.recall_matrix(bf16_ids, exact_ids)
    use_bf16 = recall_bf16 >= 0.99
    head_mode = fknn.MODE_BF16_RERANK if use_bf16 else fknn.MODE_EXACT_FP32
    if not use_bf16 and ex_steps != args.steps:
        # the exact path is the headline: time it over the full K steps
        ms_exact, st_exact = timed(fknn.MODE_EXACT_FP32, 0, ids, args.steps, 0)
        ex_steps = args.steps
    ms = ms_bf16 if use_bf16 else ms_exact
    value = replicas.job_value(world, nq, ms)

    # Not timed, rank 0: the exact path's ids and distances against the oracle
    # restatement of utils.h:80 on 64 queries, and both forms' recall@100
    # against an FP64 oracle on a seeded sample of the queries.
    check, f64 = None, None
    if rank == 0:
        import oracle
        sel = np.arange(0, nq, max(1, nq // 64))[:64]
        oids, od = oracle.exact_knn(vecs, labels, ts, q[sel], metas[sel])
        check = bool(np.array_equal(exact_ids[sel], oids) and
                     np.array_equal(exact_d[sel].view(np.uint32), od.view(np.uint32)))
        fsel = np.sort(np.random.default_rng(17).choice(nq, size=min(args.f64_sample, nq), replace=False))
        t0 = time.perf_counter()
        fids, _ = oracle.exact_knn(vecs, labels, ts, q[fsel], metas[fsel], f64=True)
        f64 = {"queries": int(len(fsel)), "oracle_seconds": time.perf_counter() - t0,
               "recall_at_100_bf16": datagen.recall_matrix(bf16_ids[fsel], fids),
               "recall_at_100_exact_fp32": datagen.recall_matrix(exact_ids[fsel], fids)}

    # end to end through the C ABI: pinned host buffers, copies inside the timed region
    hq = torch.empty((nq, 100), dtype=torch.float32, pin_memory=True).numpy()
    hm = torch.empty((nq, 4), dtype=torch.float32, pin_memory=True).numpy()
    hq[:] = q
    hm[:] = metas
    # the result is the ids, as the reference's batch interface returns them (hybrid_graph.h:48)
    hids = torch.empty((nq, 100), dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    for _ in range(2):
        idx.search(hq, hm, k=100, mode=head_mode, kprime=args.kprime, ids=hids, with_dists=False,
                   stream=stream.cuda_stream, graph=use_graph and use_bf16)
    barrier()
    lat = []
    for _ in range(args.steps):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record(stream)
        idx.search(hq, hm, k=100, mode=head_mode, kprime=args.kprime, ids=hids, with_dists=False,
                   stream=stream.cuda_stream, graph=use_graph and use_bf16)
        e.record(stream)
        e.synchronize()
        lat.append(s.elapsed_time(e))
    barrier()
    e2e_ms = max_over_ranks(sum(lat) / len(lat))
    e2e_value = world * nq / (e2e_ms * 1e-3)
    same = bool(np.array_equal(hids, bf16_ids if use_bf16 else exact_ids))

    if rank == 0:
        peaks = measured_peaks()
        fp32_peak = fp32_gemm_peak_tflops(torch)
        tpp = traffic_per_pair()

        def roof_exact():
            ms_s = statistics.mean(x["ms_screen"] for x in st_exact)
            pairs = st_exact[-1]["pairs_contraction"]
            ach = 2.0 * 100 * pairs / (ms_s * 1e-3) / 1e12
            # three fp16 products per pair on the tensor cores (fp16 and bf16
            # run at the same rate)
            pk = peaks.get("bf16_tflops", 1590.0) / 3
            return {"bound": "tensor", "kernel": "k_exact_screen", "achieved": ach, "peak": pk,
                    "unit": "TFLOP/s", "frac": ach / pk, "vs_fp32_sgemm": ach / fp32_peak,
                    "traffic": tpp * st_exact[-1]["pairs_screened"] if tpp else None,
                    "peak_source": "MEASURED_PEAKS.json bf16_tflops (cuBLAS bf16 burst) / 3: the screen makes three "
                                   "fp16 products per pair; vs_fp32_sgemm against a cuBLAS SGEMM 8192^3 (TF32 off) "
                                   "of this run",
                    "algorithmic": "2*d*P flops, d=100, P = passing (query,row) pairs of the contraction's queries",
                    "per_launch_ms": ms_s, "pairs_passing": pairs, "pairs_screened": st_exact[-1]["pairs_screened"]}

        def roof_bf16():
            ms_s = statistics.mean(x["ms_screen"] for x in st_bf16)
            pairs = st_bf16[-1]["pairs_contraction"]
            ach = 2.0 * 100 * pairs / (ms_s * 1e-3) / 1e12
            burst = peaks.get("bf16_tflops", 1590.0)
            # a screen inside a timed region of seconds runs under the power
            # cap: the sustained figure is its denominator, the burst one is kept beside it
            long_region = ms_bf16 * args.steps >= 2000.0
            sus = peaks.get("bf16_tflops_sustained")
            pk = sus if (long_region and sus) else burst
            tpp_tc = traffic_per_pair("k_screen_tc_traffic.json")
            return {"bound": "tensor", "kernel": "k_screen_tc", "achieved": ach, "peak": pk, "unit": "TFLOP/s",
                    "frac": ach / pk, "frac_vs_burst": ach / burst,
                    "traffic": tpp_tc * st_bf16[-1]["pairs_screened"] if tpp_tc else None,
                    "peak_source": ("MEASURED_PEAKS.json bf16_tflops_sustained (cuBLAS bf16, seconds-long loop)"
                                    if pk is sus else "MEASURED_PEAKS.json bf16_tflops (cuBLAS bf16 burst)") +
                                   (" [fallback]" if peaks.get("fallback") else ""),
                    "algorithmic": "2*d*P flops, d=100, P = passing (query,row) pairs of the contraction's queries",
                    "per_launch_ms": ms_s, "pairs_passing": pairs, "pairs_screened": st_bf16[-1]["pairs_screened"]}

        head_stats = st_bf16 if use_bf16 else st_exact
        launches = int(sum(x["kernel_launches"] for x in head_stats))
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "bf16" if use_bf16 else "f32", "data": "synthetic",
            "config": {"workload": w.name if (n, nq) == (w.n, w.nq) else f"{w.name} resized to n={n}, nq={nq}",
                       "mode": "bf16_rerank" if use_bf16 else "exact_fp32",
                       "kprime": args.kprime if use_bf16 else None, "n": n, "nq_per_gpu": nq, "k": 100, "d": 100,
                       "tuning": idx.get_tuning(head_mode),
                       "parallelism": f"replicas{world}" if world > 1 else "single",
                       "l2": f"no flush: each step streams the row orders (2 x {n * 404 / 1e9:.2f} GB FP32, "
                             f"2 x {n * 229 / 1e9:.2f} GB BF16) > 126 MB L2"},
            "recall_at_100_vs_exact": recall_bf16 if use_bf16 else 1.0,
            "exact_fp32": {"value": world * nq / (ms_exact * 1e-3), "ms_per_step": ms_exact,
                           "timed_steps": ex_steps, "ids_and_dists_bitexact_sample64": check},
            "f64_oracle_sample": f64,
            "bf16_rerank": {"value": world * nq / (ms_bf16 * 1e-3), "ms_per_step": ms_bf16, "kprime": args.kprime,
                            "recall_at_100_vs_exact_all_queries": recall_bf16,
                            "speedup_vs_exact": ms_exact / ms_bf16,
                            "n_boundary_f64_per_step": st_bf16[-1]["n_boundary_f64"],
                            "plan": ("on the device, the whole search one captured CUDA graph" if use_graph
                                     else "on the host"),
                            "ms_per_step_other_plan": ms_bf16_other},
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": int(nq * 100 * 4 + nq * 16),
                    "d2h_bytes_per_step": int(nq * 100 * 4), "same_ids_as_device_path": same,
                    "result": "ids (nq x 100 u32), as BatchSearch returns them"},
            "latency_ms": {"p50": statistics.median(lat), "p99": float(np.percentile(lat, 99)),
                           "note": "per batch of nq queries, end to end"},
            "gpu_launches": launches,
            "roofline": roof_bf16() if use_bf16 else roof_exact(),
            "roofline_exact_fp32": roof_exact(),
            "kernel_ms": {m: {"screen": statistics.mean(x["ms_screen"] for x in stx),
                              "merge": statistics.mean(x["ms_merge"] for x in stx),
                              "exact_scan": statistics.mean(x["ms_scan"] for x in stx),
                              "plan_host": statistics.mean(x["ms_plan"] for x in stx)}
                          for m, stx in (("exact_fp32", st_exact), ("bf16_rerank", st_bf16))},
            "clocks": clk,
        }
        line["filter"] = filter_measure(idx, metas[:32], labels, ts, 1, 2)
        if world == 1 and not args.no_cpu_baseline:
            line["cpu_baseline"] = cpu_baseline(vecs, labels, ts, q, metas,
                                                args.cpu_sample or default_cpu_sample(n))
        print(json.dumps(line), flush=True)
    idx.close()
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
