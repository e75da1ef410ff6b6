"""The lazily merged pool of the graph beam search (k_graph_beam): pools and
buffers at their smallest and around the 32 buffered entries, out-degrees
around the 32-entry chunks, floods of equal distances (the tie rule), lists
made of repeats, and the three places the visited bits can live in (both sets
in shared memory, one of them, none), which must give the same slots.  Ids and
distances equal the oracle's."""
import numpy as np
import pytest

import fknn
import oracle
from fknn import datagen
from graph_util import id_bounds_for, random_graph, save_bytes, windows

pytestmark = pytest.mark.gpu


def run(gs, mode, q, k, refine, bounds, ib):
    if mode == 1:
        return gs.SearchFilter(q, k, refine), None
    if mode == 2:
        return gs.SearchFilterSubTime(q, k, refine)
    if mode == 3:
        return gs.SearchCategoryRange(q, k, refine, bounds, ib), None
    if mode == 4:
        return gs.SearchRangeFilterSubTime(q, k, refine, bounds, ib)
    return gs.SearchRangeFilter(q, k, refine, bounds, ib), None


def check(gs, gb, vecs, q, mode, k, refine, ef, bounds, ib):
    gs.SetEf(ef)
    ids, dists = run(gs, mode, q, k, refine, bounds, ib)
    exp = oracle.graph_search(gb, vecs, q, mode, k, refine, bounds, ib, ef=ef, with_dists=mode in (2, 4))
    eids, edists = exp if mode in (2, 4) else (exp, None)
    np.testing.assert_array_equal(ids, eids, err_msg=f"mode {mode} k {k} refine {refine} ef {ef}")
    if edists is not None:
        np.testing.assert_array_equal(dists, edists)


@pytest.mark.parametrize("K", [1, 5, 31, 32, 33, 70])
def test_degrees_and_pool_sizes(K):
    n = 3000
    vecs, labels, ts, q, metas = datagen.make_workload(1, n=n, nq=24)
    ts = np.sort(ts)
    gb = random_graph(n, K, ts, seed=K, dup_frac=0.2)
    bounds = windows(q.shape[0], 3, log_w=(-2, 0))
    ib = id_bounds_for(ts, bounds)
    with fknn.GraphSearcher(gb, vecs) as gs:
        for mode in (1, 2, 3, 4, 5):
            for k, refine, ef in [(1, 1, 1), (2, 2, 1), (31, 31, 1), (32, 32, 1), (33, 20, 1), (65, 65, 32),
                                  (900, 150, 32)]:
                check(gs, gb, vecs, q, mode, k, refine, ef, bounds, ib)


@pytest.mark.parametrize("copies", [40, 1000])
def test_equal_distances(copies):
    """Rows in runs of identical vectors: most distances tie, and the pool
    must keep the order in which entries came."""
    n = 4000
    vecs, labels, ts, q, metas = datagen.make_workload(1, n=n // copies, nq=16)
    vecs = np.repeat(vecs, copies, axis=0)[:n]
    ts = np.sort(np.random.default_rng(1).random(n, dtype=np.float32))
    gb = random_graph(n, 32, ts, seed=2)
    bounds = windows(q.shape[0], 4, log_w=(-1, 0))
    ib = id_bounds_for(ts, bounds)
    with fknn.GraphSearcher(gb, vecs) as gs:
        for mode in (1, 2, 3, 4, 5):
            check(gs, gb, vecs, q, mode, 200, 150, 32, bounds, ib)


def test_lists_of_repeats():
    """Every list names two points many times, and some end at once."""
    rng = np.random.default_rng(3)
    n, K = 600, 40
    vecs, labels, ts, q, metas = datagen.make_workload(1, n=n, nq=16)
    ts = np.sort(ts)
    pair = rng.integers(0, n, (n, 2))
    adj = np.take_along_axis(pair, rng.integers(0, 2, (n, K)), axis=1).astype(np.int32)
    adj[::9] = -1
    ets = np.where(adj >= 0, ts[np.maximum(adj, 0)], 0).astype(np.float32)
    gb = save_bytes(adj, ets, eps=rng.choice(n, 20, replace=False).astype(np.int32))
    bounds = windows(q.shape[0], 6, log_w=(-1, 0))
    ib = id_bounds_for(ts, bounds)
    with fknn.GraphSearcher(gb, vecs) as gs:
        for mode in (1, 2, 3, 4, 5):
            check(gs, gb, vecs, q, mode, 64, 64, 32, bounds, ib)


@pytest.mark.parametrize("n", [4000, 100_000, 220_000])
def test_places_of_the_visited_bits_agree(n):
    """A few queries keep the visited bits in shared memory, thousands of them
    on a large graph do not; a query's slots do not depend on it."""
    vecs, labels, ts, q, metas = datagen.make_workload(1, n=n, nq=4800)
    ts = np.sort(ts)
    gb = random_graph(n, 32, ts, seed=8, dup_frac=0.0, pad_frac=0.0)
    bounds = windows(q.shape[0], 7, log_w=(-0.5, 0))
    ib = id_bounds_for(ts, bounds)
    with fknn.GraphSearcher(gb, vecs) as gs:
        for mode in (2, 4):
            ids, dists = run(gs, mode, q, 100, 100, bounds, ib)
            few, fd = run(gs, mode, q[:24], 100, 100, bounds[:24], ib[:24])
            np.testing.assert_array_equal(ids[:24], few)
            np.testing.assert_array_equal(dists[:24], fd)
            check(gs, gb, vecs, q[:24], mode, 100, 100, 32, bounds[:24], ib[:24])
            last, ld = run(gs, mode, q[-700:], 100, 100, bounds[-700:], ib[-700:])
            np.testing.assert_array_equal(ids[-700:], last)
