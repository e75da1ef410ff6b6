"""The exact search's tensor-core screen (exact_screen.cu) at the sizes and
values where it can go wrong: base sizes around the 64-row blocks and 128-row
sub-tiles, query counts around the 128- and 256-query tile halves, k at its
ends, rows and queries of very different scales (the norm slots' ranges, the
per-row path, zero rows and queries), seeds that lie too low (the redo pass),
and an HBM budget that holds only the smallest working set.  Ids and
distances equal the oracle's bit for bit."""
import numpy as np
import pytest

import fknn
import oracle
from fknn import datagen

pytestmark = pytest.mark.gpu


def check(vecs, labels, ts, q, metas, k=100, budget_room=None, **tuning):
    if budget_room is not None:
        with fknn.Index(vecs, labels, ts) as idx:
            size = idx.device_bytes
        idx = fknn.Index(vecs, labels, ts, hbm_budget=size + budget_room)
    else:
        idx = fknn.Index(vecs, labels, ts)
    with idx:
        if tuning:
            idx.set_tuning(fknn.MODE_EXACT_FP32, **tuning)
        ids, dists, st = idx.search(q, metas, k=k, return_stats=True)
    oids, odists = oracle.exact_knn(vecs, labels, ts, q, metas, k=k)
    np.testing.assert_array_equal(ids, oids)
    np.testing.assert_array_equal(dists.view(np.uint32), odists.view(np.uint32))
    return st


@pytest.mark.parametrize("n", [4097, 4159, 4160, 4224, 4225, 8191, 12353])
def test_base_sizes_around_blocks(n):
    vecs, labels, ts, q, metas = datagen.make_workload(1, n=n, nq=40)
    metas[:20] = (0, -1, -1, -1)  # the whole base: the contraction path
    st = check(vecs, labels, ts, q, metas)
    assert st["n_work_items"] > 0


@pytest.mark.parametrize("nq", [1, 2, 127, 128, 129, 255, 256, 257, 520])
def test_query_counts_around_tile_halves(nq):
    vecs, labels, ts, q, metas = datagen.make_workload(1, n=20000, nq=nq)
    metas[:] = (0, -1, -1, -1)
    st = check(vecs, labels, ts, q, metas)
    assert st["n_tiles"] == (nq + 255) // 256


@pytest.mark.parametrize("k", [1, 2, 100, 127, 128])
@pytest.mark.parametrize("pilot", [0, 2, 32, 1024])
def test_k_and_pilot(k, pilot):
    vecs, labels, ts, q, metas = datagen.make_workload(1, n=40000, nq=150)
    check(vecs, labels, ts, q, metas, k=k, items_per_sm=2, min_chunk_blocks=4, pilot_stride=pilot)


@pytest.mark.parametrize("case", ["large", "tiny", "row_scales", "query_scales", "zeros", "outlier", "positive"])
def test_value_scales(case):
    rng = np.random.default_rng(5)
    vecs, labels, ts, q, metas = datagen.make_workload(1, n=9000, nq=60)
    metas[:] = (0, -1, -1, -1)
    if case == "large":
        vecs, q = vecs * np.float32(2e14), q * np.float32(2e14)
    elif case == "tiny":
        vecs, q = vecs * np.float32(1e-18), q * np.float32(1e-18)
    elif case == "row_scales":  # neighbouring rows 2^40 apart: no shared scale in a sub-tile
        vecs = vecs * np.exp2(rng.integers(-20, 20, len(vecs))).astype(np.float32)[:, None]
    elif case == "query_scales":  # queries of one tile 2^60 apart: no norm slots
        q = q * np.exp2(rng.integers(-30, 30, len(q))).astype(np.float32)[:, None]
    elif case == "zeros":
        vecs[::7] = 0.0
        q[::5] = 0.0
    elif case == "outlier":
        vecs[1234] = np.float32(1e12)
    elif case == "positive":
        vecs, q = np.abs(vecs) * np.float32(100), np.abs(q) * np.float32(100)
    check(np.ascontiguousarray(vecs), labels, ts, np.ascontiguousarray(q), metas)


def test_low_seeds_are_screened_again():
    """Sixty rows near the queries stand in one sampled block, fewer than k:
    the pilot's seed is their distance, the merge finds it unproven and the
    redo pass answers."""
    vecs, labels, ts, q, metas = datagen.make_workload(1, n=40000, nq=300)
    ts = np.linspace(0, 1, len(ts), dtype=np.float32)
    rng = np.random.default_rng(9)
    vecs[:60] = q[0] + rng.normal(0, 1e-3, (60, 100)).astype(np.float32)
    q[:150] = q[0] + rng.normal(0, 1e-3, (150, 100)).astype(np.float32)
    metas[:] = (0, -1, -1, -1)
    st = check(vecs, labels, ts, q, metas, items_per_sm=1, min_chunk_blocks=64, pilot_stride=32)
    assert st["n_overflow"] == 0


@pytest.mark.parametrize("room_mb", [4, 16, 64])
def test_small_hbm_budget(room_mb):
    vecs, labels, ts, q, metas = datagen.make_workload(1, n=60000, nq=64)
    check(vecs, labels, ts, q, metas, budget_room=room_mb << 20)


def test_items_of_marked_queries():
    """A category of equal rows: the first items' pilot lists overflow and mark
    their queries, and the later items of those tiles (more items than the GPU
    takes at once) are skipped; the seeds still read every item's counts, which
    an earlier search of the other kind left behind."""
    rng = np.random.default_rng(11)
    n, same, nq = 20000, 12000, 10000
    vecs = rng.standard_normal((n, 100), dtype=np.float32)
    vecs[:same] = vecs[0]
    labels = np.where(np.arange(n) < same, 3, 4).astype(np.float32)
    ts = rng.random(n, dtype=np.float32)
    q = rng.standard_normal((nq, 100), dtype=np.float32)
    metas = np.tile(np.array([1, 3, -1, -1], np.float32), (nq, 1))
    with fknn.Index(vecs, labels, ts, build_bf16=True) as idx:
        idx.set_tuning(fknn.MODE_EXACT_FP32, items_per_sm=4, min_chunk_blocks=16, pilot_stride=2)
        other = metas[:2000].copy()
        other[:, :2] = (0, -1)
        idx.search(q[:2000], other, mode=fknn.MODE_BF16_RERANK, kprime=200)
        ids, dists, st = idx.search(q, metas, return_stats=True)
    assert st["n_work_items"] > 148 and st["n_overflow"] == nq
    # equal distances: the order is the ids'
    np.testing.assert_array_equal(ids, np.tile(np.arange(100, dtype=np.uint32), (nq, 1)))
    _, odists = oracle.exact_knn(vecs, labels, ts, q[:50], metas[:50])
    np.testing.assert_array_equal(dists[:50], odists)
