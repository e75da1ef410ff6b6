"""Queries answered row by row: slabs of a block's threads, its key buffer and
the longest planned for here, one row more and less; floods of equal distances
across the k-th place; and the search for a slab's ends (labels and times with
many repeats, windows that miss, touch and cross).  Ids, distances and counts
equal the oracle's."""
import numpy as np
import pytest

import fknn
import oracle

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 99, 100, 101, 128, 129, 511, 512, 513, 1025, 3583, 3584, 3585, 4095, 4096, 4097]


def dataset(seed, distinct):
    """Category c holds SIZES[c] rows, each of `distinct` vectors many times."""
    rng = np.random.default_rng(seed)
    labels = np.repeat(np.arange(len(SIZES)), SIZES).astype(np.float32)
    n = labels.shape[0]
    vecs = rng.standard_normal((distinct, 100), dtype=np.float32)[rng.integers(0, distinct, n)]
    perm = rng.permutation(n)
    ts = np.round(rng.random(n) * 50).astype(np.float32) / 50  # 51 times
    return vecs[perm], labels[perm], ts[perm], rng


@pytest.mark.parametrize("distinct", [3, 40_000])
@pytest.mark.parametrize("k", [1, 100, 128])
def test_slabs_of_every_size(distinct, k):
    vecs, labels, ts, rng = dataset(k, distinct)
    c = len(SIZES)
    q = rng.standard_normal((2 * c, 100), dtype=np.float32)
    metas = np.zeros((2 * c, 4), np.float32)
    metas[:, 0] = np.repeat([1, 3], c)
    metas[:, 1] = np.tile(np.arange(c), 2)
    metas[:, 2:] = [0.2, 0.8]
    with fknn.Index(vecs, labels, ts) as idx:
        ids, dists = idx.search(q, metas, k=k)
        oids, odists = oracle.exact_knn(vecs, labels, ts, q, metas, k=k)
        np.testing.assert_array_equal(ids, oids)
        np.testing.assert_array_equal(dists, odists)


def test_ends_of_a_slab():
    vecs, labels, ts, rng = dataset(7, 40_000)
    edges = np.array([-1, 0, 0.01, 0.02, 0.5, 0.51, 0.98, 1, 1.5, np.inf, -np.inf], np.float32)
    metas = [[t, v, l, r] for t in (0, 1, 2, 3) for v in (-1, 0, 5, 19, 20, 7) for l in edges for r in edges]
    metas = np.array(metas, np.float32)
    with fknn.Index(vecs, labels, ts) as idx:
        np.testing.assert_array_equal(idx.count_matches(metas), oracle.count_matches(labels, ts, metas))


@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1025, 33_000])
def test_ends_in_tables_of_any_length(n):
    rng = np.random.default_rng(n)
    vecs = rng.standard_normal((n, 100), dtype=np.float32)
    labels = rng.integers(0, 3, n).astype(np.float32)
    ts = rng.random(n, dtype=np.float32)
    metas = np.zeros((200, 4), np.float32)
    metas[:, 0] = rng.integers(0, 4, 200)
    metas[:, 1] = rng.integers(-1, 4, 200)
    metas[:, 2:] = np.sort(ts[rng.integers(0, n, (200, 2))], axis=1)
    with fknn.Index(vecs, labels, ts) as idx:
        np.testing.assert_array_equal(idx.count_matches(metas), oracle.count_matches(labels, ts, metas))


@pytest.mark.parametrize("rows", [3584, 3585, 4096])
def test_many_scans_at_the_edge_of_the_key_buffer(rows):
    """Slabs whose last step may or may not be the one before a selection, in
    every block several times over: all warps of a block decide alike."""
    rng = np.random.default_rng(rows)
    vecs = rng.standard_normal((rows + 500, 100), dtype=np.float32)
    labels = (np.arange(rows + 500) >= rows).astype(np.float32)
    ts = rng.random(rows + 500, dtype=np.float32)
    q = rng.standard_normal((3000, 100), dtype=np.float32)
    metas = np.tile(np.array([1, 0, -1, -1], np.float32), (3000, 1))
    with fknn.Index(vecs, labels, ts) as idx:
        ids, dists = idx.search(q, metas, k=100)
        oids, odists = oracle.exact_knn(vecs, labels, ts, q, metas, k=100)
        np.testing.assert_array_equal(ids, oids)
        np.testing.assert_array_equal(dists, odists)


def test_scans_that_select_many_times():
    """Near-ties that no candidate list holds: slabs of several buffers are
    scanned, with a bound that falls from one selection to the next."""
    rng = np.random.default_rng(3)
    n = 30_000
    vecs = np.repeat(rng.standard_normal((1, 100), dtype=np.float32), n, axis=0)
    vecs *= (1 + np.linspace(1e-5, 0, n, dtype=np.float32))[:, None]
    labels = (np.arange(n) >= 9000).astype(np.float32)
    ts = np.linspace(0, 1, n, dtype=np.float32)
    q = rng.standard_normal((400, 100), dtype=np.float32)
    metas = np.zeros((400, 4), np.float32)
    metas[:, 0] = np.arange(400) % 2
    with fknn.Index(vecs, labels, ts) as idx:
        ids, dists, st = idx.search(q, metas, k=100, return_stats=True)
        assert st["n_overflow"] == 400
        oids, odists = oracle.exact_knn(vecs, labels, ts, q, metas, k=100)
        np.testing.assert_array_equal(ids, oids)
        np.testing.assert_array_equal(dists, odists)


def test_more_queries_than_32_bit_threads_number():
    """2^27 queries of a warp each have 2^32 threads: the ones past that are
    counted too."""
    import torch
    rng = np.random.default_rng(5)
    vecs = rng.standard_normal((300, 100), dtype=np.float32)
    labels = (np.arange(300) % 3).astype(np.float32)
    nq = (1 << 27) + 9
    metas = torch.zeros((nq, 4), device="cuda")
    metas[-9:, 0] = 1
    metas[-9:, 1] = torch.arange(9, device="cuda") % 4
    counts = torch.full((nq,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with fknn.Index(vecs, labels, rng.random(300, dtype=np.float32)) as idx:
        assert fknn._lib.load().fknn_count_matches(idx._h, metas.data_ptr(), nq, counts.data_ptr(), None) == 0
    assert bool((counts[:-9] == 300).all())
    assert counts[-9:].tolist() == [100, 100, 100, 0] * 2 + [100]


@pytest.mark.parametrize("nq", [32767, 32768, 32769])
def test_ends_by_warps_and_by_threads(nq):
    vecs, labels, ts, rng = dataset(9, 40_000)
    metas = np.zeros((nq, 4), np.float32)
    metas[:, 0] = rng.integers(0, 4, nq)
    metas[:, 1] = rng.integers(-1, len(SIZES) + 1, nq)
    edges = np.array([-np.inf, -0.1, 0, 0.02, 0.5, 0.51, 0.98, 1, 1.5, np.inf], np.float32)
    metas[:, 2:] = edges[rng.integers(0, 10, (nq, 2))]
    q = rng.standard_normal((nq, 100), dtype=np.float32)
    some = rng.integers(0, nq, 200)
    with fknn.Index(vecs, labels, ts) as idx:
        np.testing.assert_array_equal(idx.count_matches(metas), oracle.count_matches(labels, ts, metas))
        ids, dists = idx.search(q, metas, k=20)
        oids, odists = oracle.exact_knn(vecs, labels, ts, q[some], metas[some], k=20)
        np.testing.assert_array_equal(ids[some], oids)
        np.testing.assert_array_equal(dists[some], odists)


@pytest.mark.parametrize("distinct", [3, 40_000])
def test_many_slabs_of_every_size(distinct):
    """As many queries as take blocks of 256 threads and buffers of 2,048 keys."""
    rng = np.random.default_rng(distinct)
    sizes = SIZES + [255, 256, 257, 1791, 1792, 1793, 2047, 2048, 2049, 2304]
    labels = np.repeat(np.arange(len(sizes)), sizes).astype(np.float32)
    n = labels.shape[0]
    vecs = rng.standard_normal((distinct, 100), dtype=np.float32)[rng.integers(0, distinct, n)]
    ts = rng.random(n, dtype=np.float32)
    q = rng.standard_normal((900, 100), dtype=np.float32)
    metas = np.zeros((900, 4), np.float32)
    metas[:, 0] = 1
    metas[:, 1] = np.arange(900) % len(sizes)
    with fknn.Index(vecs, labels, ts, build_bf16=True) as idx:
        for k in (1, 100, 128):
            oids, odists = oracle.exact_knn(vecs, labels, ts, q, metas, k=k)
            ids, dists = idx.search(q, metas, k=k)
            np.testing.assert_array_equal(ids, oids)
            np.testing.assert_array_equal(dists, odists)
            # a captured search goes by a share of its queries
            ids, dists = idx.search(np.tile(q, (4, 1)), np.tile(metas, (4, 1)), k=k, mode=fknn.MODE_BF16_RERANK,
                                    kprime=200, graph=True)
            scanned = np.tile(np.array(sizes)[np.arange(900) % len(sizes)] <= 4096, 4)
            np.testing.assert_array_equal(ids[scanned], np.tile(oids, (4, 1))[scanned])
            np.testing.assert_array_equal(dists[scanned], np.tile(odists, (4, 1))[scanned])
