"""The BF16 screen at the edges of its tiles: one and two query halves, row
blocks of 256 and a short last one, lists of every register class, with and
without a pilot, host and device plans.  The vectors are multiples of 1/8 up to
2, so BF16 operands, products, norms and sums are exact, the screening order is
the exact one, and ids and distances equal the oracle's (k' exceeds k by more
rows than share a distance)."""
import numpy as np
import pytest

import fknn
import oracle

pytestmark = pytest.mark.gpu


def grid(rng, shape):
    return (np.clip(np.round(rng.standard_normal(shape) * 5), -16, 16) / 8).astype(np.float32)


@pytest.fixture(scope="module")
def data():
    rng = np.random.default_rng(5)
    n = 30_011
    vecs = grid(rng, (n, 100))
    labels = (np.arange(n) % 5 == 0).astype(np.float32)  # 6,003 and 24,008 rows
    ts = rng.random(n, dtype=np.float32)
    q = grid(rng, (600, 100))
    metas = np.zeros((600, 4), np.float32)
    metas[:, 0] = rng.choice([0, 0, 0, 1, 2, 3], 600)
    metas[:, 1] = rng.integers(0, 2, 600)
    metas[:, 2] = rng.random(600) * 0.4
    metas[:, 3] = metas[:, 2] + 0.6
    want = oracle.exact_knn(vecs, labels, ts, q, metas, k=100)
    with fknn.Index(vecs, labels, ts, build_bf16=True) as idx:
        yield idx, q, metas, want


@pytest.mark.parametrize("nq", [1, 127, 128, 129, 255, 256, 257, 600])
@pytest.mark.parametrize("pilot", [0, 2, 8])
def test_tiles(data, nq, pilot):
    idx, q, metas, (ids, dists) = data
    idx.set_tuning(fknn.MODE_BF16_RERANK, 256, 3, 8, 0, pilot)
    for graph in (False, True):
        got, d = idx.search(q[:nq], metas[:nq], k=100, mode=fknn.MODE_BF16_RERANK, kprime=128, graph=graph)
        np.testing.assert_array_equal(got, ids[:nq])
        np.testing.assert_array_equal(d, dists[:nq])


@pytest.mark.parametrize("kprime", [128, 256, 257, 512, 513, 768, 769, 1024])
@pytest.mark.parametrize("slack", [256, 512])
def test_list_classes(data, kprime, slack):
    idx, q, metas, (ids, dists) = data
    for pilot in (0, 4):
        idx.set_tuning(fknn.MODE_BF16_RERANK, slack, 2, 4, 4, pilot)
        got, d = idx.search(q, metas, k=100, mode=fknn.MODE_BF16_RERANK, kprime=kprime)
        np.testing.assert_array_equal(got, ids)
        np.testing.assert_array_equal(d, dists)


@pytest.mark.parametrize("mode", ["bf16", "exact"])
def test_nearer_row_beyond_the_slab(mode):
    """The last row of a slab passes the bound but is not among the k best,
    and the row after it, outside, is the query itself: the two share a chunk
    of the screen, and the one inside must keep its own distance."""
    rng = np.random.default_rng(11)
    n, nq, k = 30_000, 96, 100
    vecs, q = grid(rng, (n, 100)), grid(rng, (nq, 100))
    ts = np.arange(n, dtype=np.float32)
    metas = np.zeros((nq, 4), np.float32)
    metas[:, 0] = 2
    end = 9000 + 211 * np.arange(nq)  # the last row inside
    metas[:, 3] = end
    for i in range(nq):
        d = ((vecs[: end[i]] - q[i]) ** 2).sum(1)
        r = np.argsort(d, kind="stable")[int(rng.integers(k + 2, 2 * k))]
        vecs[end[i]] = vecs[r]
        vecs[end[i], 0] += np.float32(0.125) * np.sign(vecs[r, 0] - q[i, 0] + np.float32(0.01))
        vecs[end[i] + 1] = q[i]
    with fknn.Index(vecs, np.zeros(n, np.float32), ts, build_bf16=True) as idx:
        ids, dists = oracle.exact_knn(vecs, np.zeros(n, np.float32), ts, q, metas, k=k)
        for pilot in (2, 4, 8):
            if mode == "bf16":
                idx.set_tuning(fknn.MODE_BF16_RERANK, 256, 3, 8, 0, pilot)
                got, gd = idx.search(q, metas, k=k, mode=fknn.MODE_BF16_RERANK, kprime=k)
            else:
                idx.set_tuning(fknn.MODE_EXACT_FP32, 0, 4, 16, 0, pilot)
                got, gd = idx.search(q, metas, k=k)
            np.testing.assert_array_equal(gd, dists)  # (rows at the same distance as the k-th may differ in bf16)
            if mode == "exact":
                np.testing.assert_array_equal(got, ids)


@pytest.mark.parametrize("room_mb", [16, 64])
@pytest.mark.parametrize("mode", [fknn.MODE_BF16_RERANK, fknn.MODE_FP8_RERANK])
def test_small_hbm_budget(room_mb, mode):
    """With little scratch a tile is one item, its results hold k' entries and
    a few ties, and fewer CTAs run; the answers are the same."""
    rng = np.random.default_rng(11)
    n, nq = 30_011, 600
    vecs, q = grid(rng, (n, 100)), grid(rng, (nq, 100))
    labels, ts = np.zeros(n, np.float32), rng.random(n, dtype=np.float32)
    metas = np.full((nq, 4), -1, np.float32)
    metas[:, 0] = 0
    form = {"build_bf16": True} if mode == fknn.MODE_BF16_RERANK else {"build_fp8": True}
    with fknn.Index(vecs, labels, ts, **form) as idx:
        size = idx.device_bytes
        want, want_d = idx.search(q, metas, k=100, mode=mode, kprime=128)
    with fknn.Index(vecs, labels, ts, hbm_budget=size + (room_mb << 20), **form) as idx:
        for graph in (False, True):
            for m in (1, nq):
                got, d = idx.search(q[:m], metas[:m], k=100, mode=mode, kprime=128, graph=graph)
                np.testing.assert_array_equal(got, want[:m])
                np.testing.assert_array_equal(d, want_d[:m])


def test_captured_plan_of_many_short_categories():
    """Categories too short for the contraction are no tiles of a captured
    search: neither its scratch nor the cutting of its tiles depends on them."""
    rng = np.random.default_rng(17)
    n, nq, k = 60_000, 3000, 20
    vecs, q = grid(rng, (n, 100)), grid(rng, (nq, 100))
    labels = np.where(np.arange(n) < 20_000, 0, np.arange(n)).astype(np.float32)  # one long category, 40,000 of one row
    ts = rng.random(n, dtype=np.float32)
    metas = np.zeros((nq, 4), np.float32)
    metas[:, 0] = np.arange(nq) % 4
    metas[1::8, 1] = n - 1
    metas[:, 3] = 0.9
    with fknn.Index(vecs, labels, ts, build_bf16=True) as idx:
        before = idx.device_bytes
        ids, dists, st = idx.search(q, metas, k=k, mode=fknn.MODE_BF16_RERANK, kprime=1024, graph=True, return_stats=True)
        assert st["n_work_items"] > 2 * st["n_tiles"]
        assert idx.device_bytes - before < 3 << 30
        want, want_d = idx.search(q, metas, k=k, mode=fknn.MODE_BF16_RERANK, kprime=1024)
    np.testing.assert_array_equal(ids, want)
    np.testing.assert_array_equal(dists, want_d)
    got, got_d = oracle.exact_knn(vecs, labels, ts, q, metas, k=k)
    np.testing.assert_array_equal(ids, got)
    np.testing.assert_array_equal(dists, got_d)


def test_slabs_around_the_pilots_forms():
    """Slabs whose sample is ranked by rows and by the best of every 8, 32 and
    128: all are seeded, so none falls to the exact scan, and the answers are
    the oracle's."""
    rng = np.random.default_rng(23)
    sizes = [4100, 4300, 6300, 7000, 10_000, 12_500, 17_600, 26_000, 31_000, 70_000]
    labels = np.repeat(np.arange(len(sizes)), sizes).astype(np.float32)
    n, nq = len(labels), 900
    vecs, q = grid(rng, (n, 100)), grid(rng, (nq, 100))
    ts = rng.random(n, dtype=np.float32)
    metas = np.full((nq, 4), -1, np.float32)
    metas[:, 0] = 1
    metas[:, 1] = np.arange(nq) % len(sizes)
    ids, dists = oracle.exact_knn(vecs, labels, ts, q, metas, k=100)
    with fknn.Index(vecs, labels, ts, build_bf16=True) as idx:
        for kprime in (128, 400, 1024):
            for m in (9, nq):
                for graph in (False, True):
                    got, d, st = idx.search(q[:m], metas[:m], k=100, mode=fknn.MODE_BF16_RERANK, kprime=kprime, graph=graph,
                                            return_stats=True)
                    np.testing.assert_array_equal(got, ids[:m])
                    np.testing.assert_array_equal(d, dists[:m])
                    assert st["n_overflow"] <= m // 100, (kprime, m, graph, st)
