"""The SQ8 slab brute force over the edges of its parts (the replayed prefix,
the end of the first screened part, the last short tile) and of its heap (one
node, a level more or less, the largest k), with floods of equal distances,
and in an order of rows that fills the candidate lists; the heap array of every
query equals the oracle's."""
import numpy as np
import pytest

import fknn
import oracle

pytestmark = pytest.mark.gpu


def check(codes, alpha, qv, k):
    npoints, nq = codes.shape[0], qv.shape[0]
    ids = np.empty((nq, k), dtype=np.int32)
    d = np.empty((nq, k), dtype=np.float32)
    fknn.bruteforce_subgraph(100, k, ids, d, npoints, codes, alpha, nq, qv)
    for i in range(nq):
        oi, od = oracle.sq8_bruteforce(k, codes, alpha, qv[i], with_dists=True)
        np.testing.assert_array_equal(ids[i], oi, err_msg=f"n {npoints} k {k} query {i}")
        np.testing.assert_array_equal(d[i], od)


@pytest.mark.parametrize("npoints", [1, 127, 129, 8191, 8192, 8193, 8320, 65536, 65537, 66000, 140_001])
def test_part_edges(npoints):
    rng = np.random.default_rng(npoints)
    vecs = np.repeat(rng.standard_normal((npoints // 4 + 1, 100), dtype=np.float32), 4, axis=0)[:npoints]
    alpha, codes = oracle.sq8_sym_train(vecs)
    qv = oracle.sq8_sym_encode(rng.standard_normal((3, 100), dtype=np.float32), alpha)
    for k in (1, 2, 3, 4, 7, 8, 127, 128, 129, 1023, 1024, 2048):
        if k <= npoints:
            check(codes, alpha, qv, k)


@pytest.mark.parametrize("nq", [1, 33, 130])
def test_queries_around_the_tiles(nq):
    rng = np.random.default_rng(nq)
    alpha, codes = oracle.sq8_sym_train(rng.standard_normal((70_000, 100), dtype=np.float32))
    qv = oracle.sq8_sym_encode(rng.standard_normal((nq, 100), dtype=np.float32), alpha)
    check(codes, alpha, qv, 140)


@pytest.mark.parametrize("npoints", [20_000, 80_000])
def test_rows_that_come_nearer_fill_the_lists(npoints):
    """Every row is nearer to the queries than the ones before: each enters
    the heap, the lists overflow and the codes are scanned instead."""
    rng = np.random.default_rng(npoints)
    q = rng.standard_normal((2, 100), dtype=np.float32)
    far = np.linspace(4.0, 0.0, npoints, dtype=np.float32)[:, None]
    vecs = q[:1] + far * rng.standard_normal((npoints, 100), dtype=np.float32)
    alpha, codes = oracle.sq8_sym_train(vecs)
    check(codes, alpha, oracle.sq8_sym_encode(q, alpha), 140)


@pytest.mark.parametrize("npoints", [300, 9000])
def test_more_queries_than_are_replayed_at_once(npoints):
    rng = np.random.default_rng(npoints)
    alpha, codes = oracle.sq8_sym_train(rng.standard_normal((npoints, 100), dtype=np.float32))
    nq, k = 6200, 10  # 4,736 and 1,464 where the slab is long enough
    qv = oracle.sq8_sym_encode(rng.standard_normal((nq, 100), dtype=np.float32), alpha)
    ids = np.empty((nq, k), dtype=np.int32)
    d = np.empty((nq, k), dtype=np.float32)
    fknn.bruteforce_subgraph(100, k, ids, d, npoints, codes, alpha, nq, qv)
    for i in [0, 1, 4735, 4736, 4737, *range(nq - 10, nq)]:
        oi, od = oracle.sq8_bruteforce(k, codes, alpha, qv[i], with_dists=True)
        np.testing.assert_array_equal(ids[i], oi, err_msg=f"query {i}")
        np.testing.assert_array_equal(d[i], od)


def test_scratch_of_a_short_slab_is_bounded():
    """The prefix's distances are made for as many queries as are replayed at
    once, however many the call has."""
    import threading

    import torch
    n, nq, k = 8192, 8192, 10
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    codes = torch.randint(-127, 128, (n, 112), generator=g, device="cuda", dtype=torch.int8)
    q = torch.randint(-127, 128, (nq, 112), generator=g, device="cuda", dtype=torch.int8)
    codes[:, 100:] = 0
    q[:, 100:] = 0
    out = torch.empty((nq, k), dtype=torch.int32, device="cuda")
    d = torch.empty((nq, k), device="cuda")
    torch.cuda.synchronize()
    used = []

    def call():  # a thread has a scratch of its own
        before = torch.cuda.mem_get_info()[0]
        fknn.bruteforce_subgraph(100, k, out, d, n, codes, 1.0, nq, q)
        used.append(before - torch.cuda.mem_get_info()[0])
        fknn._lib.load().fknn_sq8_release_thread_scratch()

    t = threading.Thread(target=call)
    t.start()
    t.join()
    assert used and used[0] < 180 << 20, used
