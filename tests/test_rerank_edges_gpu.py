"""fknn_rerank around the number of candidates a block's threads hold one each
of, where places are counted, and above, where the keys are sorted: repeats,
empty slots and rows at equal distances."""
import numpy as np
import pytest

import fknn
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [1, 2, 31, 32, 33, 255, 256, 257, 511])
def test_places(nc):
    rng = np.random.default_rng(nc)
    n, nq = 3000, 9
    vecs = np.repeat(rng.standard_normal((n // 3, 100), dtype=np.float32), 3, axis=0)
    q = rng.standard_normal((nq, 100), dtype=np.float32)
    cand = rng.integers(0, n, (nq, nc)).astype(np.uint32)
    cand[2, nc // 2:] = cand[2, 0]
    cand[3, ::2] = 0xFFFFFFFF
    cand[4, :] = 0xFFFFFFFF
    with fknn.Index(vecs, np.zeros(n, np.float32), np.zeros(n, np.float32)) as idx:
        for k in {1, (nc + 1) // 2, nc}:
            ids, d = idx.rerank(q, cand, k=k)
            for i in range(nq):
                c = np.unique(cand[i][cand[i] != 0xFFFFFFFF])
                dist = np.array([oracle.lib().oracle_normal_l2(vecs[j].ctypes.data, q[i].ctypes.data, 100) for j in c],
                                np.float32)
                order = np.lexsort((c, dist))[:k]
                m = order.shape[0]
                np.testing.assert_array_equal(ids[i, :m], c[order])
                np.testing.assert_array_equal(d[i, :m], dist[order])
                assert (ids[i, m:] == 0xFFFFFFFF).all() and np.isinf(d[i, m:]).all()
