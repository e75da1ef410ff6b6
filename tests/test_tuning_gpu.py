"""A tuning holds as it was given: row blocks in their unit, and work items per
SM also in small calls, where only the default counts as one.  Results do not
depend on either."""
import numpy as np
import pytest

import fknn

pytestmark = pytest.mark.gpu
N = 40_000


@pytest.fixture(scope="module")
def data():
    rng = np.random.default_rng(2)
    vecs = rng.standard_normal((N, 100), dtype=np.float32)
    q = rng.standard_normal((1100, 100), dtype=np.float32)
    metas = np.tile(np.array([0, -1, -1, -1], np.float32), (1100, 1))
    with fknn.Index(vecs, np.zeros(N, np.float32), rng.random(N, dtype=np.float32), build_bf16=True,
                    build_fp8=True) as idx:
        yield idx, q, metas


MODES = [(fknn.MODE_EXACT_FP32, 64, 0, 4), (fknn.MODE_BF16_RERANK, 128, 256, 3), (fknn.MODE_FP8_RERANK, 128, 256, 3)]


@pytest.mark.parametrize("mode,rows,slack,default", MODES)
def test_shortest_chunk(data, mode, rows, slack, default):
    idx, q, metas = data
    idx.set_tuning(mode, slack, 64, 64, 0, 8)
    want = idx.search(q, metas, mode=mode, kprime=200, return_stats=True)
    st = want[2]
    assert st["n_work_items"] == st["n_tiles"] * -(-N // (64 * rows))
    idx.set_tuning(mode, slack, 64, 8, 0, 8)
    got = idx.search(q, metas, mode=mode, kprime=200)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("mode,rows,slack,default", MODES)
def test_items_per_sm_of_a_small_call(data, mode, rows, slack, default):
    idx, q, metas = data
    out = {}
    for items in (1, 2, default):
        idx.set_tuning(mode, slack, items, 2, 0, 8)
        out[items] = idx.search(q[:300], metas[:300], mode=mode, kprime=200, return_stats=True)
        np.testing.assert_array_equal(out[items][0], out[1][0])
        np.testing.assert_array_equal(out[items][1], out[1][1])
    n = {items: o[2]["n_work_items"] for items, o in out.items()}
    assert n[2] > 1.5 * n[1] and n[default] == n[1]
