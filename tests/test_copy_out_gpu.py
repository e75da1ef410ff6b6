"""Results to host memory of any size: below, at and above what several threads
copy, in whole and part pieces, with and without distances, pageable and
pinned; equal to the results left on the device."""
import numpy as np
import pytest

import fknn
from fknn import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 1310, 1311, 2621, 2622, 6000])
def test_host_results(nq):
    torch = pytest.importorskip("torch")
    vecs, labels, ts, q, metas = datagen.make_workload(1, n=20_000, nq=nq)
    with fknn.Index(vecs, labels, ts) as idx:
        d_ids, d_dists = idx.search(torch.from_numpy(q).cuda(), torch.from_numpy(metas).cuda(), k=100)
        want, wd = d_ids.cpu().numpy().view(np.uint32), d_dists.cpu().numpy()
        for _ in range(2):
            ids, dists = idx.search(q, metas, k=100)
            np.testing.assert_array_equal(ids, want)
            np.testing.assert_array_equal(dists, wd)
        pin = torch.empty((nq, 100), dtype=torch.int32).pin_memory().numpy().view(np.uint32)
        dd = np.empty((nq, 100), np.float32)
        idx.search(q, metas, k=100, ids=pin, dists=dd)
        np.testing.assert_array_equal(pin, want)
        np.testing.assert_array_equal(dd, wd)
