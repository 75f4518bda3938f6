"""Searches with the reference's round cap and lists of 257 to 2,048 entries in
shared memory: every length launches, also where the lists and the kernel's own
arrays pass 48 KB only together."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [257, 1_000, 1_280, 1_400, 1_500, 1_536, 1_537, 2_048])
def test_partial_results_long_lists(rtd, orc, cuda, k):
    import torch
    rng = np.random.default_rng(k)
    pts = rng.random((3_000, 3), dtype=np.float32)
    q = rng.random((20, 3), dtype=np.float32)
    # a first radius that reaches every point: the capped rounds are exact
    s = rtd.default_schedule(partial_results=1, max_rounds=1, radius_heuristic=rtd.RADIUS_FIXED, radius_param=4.0)
    ids, d2 = rtd.Index().build(torch.from_numpy(pts).cuda(), s).knn(torch.from_numpy(q).cuda(), k, s)
    oi, od = orc.knn(pts, q, k)
    np.testing.assert_array_equal(ids.cpu().numpy().view(np.uint32), oi)
    np.testing.assert_array_equal(d2.cpu().numpy().view(np.uint32), od.view(np.uint32))
