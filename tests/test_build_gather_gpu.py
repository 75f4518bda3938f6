"""The build's gather of the points in key order: counts on both sides of 2^16
(up to there the low key bits ride with the index, above the keys are made again
from the points), counts mod 4, arrays off 16-byte alignment, non-finite points;
every point must find itself, and tree searches must match the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65_535, 65_536, 65_537, 65_538, 65_539, 65_540])
@pytest.mark.parametrize("skip", [0, 1, 2, 3])
def test_gathered_points(rtd, orc, cuda, n, skip):
    import torch
    rng = np.random.default_rng(n + skip)
    pts = rng.random((n, 3)).astype(np.float32)
    pts[5::9001] = np.nan
    pts[7::9001, 1] = np.inf
    P = torch.from_numpy(np.concatenate([np.zeros((skip, 3), np.float32), pts])).cuda()[skip:]
    finite = np.isfinite(pts).all(1)
    s = rtd.default_schedule(lanes_per_query=1)
    ids, d2 = rtd.Index().k_nn(P, P, 1, s)
    own = np.nonzero(finite)[0]
    np.testing.assert_array_equal(ids.cpu().numpy()[own, 0], own)
    assert not d2.cpu().numpy()[own].any()
    q = np.concatenate([rng.random((40, 3)), pts[-20:]]).astype(np.float32)
    ids, d2 = rtd.Index().k_nn(P, torch.from_numpy(q).cuda(), 5, s)
    rid, rd2 = orc.knn(pts, q, 5)
    np.testing.assert_array_equal(ids.cpu().numpy().view(np.uint32), rid)
    np.testing.assert_array_equal(d2.cpu().numpy().view(np.uint32), rd2.view(np.uint32))
