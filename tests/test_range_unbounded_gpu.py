"""Points with NaN coordinates lie in boxes without bounds.  A squared radius
of +inf reaches every finite point and none of those, whichever kernel counts:
131,071 queries are counted a warp each, 131,072 with few hits a thread each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [131_071, 131_072])
@pytest.mark.parametrize("leaf", [1, 12])
def test_range_unbounded_boxes_many_queries(rtd, orc, cuda, nq, leaf):
    import torch
    rng = np.random.default_rng(nq)
    pts = rng.normal(size=(2_000, 3)).astype(np.float32)
    pts[rng.permutation(2_000)[:1_975], 1] = np.nan
    q = rng.normal(size=(nq, 3)).astype(np.float32)
    finite = np.flatnonzero(np.isfinite(pts).all(axis=1)).astype(np.uint32)
    s = rtd.default_schedule(leaf_size=leaf)
    Q = torch.from_numpy(q).cuda()
    ix = rtd.Index().build(torch.from_numpy(pts).cuda(), s)
    for r in (1.0, 1e30):   # 1e30 squares to +inf
        if r > 1e20:
            want = np.stack([np.repeat(np.arange(nq, dtype=np.uint32), 25), np.tile(finite, nq)], 1)
        else:
            want = orc.range_pairs(pts[finite], q, r)
            want[:, 1] = finite[want[:, 1]]
        for _ in range(2):   # the second count pushes its pairs
            counts, total = ix.range_count(Q, r, s)
            assert total == len(want)
            np.testing.assert_array_equal(counts.cpu().numpy().view(np.uint32),
                                          np.bincount(want[:, 0], minlength=nq))
            pairs = ix.range_fill(Q, r, total, sort_pairs=True, schedule=s)
            np.testing.assert_array_equal(pairs.cpu().numpy().view(np.uint32), want)
        other = rtd.Index().build(torch.from_numpy(pts).cuda(), s)   # a fill without a count
        pairs = other.range_fill(Q, r, len(want), sort_pairs=True, schedule=s)
        np.testing.assert_array_equal(pairs.cpu().numpy().view(np.uint32), want)
