"""Counts and fills a thread per query (131,072 queries and more with few hits
each) and the edges of the rule that chooses them from a sample of every
nq / 1,024-th query: 64 hits on average, at 131,072 queries 128 hits of one
query, and 6.84 on average for pushing counts over leaves of up to 5 points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(rtd, orc, pts, q, r, leaf):
    import torch
    want = orc.range_pairs(pts, q, r)
    s = rtd.default_schedule(leaf_size=leaf)
    P, Q = torch.from_numpy(pts).cuda(), torch.from_numpy(q).cuda()
    ix = rtd.Index().build(P, s)
    pairs = ix.range_fill(Q, r, len(want) + 3, sort_pairs=True, schedule=s)   # a fill without a count
    np.testing.assert_array_equal(pairs.cpu().numpy().view(np.uint32), want)
    if len(want):
        with pytest.raises(rtd.RtdError):   # too small a buffer
            ix.range_fill(Q, r, len(want) - 1, schedule=s)
    for turn in range(3):   # the first fill walks, the later ones scatter the count's pairs
        counts, total = ix.range_count(Q, r, s)
        assert total == len(want)
        np.testing.assert_array_equal(counts.cpu().numpy().view(np.uint32), np.bincount(want[:, 0], minlength=len(q)))
        pairs = ix.range_fill(Q, r, total, sort_pairs=turn != 1, schedule=s).cpu().numpy().view(np.uint32)
        if turn == 1:   # grouped by query in any order
            pairs = pairs[np.lexsort((pairs[:, 1], pairs[:, 0]))]
        np.testing.assert_array_equal(pairs, want)


@pytest.mark.parametrize("nq", [131_071, 131_072, 150_001])
@pytest.mark.parametrize("hits", [0, 1, 6, 7, 63, 64, 127, 128])
@pytest.mark.parametrize("every,leaf", [(1, 5), (1, 6), (0, 4)])
def test_range_sample_edges(rtd, orc, cuda, nq, hits, every, leaf):
    """hits points at one place and a query there in every sampled position
    (or in the first alone); the others find one point or none."""
    rng = np.random.default_rng(nq + hits)
    pts = np.concatenate([np.full((hits, 3), 0.25), rng.random((700, 3)) + 1.0]).astype(np.float32)
    pts = np.ascontiguousarray(pts[rng.permutation(len(pts))])
    q = (rng.random((nq, 3)) + 1.0).astype(np.float32)
    q[::2] = rng.random((len(q[::2]), 3)) * 7 + 3   # nothing there
    q[:: nq // 1024 if every else nq] = 0.25
    check(rtd, orc, pts, q, 0.03, leaf)


@pytest.mark.parametrize("leaf", [1, 8, 64])
def test_range_contained_runs(rtd, orc, cuda, leaf):
    """Clumps of 1 to 90 points well inside the ball: contained subtrees below
    and above the 32 points from which the whole warp copies them."""
    rng = np.random.default_rng(leaf)
    sizes = rng.integers(1, 91, 150)
    centres = rng.random((150, 3)) * 40
    pts = np.repeat(centres, sizes, axis=0) + rng.normal(0, 1e-3, (sizes.sum(), 3))
    pts = np.ascontiguousarray(pts[rng.permutation(len(pts))].astype(np.float32))
    q = (centres[rng.integers(0, 150, 140_000)] + rng.normal(0, 0.05, (140_000, 3))).astype(np.float32)
    q[::500] = np.nan
    check(rtd, orc, pts, q, 0.1, leaf)
