"""The range kernels and the sorts of the pairs at the edges of the rules that
choose them: pyramid sizes, queries in order or not, thread or warp counting
with and without very long segments, and the segment sorts' sizes, against
the oracle."""
import numpy as np
import pytest

from rtdsl import workloads

pytestmark = pytest.mark.gpu


def check(rtd, orc, pts, q, r, passes=2, **sched):
    import torch
    s = rtd.default_schedule(**sched)
    P, Q = torch.from_numpy(pts).cuda(), torch.from_numpy(q).cuda()
    ix = rtd.Index().build(P, s)
    rc, rtotal = orc.range_count(pts, q, r)
    want = orc.range_pairs(pts, q, r) if rtotal < 4_000_000 else None
    for _ in range(passes):   # the second count pushes its pairs
        counts, total = ix.range_count(Q, r, s)
        assert total == rtotal
        np.testing.assert_array_equal(counts.cpu().numpy().view(np.uint32), rc)
        pairs = ix.range_fill(Q, r, total, sort_pairs=True, schedule=s).cpu().numpy().view(np.uint32)
        assert len(pairs) == rtotal
        keys = pairs[:, 0].astype(np.uint64) << np.uint64(32) | pairs[:, 1]
        assert np.all(keys[1:] > keys[:-1])
        np.testing.assert_array_equal(np.bincount(pairs[:, 0], minlength=len(q)), rc)
        if want is not None:
            np.testing.assert_array_equal(pairs, want)


@pytest.mark.parametrize("n", [1, 7, 8, 63, 64, 65, 256, 257, 2_048, 2_049, 16_385, 140_000])
@pytest.mark.parametrize("leaf", [1, 64])
def test_range_pyramid_sizes(rtd, orc, cuda, n, leaf):
    rng = np.random.default_rng(n)
    pts = rng.random((n, 3), dtype=np.float32)
    q = np.concatenate([rng.random((50, 3)), [[np.nan, 0, 0], [9, 9, 9], [0.5, 0.5, 0.5]]]).astype(np.float32)
    for r in (0.0, 0.08, 0.3 if n < 20_000 else 0.1, 3.0):
        check(rtd, orc, pts, q, r, leaf_size=leaf)


@pytest.mark.parametrize("c", [2, 32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 1_025, 4_097, 16_384, 16_385])
def test_range_segment_sizes(rtd, orc, cuda, c):
    """One query with exactly c hits, and neighbours with few or none."""
    rng = np.random.default_rng(c)
    pts = np.concatenate([rng.random((c, 3)) * 0.01, rng.random((500, 3)) * 5 + 1]).astype(np.float32)
    pts = np.ascontiguousarray(pts[rng.permutation(len(pts))])
    q = np.concatenate([[[0.005, 0.005, 0.005], [-7, 0, 0]], pts[:6]]).astype(np.float32)
    check(rtd, orc, pts, q, 0.05)


@pytest.mark.parametrize("nq", [49_151, 49_152, 131_071, 131_072])
@pytest.mark.parametrize("dense", [False, True])
def test_range_count_rules(rtd, orc, cuda, nq, dense):
    pts, q = workloads.clustered(n=20_000, nq=nq, seed=nq, n_clusters=20, box=10.0)
    if dense:   # every 40th query finds 300 points at one place
        pts[:300] = 2.5
        q[::40] = 2.5
    check(rtd, orc, pts, q, 0.02)


def test_range_non_finite_unbounded(rtd, orc, cuda):
    rng = np.random.default_rng(5)
    pts = rng.normal(size=(3_000, 3)).astype(np.float32)
    pts[::50, 1] = np.nan
    pts[7::70, 0] = np.inf
    q = rng.normal(size=(40, 3)).astype(np.float32)
    for r in (1.0, 1e30):   # 1e30 squares to +inf
        check(rtd, orc, pts, q, r)
