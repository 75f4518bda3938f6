"""DBSCAN from 131,072 points on, where the queries run in the index's own order
and a sample of them chooses the counting kernel, and on both sides of the rule
for a second hooking round (7 neighbours a point): against labels made from
the oracle's neighbour pairs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def labels_of_pairs(pairs, n, min_pts):
    """Clusters numbered by their smallest core point; a border point takes the
    smallest number among its core neighbours; noise -1."""
    from scipy.sparse import coo_matrix
    from scipy.sparse.csgraph import connected_components
    a, b = pairs[:, 0].astype(np.int64), pairs[:, 1].astype(np.int64)
    core = np.bincount(a, minlength=n) >= min_pts
    both = core[a] & core[b]
    comp = connected_components(coo_matrix((np.ones(both.sum(), np.int8), (a[both], b[both])), shape=(n, n)),
                                directed=False)[1]
    ids = np.flatnonzero(core)
    first = np.full(comp.max() + 1, n)
    np.minimum.at(first, comp[ids], ids)
    number = np.full(comp.max() + 1, -1)
    real = np.flatnonzero(first < n)
    number[real[np.argsort(first[real])]] = np.arange(len(real))
    labels = np.full(n, np.iinfo(np.int32).max)
    border = ~core[a] & core[b]
    np.minimum.at(labels, a[border], number[comp[b[border]]])
    labels[core] = number[comp[core]]
    labels[labels == np.iinfo(np.int32).max] = -1
    return labels, len(real)


def cloud(kind, n):
    rng = np.random.default_rng(n)
    if kind == "uniform":       # one component through the whole cloud
        return rng.random((n, 3)), (8 / n / 4.19) ** (1 / 3), 5
    if kind == "crowded":       # 40 neighbours a point
        return rng.random((n, 3)), (40 / n / 4.19) ** (1 / 3), 20
    if kind == "sparse":        # mostly noise
        return rng.random((n, 3)), (2 / n / 4.19) ** (1 / 3), 4
    if kind == "dense place":   # the sample finds it: counted a warp per query
        p = rng.random((n, 3))
        p[rng.permutation(n)[:1500]] = 0.5
        return p, (4 / n / 4.19) ** (1 / 3), 5
    # points along a curve, in order or in reverse: long chains of parents
    t = np.arange(n)[:: 1 if kind == "curve" else -1]
    return np.stack([np.cos(t * 1e-3) * 50, np.sin(t * 1e-3) * 50, t * 1e-4], 1), 0.12, 3


@pytest.mark.parametrize("n", [131_071, 131_072, 150_001])
@pytest.mark.parametrize("kind", ["uniform", "crowded", "sparse", "dense place", "curve", "curve reversed"])
def test_dbscan_large(rtd, orc, cuda, kind, n):
    pts, eps, min_pts = cloud(kind, n)
    pts = np.ascontiguousarray(pts, dtype=np.float32)
    want, clusters = labels_of_pairs(orc.KdTree(pts).range_pairs(pts, eps), n, min_pts)
    P = torch.from_numpy(pts).cuda()
    ix = rtd.Index().build(P)
    for _ in range(2):   # the second count pushes its pairs
        labels, nc = rtd.dbscan(P, eps, min_pts, index=ix)
        np.testing.assert_array_equal(labels.cpu().numpy(), want)
        assert nc == clusters
