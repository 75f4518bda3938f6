"""The one-launch build of small clouds: element counts around its block sizes,
leaf sizes, key widths, ties and non-finite points; searches of both kinds and
the range query against the oracle, the node count against a radix tree over
the oracle's Morton codes, and the switch to the larger build."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cloud(n, kind, seed):
    rng = np.random.default_rng(seed)
    p = rng.random((n, 3)).astype(np.float32)
    if kind == "ties":
        p = (rng.integers(0, 3, size=(n, 3)) / 2).astype(np.float32)
    elif kind == "clusters":
        p = (rng.random((8, 3))[rng.integers(0, 8, n)] + rng.normal(size=(n, 3)) * 1e-3).astype(np.float32)
    elif kind == "nonfinite":
        p[::7, 0] = np.nan
        p[3::11, 2] = np.inf
    return p


def kept_nodes(codes, leaf):
    """Nodes with more than `leaf` points of the radix tree over (code, rank)."""
    keys = np.sort(codes.astype(np.uint64)) << np.uint64(32) | np.arange(len(codes), dtype=np.uint64)
    count, todo = 0, [(0, len(keys))]
    while todo:
        a, b = todo.pop()
        if b - a <= max(leaf, 1):
            continue
        count += 1
        bit = int(keys[a] ^ keys[b - 1]).bit_length() - 1
        split = a + int(np.searchsorted(keys[a:b] >> np.uint64(bit), (keys[a] >> np.uint64(bit)) + np.uint64(1)))
        todo += [(a, split), (split, b)]
    return count


@pytest.mark.parametrize("n", [1, 2, 4, 5, 63, 64, 65, 72, 513, 1_023, 1_024, 1_025, 2_047, 2_048, 2_049, 4_095,
                               4_096, 4_097])
@pytest.mark.parametrize("leaf,bits", [(1, 63), (4, 48), (64, 30), (5, 39)])
@pytest.mark.parametrize("kind", ["uniform", "ties", "clusters", "nonfinite"])
def test_small_build(rtd, orc, cuda, n, leaf, bits, kind):
    import torch
    pts = cloud(n, kind, n)
    q = np.concatenate([cloud(40, "uniform", 1), cloud(20, "nonfinite", 2), pts[:20]]).astype(np.float32)
    P, Q = torch.from_numpy(pts).cuda(), torch.from_numpy(q).cuda()
    ix = rtd.Index()
    for k, lanes in ((3, 1), (9, 32)):
        s = rtd.default_schedule(leaf_size=leaf, morton_bits=bits, lanes_per_query=lanes)
        ids, d2 = ix.k_nn(P, Q, k, s)
        rid, rd2 = orc.knn(pts, q, k)
        np.testing.assert_array_equal(ids.cpu().numpy().view(np.uint32), rid)
        np.testing.assert_array_equal(d2.cpu().numpy().view(np.uint32), rd2.view(np.uint32))
    info = ix.info()
    counts, total = ix.range_count(Q, 0.11, s)
    rc, rt = orc.range_count(pts, q, 0.11)
    assert total == rt
    np.testing.assert_array_equal(counts.cpu().numpy().view(np.uint32), rc)
    if bits == 30 and kind != "nonfinite":
        assert info["n_internal"] == kept_nodes(orc.morton_codes(pts), leaf)
        np.testing.assert_array_equal(np.float32(info["lo"]), pts.min(0))
        np.testing.assert_array_equal(np.float32(info["hi"]), pts.max(0))


@pytest.mark.parametrize("heuristic,param", [(0, 0.0625), (1, 0.1), (3, 1.0)])
def test_small_build_radius_samples(rtd, orc, cuda, heuristic, param):
    """The radius rounds (partial lists allowed) start from the build's samples."""
    import torch
    pts, q = cloud(3_001, "uniform", 5), cloud(50, "uniform", 6)
    s = rtd.default_schedule(radius_heuristic=heuristic, radius_param=param, partial_results=1)
    ids, _ = rtd.Index().k_nn(torch.from_numpy(pts).cuda(), torch.from_numpy(q).cuda(), 6, s)
    np.testing.assert_array_equal(ids.cpu().numpy().view(np.uint32), orc.knn(pts, q, 6)[0])
