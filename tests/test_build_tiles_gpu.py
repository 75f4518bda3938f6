"""Tree nodes of clouds of more than one tile of sorted points: sizes around the
tiles, leaf sizes, key widths, ties and non-finite points; tree searches and the
range query against the oracle, and the node count against a radix tree over
the oracle's Morton codes."""
import numpy as np
import pytest
from test_small_build_gpu import cloud, kept_nodes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4_097, 5_119, 5_120, 5_121, 6_145, 33_000])
@pytest.mark.parametrize("leaf,bits", [(1, 63), (4, 48), (64, 30), (5, 39)])
@pytest.mark.parametrize("kind", ["uniform", "ties", "clusters", "nonfinite"])
def test_build_tiles(rtd, orc, cuda, n, leaf, bits, kind):
    import torch
    pts = cloud(n, kind, n)
    q = np.concatenate([cloud(60, "uniform", 1), cloud(20, "nonfinite", 2), pts[:: n // 30]]).astype(np.float32)
    P, Q = torch.from_numpy(pts).cuda(), torch.from_numpy(q).cuda()
    ix = rtd.Index()
    rid, rd2 = orc.knn(pts, q, 5)
    s = rtd.default_schedule(leaf_size=leaf, morton_bits=bits, lanes_per_query=1)
    ids, d2 = ix.k_nn(P, Q, 5, s)
    np.testing.assert_array_equal(ids.cpu().numpy().view(np.uint32), rid)
    np.testing.assert_array_equal(d2.cpu().numpy().view(np.uint32), rd2.view(np.uint32))
    info = ix.info()
    counts, total = ix.range_count(Q, 0.05, s)
    rc, rt = orc.range_count(pts, q, 0.05)
    assert total == rt
    np.testing.assert_array_equal(counts.cpu().numpy().view(np.uint32), rc)
    if bits == 30 and kind != "nonfinite":
        assert info["n_internal"] == kept_nodes(orc.morton_codes(pts), leaf)
