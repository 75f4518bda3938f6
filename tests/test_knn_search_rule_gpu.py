"""The automatic choice between a thread and a warp per query, at both sides of
its lines: the same neighbours either way, and the oracle's."""
import numpy as np
import pytest

from rtdsl import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,line", [(3_000, 1, 26_500), (3_000, 8, 58_000), (70_000, 5, 44_500), (3_000, 9, 72_000),
                                      (40_000, 12, 96_000), (700, 13, 156_000), (131_072, 16, 192_000),
                                      (131_073, 16, 192_000), (15, 16, 192_000), (900, 1, 10_500), (30_000, 5, 36_500)])
@pytest.mark.parametrize("over", [0, 1])
def test_knn_both_sides_of_the_line(rtd, orc, cuda, n, k, line, over):
    import torch
    pts, q = workloads.clustered(n=n, nq=line + over, seed=n + k, n_clusters=7, box=4.0)
    P, Q = torch.from_numpy(pts).cuda(), torch.from_numpy(q).cuda()
    ix = rtd.Index().build(P)
    ids, d2 = ix.knn(Q, k)
    ids2, d22 = rtd.Index().k_nn(P, Q, k)
    for lanes in (1, 32):
        other_ids, other_d2 = ix.knn(Q, k, rtd.default_schedule(lanes_per_query=lanes))
        for a, b in ((ids, other_ids), (ids2, other_ids), (d2, other_d2), (d22, other_d2)):
            assert torch.equal(a, b)
    some = slice(0, len(q), 997)
    oi, od = orc.KdTree(pts).knn(q[some], k)
    np.testing.assert_array_equal(ids[some].cpu().numpy().view(np.uint32), oi)
    np.testing.assert_array_equal(d2[some].cpu().numpy().view(np.uint32), od.view(np.uint32))
