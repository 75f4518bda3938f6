"""The batched search's list classes at their edges, alone and mixed, on
clouds around the sizes at which a window or a pyramid level is the whole
cloud: every query equal to the oracle, eager, captured and with NULL d2."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 7, 8, 64, 65, 257, 2_049, 5_000]


def clouds(seed, ks, empty=False):
    rng = np.random.default_rng(seed)
    out = []
    for i, k in enumerate(ks):
        n = SIZES[(i + seed) % len(SIZES)]
        p = rng.normal(size=(n, 3)).astype(np.float32)
        q = rng.normal(size=(11 + 5 * i, 3)).astype(np.float32)
        if i % 3 == 0:
            p[n // 2:] = p[: n - n // 2]          # duplicates
        if i % 4 == 1:
            p[0, 0], q[0, 1] = np.nan, np.nan
        out.append((p, q, k))
        if empty:
            out.append((np.zeros((0, 3), np.float32), q[:3], k))
    return out


@pytest.mark.parametrize("ks", [[1] * 8, [9] * 8, [64] * 8, [512, 513] * 4, [1, 5, 6, 8, 9, 16, 17, 33, 65, 256, 300, 600],
                                [2, 3], [40, 20]])
@pytest.mark.parametrize("graph", [False, True])
def test_batch_list_classes(rtd, orc, cuda, ks, graph):
    import torch
    for seed, empty in ((0, False), (3, True)):
        cl = clouds(seed, ks, empty)
        b = rtd.Batch([(len(p), len(q), k) for p, q, k in cl])
        P = torch.from_numpy(np.concatenate([c[0] for c in cl])).cuda()
        Q = torch.from_numpy(np.concatenate([c[1] for c in cl])).cuda()
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(2 if graph else 1):
                ids, d2 = b.knn(P, Q, use_graph=graph)
            only, none = b.knn(P, Q, with_d2=False)
            torch.cuda.synchronize()
        assert none is None and torch.equal(only, ids)
        for (p, q, k), i, d in zip(cl, b.split(ids.cpu().numpy().view(np.uint32)), b.split(d2.cpu().numpy())):
            rid, rd2 = orc.knn(p, q, k)
            np.testing.assert_array_equal(i, rid)
            np.testing.assert_array_equal(d.view(np.uint32), rd2.view(np.uint32))
