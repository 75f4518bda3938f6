"""The collecting warp search (knn_collect.cuh) against the oracle: list and
candidate-buffer edges, pyramid edges, ties across the cut, non-finite
coordinates, and the rules that choose between it and a thread per query."""
import numpy as np
import pytest

from rtdsl import workloads

pytestmark = pytest.mark.gpu


def check(rtd, orc, pts, q, k, **sched):
    import torch
    s = rtd.default_schedule(**sched)
    P, Q = torch.from_numpy(pts).cuda(), torch.from_numpy(q).cuda()
    ix = rtd.Index()
    rid, rd2 = orc.knn(pts, q, k)
    for ids, d2 in (ix.k_nn(P, Q, k, s), ix.build(P, s).knn(Q, k, s)):
        np.testing.assert_array_equal(ids.cpu().numpy().view(np.uint32), rid)
        np.testing.assert_array_equal(d2.cpu().numpy().view(np.uint32), rd2.view(np.uint32))
    ix.info()   # raises on a device error flag


@pytest.mark.parametrize("k", [1, 5, 16, 17, 22, 23, 32, 33, 51, 52, 64, 65, 128, 255, 256, 257, 410, 513, 1000, 2047,
                               2048, 2049])
def test_collect_list_sizes(rtd, orc, cuda, k):
    pts, q = workloads.clustered(n=9_001, nq=301, seed=k, n_clusters=9, box=10.0)
    check(rtd, orc, pts, q, k, lanes_per_query=32)


@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 65, 72, 256, 257, 2048, 2049, 2056, 16_385, 131_073])
@pytest.mark.parametrize("bits", [30, 48])
def test_collect_pyramid_sizes(rtd, orc, cuda, n, bits):
    rng = np.random.default_rng(n)
    pts = rng.random((n, 3), dtype=np.float32)
    q = np.concatenate([rng.random((60, 3)), rng.random((10, 3)) * 40 - 20]).astype(np.float32)
    check(rtd, orc, pts, q, 20, morton_bits=bits, lanes_per_query=32)


@pytest.mark.parametrize("k", [4, 30, 100, 700])
def test_collect_ties_and_duplicates(rtd, orc, cuda, k):
    rng = np.random.default_rng(k)
    grid = rng.integers(0, 4, size=(4_000, 3)).astype(np.float32)   # 64 places, about 62 points each
    q = np.concatenate([grid[:60], rng.random((20, 3)) * 4]).astype(np.float32)
    check(rtd, orc, grid, q, k, lanes_per_query=32)
    same = np.full((3_000, 3), 0.25, np.float32)
    check(rtd, orc, same, q[:20], k, lanes_per_query=32)


@pytest.mark.parametrize("k", [5, 40, 300])
def test_collect_non_finite(rtd, orc, cuda, k):
    rng = np.random.default_rng(3)
    pts = rng.normal(size=(2_000, 3)).astype(np.float32)
    pts[::17, 0] = np.nan
    pts[5::41, 1] = np.inf
    pts[7::43, 2] = -np.inf
    pts[11::301] = 3e38
    q = rng.normal(size=(64, 3)).astype(np.float32)
    q[3, 2] = np.nan
    q[4, 0] = np.inf
    q[5] = -3e38
    check(rtd, orc, pts, q, k, lanes_per_query=32)


@pytest.mark.parametrize("nq,k", [(7_999, 1), (8_000, 1), (8_001, 1), (24_000, 3), (24_001, 3), (49_151, 17),
                                  (49_152, 17), (94_720, 13), (96_001, 12), (189_440, 14), (378_881, 13)])
def test_search_and_order_rules(rtd, orc, cuda, nq, k):
    pts, q = workloads.clustered(n=6_000, nq=nq, seed=nq, n_clusters=9, box=10.0)
    check(rtd, orc, pts, q, k)
