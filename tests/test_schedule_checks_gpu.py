"""Schedules that no search takes are refused whichever kernel the search
would run."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,k", [(10, 1), (10, 5), (40_000, 1), (100, 300), (20, 3_000)])
@pytest.mark.parametrize("partial", [0, 1])
@pytest.mark.parametrize("heuristic", [-1, 5, 77])
def test_unknown_radius_heuristic_refused(rtd, cuda, nq, k, partial, heuristic):
    import torch
    p, q = torch.rand((4_000, 3), device=cuda), torch.rand((nq, 3), device=cuda)
    s = rtd.default_schedule(radius_heuristic=heuristic, partial_results=partial)
    ix = rtd.Index().build(p)
    with pytest.raises(rtd.RtdError, match="radius heuristic"):
        ix.knn(q, k, s)
    with pytest.raises(rtd.RtdError, match="radius heuristic"):
        ix.k_nn(p, q, k, s)
    with pytest.raises(rtd.RtdError, match="radius heuristic"):
        rtd.KnnGraph(p, q, k, s)
    ids, _ = ix.knn(q, k)   # the index is as it was
    assert int(ids[:, 0].min()) >= 0
