"""knn_distances and the index it keeps per thread, as far as that goes
without a GPU: what is refused."""
import pytest
import torch


@pytest.mark.parametrize("queries,points,error", [
    (torch.rand(5, 3), torch.rand(5, 3), "CUDA"),
    (torch.rand(5, 3), torch.tensor(1.0), "CUDA"),
    (torch.tensor(1.0), torch.rand(5, 3), "CUDA"),
])
def test_knn_distances_refuses_host_tensors(rtd, queries, points, error):
    from rtdsl import torch_ops
    with pytest.raises(TypeError, match=error):
        torch_ops.knn_distances(queries, points, 2)
