"""knn_distances keeps one index per thread between calls: results must not
depend on what the index held before, on the stream, or on the thread."""
import threading

import numpy as np
import pytest

from rtdsl import workloads

pytestmark = pytest.mark.gpu


def test_kept_index_sizes_streams_threads(rtd, orc, cuda):
    import torch
    from rtdsl import torch_ops
    sets = []
    for n, nq, k in ((4_000, 900, 5), (300, 50, 16), (9_000, 3_000, 3), (40, 7, 60), (6_000, 2_000, 20)):
        pts, q = workloads.clustered(n=n, nq=nq, seed=n, n_clusters=5, box=10.0)
        sets.append((pts, q, k, orc.knn(pts, q, k)))

    failed = []

    def work(order):
        try:
            streams = [torch.cuda.Stream() for _ in range(2)]
            for turn, i in enumerate(order):
                pts, q, k, (rid, rd2) = sets[i]
                with torch.cuda.stream(streams[turn % 2]):
                    P = torch.from_numpy(pts).cuda().requires_grad_()
                    Q = torch.from_numpy(q).cuda().requires_grad_()
                    d2, ids = torch_ops.knn_distances(Q, P, k)
                    real = ids >= 0
                    gq, = torch.autograd.grad(d2[real].sum(), Q)
                    got = ids.cpu().numpy().view(np.uint32), d2.detach().cpu().numpy()
                np.testing.assert_array_equal(got[0], rid)
                np.testing.assert_array_equal(got[1].view(np.uint32), rd2.view(np.uint32))
                assert torch.isfinite(gq).all()
            rtd.release_kept_index()
        except Exception as e:   # noqa: BLE001 - reported by the main thread
            failed.append(e)

    threads = [threading.Thread(target=work, args=(o,)) for o in ([0, 1, 2, 3, 4, 2], [4, 3, 2, 1, 0, 0])]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


def test_kept_index_after_an_error(rtd, cuda):
    import torch
    from rtdsl import torch_ops
    p = torch.rand((100, 3), device=cuda)
    torch_ops.knn_distances(p, p, 3)
    with pytest.raises(rtd.RtdError):
        torch_ops.knn_distances(p, p, 0)
    d2, ids = torch_ops.knn_distances(p, p, 1)
    assert torch.equal(ids[:, 0], torch.arange(100, device=cuda, dtype=torch.int32)) and not d2.any()
