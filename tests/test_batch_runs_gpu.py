"""The batched build's boxes and gather where a warp's run of points meets many
clouds: clouds of 0 to 70 points between larger ones, non-finite points, a cloud
without a finite coordinate, arrays off 16-byte alignment."""
import numpy as np
import pytest
from test_batch_gpu import check_against_oracle, packed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skip", [0, 1, 2])
@pytest.mark.parametrize("clouds", [3, 400])
def test_batch_runs(rtd, orc, cuda, skip, clouds):
    import torch
    rng = np.random.default_rng(clouds + skip)
    cl = []
    for c in range(clouds):
        n = 9_000 if c % 97 == 1 else int(rng.integers(0, 71))
        p = (rng.random((n, 3)) * (1 + c % 5) - c).astype(np.float32)
        if c % 7 == 3:
            p[::5, c % 3] = np.nan
            p[1::9, 1] = np.inf
        if c % 50 == 20:
            p[:] = np.nan
        q = (rng.random((11, 3)) * (1 + c % 5) - c).astype(np.float32)
        cl.append({"points": p, "queries": q, "k": (1, 6, 12)[c % 3]})
    pts, q, sizes = packed(cl)
    P = torch.from_numpy(np.concatenate([np.zeros((skip, 3), np.float32), pts])).cuda()[skip:]
    b = rtd.Batch(sizes)
    ids, d2 = b.knn(P, torch.from_numpy(q).cuda())
    check_against_oracle(orc, b, cl, ids, d2)
