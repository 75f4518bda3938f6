"""Points that another stream rewrites while DBSCAN runs: the fill may then
find other neighbours than the count and leave slots of the pair buffer
unwritten.  The call reports that, or labels one of the states it saw; it
never uses what was not written, and the index stays usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3_000, 140_000])
def test_dbscan_while_points_change(rtd, orc, cuda, n):
    import torch
    rng = np.random.default_rng(n)
    close = (rng.random((n, 3)) * (n / 20.0) ** (1 / 3)).astype(np.float32)   # some 20 points a unit cube
    A = torch.from_numpy(close).cuda()
    B = A * 50.0 + 1000.0   # no neighbours, and far from the index's points
    P = A.clone()
    ix = rtd.Index().build(P)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    for _ in range(10):
        with torch.cuda.stream(side):
            torch.cuda._sleep(4_000_000)   # about 2 ms, in which the copies queue up
            for _ in range(300):
                P.copy_(B)
                P.copy_(A)
            done.record()
        while not done.query():
            try:
                labels, nc = rtd.dbscan(P, 0.6, 4, index=ix)
                got = labels.cpu().numpy()
                assert got.min() >= -1 and got.max() < max(nc, 1)
            except rtd.RtdError:
                pass   # most calls: count and fill disagree
    torch.cuda.synchronize()
    labels, nc = rtd.dbscan(P, 0.6, 4, index=ix)
    if n < 10_000:
        ref, ref_nc = orc.dbscan(close, 0.6, 4)
    else:
        ref, ref_nc = rtd.dbscan(A, 0.6, 4)
        ref = ref.cpu().numpy()
    np.testing.assert_array_equal(labels.cpu().numpy(), ref)
    assert nc == ref_nc
