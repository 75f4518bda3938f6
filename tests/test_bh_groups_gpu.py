"""Plummer walks at the edges of the warp groups (32 bodies), of the tiles
(32 interactions, odd last pairs) and of the rule that lets a block share a
group: forward against the FP64 evaluation with the same decisions, adjoint
against the FP64 gradient of the direct sum (theta 0, where both are the
same sum) and against the adjoint that walks instead of replaying."""
import numpy as np
import pytest

from rtdsl import BH_LAW_PLUMMER, default_bh_params, workloads
from rtdsl.bh import BarnesHut

pytestmark = pytest.mark.gpu
SHARED = 148 * 5 * 32   # bodies up to which a block shares a group


def bodies(n):
    pos, mass = workloads.plummer(n, seed=n)
    return pos, (mass * (1.0 + np.arange(n) % 5)).astype(np.float32)


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("quad", [0, 1])
@pytest.mark.parametrize("n,bucket", [(2, 1), (31, 4), (32, 4), (33, 4), (65, 100), (1_000, 40), (SHARED, 16),
                                      (SHARED + 1, 16), (SHARED + 33, 50)])
def test_forward_group_edges(orc, cuda, n, bucket, quad):
    # 2e-5: FP32 sums of a few thousand terms, as for the other frozen checks
    import torch
    pos, mass = bodies(n)
    p = default_bh_params(law=BH_LAW_PLUMMER, theta=0.6, eps=1e-2, G=1.0, bucket=bucket, quadrupole=quad)
    bh = BarnesHut().build(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda(), p)
    acc, phi = bh.forward(p)
    _, ophi, oacc = orc.PlummerFrozen(pos, mass, theta=0.6, bucket=bucket).eval(pos, mass, eps=1e-2, G=1.0,
                                                                               quad=bool(quad))
    assert rel(acc.cpu().numpy(), oacc) < 2e-5 and rel(phi.cpu().numpy(), ophi) < 2e-5


@pytest.mark.parametrize("n", [2, 3, 31, 33, 64, 97, 2_049])
def test_adjoint_group_edges_direct(orc, cuda, n):
    # 1e-3: a pair's FP32 derivative is good to about 20 roundings (1e-6) and
    # close pairs dominate the norm; one lost pair among 2,049 bodies is not
    # visible, one lost lane, source or tile is
    import torch
    pos, mass = bodies(n)
    p = default_bh_params(law=BH_LAW_PLUMMER, theta=0.0, eps=5e-2, G=1.0, bucket=8)
    bh = BarnesHut().build(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda(), p)
    _, _, acc64, gp64, gm64 = orc.direct_plummer_f64(pos, mass, 5e-2, 1.0, grad=True)
    for _ in range(4):   # walked, then recorded and replayed
        acc, phi = bh.forward(p)
        gp, gm = bh.backward(acc, torch.ones_like(phi), p)
        assert rel(gp.cpu().numpy(), gp64) < 1e-3 and rel(gm.cpu().numpy(), gm64) < 1e-3


@pytest.mark.parametrize("quad", [0, 1])
@pytest.mark.parametrize("n", [40, 1_025, SHARED, SHARED + 1])
def test_adjoint_walked_and_replayed(cuda, n, quad):
    import torch
    pos, mass = bodies(n)
    p = default_bh_params(law=BH_LAW_PLUMMER, theta=0.7, eps=1e-2, G=1.0, bucket=20, quadrupole=quad)
    bh = BarnesHut().build(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda(), p)
    outs = []
    for _ in range(4):
        acc, phi = bh.forward(p)
        gp, gm = bh.backward(acc, torch.ones_like(phi), p)
        outs.append((gp.cpu().numpy(), gm.cpu().numpy()))
    assert bh.info()["log_pages"] > 0
    for gp, gm in outs[1:]:   # the same terms, FP32 atomics in another order
        assert rel(gp, outs[0][0]) < 1e-5 and rel(gm, outs[0][1]) < 1e-5
