"""Reference-law walk on the GPU at the sizes where the number of bodies a
warp takes changes, and at partly filled last warps: bitwise equal to the
oracle's walk."""
import numpy as np
import pytest

from rtdsl import BH_LAW_REFERENCE, default_bh_params, workloads
from rtdsl.bh import BarnesHut

pytestmark = pytest.mark.gpu
FULL = 148 * 42


@pytest.mark.parametrize("n", [1, 3, 33, 2 * FULL, 2 * FULL + 1, 4 * FULL + 3, 32 * FULL, 32 * FULL + 5])
def test_reference_walk_bitwise_at_group_edges(orc, cuda, n):
    import torch
    pos, mass = workloads.plummer(n, seed=n)
    mass = (mass * (1.0 + (np.arange(n) % 7))).astype(np.float32)
    nodes, order, _ = orc.bh_build(pos, mass, bucket=128)
    bh = BarnesHut().build(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda(),
                           default_bh_params(law=BH_LAW_REFERENCE))
    out, _ = bh.forward(default_bh_params(law=BH_LAW_REFERENCE, theta=0.8, G=1.0))
    sel = np.unique(np.concatenate([np.arange(min(n, 40)), np.arange(max(0, n - 40), n),
                                    np.random.default_rng(1).integers(0, n, 400)])).astype(np.uint32)
    ref = orc.bh_ref_forces_at(pos, mass, nodes, order, sel, 0.8, 1.0)
    got = out.cpu().numpy()[sel]
    assert np.array_equal(got.view(np.uint32), np.asarray(ref, np.float32).view(np.uint32))
