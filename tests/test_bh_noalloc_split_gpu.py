"""rtd_bh_forward_noalloc where the warps of a block share a group: the bits of
rtd_bh_forward, also with more groups than the fixed stacks have blocks."""
import ctypes as C

import numpy as np
import pytest
import torch

from rtdsl import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 4_700, 4_800, 23_680, 23_681])
@pytest.mark.parametrize("quad", [0, 1])
def test_noalloc_equals_forward_in_shared_groups(rtd, cuda, n, quad):
    pos, mass = workloads.plummer(n, seed=n)
    p = rtd.default_bh_params(law=rtd.BH_LAW_PLUMMER, theta=0.6, eps=1e-3, G=1.0, bucket=16, quadrupole=quad)
    bh = rtd.BarnesHut().build(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda(), p)
    acc, phi = torch.full((n, 3), np.nan, device=cuda), torch.full((n,), np.nan, device=cuda)
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert rtd.load().rtd_bh_forward_noalloc(bh._h, C.byref(p), C.c_void_p(acc.data_ptr()),
                                             C.c_void_p(phi.data_ptr()), st) == 0
    ref_acc, ref_phi = bh.forward(p)
    for got, ref in ((acc, ref_acc), (phi, ref_phi)):
        assert torch.isfinite(got).all()
        np.testing.assert_array_equal(got.cpu().numpy().view(np.uint32), ref.cpu().numpy().view(np.uint32))
