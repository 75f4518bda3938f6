"""Cells and bodies without a finite place.  A cell whose mass-weighted
coordinates overflow to +inf and -inf has a NaN in its centre of mass.  No body
accepts such a cell, so its bodies are summed one by one, however far the cell
lies on its other axes.  And a body without a finite place reaches the bodies
that open its leaf, not those beside them that do not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6, 32, 33, 400])
@pytest.mark.parametrize("quad", [0, 1])
def test_plummer_opens_cells_with_a_nan_centre(rtd, cuda, n, quad):
    import torch
    rng = np.random.default_rng(n)
    # x of both signs and y of one sign: with these masses the products with x
    # sum to inf - inf, those with y to inf, those with z to a number
    pos = np.stack([np.where(np.arange(n) % 2, 1.0, -1.0) * rng.uniform(50, 100, n), rng.uniform(50, 100, n),
                    rng.uniform(-1e-3, 1e-3, n)], 1).astype(np.float32)
    mass = rng.uniform(1e37, 2e37, n).astype(np.float32) / np.float32(n)
    mass[:6] = 1e37   # (the sums stay finite, the products do not)
    p = rtd.default_bh_params(law=rtd.BH_LAW_PLUMMER, theta=0.5, eps=1e-3, G=1e-30, quadrupole=quad, bucket=512)
    bh = rtd.BarnesHut().build(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda(), p)
    acc, phi = bh.forward(p)
    x, m = pos.astype(np.float64), mass.astype(np.float64)
    d = x[None] - x[:, None]
    i1 = 1.0 / np.sqrt((d ** 2).sum(-1) + 1e-6)
    np.fill_diagonal(i1, 0.0)
    want = 1e-30 * (d * (m[None, :] * i1 ** 3)[..., None]).sum(1)
    want_phi = -1e-30 * (m[None, :] * i1).sum(1)
    # FP32 sums of n terms of either sign, each of some 16 roundings
    rel = (n + 16) * 2.0 ** -23
    scale = 1e-30 * np.abs(d * (m[None, :] * i1 ** 3)[..., None]).sum(1)
    fits = (m[None, :] * i1 ** 3).max(1) < 1e38   # mass / distance^3 of every pair within FP32
    assert fits.sum() >= n - 2
    assert np.all((np.abs(acc.cpu().numpy() - want) <= rel * scale)[fits])
    np.testing.assert_allclose(phi.cpu().numpy(), want_phi, rtol=rel)


@pytest.mark.parametrize("n", [17, 31, 40])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_plummer_bodies_beside_one_that_is_nowhere(rtd, cuda, n, axis):
    """Negative masses leave the root's centre at the origin, body 0 among them:
    the bodies far enough from it take the root, the near ones open it."""
    import torch
    rng = np.random.default_rng(n + axis)
    pos = (rng.normal(size=(n, 3)) * 10).astype(np.float32)
    pos[0, axis] = np.nan
    mass = -rng.uniform(0.5, 1.0, n).astype(np.float32)
    p = rtd.default_bh_params(law=rtd.BH_LAW_PLUMMER, theta=3.0, eps=1e-3, G=1.0, quadrupole=0, bucket=64)
    bh = rtd.BarnesHut().build(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda(), p)
    acc, phi = (t.cpu().numpy() for t in bh.forward(p))
    x = pos.astype(np.float64)
    width = float(np.subtract(*[np.asarray(bh.info()[k]) for k in ("root_max", "root_min")]).max())
    r = np.sqrt((x ** 2).sum(1))
    far = r * 3.0 > width * 1.001
    assert 2 < far.sum() < n - 2
    total = mass.astype(np.float64).sum()
    np.testing.assert_allclose(phi[far], -total / np.sqrt(r[far] ** 2 + 1e-6), rtol=(n + 16) * 2.0 ** -23)
    np.testing.assert_allclose(acc[far], -total * x[far] / (r[far] ** 2 + 1e-6)[:, None] ** 1.5,
                               rtol=(n + 16) * 2.0 ** -23)
    assert np.isnan(acc[r * 3.0 < width * 0.999]).all()
