"""A non-finite coefficient in a band of weight zero: every route of the density
gives a non-finite density of its spin, as the sum of 0 * |psi|^2 does, and
leaves the other spin as it was."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("mask", ["sphere", "cubic"])      # column-first and plane-first transforms
@pytest.mark.parametrize("prec", [32, 64])
def test_empty_band_with_a_nonfinite_coefficient(prec, mask, bad):
  import torch
  from jrystal_gb300.engine import PlaneWavePlan
  from tests.systems import make_system, random_params
  sysm = make_system(kind="si2", grid=(24, 24, 24), kgrid=(2, 1, 1), nb=35, nocc=2, mask=mask)
  plan = PlaneWavePlan(sysm.cell_vectors, sysm.positions, sysm.charges, sysm.grid, sysm.mask,
                       sysm.kpts, 35, 2, prec, sysm.xc)
  w = [torch.tensor(x, device="cuda").to(plan.rdtype) for x in random_params(sysm, seed=7, ns=2)]
  c = plan.coeff(*w)
  occ = np.zeros((2, 2, 35))
  occ[..., :30] = 0.5
  occ[:, 1, 3] = 0.0
  rho = plan.density(c, occ).clone()
  assert torch.isfinite(rho).all()
  for s, k, g, b in ((0, 1, 5, 3), (1, 0, c.shape[2] - 1, 34)):
    d = c.clone()
    torch.view_as_real(d)[s, k, g, b, 1] = bad
    out = plan.density(d, occ)
    assert not torch.isfinite(out[s]).any()
    assert torch.equal(out[1 - s], rho[1 - s])
  assert torch.equal(plan.density(c, occ), rho)            # nothing of it is kept
  plan.close()
