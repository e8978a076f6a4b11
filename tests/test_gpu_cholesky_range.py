"""Coefficient map of FP32 parameters scaled by powers of two.

C = W R^-1 does not change when W is multiplied by 2^s, and neither does the
condition estimate.  Pivots up to 2^126 only shift their exponents.  Above, the
reciprocal of a pivot is a subnormal float, good to 2^-22: with nb eliminations of
nearly orthogonal columns (each takes away less than a tenth of a column) C moves by
less than nb * 0.1 * 2^-22 = 1e-6 at 40 bands.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s", [60, 62, 63])       # pivots near 2^120.9, 2^124.9, 2^126.9
@pytest.mark.parametrize("nb", [1, 4, 12, 40])
def test_coefficients_of_scaled_parameters(nb, s):
  import torch
  from jrystal_gb300.engine import PlaneWavePlan
  from tests.systems import make_system, random_params
  sysm = make_system(kind="si2", grid=(24, 24, 24), kgrid=(2, 1, 1), nb=nb, nocc=1)
  plan = PlaneWavePlan(sysm.cell_vectors, sysm.positions, sysm.charges, sysm.grid, sysm.mask,
                       sysm.kpts, nb, 1, 32, sysm.xc)
  w = np.stack(random_params(sysm, seed=nb))
  w *= np.sqrt(2.0 ** 0.9 / (w ** 2).sum((0, -2)))[..., None, :]     # column norms^2 of 2^0.9
  w = [torch.tensor(x.astype(np.float32), device="cuda") for x in w]
  ws = [x * 2.0 ** s for x in w]
  c0 = plan.coeff(*w).cpu().numpy()
  e0 = plan.energy_and_grad(*w, sysm.occupation, with_grad=False)[0].cpu().numpy()
  c1 = plan.coeff(*ws).cpu().numpy()
  e1 = plan.energy_and_grad(*ws, sysm.occupation, with_grad=False)[0].cpu().numpy()
  assert np.abs(c1 - c0).max() <= 1e-6 * np.abs(c0).max()
  assert e1[6] == 0 and abs(e1[5] - e0[5]) <= 1e-6 * e0[5]
  plan.close()
