"""FP64 contractions at the band counts where their tiles change: Gram row blocks of
four (4, 12, 20, 28 bands end one early), rotation tiles of 10, 12, 14 and 16 columns,
odd counts (unaligned rows).  Against the FP64 oracle, at the parity tests' tolerances."""
import numpy as np
import pytest

from oracle import restatement as R
from tests.systems import make_system, random_params
from tests.test_gpu_parity import TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 3, 4, 5, 10, 11, 12, 13, 14, 18, 20, 21, 25, 27, 28, 29, 42, 45])
def test_band_count(nb):
  import torch
  from jrystal_gb300.engine import PlaneWavePlan
  sysm = make_system(kind="si2", grid=(18, 18, 18), kgrid=(2, 1, 1), nb=nb, nocc=max(1, nb // 2))
  w = random_params(sysm, seed=nb)
  terms, gr, gi, _ = R.energy_terms(*w, sysm)
  plan = PlaneWavePlan(sysm.cell_vectors, sysm.positions, sysm.charges, sysm.grid, sysm.mask,
                       sysm.kpts, nb, 1, 64, sysm.xc)
  t = [torch.tensor(x, device="cuda") for x in w]
  e, g1, g2 = plan.energy_and_grad(*t, sysm.occupation)
  e = e.cpu().numpy()
  tol = TOL[64]
  for i, name in enumerate(["kinetic", "external", "hartree", "xc", "total"]):
    assert abs(e[i] - terms[name]) <= tol["e_rel"] * max(1.0, abs(terms[name])), name
  scale = max(np.abs(gr).max(), np.abs(gi).max())
  assert max(np.abs(g1.cpu().numpy() - gr).max(), np.abs(g2.cpu().numpy() - gi).max()) <= tol["g_rel"] * scale
  plan.close()
