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


@pytest.mark.parametrize("prec,nb", [(64, 9), (64, 12), (64, 14), (64, 27), (64, 28), (32, 27), (32, 32), (32, 45)])
def test_adam_epilogue_of_the_rotation(prec, nb):
  """The single-stream step (Adam inside the adjoint rotation) against gradient and
  update in two calls: the same arithmetic, a few roundings apart."""
  import torch
  from jrystal_gb300 import _lib
  from jrystal_gb300.engine import PlaneWavePlan, adam_update
  lib = _lib.load()
  sysm = make_system(kind="si2", grid=(18, 18, 18), kgrid=(2, 1, 1), nb=nb, nocc=max(1, nb // 2))
  plan = PlaneWavePlan(sysm.cell_vectors, sysm.positions, sysm.charges, sysm.grid, sysm.mask,
                       sysm.kpts, nb, 1, prec, sysm.xc)
  occ = torch.tensor(sysm.occupation, device="cuda")
  p1 = torch.tensor(np.stack(random_params(sysm, seed=nb)), device="cuda").to(plan.rdtype)
  p2, g1 = p1.clone(), torch.empty_like(p1)
  m1, v1, m2, v2 = (torch.zeros_like(p1) for _ in range(4))
  prev = lib.jrg_pipeline(0)
  try:
    for t in (1, 2):
      plan.energy_and_grad(p1[0], p1[1], occ, g1[0], g1[1])
      adam_update(p1, g1, m1, v1, t, 1e-2)
      plan.energy_grad_adam(p2, m2, v2, occ, t, 1e-2)
  finally:
    lib.jrg_pipeline(prev)
  tol = dict(rtol=1e-12, atol=1e-14) if prec == 64 else dict(rtol=2e-5, atol=1e-6)   # as test_gpu_fused_step.py
  for a, b in ((m1, m2), (p1, p2)):
    np.testing.assert_allclose(b.cpu().numpy(), a.cpu().numpy(), **tol)
  plan.close()
