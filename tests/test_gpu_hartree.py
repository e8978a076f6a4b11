"""Hartree term of the energy path (x forward, 4 pi/G^2, x inverse in one kernel)
against the density's Hartree energy by numpy, over the register-resident lengths,
odd ones, mixed axes and a grid with more rows than energy slots.

FP64 sums of up to 64^3 terms of one sign: relative rounding below
log2(N) eps ~ 4e-15 of a term plus the transforms' 18 * 8 eps; 1e-12 bounds it.
FP32: the density and its transform carry relative errors of a few 1e-7 that
average out in the sum; 2e-6 as for the other energy terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("grid", [(16, 16, 16), (24, 24, 24), (27, 27, 27), (32, 32, 32), (36, 36, 36), (48, 48, 48),
                                  (64, 64, 64), (45, 45, 45), (9, 10, 12), (20, 30, 25), (8, 280, 6)])
@pytest.mark.parametrize("ns", [1, 2])
def test_hartree_energy(grid, prec, ns):
  import torch
  from jrystal_gb300 import grid as g
  from jrystal_gb300.engine import PlaneWavePlan
  cell = np.diag([0.16 * v for v in grid])
  rmax = np.pi / 0.16
  mask = g.spherical_mask(cell, grid, 0.5 * (0.5 * rmax) ** 2 * (1 - 1e-9))
  kpts = g.k_vectors(cell, (2, 1, 1))
  plan = PlaneWavePlan(cell, np.zeros((1, 3)), np.ones(1), grid, mask, kpts, 3, ns, prec)
  rng = np.random.default_rng(2)
  w = torch.tensor(rng.standard_normal((2,) + plan.param_shape), dtype=plan.rdtype, device="cuda")
  occ = rng.uniform(0.2, 0.6, (ns, 2, 3))
  e = plan.energy_and_grad(w[0], w[1], occ)[0].cpu().numpy()
  rho = plan.density(plan.coeff(w[0], w[1]), occ).double().cpu().numpy().sum(0)
  gv = g.g_vectors(cell, grid)
  g2 = np.sum(gv * gv, -1)
  rg = np.fft.fftn(rho)
  rg[0, 0, 0] = 0.0
  g2[0, 0, 0] = 1.0
  want = 0.5 * np.sum(4 * np.pi / g2 * np.abs(rg) ** 2) * plan.vol / rho.size ** 2
  assert abs(e[2] - want) <= (1e-12 if prec == 64 else 2e-6) * abs(want)
