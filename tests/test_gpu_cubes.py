"""Slab kernels of cubic grids (every length of the column-first transforms, z lines
by pairs of threads above 64 points) against the generic shared-memory kernels of
the same plan, at the tolerances of test_gpu_columns.py: a band alone, a tile that
is not full, several tiles with empty bands in between.  And the Hartree term of a
96^3 density, whose line kernel no smaller grid uses."""
import numpy as np
import pytest

from tests.test_gpu_columns import LENGTHS, _check, _plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,prec", [(n, 32) for n in LENGTHS] + [(n, 64) for n in LENGTHS if n <= 72])
def test_cube(n, prec):
  for nb, empty in ((1, []), (7, [2]), (23, [0, 5, 6, 21])):
    if nb == 23 and prec == 64 and n > 56:
      continue                      # minutes of FP64 for what 7 bands show
    plan = _plan((n, n, n), nb, prec)
    rng = np.random.default_rng(n + nb)
    occ = rng.uniform(0.2, 1.0, (1, 2, nb))
    occ[0, 1, empty] = 0.0
    _check(plan, occ, n)
    plan.close()


def test_hartree_energy_96():
  import torch
  from jrystal_gb300 import grid as g
  n = 96
  plan = _plan((n, n, n), 3, 32)
  w = torch.randn((2,) + plan.param_shape, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda")
  occ = np.full((1, 2, 3), 0.4)
  e = plan.energy_and_grad(w[0], w[1], occ)[0].cpu().numpy()
  rho = plan.density(plan.coeff(w[0], w[1]), occ)[0].double()
  cell = np.eye(3) * 10.26 / 64 * n
  g2 = torch.as_tensor(np.sum(g.g_vectors(cell, (n, n, n)) ** 2, -1), device="cuda")
  g2[0, 0, 0] = float("inf")
  want = 0.5 * (4 * np.pi / g2 * torch.fft.fftn(rho).abs() ** 2).sum().item() * plan.vol / n ** 6
  assert abs(e[2] - want) <= 2e-6 * abs(want)      # as the other lengths in test_gpu_hartree.py
  plan.close()
