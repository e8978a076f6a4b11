"""Integral of the FP32 density against Parseval's sum: vol/N sum rho = sum w |c|^2.

Roundings of the arithmetic average out over the 4096 or more points (below 2e-9);
what is left is the norm of the transforms' FP32 constants along the three axes, a
fixed factor for each length.  From the tables it is at most 6.0e-8 (60^3); 7e-8, a
little more than one rounding of a float, is allowed.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 18, 20, 21, 24, 25, 27, 28, 30, 32, 35, 36, 40, 42, 45, 48, 49, 50, 54,
                               56, 60, 63, 64, 70, 72, 80, 84, 90, 96])
def test_density_norm(n):
  import torch
  from jrystal_gb300 import grid as g
  from jrystal_gb300.engine import PlaneWavePlan
  spacing, nb = 10.26 / 64, 6
  cell = np.eye(3) * spacing * n
  mask = g.spherical_mask(cell, (n, n, n), 0.5 * (0.5 * np.pi / spacing) ** 2 * (1 - 1e-9))
  kpts = g.k_vectors(cell, (2, 1, 1))
  plan = PlaneWavePlan(cell, np.zeros((1, 3)), np.ones(1), (n, n, n), mask, kpts, nb, 1, 32)
  gk = torch.as_tensor(g.g_vectors(cell, (n, n, n))[mask][None] + kpts[:, None], device="cuda")
  damp = 1.0 / (1.0 + 0.25 * (gk * gk).sum(-1)) + 0.02
  gen = torch.Generator(device="cuda")
  gen.manual_seed(n)
  c = torch.randn(plan.param_shape, generator=gen, device="cuda", dtype=torch.complex128) * damp[None, :, :, None]
  c = (c / torch.linalg.vector_norm(c, dim=2, keepdim=True)).to(torch.complex64)
  w = np.random.default_rng(n).uniform(0.3, 1.0, (1, 2, nb))
  rho = plan.density(c, w)
  got = rho.double().sum().item() * plan.vol / n ** 3
  want = (c.to(torch.complex128).abs() ** 2 * torch.as_tensor(w, device="cuda")[:, :, None]).sum().item()
  assert abs(got / want - 1.0) <= 7e-8
  plan.close()
