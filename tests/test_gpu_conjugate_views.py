"""Lazily conjugated tensors at the entry points that read raw memory: torch keeps
``x.conj()`` as a flag on the same memory, and the cotangent that reaches a
transform through it has that flag.

References by numpy in FP64; a 3-D transform's relative rounding is below
24 log2(N) eps = 6.4e-14 at 16^3 in the 2-norm, the coefficient map's and the
density's a few times that; 1e-12 is asked."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12
AX = (-3, -2, -1)


def _complex(rng, shape):
  return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _close(a, b):
  return np.linalg.norm(a.resolve_conj().cpu().numpy() - b) <= TOL * np.linalg.norm(b)


def test_wave_grid_cotangent_through_a_conjugate():
  """L = Re sum conj(psi) A: the gradient of L is the adjoint transform of A."""
  import torch
  from jrystal_gb300 import pw
  rng = np.random.default_rng(2)
  z, a = (_complex(rng, (1, 2, 3, 16, 16, 16)) for _ in range(2))
  c = torch.tensor(z, device="cuda", requires_grad=True)
  psi = pw.wave_grid(c, 2.0)
  (psi.conj() * torch.tensor(a, device="cuda")).real.sum().backward()
  assert _close(c.grad, np.fft.fftn(a, axes=AX) / np.sqrt(2.0))


@pytest.mark.parametrize("inverse", [False, True])
def test_transforms_of_a_conjugate(inverse):
  import torch
  from jrystal_gb300 import _ops, pw
  rng = np.random.default_rng(3)
  z = _complex(rng, (2, 16, 12, 10))
  x = torch.tensor(z, device="cuda").conj()
  want = (np.fft.ifftn if inverse else np.fft.fftn)(z.conj(), axes=AX)
  assert _close((_ops.ifftn if inverse else _ops.fftn)(x), want)
  if inverse:
    assert _close(pw.wave_grid(x, 1.0), want * 1920)


def test_plan_entry_points_take_conjugate_views():
  import torch
  from jrystal_gb300.engine import PlaneWavePlan
  from tests.systems import make_system, random_params
  sysm = make_system(kind="si2", grid=(16, 16, 16), kgrid=(2, 1, 1), nb=4, nocc=2)
  plan = PlaneWavePlan(sysm.cell_vectors, sysm.positions, sysm.charges, sysm.grid, sysm.mask,
                       sysm.kpts, 4, 1, 64, sysm.xc)
  w = [torch.tensor(x, device="cuda") for x in random_params(sysm, seed=5)]
  c = plan.coeff(*w)
  view, copy = c.conj(), c.conj().resolve_conj().clone()
  assert view.is_conj() and not copy.is_conj()
  pairs = [(plan.density(x, sysm.occupation),) + tuple(plan.coeff_adjoint(*w, x)) for x in (view, copy)]
  for a, b in zip(*pairs):
    assert _close(a, b.cpu().numpy())
  plan.close()
