"""Column-first transforms (every axis length, mixed axes, empty bands) against the
generic shared-memory kernels of the same plan, through the C ABI.

Both routes compute the same sums in the same precision.  Four transforms of
three axes in a row have a relative rounding error below 4 * 8 log2(96^3) eps,
1.4e-13 in FP64 and 7.6e-5 in FP32; independent roundings add in quadrature, so
a tenth of that is asked of the 2-norms.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPACING = 10.26 / 64
LENGTHS = [16, 18, 20, 21, 24, 25, 27, 28, 30, 32, 35, 36, 40, 42, 45, 48, 49, 50, 54, 56, 60, 63,
           64, 70, 72, 80, 84, 90, 96]
# every length on every axis once, paired with a short and a middle one
GRIDS = [(n, LENGTHS[(7 * i + 3) % 12], LENGTHS[(5 * i + 1) % 14]) for i, n in enumerate(LENGTHS)]
GRIDS += [(LENGTHS[(5 * i + 2) % 14], n, LENGTHS[(7 * i + 5) % 12]) for i, n in enumerate(LENGTHS)]
GRIDS += [(LENGTHS[(7 * i + 1) % 12], LENGTHS[(5 * i + 4) % 14], n) for i, n in enumerate(LENGTHS)]
CUBES = [(n, n, n) for n in (16, 24, 27, 32, 36, 40, 45, 48, 54, 60, 64)]


def _plan(grid, nb, prec, radius=1.0, nk=2, ns=1):
  from jrystal_gb300 import grid as g
  from jrystal_gb300.engine import PlaneWavePlan
  cell = np.diag([SPACING * v for v in grid])
  pos = np.array([[0.1, 0.2, 0.3], [0.6, 0.55, 0.7]]) @ cell
  rmax = np.pi / SPACING
  mask = g.spherical_mask(cell, grid, 0.5 * (0.5 * radius * rmax) ** 2 * (1 - 1e-9))
  kpts = g.k_vectors(cell, (nk, 1, 1))
  return PlaneWavePlan(cell, pos, np.full(2, 6.0), grid, mask, kpts, nb, ns, prec)


def _both(plan, occ, seed):
  """(energies, gradient, density) by the default and by the generic kernels."""
  import torch
  rng = np.random.default_rng(seed)
  shape = plan.param_shape
  w = torch.tensor(rng.standard_normal((2,) + shape), dtype=plan.rdtype, device="cuda")
  out = []
  for fast in (1, 0):
    prev = plan.lib.jrg_fast_paths(fast)
    try:
      e, gr, gi = plan.energy_and_grad(w[0], w[1], occ)
      c = plan.coeff(w[0], w[1])
      rho = plan.density(c, occ)
      out.append([x.double().cpu().numpy() for x in (e, torch.stack([gr, gi]), rho)])
    finally:
      plan.lib.jrg_fast_paths(prev)
  return out


def _check(plan, occ, seed):
  tol = 1.4e-14 if plan.precision == 64 else 7.6e-6
  a, b = _both(plan, occ, seed)
  for x, y in zip(a, b):
    assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y), np.linalg.norm(x - y) / np.linalg.norm(y)


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("grid", GRIDS[::2] + CUBES, ids=lambda g: "x".join(map(str, g)))
def test_lengths(grid, prec):
  if prec == 64 and max(grid[1] * grid[2], grid[0] * grid[2]) > 5600:
    pytest.skip("the generic FP64 kernels do not hold this plane")
  nb = 5
  plan = _plan(grid, nb, prec)
  occ = np.zeros((1, 2, nb))
  occ[:, 0, :3] = 1.0
  occ[:, 1, [0, 2, 4]] = 0.7       # empty bands in between
  _check(plan, occ, 3)


@pytest.mark.parametrize("grid", GRIDS[1::2], ids=lambda g: "x".join(map(str, g)))
def test_lengths_fp32_rest(grid):
  plan = _plan(grid, 4, 32, radius=0.8)
  occ = np.full((1, 2, 4), 0.5)
  _check(plan, occ, 4)


@pytest.mark.parametrize("nb", [1, 2, 33, 70])
@pytest.mark.parametrize("grid", [(24, 24, 24), (20, 18, 30)])
def test_band_counts_spin_and_empty_blocks(grid, nb):
  plan = _plan(grid, nb, 32, nk=3, ns=2)
  rng = np.random.default_rng(nb)
  occ = rng.uniform(0.1, 1.0, (2, 3, nb))
  occ[1, 1] = 0.0                  # a (spin, k) block without an occupied band
  occ[0, 2, nb // 2:] = 0.0
  _check(plan, occ, 5)


def test_band_trace_with_zero_weights():
  import torch
  plan = _plan((32, 27, 40), 6, 64)
  rng = np.random.default_rng(8)
  w = torch.tensor(rng.standard_normal((2,) + plan.param_shape), device="cuda")
  v = torch.tensor(rng.standard_normal(plan.grid), device="cuda")
  wts = np.ones((1, 2, 6))
  wts[0, 1, ::2] = 0.0
  out = []
  for fast in (1, 0):
    prev = plan.lib.jrg_fast_paths(fast)
    try:
      t, gr, gi, h = plan.band_trace_grad(w[0], w[1], v, wts, hmat=True)
      out.append([x.cpu().numpy() for x in (t, gr, gi, h)])
    finally:
      plan.lib.jrg_fast_paths(prev)
  for x, y in zip(*out):
    assert np.linalg.norm(x - y) <= 1.4e-14 * np.linalg.norm(y)


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("shape", [(1, 2, 3, 24, 24, 24), (5, 20, 27, 16), (16, 16, 16)])
def test_wave_grid_and_its_adjoint(shape, prec):
  """Factor applied inside the transform, value and vector-Jacobian product against
  numpy (a transform's rounding, 24 log2(N) eps at most)."""
  import torch
  from jrystal_gb300 import pw
  rng = np.random.default_rng(4)
  z = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
  g = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
  dt = torch.complex64 if prec == 32 else torch.complex128
  c = torch.tensor(z, dtype=dt, device="cuda", requires_grad=True)
  w = pw.wave_grid(c, 37.5)
  w.backward(torch.tensor(g, dtype=dt, device="cuda"))
  ax = (-3, -2, -1)
  n = np.prod(shape[-3:])
  tol = 24 * np.log2(n) * (1.2e-7 if prec == 32 else 2.2e-16)
  want = np.fft.ifftn(z, axes=ax) * n / np.sqrt(37.5)
  adj = np.fft.fftn(g, axes=ax) / np.sqrt(37.5)
  for a, b in ((w.detach(), want), (c.grad, adj)):
    assert np.linalg.norm(a.cpu().numpy() - b) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("nb", [1, 7, 8, 9, 16, 17, 24, 32])
@pytest.mark.parametrize("grid,nk", [((16, 16, 16), 2), ((30, 24, 32), 3), ((40, 40, 40), 5)])
def test_gram_splits_summed_by_their_consumers(grid, nk, nb):
  """One to many G splits of the Gram products (summed in the Cholesky and adjoint
  kernels while few): FP32 against the FP64 plan, at the FP32 path's tolerances."""
  import torch
  rng = np.random.default_rng(nb)
  out = []
  w = None
  for prec in (64, 32):
    plan = _plan(grid, nb, prec, nk=nk)
    if w is None:
      w = rng.standard_normal((2,) + plan.param_shape)
    occ = np.full((1, nk, nb), 1.3 / nk)
    x = torch.tensor(w, dtype=plan.rdtype, device="cuda")
    e, gr, gi = plan.energy_and_grad(x[0], x[1], occ)
    out.append((e[:5].cpu().numpy(), torch.stack([gr, gi]).double().cpu().numpy()))
  (e64, g64), (e32, g32) = out
  assert np.all(np.abs(e32 - e64) <= 2e-6 * np.maximum(np.abs(e64), 1.0))
  assert np.abs(g32 - g64).max() <= 1e-4 * np.abs(g64).max()
