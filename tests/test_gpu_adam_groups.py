"""The optimiser step with one and with two 16-byte groups per thread, around
the size where the second begins, aligned and not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGE = 152 * 8 * 256 * 4      # elements of the last launch with one group per thread


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("n", [1, 1023, EDGE, EDGE + 1, EDGE + 4, EDGE + 2051])
def test_adam_update_sizes(n, off):
  import torch
  from jrystal_gb300.engine import adam_update
  rng = np.random.default_rng(n + off)
  f = lambda a: a.astype(np.float32)
  p, g = f(rng.normal(size=n)), f(rng.normal(size=n))
  # moments of the gradient's sign: no cancellation, so that every factor of
  # the increment is good to a few roundings
  m, v = f(np.abs(rng.normal(size=n))) * np.sign(g), f(rng.normal(size=n) ** 2)
  s = f(rng.uniform(0.5, 1.5, size=n))

  def dev(a):
    b = torch.empty(n + 8, device="cuda", dtype=torch.float32)[off:off + n]
    b.copy_(torch.tensor(a))
    return b
  dp, dg, dm, dv, ds = (dev(a) for a in (p, g, m, v, s))
  b1, b2, lr, step = 0.875, 0.9375, 0.0078125, 3     # exact in FP32, and so are 1 - b1 and 1 - b2
  adam_update(dp, dg, dm, dv, step, lr, b1, b2, 1e-8, scale=ds)
  p, g, m, v, s = (a.astype(np.float64) for a in (p, g, m, v, s))
  m = b1 * m + (1 - b1) * g
  v = b2 * v + (1 - b2) * g * g
  inc = -s * lr * (m / (1 - b1**step)) / (np.sqrt(v / (1 - b2**step)) + 1e-8)
  eps = 2.0**-24
  # two products and a sum for each moment; the increment: both moments, two
  # rounded factors, two products, root, sum, division, scale; then the last sum
  assert (np.abs(dm.cpu().numpy() - m) <= 4 * eps * np.abs(m) + 1e-38).all()
  assert (np.abs(dv.cpu().numpy() - v) <= 5 * eps * v + 1e-38).all()
  assert (np.abs(dp.cpu().numpy() - (p + inc)) <= 16 * eps * np.abs(inc) + 2 * eps * np.abs(p + inc) + 1e-38).all()


def test_pipelined_halves_with_two_groups():
  import torch
  from jrystal_gb300.engine import PlaneWavePlan, adam_update
  from tests.systems import make_system, random_params
  sysm = make_system(kind="si2", grid=(48, 48, 48), kgrid=(4, 4, 2), nb=8, nocc=4)
  plan = PlaneWavePlan(sysm.cell_vectors, sysm.positions, sysm.charges, sysm.grid, sysm.mask,
                       sysm.kpts, 8, 1, 32, sysm.xc)
  wr, wi = random_params(sysm, seed=3, dtype=np.float32)
  p1 = torch.tensor(np.stack([wr, wi]), device="cuda").contiguous()
  assert p1[0].numel() // 2 > EDGE // 2        # each half launches both parts
  occ = torch.tensor(sysm.occupation, device="cuda")
  p2, g1 = p1.clone(), torch.empty_like(p1)
  m1, v1, m2, v2 = (torch.zeros_like(p1) for _ in range(4))
  for t in (1, 2):
    plan.energy_and_grad(p1[0], p1[1], occ, g1[0], g1[1])
    adam_update(p1, g1, m1, v1, t, 1e-2)
    plan.energy_grad_adam(p2, m2, v2, occ, t, 1e-2)
    for a, b in ((m1, m2), (p1, p2)):
      np.testing.assert_allclose(b.cpu().numpy(), a.cpu().numpy(), rtol=2e-5, atol=1e-6)
  plan.close()
