"""Spheres and masks that reach past the window |i| < N/4 keep the plane-first kernels.
The largest alias-free sphere, which the other full-size cases use, takes the
column-first ones, so that the passes with several bands per CTA are reached here:
enough (k, band) planes for them in each half of the two-way pipeline, with the known
zeros of 32^3 and 64^3 left out (cubic mask) and not (48^3, a larger sphere).

Against the generic kernels at the tolerances of test_gpu_columns.py."""
import numpy as np
import pytest

from tests.test_gpu_columns import SPACING, _check, _plan

pytestmark = pytest.mark.gpu


def _masked(n, mask, nb, prec, nk):
  from jrystal_gb300 import grid as g
  from jrystal_gb300.engine import PlaneWavePlan
  cell = np.eye(3) * SPACING * n
  pos = np.array([[.1, .2, .3], [.6, .55, .7]]) @ cell
  return PlaneWavePlan(cell, pos, np.full(2, 6.0), (n, n, n), mask, g.k_vectors(cell, (nk, 1, 1)), nb, 1, prec)


def _occ(nk, nb):
  occ = np.random.default_rng(nk).uniform(0.2, 1.0, (1, nk, nb)) / nk
  occ[0, 1, 2:] = 0.0
  return occ


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("n,nk,kind", [(32, 40, "cubic"), (48, 30, "cubic"), (64, 24, "cubic"), (64, 24, "sphere"),
                                       (24, 3, "cubic"), (40, 3, "cubic")])
def test_masks_past_the_window(n, nk, kind, prec):
  from jrystal_gb300 import grid as g
  mask = g.cubic_mask((n, n, n)) if kind == "cubic" else \
    g.spherical_mask(np.eye(3) * SPACING * n, (n, n, n), 0.5 * (0.65 * np.pi / SPACING) ** 2)
  plan = _masked(n, mask, 8, prec, nk)
  _check(plan, _occ(nk, 8), n)
  plan.close()


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [24, 27, 30])
def test_edge_of_the_window(n, axis, prec):
  """One G vector at the last index of the window, and at the one after it, on either side."""
  from jrystal_gb300 import grid as g
  h = (n - 1) // 4
  for i in (h, -h, h + 1, -h - 1):
    mask = g.spherical_mask(np.eye(3) * SPACING * n, (n, n, n), 0.5 * (0.35 * np.pi / SPACING) ** 2)
    mask[tuple(i if a == axis else 0 for a in range(3))] = True
    plan = _masked(n, mask, 4, prec, 2)
    _check(plan, _occ(2, 4), n + i)
    plan.close()


@pytest.mark.parametrize("prec", [32, 64])
def test_bounded_workspace_with_empty_bands(prec):
  """Columns recomputed block by block: empty bands, and blocks without an occupied one."""
  plan = _plan((20, 27, 24), 6, prec, nk=5)
  occ = _occ(5, 6)
  occ[0, 3] = 0.0
  for limit in (plan.workspace_bytes // 2, 1):
    assert plan.set_memory_limit(limit) < 5
    _check(plan, occ, 6)
  plan.close()
