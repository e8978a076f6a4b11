"""Plans of different band counts on the same grid, one host thread and one stream
each, at the same time: no call is refused and every result is bit for bit that of
the plan on its own (the kernels, and their shared-memory limits, are common to all)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plans", [
  [((24, 24, 24), 4, 64), ((24, 24, 24), 28, 64), ((24, 24, 24), 9, 32), ((24, 24, 24), 40, 32)],
  [((48, 48, 48), 4, 32), ((48, 48, 48), 40, 32)],
  [((20, 27, 24), 3, 32), ((20, 27, 24), 28, 32), ((20, 27, 24), 12, 64)],
])
def test_energies_from_several_threads(plans):
  import torch
  from tests.test_gpu_columns import _plan
  work, errors, results = [], [], []
  for i, (grid, nb, prec) in enumerate(plans):
    plan = _plan(grid, nb, prec)
    w = torch.tensor(np.random.default_rng(i).standard_normal((2,) + plan.param_shape), dtype=plan.rdtype,
                     device="cuda")
    occ = torch.full((1, 2, nb), 0.5, dtype=torch.float64, device="cuda")
    e, gr, gi = plan.energy_and_grad(w[0], w[1], occ)
    work.append((plan, w, occ, e.clone(), torch.stack([gr, gi])))
    results.append([])
  torch.cuda.synchronize()

  def run(i):
    plan, w, occ, _, _ = work[i]
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
      for _ in range(300):
        try:
          e, gr, gi = plan.energy_and_grad(w[0], w[1], occ)
          results[i].append(e.clone())
        except Exception as ex:
          errors.append(f"{plans[i]}: {ex}")
      results[i].append(torch.stack([gr, gi]))
    stream.synchronize()

  threads = [threading.Thread(target=run, args=(i,)) for i in range(len(plans))]
  for t in threads:
    t.start()
  for t in threads:
    t.join()
  assert not errors, (len(errors), errors[0])
  for (plan, _, _, e, g), got in zip(work, results):
    assert all(torch.equal(e, x) for x in got[:-1]) and torch.equal(g, got[-1])
    plan.close()
