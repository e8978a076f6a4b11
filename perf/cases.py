"""Performance cases: what programs built on this package have the GPU do.

Kinds (``case["kind"]``), each a call a program makes over and over:

  step       one optimiser step (energy, gradient, Adam) through
             ``calc.Minimizer.step``, the ground-state loop's iteration;
  grad       energy and gradient without the update (an outer optimiser);
  bands      energy, gradient and band energies (learnable occupations);
  trace      band trace, its gradient and the band Hamiltonian in a fixed
             potential (the band-structure loop's iteration);
  field      coefficients -> density -> effective potential (what follows a
             ground state: post-processing, start of a band structure);
  wave       wave functions on the dense grid through ``pw.wave_grid``.

Grids, cells, k-point sets, band counts and precisions are those of the named
workloads, the strained training cells and the tests, and generic orthorhombic
boxes for grids with different axes.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import jrystal_gb300.grid as grid
from jrystal_gb300 import calc, cells, pw, workloads
from jrystal_gb300.engine import PlaneWavePlan

LDA = "lda_x+lda_c_vwn"
PBE = "gga_x_pbe+gga_c_pbe"
SPACING = 10.26 / 64   # bohr per grid point of the generic boxes (the Si8 64^3 density)


def _case(name, kind, cell, n, k, nb, nocc, prec, spin=1, xc=LDA, proj=0, radius=1.0):
  return dict(name=name, kind=kind, cell=cell, nx=n[0], ny=n[1], nz=n[2], k1=k[0], k2=k[1],
              k3=k[2], nb=nb, nocc=nocc, prec=prec, spin=spin, xc=xc, proj=proj, radius=radius)


def listed():
  cube = lambda n: (n, n, n)
  return [
    # the headline workload: all-electron Si8, 27 k-points, 24 bands, FP32 Adam step
    _case("si8_step", "step", "si8", cube(64), (3, 3, 3), 24, 16, 32),
    # the scale workload: Si64 supercell, Gamma + 2x2x2, 160 bands
    _case("si64_step", "step", "si64", cube(96), (2, 2, 2), 160, 128, 32),
    # smallest training cell: one Al atom, latency of a whole step
    _case("al_step_small", "step", "al", cube(24), (2, 2, 2), 8, 4, 32),
    # middle training cell with an odd band count
    _case("c2_step_odd", "step", "c", cube(36), (2, 2, 2), 13, 6, 32),
    # a box whose axes differ (slab, wire, low-symmetry cell), odd and 5-smooth sizes
    _case("box_step_ragged", "step", "box", (30, 45, 64), (2, 2, 1), 21, 14, 32),
    # the reference's default precision: Si2 primitive cell, FP64
    _case("si2_grad_fp64", "grad", "si2", cube(48), (2, 2, 2), 8, 4, 64),
    # open-shell run: two spin channels
    _case("si2_grad_spin", "grad", "si2", cube(32), (2, 2, 2), 10, 4, 32, spin=2),
    # metal with fractional occupations, PBE, FP64
    _case("al_bands_pbe_fp64", "bands", "al", cube(32), (3, 3, 3), 9, 7, 64, xc=PBE),
    # norm-conserving pseudopotential: 4 projector rows per atom
    _case("si8_step_nc", "step", "si8", cube(48), (2, 2, 2), 20, 16, 32, proj=4),
    # band structure: 30 points of a k path in one call
    _case("si2_trace_path", "trace", "si2", cube(48), (30, 1, 1), 8, 8, 32),
    # density and potentials of a converged state, FP64
    _case("si2_field_fp64", "field", "si2", cube(48), (2, 2, 2), 8, 4, 64),
    # wave functions on the grid for plotting and analysis
    _case("si8_wave", "wave", "si8", cube(48), (2, 2, 2), 16, 16, 32),
  ]


SMOOTH = [n for n in range(16, 97)
          if all(n % p or p in (2, 3, 5, 7) for p in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37,
                                                      41, 43, 47, 53, 59, 61, 67, 71, 73, 79, 83, 89))]


def _log_int(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
  """A grid size of the reference's table (7-smooth) in [lo, hi], spread over the logarithm."""
  v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
  return min((n for n in SMOOTH if lo <= n <= hi), key=lambda n: abs(n - v))


def draw(rng):
  kind = rng.choice(["step", "step", "step", "step", "grad", "grad", "bands", "trace", "field", "wave"])
  prec = 32 if kind in ("step", "trace", "wave") else rng.choice([32, 64])
  radius = rng.choice([1.0, 1.0, rng.uniform(0.7, 1.0)])
  spin, xc, proj = 1, LDA, 0
  while True:
    cell = rng.choice(["si2", "c", "al", "si8", "box"])
    if cell == "box":
      n = tuple(_size(rng, 18, 80 if prec == 32 else 60) for _ in range(3))
      k = rng.choice([(1, 1, 1), (2, 2, 1), (2, 2, 2), (3, 2, 1)])
    else:
      # cubic grids as the package's cells use them, up to 64^3 (FP64) and 96^3 (FP32)
      sizes = [24, 27, 32, 36, 40, 45, 48, 54, 60, 64] + ([72, 80, 96] if prec == 32 else [])
      n = (rng.choice(sizes),) * 3
      k = rng.choice([(1, 1, 1), (2, 2, 1), (2, 2, 2), (3, 3, 3)])
    if kind == "trace":
      k = (rng.choice([8, 20, 30, 40]), 1, 1)
    nb = _log_int(rng, 4, 96 if cell in ("si8", "box") else 16)
    if kind in ("grad", "field") and cell != "box":
      spin = rng.choice([1, 1, 2])
    if kind in ("step", "bands") and nb <= 32 and rng.random() < 0.3:
      xc = PBE
    if kind in ("step", "grad") and xc == LDA and rng.random() < 0.25:
      proj = 4
    case = _case(None, kind, cell, n, k, nb, max(1, (2 * nb) // 3), prec, spin, xc, proj, radius)
    del case["name"]
    w = work(case)
    # no more than the Si64 step in work; FP64 transforms, dense wave grids and
    # projector tables (atoms x k-points on the host) bounded to ordinary sizes
    points = spin * k[0] * k[1] * k[2] * nb * n[0] * n[1] * n[2]
    top = 2.5e8 if kind == "wave" or prec == 64 else 4e8 if kind != "step" else 1.2e9
    if points <= top and w["flops"] < 3e11 and proj * k[0] * k[1] * k[2] * n[0] * n[1] * n[2] < 4e7:
      return case


# ---- what the program has in hand -------------------------------------------

_GEOMETRY = ("kind", "cell", "nx", "ny", "nz", "k1", "k2", "k3", "proj", "radius")


def _geometry(case):
  return _geometry_of(*(case[k] for k in _GEOMETRY))


@functools.lru_cache(maxsize=4)
def _geometry_of(kind, cell_name, nx, ny, nz, k1, k2, k3, proj, radius):
  """(cell, positions, charges, mask, kpts, G vectors, projector tables)."""
  n = (nx, ny, nz)
  if cell_name == "si2":
    base = workloads.si2_fcc()
    cell, pos, chg = base.cell, base.positions, base.charges
  elif cell_name == "si8":
    base = workloads.si8_cubic()
    cell, pos, chg = base.cell, base.positions, base.charges
  elif cell_name == "si64":
    base = workloads.si64_supercell()
    cell, pos, chg = base.cell, base.positions, base.charges
  elif cell_name in ("al", "c"):
    base = cells.strained_cell(np.random.default_rng(7), kind=cell_name, grids=(n[0],))
    cell, pos, chg = base.cell, base.positions, base.charges
  else:
    cell = np.diag([SPACING * v for v in n])
    pos = workloads._diamond_basis() @ cell
    chg = np.full(8, 14.0)
  # largest alias-free sphere (times radius): half the inscribed frequency ball
  rmax = min(n[i] * math.pi / np.linalg.norm(cell[i]) for i in range(3))
  mask = grid.spherical_mask(cell, n, 0.5 * (0.5 * radius * rmax) ** 2 * (1 - 1e-9))
  if kind == "trace":   # a straight path Gamma - X - L like the band driver's
    b = grid.reciprocal_vectors(cell)
    t = np.linspace(0.0, 1.0, k1)[:, None]
    kpts = (t * np.array([[0.5, 0.0, 0.5]]) + t * t * np.array([[0.0, 0.4, 0.0]])) @ b
  else:
    kpts = grid.k_vectors(cell, (k1, k2, k3))
    if cell_name == "si64":
      kpts = np.concatenate([np.zeros((1, 3)), kpts])
  g = grid.g_vectors(cell, n)
  tables = _projectors(cell, pos, mask, kpts, g) if proj else None
  return cell, pos, chg, mask, kpts, g, tables


def _projectors(cell, pos, mask, kpts, g, z_val=4.0):
  """Analytic norm-conserving tables: local -z erf(r/rc)/r (closed form in G)
  and Gaussian s and p projectors on every atom, (V_loc(G) grid, rows [K, 4A, G])."""
  vol = abs(np.linalg.det(cell))
  num = float(np.prod(mask.shape))
  g2 = np.sum(g * g, axis=-1)
  shape = np.exp(-g2 * 0.8 ** 2 / 4) * 4 * np.pi * z_val / np.where(g2 > 0, g2, 1.0)
  shape[0, 0, 0] = 0.0
  phase = sum(np.exp(-1j * (g @ p)) for p in pos)
  v_local = -num / vol * shape * phase
  q = g[mask][None] + kpts[:, None]                       # (K, G, 3)
  q2 = np.sum(q * q, axis=-1)
  radial = np.exp(-q2 * 0.9 ** 2 / 4)
  rows = []
  for p in pos:
    e = np.exp(-1j * (q @ p)) * radial
    rows.append(2.2 * e)
    rows += [1.1j * q[..., a] * e for a in range(3)]
  return v_local, np.ascontiguousarray(np.stack(rows, axis=1))


def _occupation(case, nk):
  """2/K per doubly occupied band; per channel 1/K with two spins (the channels
  differ by two electrons); fractional around the last bands for a metal."""
  nb, nocc = case["nb"], case["nocc"]
  occ = np.zeros((case["spin"], nk, nb))
  if case["kind"] == "bands":
    x = (np.arange(nb) - nocc + 0.5) / 1.5
    occ[:] = 2.0 / nk / (1.0 + np.exp(x))[None, None]
  elif case["spin"] == 2:
    occ[0, :, :min(nb, nocc + 1)] = 1.0 / nk
    occ[1, :, :max(1, nocc - 1)] = 1.0 / nk
  else:
    occ[:, :, :nocc] = 2.0 / nk
  return occ


def _inputs(case, seed):
  """Device inputs from the seed: parameters of smooth orbitals (N(0,1) damped
  at large |G+k| as a few steps of minimisation leave them), Adam moments,
  a potential of screened atomic wells."""
  cell, pos, chg, mask, kpts, g, _ = _geometry(case)
  dev = torch.device("cuda")
  dt = torch.float64 if case["prec"] == 64 else torch.float32
  gen = torch.Generator(device=dev)
  gen.manual_seed(1_000_003 * (seed % 2_000_000_011) + 17)
  ng = int(mask.sum())
  shape = (2, case["spin"], len(kpts), ng, case["nb"])
  gk = torch.as_tensor(g[mask][None] + kpts[:, None], device=dev)
  damp = (1.0 / (1.0 + 0.25 * (gk * gk).sum(-1))).to(dt)[None, None, :, :, None]
  out = {"params": torch.randn(shape, generator=gen, device=dev, dtype=dt) * damp + 0.02 *
                   torch.randn(shape, generator=gen, device=dev, dtype=dt)}
  if case["kind"] == "step":
    out["m"] = 1e-4 * torch.randn(shape, generator=gen, device=dev, dtype=dt)
    out["v"] = 1e-8 * (0.2 + torch.rand(shape, generator=gen, device=dev, dtype=dt))
  if case["kind"] == "trace":
    gg = torch.as_tensor(g, device=dev)
    g2 = (gg * gg).sum(-1)
    shift = 0.02 * torch.randn(pos.shape, generator=gen, device=dev, dtype=torch.float64)
    p = torch.as_tensor(pos, device=dev) + shift
    s = sum(torch.exp(-1j * (gg @ p[i])) for i in range(len(pos)))
    w = torch.exp(-0.3 * g2) / torch.where(g2 > 0, g2, torch.ones_like(g2)) * (g2 > 0)
    vol = abs(np.linalg.det(cell))
    out["v_eff"] = torch.fft.ifftn(-4 * math.pi * 4.0 / vol * w * s).real.mul(g2.numel()).to(dt)
  return out


def prepare(case, seed):
  cell, pos, chg, mask, kpts, g, tables = _geometry(case)
  n = (case["nx"], case["ny"], case["nz"])
  s = {"case": case, **_inputs(case, seed)}
  if case["kind"] == "wave":   # dense coefficients, as pw.coeff gives them
    c = torch.complex(s["params"][0], s["params"][1]).transpose(-1, -2)
    c = c / torch.linalg.vector_norm(c, dim=-1, keepdim=True)
    full = torch.zeros(c.shape[:3] + (int(np.prod(n)),), dtype=c.dtype, device=c.device)
    full[..., torch.as_tensor(np.flatnonzero(mask.reshape(-1)), device=c.device)] = c
    del s["params"]
    s["coeff"] = full.reshape(c.shape[:3] + n)
    s["vol"] = float(abs(np.linalg.det(cell)))
    return s
  plan = PlaneWavePlan(cell, pos, chg, n, mask, kpts, case["nb"], case["spin"], case["prec"],
                       case["xc"])
  if tables is not None:
    plan.set_pseudopotential(*tables)
  s["plan"] = plan
  s["occ"] = torch.as_tensor(_occupation(case, len(kpts)), device=plan.device)
  if case["kind"] == "step":
    opt = calc.Minimizer(plan, s["occ"].cpu(), s.pop("params"))
    opt.m.copy_(s.pop("m"))
    opt.v.copy_(s.pop("v"))
    opt.t = 50
    s["opt"] = opt
  else:
    s["grads"] = torch.empty_like(s["params"])
  return s


# ---- one pass ---------------------------------------------------------------
# Energies and band quantities are kept in the plan's real type, the type the
# path computes them in.

def run(s):
  kind = s["case"]["kind"]
  if kind == "wave":
    return pw.wave_grid(s["coeff"], s["vol"])
  plan = s["plan"]
  if kind == "step":
    opt = s["opt"]
    return {"energies": opt.step().to(plan.rdtype), "params": opt.params, "m": opt.m, "v": opt.v}
  p, gr = s["params"], s["grads"]
  if kind == "grad":
    e, _, _ = plan.energy_and_grad(p[0], p[1], s["occ"], gr[0], gr[1])
    return {"energies": e.to(plan.rdtype), "grad": gr}
  if kind == "bands":
    e, _, _, eps = plan.energy_grad_bands(p[0], p[1], s["occ"], gr[0], gr[1])
    return {"energies": e.to(plan.rdtype), "grad": gr, "eps": eps.to(plan.rdtype)}
  if kind == "trace":
    out, _, _, h = plan.band_trace_grad(p[0], p[1], s["v_eff"], None, gr[0], gr[1], hmat=True)
    return {"trace": out.to(plan.rdtype), "grad": gr, "hmat": h.to(plan.cdtype)}
  c = plan.coeff(p[0], p[1])
  rho = plan.density(c, s["occ"])
  return {"coeff": c, "density": rho, "potential": plan.potential(rho, kohn_sham=True)}


def work(case):
  """Compulsory bytes (inputs read once, outputs written once) and operations
  of one pass: sphere-pruned transforms (z on the rows the sphere touches, y on
  its planes, x on all), one inverse and, with a gradient, one forward;
  Hermitian halves of the Gram products, triangular rotations."""
  n = (case["nx"], case["ny"], case["nz"])
  r = case["prec"] // 8
  nk = case["k1"] * case["k2"] * case["k3"] + (case["cell"] == "si64")
  nsk, nb = case["spin"] * nk, case["nb"]
  num = float(n[0] * n[1] * n[2])
  bands = nsk * nb
  log = [math.log2(v) for v in n]
  if case["kind"] == "wave":
    return {"bytes": 2 * bands * num * 2 * r, "flops": bands * num * (5 * sum(log) + 2)}
  rad = case["radius"]
  fcc = 0.707 if case["cell"] in ("si2", "c", "al") else 1.0   # skewed cells: smaller ball
  ng = num * math.pi / 48 * rad ** 3 * fcc
  fft = 5 * num * (math.pi / 16 * rad ** 2 * log[2] + 0.5 * rad * log[1] + log[0])
  params = 2 * nsk * ng * nb * r
  gram = 4 * ng * nb * nb * nsk
  proj = 8.0 * case["proj"] * (8 if case["cell"] in ("si8", "box") else 2) * ng * bands
  if case["kind"] == "field":
    return {"bytes": 2 * params + 8 * num * r, "flops": 2 * gram + bands * (fft + 4 * num)}
  flops = 6 * gram + bands * (2 * fft + 12 * num) + 2 * proj
  return {"bytes": (6 if case["kind"] == "step" else 2) * params + 3 * num * r, "flops": flops}


# ---- the same in 64 bits ----------------------------------------------------

def _vwn(x, a, b, c, x0):
  """One correlation fit of Vosko, Wilk & Nusair (1980) in x = sqrt(r_s)."""
  q = math.sqrt(4 * c - b * b)
  at = torch.atan(q / (2 * x + b))
  xx = x * x + b * x + c
  return a * (torch.log(x * x / xx) + 2 * b / q * at - b * x0 / (x0 * x0 + b * x0 + c) *
              (torch.log((x - x0) ** 2 / xx) + 2 * (b + 2 * x0) / q * at))


_PARA = (0.0310907, 3.72744, 12.9352, -0.10498)
_FERRO = (0.01554535, 7.06042, 18.0578, -0.32500)
_STIFF = (-1 / (6 * math.pi ** 2), 1.13107, 13.0045, -0.0047584)


def _slater(rho):
  return -0.75 * (3 / math.pi) ** (1 / 3) * rho ** (1 / 3)


def _eps_lda(rho):
  """Energy per particle of a (S, ...) density, S = 1 or 2."""
  tot = rho.sum(0)
  x = (3 / (4 * math.pi * tot)) ** (1 / 6)
  if rho.shape[0] == 1:
    return _slater(tot) + _vwn(x, *_PARA)
  z = (rho[0] - rho[1]) / tot
  f = ((1 + z) ** (4 / 3) + (1 - z) ** (4 / 3) - 2) / (2 ** (4 / 3) - 2)
  fpp = 4 / (9 * (2 ** (1 / 3) - 1))
  p = _vwn(x, *_PARA)
  ec = p + _vwn(x, *_STIFF) * f * (1 - z ** 4) / fpp + (_vwn(x, *_FERRO) - p) * f * z ** 4
  return 0.5 * (_slater(2 * rho[0]) + _slater(2 * rho[1])) + ec


def _eps_pbe(rho, sigma):
  """Perdew, Burke & Ernzerhof (1996) on top of Perdew & Wang (1992)."""
  kf = (3 * math.pi ** 2 * rho) ** (1 / 3)
  s2 = sigma / (4 * kf * kf * rho * rho)
  ex = _slater(rho) * (1.804 - 0.804 / (1 + 0.2195149727645171 * s2 / 0.804))
  rs = (3 / (4 * math.pi * rho)) ** (1 / 3)
  den = 2 * 0.0310907 * (7.5957 * rs ** 0.5 + 3.5876 * rs + 1.6382 * rs ** 1.5 + 0.49294 * rs * rs)
  ec = -2 * 0.0310907 * (1 + 0.2137 * rs) * torch.log(1 + 1 / den)
  gam, beta = (1 - math.log(2)) / math.pi ** 2, 0.06672455060314922
  t2 = sigma / (16 * kf / math.pi * rho * rho)
  a = beta / gam / (torch.exp(-ec / gam) - 1)
  at = a * t2
  return ex + ec + gam * torch.log(1 + beta / gam * t2 * (1 + at) / (1 + at + at * at))


class _Exact:
  """The plane-wave path in complex128: plain torch operations, gradients of
  the orthonormalisation, transforms and functionals by torch autograd."""

  def __init__(self, case):
    cell, pos, chg, mask, kpts, g, tables = _geometry(case)
    dev = torch.device("cuda")
    self.case, self.n = case, (case["nx"], case["ny"], case["nz"])
    self.num = float(np.prod(self.n))
    self.vol = float(abs(np.linalg.det(cell)))
    self.idx = torch.as_tensor(np.flatnonzero(mask.reshape(-1)), device=dev)
    self.g = torch.as_tensor(g, device=dev)
    self.g2 = (self.g * self.g).sum(-1)
    self.tk = torch.as_tensor(0.5 * np.sum((g[mask][None] + kpts[:, None]) ** 2, -1), device=dev)
    self.occ = torch.as_tensor(_occupation(case, len(kpts)), device=dev)
    self.proj = None
    if tables is not None:
      self.v_ext = torch.as_tensor(tables[0], device=dev)
      self.proj = torch.as_tensor(tables[1], device=dev)
    else:
      s = sum(float(chg[i]) * torch.exp(-1j * (self.g @ torch.as_tensor(pos[i], device=dev)))
              for i in range(len(pos)))
      k = 4 * math.pi / (self.g2 + 1e-10)
      k[0, 0, 0] = 0.0
      self.v_ext = -k * s * self.num / self.vol
    self.hart = 4 * math.pi / torch.where(self.g2 > 0, self.g2, torch.ones_like(self.g2)) * (self.g2 > 0)

  def orth(self, w):
    """(C, Cholesky factor) of W^H W = L L^H, C = W L^-H."""
    low = torch.linalg.cholesky(w.mH @ w)
    c = torch.linalg.solve_triangular(low, w.mH, upper=False).mH
    return c, low

  def psi(self, c):
    full = torch.zeros((c.shape[1], int(self.num)), dtype=c.dtype, device=c.device)
    full = full.index_copy(1, self.idx, c.T)
    return torch.fft.ifftn(full.reshape((-1,) + self.n), dim=(1, 2, 3)) * (self.num / math.sqrt(self.vol))

  def xc_density(self, rho):
    """E_xc per volume element on the grid."""
    tot = rho.sum(0)
    if self.case["xc"] == LDA:
      return _eps_lda(rho) * tot
    rg = torch.fft.fftn(rho[0])
    grad = [torch.fft.ifftn(1j * self.g[..., a] * rg).real for a in range(3)]
    return _eps_pbe(rho[0], sum(x * x for x in grad)) * tot

  def grid_terms(self, rho):
    """(external, Hartree, xc) energies and each spin's dE/drho N/vol."""
    rho = rho.detach().requires_grad_(True)
    rg = torch.fft.fftn(rho.sum(0))
    f = self.vol / self.num ** 2
    ext = (rg.conj() * self.v_ext).real.sum() * f
    har = 0.5 * (self.hart * rg.abs() ** 2).sum() * f
    xc = self.xc_density(rho).sum() * self.vol / self.num
    v, = torch.autograd.grad(ext + har + xc, rho)
    return [x.detach() for x in (ext, har, xc)], v * (self.num / self.vol)

  def block(self, w, k, weight, v):
    """Weighted <T + V + V_nl> of one (s, k) block as a function of W: (sum,
    band expectations, kinetic part, nonlocal part, H c, C)."""
    c, _ = self.orth(w)
    t = (self.tk[k][:, None] * c.abs() ** 2).sum(0)
    dens = self.psi(c).abs() ** 2
    ev = (dens * v).sum((1, 2, 3)) * (self.vol / self.num)
    nl = torch.zeros_like(t)
    if self.proj is not None:
      nl = ((self.proj[k] @ c).abs() ** 2).sum(0) / self.vol
    eps = t + ev + nl
    return (weight * eps).sum(), eps.detach(), (weight * t).sum().detach(), (weight * nl).sum().detach(), c

  def pass_(self, params, v_fixed=None, weights=None, hmat=False):
    """energies[8] (or trace pair), gradient, band energies, band Hamiltonian."""
    w_all = torch.complex(params[0].double(), params[1].double())
    ns, nk = w_all.shape[:2]
    occ = self.occ if weights is None else weights
    cond = 1.0
    if v_fixed is None:
      rho = torch.zeros((ns,) + self.n, dtype=torch.float64, device=w_all.device)
      for s in range(ns):
        for k in range(nk):
          c, low = self.orth(w_all[s, k])
          rho[s] += (self.psi(c).abs() ** 2 * occ[s, k][:, None, None, None]).sum(0)
          d = torch.diagonal(low).real ** 2
          cond = max(cond, float(((w_all[s, k].abs() ** 2).sum(0) / d).max()))
          del c
      (ext, har, xc), v = self.grid_terms(rho)
    else:
      v = v_fixed[None].expand((ns,) + self.n)
    grad = torch.empty_like(params, dtype=torch.float64)
    eps = torch.empty_like(occ)
    kin = nlo = tot = 0.0
    hm = []
    for s in range(ns):
      for k in range(nk):
        w = w_all[s, k].detach().requires_grad_(True)
        total, eps[s, k], t, nl, c = self.block(w, k, occ[s, k], v[s])
        gw, = torch.autograd.grad(total, w)
        grad[0, s, k], grad[1, s, k] = gw.real, gw.imag
        kin, nlo, tot = kin + t, nlo + nl, tot + total.detach()
        if hmat:
          c = c.detach()
          hp = torch.fft.fftn(self.psi(c) * v[s], dim=(1, 2, 3)).reshape(c.shape[1], -1)[:, self.idx]
          hc = self.tk[k][:, None] * c + hp.T * (math.sqrt(self.vol) / self.num)
          hm.append((c.mH @ hc) * occ[s, k][None])
        del total, gw, w, c
    if v_fixed is not None:
      return torch.stack([tot, kin]), grad, eps, torch.stack(hm).reshape(ns, nk, *hm[0].shape)
    zero = torch.zeros_like(xc)
    e = torch.stack([kin, ext + nlo, har, xc, kin + ext + nlo + har + xc, zero + cond, zero, zero + nlo])
    return e, grad, eps, None


def exact(case, seed):
  x = _inputs(case, seed)
  if case["kind"] == "wave":
    s = prepare(case, seed)
    num = float(np.prod(s["coeff"].shape[-3:]))
    c = s["coeff"].to(torch.complex128)
    return torch.fft.ifftn(c, dim=(-3, -2, -1)) * (num / math.sqrt(s["vol"]))
  ex = _Exact(case)
  p = x["params"]
  if case["kind"] == "trace":
    out, grad, _, h = ex.pass_(p, v_fixed=x["v_eff"].double(), weights=torch.ones_like(ex.occ), hmat=True)
    return {"trace": out, "grad": grad, "hmat": h}
  if case["kind"] == "field":
    w = torch.complex(p[0].double(), p[1].double())
    c = torch.empty_like(w)
    rho = torch.zeros((w.shape[0],) + ex.n, dtype=torch.float64, device=w.device)
    for s in range(w.shape[0]):
      for k in range(w.shape[1]):
        c[s, k], _ = ex.orth(w[s, k])
        rho[s] += (ex.psi(c[s, k]).abs() ** 2 * ex.occ[s, k][:, None, None, None]).sum(0)
    vh = torch.fft.ifftn(ex.hart * torch.fft.fftn(rho.sum(0))).real
    ve = torch.fft.ifftn(ex.v_ext).real
    r = rho.detach().requires_grad_(True)
    if w.shape[0] == 1:
      vx, = torch.autograd.grad(ex.xc_density(r).sum(), r)
    else:   # the reference's polarised form: eps + rho_s d eps / d rho_s
      e = _eps_lda(r)
      d, = torch.autograd.grad(e.sum(), r)
      vx = e.detach()[None] + rho * d
    return {"coeff": c, "density": rho, "potential": torch.cat([vh[None], ve[None], vx])}
  e, grad, eps, _ = ex.pass_(p)
  if case["kind"] == "grad":
    return {"energies": e, "grad": grad}
  if case["kind"] == "bands":
    return {"energies": e, "grad": grad, "eps": eps}
  # optax.adam's update of step 51 from the given moments
  lr, b1, b2, eps_a, t = 1e-2, 0.9, 0.99, 1e-8, 51
  m = b1 * x["m"].double() + (1 - b1) * grad
  v = b2 * x["v"].double() + (1 - b2) * grad * grad
  new = p.double() - lr * (m / (1 - b1 ** t)) / (torch.sqrt(v / (1 - b2 ** t)) + eps_a)
  return {"energies": e, "params": new, "m": m, "v": v}
