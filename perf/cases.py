"""The framework's work as a set of timed cases.

Every case goes through the public entry points that a program uses:

* ``pair``: ``Grid.to_nodal`` then ``Grid.to_modal`` of a batch of fields (the
  transforms of regridding, diagnostics and filtering programs);
* ``step``: filtered SIL3 steps of the primitive equations, ``repeated(
  step_with_filters(imex_rk_sil3(eq, dt), [filter]), n)`` on sigma levels (dry,
  moist with tracers, or with Held-Suarez forcing) or on hybrid levels;
* ``grad``: a rollout of such steps and the gradient of a tracking loss with
  respect to the initial state (data assimilation, training);
* ``shallow``: filtered SIL3 steps of the multi-layer shallow-water equations.

``listed`` names twelve of them; ``draw`` gives others of the same ranges.
``exact`` evaluates a case in 64-bit torch, written from the equations and
without this package.
"""

import functools
import math

import numpy as np
import torch

from dinosaur_b200 import coordinate_systems
from dinosaur_b200 import held_suarez
from dinosaur_b200 import hybrid_coordinates
from dinosaur_b200 import layer_coordinates
from dinosaur_b200 import primitive_equations as pe
from dinosaur_b200 import shallow_water as sw
from dinosaur_b200 import sigma_coordinates
from dinosaur_b200 import spherical_harmonic as sh
from dinosaur_b200 import time_integration as ti
from dinosaur_b200 import units

MINUTE = 60.0 * 2 * 7.292e-5  # one minute in units of 1 / (2 Omega)

# Largest wavenumber and latitude nodes of the grid constructors (a grid has
# twice as many longitudes as latitudes).
GRIDS = {'T21': (21, 32), 'T31': (31, 48), 'TL47': (47, 48), 'T42': (42, 64),
         'TL63': (63, 64), 'TL95': (95, 96), 'T85': (85, 128), 'TL127': (127, 128),
         'T106': (106, 160), 'TL159': (159, 160), 'T119': (119, 180),
         'TL179': (179, 180), 'T170': (170, 256), 'TL255': (255, 256),
         'T213': (213, 320), 'T340': (340, 512)}


def _pair(name, grid, fields, precision):
  return dict(name=name, kind='pair', grid=grid, fields=fields, precision=precision)


def _step(name, grid, layers, members, physics, precision, steps, kind='step'):
  return dict(name=name, kind=kind, grid=grid, layers=layers, members=members,
              physics=physics, precision=precision, steps=steps)


def listed():
  return [
      # A diagnostic on a handful of fields of the smallest grid: latency.
      _pair('pair T21 x6', 'T21', 6, 'fp32'),
      # The transform benchmark's two grids, at the precision it runs them.
      _pair('pair T85 x128 bf16x3', 'T85', 128, 'bf16x3'),
      _pair('pair TL255 x128 bf16x3', 'TL255', 128, 'bf16x3'),
      # Three variables on 25 levels of a linear grid, default precision.
      _pair('pair TL159 x75', 'TL159', 75, 'fp32'),
      # One hour of the smallest baroclinic-wave configuration.
      _step('step T21/12', 'T21', 12, 1, 'dry', 'fp32', 4),
      # The Held-Suarez ensemble, one step per call.
      _step('step T42/24 hs x16', 'T42', 24, 16, 'hs', 'fp32', 1),
      # A moist ensemble of three on an odd number of levels.
      _step('step TL95/19 moist x3', 'TL95', 19, 3, 'moist', 'fp32', 1),
      # The forecast grid on hybrid levels, at the more accurate split form.
      _step('step T170/32 hybrid tf32x3', 'T170', 32, 1, 'hybrid', 'tf32x3', 1),
      # The large dry configuration.
      _step('step TL255/32 bf16x3', 'TL255', 32, 1, 'dry', 'bf16x3', 1),
      # The large moist ensemble with two passive tracers.
      _step('step TL255/32 moist x4 bf16x3', 'TL255', 32, 4, 'moist', 'bf16x3', 1),
      # A gradient through a rollout.
      _step('grad T42/20', 'T42', 20, 1, 'dry', 'fp32', 6, kind='grad'),
      # Three shallow-water layers.
      dict(name='shallow T85/3', kind='shallow', grid='T85', layers=3, members=1,
           precision='fp32', steps=4),
  ]


def draw(rng):
  """A case of the same ranges (sizes spread over their logarithm)."""
  log_int = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
  names = list(GRIDS)
  known = [{k: v for k, v in c.items() if k != 'name'} for c in listed()]
  # Points times fields of the largest listed case, whose cost bounds a draw.
  most = 0.5 * 512 * 256 * 32 * 4
  while True:
    kind = rng.choice(['pair', 'pair', 'step', 'step', 'step', 'grad', 'shallow'])
    grid = rng.choice(names)
    wn, lat = GRIDS[grid]
    points = 2 * lat * lat
    # The split forms are for grids from T85 on.
    precision = rng.choice(['fp32', 'bf16x3', 'tf32x3']) if wn >= 85 else 'fp32'
    if kind == 'pair':
      case = _pair('', grid, log_int(1, 512), precision)
      cost = case['fields'] * points / 8
    elif kind == 'shallow':
      case = dict(kind='shallow', grid=grid, layers=log_int(1, 12),
                  members=log_int(1, 8), precision=precision, steps=rng.randint(1, 6))
      cost = case['layers'] * case['members'] * points * case['steps']
    else:
      physics = (rng.choice(['dry', 'moist', 'hs']) if kind == 'grad' else
                 rng.choice(['dry', 'moist', 'hs', 'hybrid']))
      case = _step('', grid, log_int(4, 40), log_int(1, 16), physics, precision,
                   rng.randint(1, 6), kind=kind)
      cost = case['layers'] * case['members'] * points * case['steps'] * (
          4 if kind == 'grad' else 1) * (2 if physics == 'moist' else 1)
      if wn > 255:
        continue
    case.pop('name', None)
    if cost <= most and case not in known:
      return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------


def _modal_random(gen, grid, lead, power):
  """Coefficients of a smooth random field: N(0, 1) (l + 1)^-power for
  |m| <= l, the highest total wavenumber zero."""
  wn, _ = GRIDS[grid]
  m_rows, n_l = 2 * wn + 1, wn + 2
  x = torch.randn(tuple(lead) + (m_rows, n_l), generator=gen, device='cuda',
                  dtype=torch.float32)
  l = torch.arange(n_l, device='cuda')
  m = (torch.arange(m_rows, device='cuda') + 1) // 2
  scale = torch.where((m[:, None] <= l) & (l < n_l - 1), (l + 1.0) ** -power, 0.0)
  return x * scale.float()


def _column_random(gen, grid, members, layers, power):
  """Random fields that vary smoothly over the levels: four vertical modes."""
  modes = _modal_random(gen, grid, (members, 4), power)
  s = (torch.arange(layers, device='cuda') + 0.5) / layers
  j = torch.arange(4, device='cuda')
  profile = torch.cos(math.pi * j * s[:, None]) / (j + 1.0)
  return torch.einsum('kj,bjml->bkml', profile, modes).contiguous()


def _constant(value):
  """Modal coefficient of a constant field."""
  return 2 * math.sqrt(math.pi) * value


def _reference_temperature(case):
  k = case['layers']
  if case['physics'] == 'hs':
    return np.full((k,), 285.0)
  return np.maximum(200.0, 288.0 * ((np.arange(k) + 0.5) / k) ** 0.19)


def _time_step(case):
  return min(15.0, 1500.0 / GRIDS[case['grid']][0]) * MINUTE


def _filter_options(case):
  if case.get('physics') == 'hs':
    return dict(tau=0.0087504, order=1.5, cutoff=0.8)
  return {}


def _orography(grid):
  gen = torch.Generator(device='cuda').manual_seed(17)
  return 3e-4 * _modal_random(gen, grid, (), 2.0)


def _tracer_names(case):
  return ('specific_humidity', 'tracer_a', 'tracer_b') if case['physics'] == 'moist' else ()


def _pe_arrays(case, seed):
  """Leaves of a state: [members, layers, M, L] each, ln p_s with one level."""
  gen = torch.Generator(device='cuda').manual_seed(seed)
  b, k, grid = case['members'], case['layers'], case['grid']
  out = {
      'vorticity': 0.05 * _column_random(gen, grid, b, k, 1.0),
      'divergence': 0.005 * _column_random(gen, grid, b, k, 1.0),
      'temperature_variation': 10.0 * _column_random(gen, grid, b, k, 1.5),
      'log_surface_pressure': 0.05 * _modal_random(gen, grid, (b, 1), 2.0),
  }
  out['log_surface_pressure'][..., 0, 0] += _constant(math.log(units.nondim_pressure(1e5)))
  for name, mean in zip(_tracer_names(case), (5e-3, 1.0, 2.0)):
    out[name] = 0.2 * mean * _column_random(gen, grid, b, k, 1.5)
    out[name][..., 0, 0] += _constant(mean)
  return out


def _sw_parameters(case):
  """Mean potentials and densities of the layers."""
  k = case['layers']
  return np.linspace(0.04, 0.06, k), np.linspace(1.0, 1.5, k)


def _sw_arrays(case, seed):
  gen = torch.Generator(device='cuda').manual_seed(seed)
  b, k, grid = case['members'], case['layers'], case['grid']
  return {'vorticity': 0.05 * _modal_random(gen, grid, (b, k), 1.0),
          'divergence': 0.005 * _modal_random(gen, grid, (b, k), 1.0),
          'potential': 0.005 * _modal_random(gen, grid, (b, k), 1.5)}


# ---------------------------------------------------------------------------
# What a program builds once and keeps: grids, equations, step functions
# ---------------------------------------------------------------------------


@functools.lru_cache(maxsize=2)
def _grid(name, precision):
  impl = functools.partial(sh.CudaSphericalHarmonics, precision=precision)
  return getattr(sh.Grid, name)(spherical_harmonics_impl=impl)


@functools.lru_cache(maxsize=1)
def _pe_step(items):
  case = dict(items)
  grid = _grid(case['grid'], case['precision'])
  tref, orography = _reference_temperature(case), _orography(case['grid'])
  specs = units.SimUnits()
  if case['physics'] == 'hybrid':
    levels = hybrid_coordinates.HybridCoordinates.analytic_levels(case['layers'])
    coords = coordinate_systems.CoordinateSystem(grid, levels)
    eq = pe.PrimitiveEquationsHybrid(tref, orography, coords, specs)
  else:
    levels = sigma_coordinates.SigmaCoordinates.equidistant(case['layers'])
    coords = coordinate_systems.CoordinateSystem(grid, levels)
    eq = pe.PrimitiveEquationsSigma(
        tref, orography, coords, specs,
        humidity_key='specific_humidity' if case['physics'] == 'moist' else None)
  if case['physics'] == 'hs':
    eq = ti.compose_equations([eq, held_suarez.HeldSuarezForcingSigma(coords, specs, tref)])
  dt = _time_step(case)
  step = ti.step_with_filters(ti.imex_rk_sil3(eq, dt), [
      ti.exponential_step_filter(grid, dt, **_filter_options(case))])
  return ti.repeated(step, case['steps'])


@functools.lru_cache(maxsize=1)
def _sw_step(items):
  case = dict(items)
  grid = _grid(case['grid'], case['precision'])
  potential, densities = _sw_parameters(case)
  coords = coordinate_systems.CoordinateSystem(
      grid, layer_coordinates.LayerCoordinates(case['layers']))
  eq = sw.ShallowWaterEquations(coords, units.SimUnits(), _orography(case['grid']),
                                potential, densities=densities)
  dt = _time_step(case)
  step = ti.step_with_filters(ti.imex_rk_sil3(eq, dt), [
      ti.exponential_step_filter(grid, dt)])
  return ti.repeated(step, case['steps'])


def _key(case):
  return tuple(sorted((k, v) for k, v in case.items() if k != 'name'))


def _pe_state(arrays, members):
  one = (lambda x: x[0]) if members == 1 else (lambda x: x)
  leaf = lambda k: one(arrays[k])
  names = ('vorticity', 'divergence', 'temperature_variation', 'log_surface_pressure')
  return pe.State(*[leaf(k) for k in names],
                  tracers={k: leaf(k) for k in arrays if k not in names})


def _pe_leaves(state):
  return dict({'vorticity': state.vorticity, 'divergence': state.divergence,
               'temperature_variation': state.temperature_variation,
               'log_surface_pressure': state.log_surface_pressure}, **state.tracers)


# Weights of the tracking loss, which bring the leaves to one scale.
LOSS_WEIGHT = {'vorticity': 20.0, 'divergence': 200.0, 'temperature_variation': 0.1,
               'log_surface_pressure': 20.0, 'specific_humidity': 200.0,
               'tracer_a': 1.0, 'tracer_b': 1.0}


def prepare(case, seed):
  kind = case['kind']
  if kind == 'pair':
    gen = torch.Generator(device='cuda').manual_seed(seed)
    grid = _grid(case['grid'], case['precision'])
    grid.plan  # built with the grid, before the first transform
    return dict(kind=kind, grid=grid,
                x=_modal_random(gen, case['grid'], (case['fields'],), 1.5))
  if kind == 'shallow':
    arrays = _sw_arrays(case, seed)
    one = (lambda x: x[0]) if case['members'] == 1 else (lambda x: x)
    return dict(kind=kind, step=_sw_step(_key(case)),
                state=sw.State(*[one(arrays[k])
                                 for k in ('vorticity', 'divergence', 'potential')]))
  out = dict(kind=kind, step=_pe_step(_key(case)),
             state=_pe_state(_pe_arrays(case, seed), case['members']))
  if kind == 'grad':
    out['target'] = _pe_state(_pe_arrays(case, seed + 1000003), case['members'])
  return out


def run(state):
  kind = state['kind']
  if kind == 'pair':
    nodal = state['grid'].to_nodal(state['x'])
    return nodal, state['grid'].to_modal(nodal)
  if kind == 'shallow':
    s = state['step'](state['state'])
    return s.vorticity, s.divergence, s.potential
  if kind == 'step':
    return _pe_leaves(state['step'](state['state']))
  # grad
  leaves = {k: v.detach().requires_grad_(True) for k, v in _pe_leaves(state['state']).items()}
  members = 1 if leaves['vorticity'].ndim == 3 else leaves['vorticity'].shape[0]
  lead = (lambda x: x[None]) if members == 1 else (lambda x: x)
  final = _pe_leaves(state['step'](_pe_state({k: lead(v) for k, v in leaves.items()}, members)))
  target = _pe_leaves(state['target'])
  loss = sum(0.5 * ((final[k] - target[k]) * LOSS_WEIGHT[k]).square().sum() for k in final)
  loss.backward()
  return {'final': {k: v.detach() for k, v in final.items()},
          'gradient': {k: v.grad for k, v in leaves.items()}}


# ---------------------------------------------------------------------------
# Work and tolerances
# ---------------------------------------------------------------------------


def _counts(case):
  """(nodal points, modal coefficients, Legendre multiply-adds) per field,
  with the even and odd wavenumbers summed over one hemisphere."""
  wn, lat = GRIDS[case['grid']]
  lw, n_l = wn + 1, wn + 2
  modal = n_l + 2 * sum(n_l - m for m in range(1, lw))
  return 2 * lat * lat, modal, modal * (lat // 2)


def work(case):
  """One pass: inputs once, outputs once; transforms by their folded Legendre
  sums and real FFTs, and the implicit solves by their per-l operators."""
  points, modal, legendre = _counts(case)
  lat = GRIDS[case['grid']][1]
  transform = 2.0 * legendre + 2.5 * points * math.log2(2 * lat)
  if case['kind'] == 'pair':
    f = case['fields']
    return {'bytes': 4.0 * f * (2 * points + 2 * modal), 'flops': 2 * f * transform}
  f = case['layers'] * case['members']
  if case['kind'] == 'shallow':
    return {'bytes': 4.0 * modal * 6 * f, 'flops': case['steps'] * 3 * 9 * f * transform}
  nt = len(_tracer_names(case))
  state = (3 + nt) * f + case['members']
  inv = state + 2 * f + 2 * case['members'] + (2 * f if nt else 0)
  fwd = 6 * f + 3 * nt * f + case['members'] + (3 * f if nt else 0)
  if case['physics'] == 'hs':
    fwd += f
  n = 2 * case['layers'] + 1
  solve = 2.0 * n * n * modal * case['members']
  flops = case['steps'] * (3 * (inv + fwd) * transform + 5 * solve)
  nbytes = 8.0 * modal * state
  if case['kind'] == 'grad':
    flops, nbytes = 3 * flops, 2.5 * nbytes
  return {'bytes': nbytes, 'flops': flops}


def tolerance(case):
  # Against `exact`, measured: pairs 5e-7 (bf16x3 6e-6); steps and gradients
  # 2e-6 (bf16x3 2e-5; hybrid levels 5e-6), in the divergence.
  split = case['precision'] == 'bf16x3'
  if case['kind'] == 'pair':
    return {'rel': 2.5e-5 if split else 2e-6}
  hybrid = case.get('physics') == 'hybrid'
  return {'rel': 1e-4 if split else 2e-5 if hybrid else 1e-5}


# ---------------------------------------------------------------------------
# The same in 64-bit torch
# ---------------------------------------------------------------------------


class _Sphere64:
  """Transforms and spectral operators as dense 64-bit products."""

  def __init__(self, grid):
    wn, lat = GRIDS[grid]
    self.lw, self.n_l, self.n_lat, self.n_lon = wn + 1, wn + 2, lat, 2 * lat
    x, w = np.polynomial.legendre.leggauss(lat)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device='cuda', dtype=torch.float64)
    self.sin = t(x)
    self.sec2, self.cos2 = 1 / (1 - self.sin ** 2), 1 - self.sin ** 2
    self.weights = t(w * 2 * np.pi / self.n_lon)
    p = np.zeros((self.lw, lat, self.n_l))
    root = np.sqrt(1 - x * x)
    pmm = np.full(lat, math.sqrt(0.5))
    for m in range(self.lw):
      if m:
        pmm = -math.sqrt(1 + 0.5 / m) * root * pmm
      p[m, :, m] = pmm
    m = np.arange(self.lw)[:, None].astype(np.float64)
    for l in range(1, self.n_l):
      low = np.arange(self.lw) < l
      mm = m[low]
      a = np.sqrt((4.0 * l * l - 1) / (l * l - mm * mm))
      b = np.sqrt(np.maximum((l - 1.0) ** 2 - mm * mm, 0.0) / (4.0 * (l - 1.0) ** 2 - 1)) if l > 1 else 0 * mm
      prev = p[low, :, l - 2] if l > 1 else 0.0
      p[low, :, l] = a * (x * p[low, :, l - 1] - b * prev)
    rows = (np.arange(2 * self.lw - 1) + 1) // 2
    self.p = t(p)[torch.as_tensor(rows, device='cuda')]  # [M, J, L]
    lon = 2 * np.pi * np.arange(self.n_lon) / self.n_lon
    f = np.empty((self.n_lon, 2 * self.lw - 1))
    f[:, 0] = 1 / np.sqrt(2 * np.pi)
    k = np.arange(1, self.lw)
    f[:, 1::2] = np.cos(np.outer(lon, k)) / np.sqrt(np.pi)
    f[:, 2::2] = np.sin(np.outer(lon, k)) / np.sqrt(np.pi)
    self.f = t(f)
    l = np.arange(self.n_l).astype(np.float64)
    self.lap = t(-l * (l + 1))
    self.inv_lap = torch.where(self.lap == 0, 0.0, 1 / self.lap)
    mr = rows[:, None].astype(np.float64)
    mask = mr <= l
    a = np.sqrt(mask * np.maximum(l ** 2 - mr ** 2, 0) / np.where(l > 0, 4 * l ** 2 - 1, 1))
    b = np.sqrt(mask * np.maximum((l + 1) ** 2 - mr ** 2, 0) / (4 * (l + 1) ** 2 - 1))
    a[:, 0] = 0
    b[:, -1] = 0
    self.d_cos = t((l + 1) * a), t(-l * b)
    self.d_sec = t((l - 1) * a), t(-(l + 2) * b)
    self.m_rows = t(rows)[:, None]

  def to_nodal(self, x):
    y = torch.einsum('mjl,...ml->...mj', self.p, x)
    return torch.matmul(self.f, y)

  def to_modal(self, z):
    y = torch.matmul(self.f.T, z * self.weights)
    return torch.einsum('mjl,...mj->...ml', self.p, y)

  def d_dlon(self, x):
    swapped = torch.zeros_like(x)
    swapped[..., 1::2, :] = x[..., 2::2, :]
    swapped[..., 2::2, :] = -x[..., 1::2, :]
    return swapped * self.m_rows

  @staticmethod
  def _recurrence(tables, x):
    up, down = tables[0] * x, tables[1] * x
    pad = torch.zeros_like(x[..., :1])
    return (torch.cat([up[..., 1:], pad], -1) + torch.cat([pad, down[..., :-1]], -1))

  def cos_lat_grad(self, x):
    return self.d_dlon(x), self._recurrence(self.d_cos, x)

  def div(self, u, v):
    return self.d_dlon(u) + self._recurrence(self.d_sec, v)

  def curl(self, u, v):
    return self.d_dlon(v) - self._recurrence(self.d_sec, u)

  def wind(self, vorticity, divergence):
    ax, ay = self.cos_lat_grad(divergence * self.inv_lap)
    bx, by = self.cos_lat_grad(vorticity * self.inv_lap)
    return ax - by, ay + bx

  def clip(self, x):
    return torch.cat([x[..., :-1], torch.zeros_like(x[..., :1])], -1)


_sphere64 = functools.lru_cache(maxsize=1)(_Sphere64)


def _t64(a):
  return torch.as_tensor(np.ascontiguousarray(a), device='cuda', dtype=torch.float64)


def _col(a):
  return _t64(a)[:, None, None]


class _Equations64:
  """Explicit and implicit terms of the primitive equations on sigma or hybrid
  levels; states are dicts of [members, layers, M, L] arrays."""

  def __init__(self, case):
    self.sphere = _sphere64(case['grid'])
    self.physics, self.k = case['physics'], case['layers']
    self.tracers = _tracer_names(case)
    self.spec = units.SimUnits()
    self.tref = _reference_temperature(case)
    self.orography = _orography(case['grid']).double()
    k, spec, tref = self.k, self.spec, self.tref
    lower = np.tril(np.ones((k, k)))
    if self.physics == 'hybrid':
      lev = hybrid_levels64(k)
      self.a, self.b = units.nondim_pressure(lev[0] * 100.0), lev[1]
      self.ps_ref = units.nondim_pressure(101325.0)
      alpha, ratio, dp, weight = (x.flatten().cpu().numpy() for x in self.pressure_terms(
          _col([self.ps_ref])))
      self.alpha = alpha
      self.g = spec.R * (np.diag(alpha) + np.triu(np.tile(ratio, (k, 1)), 1))
      self.row = np.diff(self.a) / self.ps_ref + np.diff(self.b)
      self.column = spec.R * tref * weight * self.ps_ref / dp
      thick, sums, scale = dp, np.cumsum(np.diff(self.b)), dp
    else:
      bounds = np.linspace(0, 1, k + 1, dtype=np.float32)  # the levels' own type
      b64 = bounds.astype(np.float64)
      self.centers = ((b64[1:] + b64[:-1]) / 2).astype(np.float32)
      ds32 = np.diff(b64).astype(np.float32)
      self.ds = ds32.astype(np.float64)
      c2c = np.diff(self.centers.astype(np.float64)).astype(np.float32)
      self.inv_c2c = (1 / c2c).astype(np.float64)
      logs = np.log(self.centers)
      alpha = np.empty(k, np.float32)
      alpha[:-1], alpha[-1] = np.diff(logs) / 2, -logs[-1]
      self.alpha = alpha = alpha.astype(np.float64)
      pair_sum = np.concatenate([[0.0], alpha[1:] + alpha[:-1]])
      self.g = spec.R * (np.diag(alpha) + np.triu(np.tile(pair_sum, (k, 1)), 1))
      self.row, self.column = self.ds, spec.R * tref
      thick, sums, scale = self.ds, np.cumsum(ds32).astype(np.float64), self.ds
    up = lambda x: np.concatenate([np.zeros((1, k)), x[:-1]])
    pa = lower * self.alpha[:, None]
    pairs = thick[:-1] + thick[1:]
    kk = np.concatenate([np.diff(tref) / pairs, [0]])[:, None] * (lower - sums[:, None])
    self.h = (spec.kappa * tref[:, None] * (pa + up(pa)) / thick[:, None] - kk - up(kk)) * scale

  # -- implicit part ---------------------------------------------------------
  @functools.cached_property
  def operator(self):
    """[L, n, n] matrices of the implicit terms on (div, T', ln p_s)."""
    k, n = self.k, 2 * self.k + 1
    m = torch.zeros((self.sphere.n_l, n, n), device='cuda', dtype=torch.float64)
    lap = self.sphere.lap[:, None, None]
    m[:, :k, k:2 * k] = -lap * _t64(self.g)
    m[:, :k, 2 * k:] = -lap * _t64(self.column)[:, None]
    m[:, k:2 * k, :k] = -_t64(self.h)
    m[:, 2 * k, :k] = -_t64(self.row)
    return m

  def apply(self, matrix, s):
    y = torch.cat([s['divergence'], s['temperature_variation'], s['log_surface_pressure']], -3)
    y = torch.einsum('lij,bjml->biml', matrix, y)
    k = self.k
    return {'divergence': y[:, :k], 'temperature_variation': y[:, k:2 * k],
            'log_surface_pressure': y[:, 2 * k:]}

  def implicit(self, s):
    return {**{k: torch.zeros_like(v) for k, v in s.items()}, **self.apply(self.operator, s)}

  def inverse(self, s, eta):
    n = 2 * self.k + 1
    eye = torch.eye(n, device='cuda', dtype=torch.float64)
    return {**s, **self.apply(torch.linalg.inv(eye - eta * self.operator), s)}

  # -- explicit part ---------------------------------------------------------
  def pressure_terms(self, ps):
    """alpha, log pressure ratio, layer thickness and pressure-gradient weight
    of every hybrid layer at surface pressure ps."""
    a, b = _col(self.a), _col(self.b)
    p, floor = a + b * ps, 1e-6 * ps
    lo, hi = p[..., :-1, :, :], p[..., 1:, :, :]
    dp = hi - lo
    ratio = torch.log(torch.maximum(hi, floor) / torch.maximum(lo, floor))
    alpha = 1 - lo / dp * ratio
    return alpha, ratio, dp, ratio * b[:-1] + alpha * (b[1:] - b[:-1])

  def explicit(self, s):
    sp, spec = self.sphere, self.spec
    sec2, nodal = sp.sec2, sp.to_nodal
    zeta, div = nodal(s['vorticity']), nodal(s['divergence'])
    temp = nodal(s['temperature_variation'])
    q = {n: nodal(s[n]) for n in self.tracers}
    u, v = (nodal(c) for c in sp.wind(s['vorticity'], s['divergence']))
    gx, gy = (nodal(c) for c in sp.cos_lat_grad(s['log_surface_pressure']))
    ug = (u * gx + v * gy) * sec2
    tref = _col(self.tref)
    coriolis = 2 * spec.angular_velocity * sp.sin
    shift = lambda x: torch.cat([torch.zeros_like(x[..., :1, :, :]), x[..., :-1, :, :]], -3)
    zero = torch.zeros_like(u[..., :1, :, :])
    hybrid = self.physics == 'hybrid'
    if hybrid:
      ps = torch.exp(nodal(s['log_surface_pressure']))
      alpha, ratio, dp, weight = self.pressure_terms(ps)
      db = _col(np.diff(self.b))
      layer_full, layer_adv = dp * div + db * ps * ug, db * ps * ug
      sums, w_scale = _col(np.cumsum(np.diff(self.b))), dp
      grad_p = ug * ps * weight / dp
    else:
      layer_full, layer_adv = _col(self.ds) * (div + ug), _col(self.ds) * ug
      sums, w_scale, grad_p = _col(np.cumsum(self.ds)), 1.0, ug
      dp = _col(self.ds)

    def flux(x):
      c = torch.cumsum(x, -3)
      return (sums * c[..., -1:, :, :] - c)[..., :-1, :, :]

    full, adv = flux(layer_full), flux(layer_adv)

    def vertical(w, x):
      d = x[..., 1:, :, :] - x[..., :-1, :, :]
      y = torch.cat([zero, w * (d if hybrid else d * _col(self.inv_c2c)), zero], -3)
      return -0.5 * (y[..., 1:, :, :] + y[..., :-1, :, :]) / w_scale

    def omega(field, total):
      af = _col(self.alpha) * torch.cumsum(total, -3)
      return field * (grad_p - (af + shift(af)) / dp)

    moist = self.physics == 'moist'
    ratio_r, ratio_c = spec.R_vapor / spec.R, spec.Cp_vapor / spec.Cp
    hum = q['specific_humidity'] if moist else None
    virtual = 1 + (ratio_r - 1) * hum if moist else 1.0
    if hybrid:
      pgf = spec.R * (temp + tref) * weight * ps / dp - _col(self.column)
    else:
      pgf = spec.R * temp * virtual
    au = -v * (zeta + coriolis) - vertical(full, u) + pgf * gx
    av = u * (zeta + coriolis) - vertical(full, v) + pgf * gy
    d_temp = temp * div + vertical(full, temp)
    if np.unique(self.tref).size > 1:
      d_temp = d_temp + vertical(adv, tref.expand(temp.shape))
    field = temp
    if moist:
      field = (temp * virtual + tref * (ratio_r - ratio_c) * hum) / (1 + (ratio_c - 1) * hum)
    d_temp = d_temp + spec.kappa * (omega(tref, layer_adv) + omega(field, layer_full))
    energy = 0.5 * (u * u + v * v) * sec2
    if hybrid:
      t_all = temp + tref
      below = torch.flip(torch.cumsum(torch.flip(t_all * ratio, (-3,)), -3), (-3,))
      phi = spec.R * (below - t_all * ratio + alpha * t_all)
      energy = energy + phi - torch.einsum('gh,...hij->...gij', _t64(self.g), temp)
      da = _col(np.diff(self.a))
      d_lnps = -torch.sum(da * div * (1 / ps - 1 / self.ps_ref) + ug * db, -3, keepdim=True)
    else:
      d_lnps = -torch.sum(layer_adv, -3, keepdim=True)
    extra = 0.0
    if self.physics == 'hs':
      cut = np.maximum(0, (self.centers.astype(np.float64) - 0.7) / 0.3)
      rate = 1 / units.nondim_time(86400.0)
      au = au + _col(rate * cut) * u
      av = av + _col(rate * cut) * v
      lp = nodal(s['log_surface_pressure']) + _col(np.log(
          self.centers.astype(np.float64))) - math.log(units.nondim_pressure(1e5))
      teq = torch.exp(spec.kappa * lp) * (315.0 - 60.0 * sp.sin ** 2 - 10.0 * lp * sp.cos2)
      kt = rate / 40 + (rate / 4 - rate / 40) * _col(cut) * sp.cos2 ** 2
      extra = sp.to_modal(-kt * (temp + tref - torch.clamp(teq, min=200.0)))
    au, av = sp.to_modal(au * sec2), sp.to_modal(av * sec2)
    d_vort = -sp.curl(au, av)
    d_div = -sp.div(au, av) - sp.lap * (sp.to_modal(energy) + spec.g * self.orography)
    if moist:
      coef = tref * (spec.R_vapor - spec.R)
      hx, hy = (nodal(c) for c in sp.cos_lat_grad(s['specific_humidity']))
      lap_p = nodal(s['log_surface_pressure'] * sp.lap)
      d_vort = d_vort + sp.to_modal(coef * sec2 * (gx * hy - gy * hx))
      phi = torch.einsum('gh,...hij->...gij', _t64(self.g), hum * (temp + tref) * (ratio_r - 1))
      d_div = d_div - sp.lap * sp.to_modal(phi) - sp.to_modal(
          coef * (sec2 * (gx * hx + gy * hy) + hum * lap_p))

    def advected(x, nodal_part):
      return sp.to_modal(nodal_part) - sp.div(sp.to_modal(u * x * sec2), sp.to_modal(v * x * sec2))

    out = {'vorticity': d_vort, 'divergence': d_div,
           'temperature_variation': advected(temp, d_temp),
           'log_surface_pressure': sp.to_modal(d_lnps)}
    for n in self.tracers:
      out[n] = advected(q[n], q[n] * div + vertical(full, q[n]))
    out = {n: sp.clip(x) for n, x in out.items()}
    out['temperature_variation'] = out['temperature_variation'] + extra
    return out


def hybrid_levels64(k):
  """a (hPa) and b of the analytic levels: eta = (i / k)^2, b = eta^3."""
  eta = np.linspace(0, 1, k + 1) ** 2
  b = eta ** 3
  a = (eta - b) * 1000.0
  a[0] = a[-1] = 0.0
  return a, b


class _Shallow64:

  def __init__(self, case):
    self.sphere = _sphere64(case['grid'])
    potential, rho = _sw_parameters(case)
    self.mean = _col(potential)
    ratios = np.minimum(rho[None, :] / rho[:, None], 1.0)
    np.fill_diagonal(ratios, 0.0)
    self.ratios = _t64(ratios)
    self.orography = _orography(case['grid']).double()

  def explicit(self, s):
    sp = self.sphere
    u, v = (sp.to_nodal(sp.clip(c)) for c in sp.wind(s['vorticity'], s['divergence']))
    zeta = sp.to_nodal(sp.clip(s['vorticity'])) + 2 * units.SimUnits().angular_velocity * sp.sin
    phi = sp.to_nodal(sp.clip(s['potential']))
    bu, bv, gu, gv = (sp.to_modal(x * sp.sec2) for x in (u * zeta, v * zeta, u * phi, v * phi))
    energy = sp.to_modal(0.5 * (u * u + v * v) * sp.sec2)
    p = torch.einsum('ij,bjml->biml', self.ratios, s['potential']) + self.orography
    return {'vorticity': sp.clip(-sp.div(bu, bv)),
            'divergence': sp.clip(-sp.lap * (p + energy) + sp.curl(bu, bv)),
            'potential': sp.clip(-sp.div(gu, gv))}

  def implicit(self, s):
    return {'vorticity': torch.zeros_like(s['vorticity']),
            'divergence': -self.sphere.lap * s['potential'],
            'potential': -self.mean * s['divergence']}

  def inverse(self, s, eta):
    lap = self.sphere.lap
    f = 1 / (1 - eta * eta * self.mean * lap)
    return {'vorticity': s['vorticity'],
            'divergence': f * (s['divergence'] - eta * lap * s['potential']),
            'potential': f * (s['potential'] - eta * self.mean * s['divergence'])}


def _sil3(eq, y, dt, scaling):
  """One filtered step of the SIL3 implicit-explicit Runge-Kutta scheme."""
  comb = lambda *terms: {k: sum(c * t[k] for c, t in terms) for k in y}
  f0, g0 = eq.explicit(y), eq.implicit(y)
  y1 = eq.inverse(comb((1, y), (dt / 3, f0), (dt / 6, g0)), dt / 6)
  f1 = eq.explicit(y1)
  y2 = eq.inverse(comb((1, y), (dt / 6, f0), (dt / 2, f1), (dt / 3, g0)), dt / 3)
  f2, g2 = eq.explicit(y2), eq.implicit(y2)
  base = comb((1, y), (dt / 2, f0), (-dt / 2, f1), (dt, f2), (3 * dt / 8, g0), (3 * dt / 8, g2))
  g3 = eq.implicit(eq.inverse(base, dt / 4))
  return {k: v * scaling for k, v in comb((1, base), (dt / 4, g3)).items()}


def _rollout64(eq, y, case):
  dt, n_l = _time_step(case), eq.sphere.n_l
  opt = dict(dict(tau=0.010938, order=18, cutoff=0.0), **_filter_options(case))
  x = np.arange(n_l) / (n_l - 1)
  x = np.maximum(0, (x - opt['cutoff']) / (1 - opt['cutoff']))
  scaling = _t64(np.exp(-dt / opt['tau'] * x ** (2 * opt['order'])))
  for _ in range(case['steps']):
    y = _sil3(eq, y, dt, scaling)
  return y


def exact(case, seed):
  kind = case['kind']
  one = (lambda x: x[0]) if case.get('members') == 1 else (lambda x: x)
  if kind == 'pair':
    gen = torch.Generator(device='cuda').manual_seed(seed)
    sp = _sphere64(case['grid'])
    nodal = sp.to_nodal(_modal_random(gen, case['grid'], (case['fields'],), 1.5).double())
    return nodal, sp.to_modal(nodal)
  if kind == 'shallow':
    y = {k: v.double() for k, v in _sw_arrays(case, seed).items()}
    y = _rollout64(_Shallow64(case), y, case)
    return tuple(one(y[k]) for k in ('vorticity', 'divergence', 'potential'))
  y = {k: v.double() for k, v in _pe_arrays(case, seed).items()}
  eq = _Equations64(case)
  if kind == 'step':
    with torch.no_grad():
      return {k: one(v) for k, v in _rollout64(eq, y, case).items()}
  points = 2 * GRIDS[case['grid']][1] ** 2
  if points * case['layers'] * case['members'] * case['steps'] > 4e6:
    return None  # the 64-bit tape of this rollout would not fit
  y = {k: v.requires_grad_(True) for k, v in y.items()}
  final = _rollout64(eq, y, case)
  target = _pe_arrays(case, seed + 1000003)
  loss = sum(0.5 * ((final[k] - target[k].double()) * LOSS_WEIGHT[k]).square().sum()
             for k in final)
  loss.backward()
  return {'final': {k: one(v.detach()) for k, v in final.items()},
          'gradient': {k: one(v.grad) for k, v in y.items()}}
