"""Dependent launches that overlap: back-to-back calls give the bits of calls
that are waited for.

Kernels of large grids start while their predecessor is finishing, so a missing
wait would let one read or overwrite what the other still uses.  Transforms
(with the real FFT and with direct sums, at all precisions), operators, and
steps and gradients of every form of the equations run in a row on alternating
inputs, without any synchronisation, on grids with one and with several chunks
per transform and grids below and above the size from which launches overlap;
every result must equal, bit for bit, the one of a call that was waited for.
"""

import functools

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from dinosaur_b200 import _lib  # noqa: E402
from dinosaur_b200 import coordinate_systems  # noqa: E402
from dinosaur_b200 import held_suarez  # noqa: E402
from dinosaur_b200 import hybrid_coordinates  # noqa: E402
from dinosaur_b200 import layer_coordinates  # noqa: E402
from dinosaur_b200 import primitive_equations as pe  # noqa: E402
from dinosaur_b200 import shallow_water  # noqa: E402
from dinosaur_b200 import sigma_coordinates  # noqa: E402
from dinosaur_b200 import spherical_harmonic as sh  # noqa: E402
from dinosaur_b200 import time_integration as ti  # noqa: E402
from dinosaur_b200 import units  # noqa: E402


def grid_of(name, precision):
  impl = functools.partial(sh.CudaSphericalHarmonics, precision=precision)
  return getattr(sh.Grid, name)(spherical_harmonics_impl=impl)


def field(grid, lead, power, seed):
  rng = np.random.default_rng(seed)
  _, l = np.meshgrid(*grid.modal_axes, indexing='ij')
  x = rng.standard_normal(lead + l.shape) * grid.mask / (l + 1.0) ** power
  return torch.as_tensor(x, device='cuda', dtype=torch.float32)


@pytest.mark.parametrize('name,fields,precision', [
    ('T21', 3, 'fp32'), ('TL95', 70, 'fp32'), ('T85', 150, 'bf16x3'),
    ('TL255', 130, 'bf16x3'), ('TL127', 40, 'tf32x3')])
def test_transforms_in_a_row(name, fields, precision):
  check_transforms_in_a_row(grid_of(name, precision), fields)


@pytest.mark.parametrize('name,fields,precision,inverse,forward', [
    ('T213', 70, 'bf16x3', '160x2', '112x2'), ('TL255', 130, 'bf16x3', '128x2', '144x2'),
    ('T106', 70, 'tf32x3', '80x2', '64x2'), ('TL127', 70, 'tf32x3', '64x2', '80x2')])
def test_contractions_that_fill_tensor_memory_in_a_row(name, fields, precision, inverse,
                                                       forward, monkeypatch):
  # Launch shapes of which one CTA takes all 512 columns of tensor memory (the
  # inverse at T213 and T106, the forward at TL255 and TL127) while the shared
  # memory holds two: the CTAs of a launch and of its dependent queue for them,
  # between a forward and the next inverse transform and in the timed launches
  # of the plan's own set-up.
  monkeypatch.setenv('DINO_B200_TC_SHAPE', f'inv:{inverse},fwd:{forward}')
  g = grid_of(name, precision)
  described = g.plan.describe()
  for shape in (inverse, forward):
    rows, stages = shape.split('x')
    assert f'ranges of {rows} rows, {stages} stages' in described, described
  check_transforms_in_a_row(g, fields)
  _lib.check(_lib.lib().dino_plan_status(g.plan.handle))


def check_transforms_in_a_row(g, fields):
  xs = [field(g, (fields,), 1.5, s) for s in (0, 1)]
  def chain(x):
    n = g.to_nodal(x)
    m = g.to_modal(n)
    return n, m, g.laplacian(m), g.to_nodal(g.d_dlon(m))
  want = []
  for x in xs:
    out = chain(x)
    torch.cuda.synchronize()
    want.append([t.clone() for t in out])
  torch.cuda.synchronize()
  got = [chain(xs[i % 2]) for i in range(8)]
  torch.cuda.synchronize()
  for i, out in enumerate(got):
    for a, b in zip(out, want[i % 2]):
      assert torch.equal(a, b)


@pytest.mark.parametrize('wavenumbers,fields', [(7, 5), (70, 30)])
def test_direct_longitude_sums_in_a_row(wavenumbers, fields):
  # 3 N + 1 longitudes: no real FFT; few and many CTAs.
  check_transforms_in_a_row(sh.Grid.with_wavenumbers(wavenumbers), fields)


def leaves(s):
  return [s.vorticity, s.divergence, s.temperature_variation, s.log_surface_pressure,
          *s.tracers.values()]


def check_in_a_row(run, states):
  """run(state) -> list of tensors: unsynchronised calls on alternating states."""
  want = []
  for s in states:
    want.append([t.clone() for t in run(s)])
    torch.cuda.synchronize()
  got = [run(states[i % 2]) for i in range(4)]
  torch.cuda.synchronize()
  for i, out in enumerate(got):
    for a, b in zip(out, want[i % 2]):
      assert torch.isfinite(a).all()
      assert torch.equal(a, b)


@pytest.mark.parametrize('form,name,layers,members,precision', [
    ('dry', 'T21', 5, 1, 'fp32'), ('dry', 'T42', 12, 6, 'fp32'), ('dry', 'TL127', 6, 1, 'fp32'),
    ('moist', 'T21', 5, 1, 'fp32'), ('moist', 'T42', 9, 6, 'fp32'),
    ('held_suarez', 'T42', 9, 6, 'fp32'), ('hybrid', 'TL127', 6, 2, 'fp32'),
    ('hybrid', 'TL127', 6, 2, 'tf32x3'), ('moist', 'TL127', 6, 2, 'bf16x3')])
def test_steps_and_gradients_in_a_row(form, name, layers, members, precision):
  g = grid_of(name, precision)
  if form == 'hybrid':
    vertical = hybrid_coordinates.HybridCoordinates.analytic_ecmwf_like(layers)
  else:
    vertical = sigma_coordinates.SigmaCoordinates.equidistant(layers)
  coords = coordinate_systems.CoordinateSystem(g, vertical)
  tref = np.linspace(220.0, 290.0, layers)
  kw = dict(humidity_key='specific_humidity') if form == 'moist' else {}
  cls = pe.PrimitiveEquationsHybrid if form == 'hybrid' else pe.PrimitiveEquationsSigma
  specs = units.SimUnits()
  eq = cls(tref, field(g, (), 2.0, 9).cpu().numpy() * 1e-4, coords, specs, **kw)
  if form == 'held_suarez':
    eq = ti.compose_equations([eq, held_suarez.HeldSuarezForcingSigma(coords, specs, tref)])
  lead = (members,) if members > 1 else ()
  def state(s):
    lnps = 0.02 * field(g, lead + (1,), 2.0, s + 3)
    lnps[..., 0, 0] += 2 * np.sqrt(np.pi) * 45.0
    tracers = {}
    if form == 'moist':
      tracers['specific_humidity'] = 1e-3 * field(g, lead + (layers,), 1.5, s + 4)
    return pe.State(0.05 * field(g, lead + (layers,), 1.0, s),
                    0.005 * field(g, lead + (layers,), 1.0, s + 1),
                    5.0 * field(g, lead + (layers,), 1.5, s + 2), lnps, tracers=tracers)
  step = ti.repeated(ti.imex_rk_sil3(eq, 0.05), 2)
  def run(s):
    if form == 'hybrid':  # no step VJP
      return leaves(step(s)) + leaves(eq.explicit_terms(s))
    xs = [x.detach().clone().requires_grad_(True) for x in leaves(s)]
    out = leaves(step(pe.State(*xs[:4], tracers=dict(zip(s.tracers, xs[4:])))))
    sum(o.square().sum() for o in out).backward()
    return leaves(step(s)) + [o.detach() for o in out] + [x.grad for x in xs]
  check_in_a_row(run, [state(10), state(20)])


@pytest.mark.parametrize('name,layers,members', [('T21', 2, 1), ('TL127', 3, 4)])
def test_shallow_water_steps_in_a_row(name, layers, members):
  g = grid_of(name, 'fp32')
  coords = coordinate_systems.CoordinateSystem(g, layer_coordinates.LayerCoordinates(layers))
  eq = shallow_water.ShallowWaterEquations(
      coords, units.SimUnits(), field(g, (), 2.0, 9).cpu().numpy() * 1e-3,
      np.linspace(0.04, 0.06, layers), densities=np.linspace(1.0, 1.5, layers))
  lead = (members, layers) if members > 1 else (layers,)
  state = lambda s: shallow_water.State(0.05 * field(g, lead, 1.0, s),
                                        0.005 * field(g, lead, 1.0, s + 1),
                                        0.005 * field(g, lead, 1.0, s + 2))
  step = ti.repeated(ti.imex_rk_sil3(eq, 0.05), 2)
  check_in_a_row(lambda s: [*vars(step(s)).values(), *vars(eq.explicit_terms(s)).values()],
                 [state(10), state(20)])
