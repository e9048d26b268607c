"""GPU parity of the shallow-water equations (dino_swe_* through the C ABI).

Against the FP64 oracle (pinned to the reference's outputs in
tests/golden/swe_T21_L2.npz): explicit / implicit terms and the implicit
inverse <= 2e-5 max-abs relative to each field's max; two filtered SIL3
steps <= 5e-5; the steady multi-layer state <= 2e-5.  The reference's own
steady geostrophic-flow test (shallow_water_test.py:100-203): mean potential
< 1e-8 and relative L2 drift < 1e-5 over 10 x 1000 steps (one layer).  With
four identical layers the steady potential of the upper three layers is
exactly zero; there the FP32 rounding of the geostrophic balance reaches the
potential through the implicit -phi_ref * divergence term with nothing to
restore it, and the drift grows linearly (measured 6.5e-7 after 1000 steps,
1.14e-5 after 10000; the FP64 oracle drifts 9e-15 over 1000 steps, so the
discretisation is exact), so that case is held to 2e-5.
"""

import os
import time

import numpy as np
import pytest
import torch

from oracle import dycore as od
from oracle import sht as osht
from oracle import swe as oswe

pytestmark = pytest.mark.gpu

from dinosaur_b200 import coordinate_systems  # noqa: E402
from dinosaur_b200 import layer_coordinates  # noqa: E402
from dinosaur_b200 import shallow_water as sw  # noqa: E402
from dinosaur_b200 import shallow_water_states as sws  # noqa: E402
from dinosaur_b200 import spherical_harmonic as sh  # noqa: E402
from dinosaur_b200 import time_integration as ti  # noqa: E402
from dinosaur_b200 import units  # noqa: E402

GOLDEN = os.path.join(os.path.dirname(__file__), 'golden')
KEYS = oswe.SWE_KEYS


def rel(a, b):
  a = a.detach().double().cpu().numpy()
  return np.abs(a - b).max() / max(np.abs(b).max(), 1e-30)


def case():
  g = np.load(os.path.join(GOLDEN, 'swe_T21_L2.npz'))
  og = osht.Grid.T21()
  grid = sh.Grid.T21()
  coords = coordinate_systems.CoordinateSystem(
      grid, layer_coordinates.LayerCoordinates(2))
  eq = sw.ShallowWaterEquations(coords, units.SimUnits(), g['orography'],
                                g['ref_potential'], densities=g['densities'])
  oeq = oswe.ShallowWaterEquations(og, od.SimUnits(), g['orography'],
                                   g['ref_potential'], g['densities'])
  st = {k: np.asarray(g[f'in_{k}'], np.float32).astype(np.float64) for k in KEYS}
  return g, og, grid, eq, oeq, st


def to_state(d):
  return sw.State(*[torch.as_tensor(d[k], device='cuda', dtype=torch.float32)
                    for k in KEYS])


def assert_close(got, ref, tol):
  for k in KEYS:
    e = rel(getattr(got, k), ref[k])
    assert e < tol, (k, e)


def test_terms_and_inverse_match_oracle():
  _, _, _, eq, oeq, st = case()
  s = to_state(st)
  assert_close(eq.explicit_terms(s), oeq.explicit_terms(st), 2e-5)
  assert_close(eq.implicit_terms(s), oeq.implicit_terms(st), 2e-6)
  for eta in (0.03, 0.2):
    assert_close(eq.implicit_inverse(s, eta), oeq.implicit_inverse(st, eta), 2e-6)


def test_filtered_sil3_steps_match_oracle():
  g, og, grid, eq, oeq, st = case()
  dt = float(g['dt'])
  step = ti.step_with_filters(ti.imex_rk_sil3(eq, dt),
                              [ti.exponential_step_filter(grid, dt)])
  ostep = oswe.filtered_step(oswe.imex_rk_sil3(oeq, dt),
                             osht.exponential_filter_scaling(og, dt / 0.010938))
  got = step(step(to_state(st)))
  ref = ostep(ostep(st))
  assert_close(got, ref, 5e-5)


def test_multi_layer_steady_state_matches_oracle():
  g, og, grid, _, _, _ = case()
  coords = coordinate_systems.CoordinateSystem(
      grid, layer_coordinates.LayerCoordinates(2))
  got = sws.multi_layer(g['u_layers'], g['densities'], coords)
  ref = oswe.multi_layer(g['u_layers'], g['densities'], og)
  assert_close(got, ref, 2e-5)


@pytest.mark.parametrize('params', [
    dict(wavenumbers=64, layers=1, velocity=lambda lat: np.cos(3 * lat) / 5,
         dt=1e-3, tol=1e-5),
    dict(wavenumbers=64, layers=4, velocity=lambda lat: np.cos(lat) / 5,
         dt=1e-3, tol=2e-5),
])
def test_reference_steady_geostrophic_flow(params):
  # shallow_water_test.py:100-203 (density ratio 0.9, mean potential 1/10,
  # 10 x 1000 filtered SIL3 steps).
  grid = sh.Grid.with_wavenumbers(params['wavenumbers'])
  layers = params['layers']
  coords = coordinate_systems.CoordinateSystem(
      grid, layer_coordinates.LayerCoordinates(layers))
  density = np.array([0.9 ** n for n in range(layers)][::-1])
  mean_potential = np.ones(layers) / 10
  dt = params['dt']
  eq = sw.ShallowWaterEquations(coords, units.SimUnits(), None, mean_potential,
                                densities=density)
  step = ti.repeated(ti.step_with_filters(
      ti.imex_rk_sil3(eq, dt), [ti.exponential_step_filter(grid, dt)]), 1000)
  lat = np.arccos(grid.cos_lat)
  velocity = np.stack([params['velocity'](lat)] * layers)
  state = sws.multi_layer(velocity, density, coords)
  init = grid.to_nodal(state.potential).double().cpu().numpy()
  init_l2 = np.sqrt(np.square(init).sum())
  w = osht.gauss_legendre_nodes(grid.latitude_nodes)[1]
  for _ in range(10):
    state = step(state)
    pot = grid.to_nodal(state.potential).double().cpu().numpy()
    mean = np.mean(w * pot / np.sum(w), axis=(-1, -2))
    assert np.all(np.abs(mean) < 1e-8), mean
    assert np.sqrt(np.square(pot - init).sum()) / init_l2 < params['tol']


@pytest.mark.parametrize('layers,members,wavenumbers', [(1, 1, 5), (3, 1, 21), (2, 3, 12)])
def test_fused_step_matches_generic_stepper(layers, members, wavenumbers):
  # The fused CUDA step against the tableau loop over the same kernels' terms:
  # both FP32, so they differ by the rounding of a few sums per stage (bound:
  # 16 roundings of 6e-8 relative to each field's maximum, three steps).
  grid = sh.Grid.with_wavenumbers(wavenumbers)
  coords = coordinate_systems.CoordinateSystem(
      grid, layer_coordinates.LayerCoordinates(layers))
  rng = np.random.default_rng(3)
  shape = (members, layers) if members > 1 else (layers,)
  _, l = np.meshgrid(*grid.modal_axes, indexing='ij')
  field = lambda a: torch.as_tensor(
      a * rng.standard_normal(shape + l.shape) * grid.mask / (l + 1.0), device='cuda',
      dtype=torch.float32)
  state = sw.State(field(0.05), field(0.005), field(0.005))
  orography = rng.standard_normal(l.shape) * grid.mask * 1e-3
  eq = sw.ShallowWaterEquations(coords, units.SimUnits(), orography,
                                np.linspace(0.04, 0.06, layers),
                                densities=np.linspace(1.0, 1.5, layers))
  dt = 0.05
  filt = ti.exponential_step_filter(grid, dt)
  fused = ti.repeated(ti.step_with_filters(ti.imex_rk_sil3(eq, dt), [filt]), 3)
  assert isinstance(fused, ti.FusedShallowWaterStep)
  generic = ti.repeated(ti.step_with_filters(
      ti.imex_runge_kutta(ti.SIL3_TABLEAU, eq, dt), [filt]), 3)
  before = state.vorticity.clone()
  got, want = fused(state), generic(state)
  assert torch.equal(state.vorticity, before)
  assert_close(got, {k: getattr(want, k).double().cpu().numpy() for k in KEYS}, 1e-6)
  # Another time step, no filter, and the first again: one capture per case.
  other = ti.imex_rk_sil3(eq, 2 * dt)(state)
  assert_close(other, {k: v.double().cpu().numpy() for k, v in vars(
      ti.imex_runge_kutta(ti.SIL3_TABLEAU, eq, 2 * dt)(state)).items()}, 1e-6)
  assert torch.equal(fused(state).potential, got.potential)


def test_fused_step_leaves_other_states_to_the_generic_stepper():
  _, _, grid, eq, _, st = case()
  step = ti.imex_rk_sil3(eq, 0.05)
  s = to_state(st)
  assert eq._fused_engine(s) is not None
  s64 = sw.State(s.vorticity.double(), s.divergence.double(), s.potential.double())
  assert eq._fused_engine(s64) is None
  assert step(s64).vorticity.dtype == torch.float64
  leaf = s.vorticity.clone().requires_grad_(True)
  assert eq._fused_engine(sw.State(leaf, s.divergence, s.potential)) is None
  with pytest.raises(ValueError):
    step(sw.State(s.vorticity[:, :-1], s.divergence[:, :-1], s.potential[:, :-1]))


def small_case(layers=2, wavenumbers=5):
  grid = sh.Grid.with_wavenumbers(wavenumbers)
  coords = coordinate_systems.CoordinateSystem(
      grid, layer_coordinates.LayerCoordinates(layers))
  rng = np.random.default_rng(11)
  _, l = np.meshgrid(*grid.modal_axes, indexing='ij')
  field = lambda a: torch.as_tensor(
      a * rng.standard_normal((layers,) + l.shape) * grid.mask / (l + 1.0), device='cuda',
      dtype=torch.float32)
  eq = sw.ShallowWaterEquations(coords, units.SimUnits(), None, np.linspace(0.04, 0.06, layers),
                                densities=np.linspace(1.0, 1.5, layers))
  return grid, eq, sw.State(field(0.05), field(0.005), field(0.005))


def test_steppers_in_turn_on_one_equation():
  # More (time step, filter) pairs than are kept, on a stream of its own and
  # without a wait in between: each gives what it gives alone.
  grid, eq, state = small_case()
  steps = []
  for i in range(11):
    dt = 0.02 + 0.005 * i
    step = ti.imex_rk_sil3(eq, dt)
    if i % 3:
      step = ti.step_with_filters(step, [ti.exponential_step_filter(grid, dt, tau=0.01 * i)])
    steps.append(step)
  want = []
  for i, step in enumerate(steps):
    out = step(state)
    torch.cuda.synchronize()
    want.append([x.clone() for x in vars(out).values()])
    ref = ti.imex_runge_kutta(ti.SIL3_TABLEAU, eq, step.dt)(state)
    for f in step.filters:
      ref = f(state, ref)
    assert_close(out, {k: v.double().cpu().numpy() for k, v in vars(ref).items()}, 1e-6)
  order = [0, 1, 0, 1, 2, 0, 3, 1] + list(range(11)) + list(range(10, -1, -1))
  stream = torch.cuda.Stream()
  stream.wait_stream(torch.cuda.current_stream())
  with torch.cuda.stream(stream):
    got = [steps[i](state) for i in order]
  torch.cuda.synchronize()
  for i, out in zip(order, got):
    for a, b in zip(vars(out).values(), want[i]):
      assert torch.equal(a, b)


def test_steppers_in_turn_cost_what_one_costs():
  # Each of a few steppers keeps its captured step: taking turns costs no
  # capture (62 us a call; 320 us when every call captures its step).
  _, eq, state = small_case()
  steps = [ti.imex_rk_sil3(eq, dt) for dt in (0.05, 0.025, -0.05)]
  def per_call(turns):
    best = np.inf
    for _ in range(5):
      torch.cuda.synchronize()
      t0 = time.perf_counter()
      for i in range(60):
        steps[i % turns](state)
      torch.cuda.synchronize()
      best = min(best, (time.perf_counter() - t0) / 60)
    return best
  per_call(3)
  one, three = per_call(1), per_call(3)
  assert three < 1.5 * one, (one, three)


def generic_stepper(eq, dt):
  return ti.imex_runge_kutta(ti.SIL3_TABLEAU, eq, dt)


@pytest.mark.parametrize('dt', [np.nan, np.inf])
def test_steppers_refuse_a_time_step_that_is_not_finite(dt):
  _, eq, state = small_case()
  for step in (generic_stepper(eq, dt), ti.imex_rk_sil3(eq, dt)):
    with pytest.raises(ValueError, match='finite'):
      step(state)


def test_repeated_takes_the_counts_that_a_loop_takes():
  _, eq, state = small_case()
  for step in (generic_stepper(eq, 0.05), ti.imex_rk_sil3(eq, 0.05)):
    assert ti.repeated(step, 0)(state) is state
    assert ti.repeated(step, -2)(state) is state
    with pytest.raises(TypeError):
      ti.repeated(step, 2.0)(state)
  two = ti.repeated(ti.imex_rk_sil3(eq, 0.05), np.int64(2))
  assert isinstance(two, ti.FusedShallowWaterStep) and two.n_steps == 2


def test_a_subclass_of_the_spectral_filter_is_called():
  grid, eq, state = small_case()

  class Halving(ti.SpectralStepFilter):

    def __call__(self, u, u_next):
      return sw.State(*[0.5 * x for x in vars(u_next).values()])

  step = ti.imex_rk_sil3(eq, 0.05)
  halved = ti.step_with_filters(step, [Halving(np.ones(grid.total_wavenumbers))])(state)
  assert torch.equal(halved.potential, 0.5 * step(state).potential)
