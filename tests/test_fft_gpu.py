"""GPU longitude transforms at every real-FFT length and at tile remainders.

Every supported half length N = I / 2 (each radix schedule), with latitude
counts that fill no 16-column tile, leave an even remainder or are odd (the
scalar row path), and odd field counts.  The longitude phase alone runs at the
widest truncation (lw = N) on random rows of the full spectrum, against NumPy's
FFT in 64 bits: no wavenumber is left out.  Bound: sqrt(log2(2 N)) * 6e-8 (one
rounding a level of the transform, adding up at random), 1.2e-7 to 2.0e-7.  Whole
transforms run against the FP64 oracle at up to 40 zonal wavenumbers (its cost
limits them) and at linear truncation for three lengths.  Bound: relative L2
2e-6, as the other FP32 transform tests (FP32 Legendre sums 3e-7, FFT rounding
below log2(2560) * 6e-8 = 7e-7).
"""

import numpy as np
import pytest
import torch

from oracle import sht as osht
from oracle import states as ost

pytestmark = pytest.mark.gpu

from dinosaur_b200 import _lib  # noqa: E402
from dinosaur_b200 import spherical_harmonic as sh  # noqa: E402

LENGTHS = (8, 16, 32, 48, 64, 96, 128, 160, 180, 256, 320, 512, 640, 1280)


def l2(a, b):
  a = a.double().cpu().numpy()
  return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize('lat', [18, 33, 48])
@pytest.mark.parametrize('n', LENGTHS)
def test_lengths(n, lat):
  # Longitude wavenumbers: up to the FFT's own limit lw = N on short rows, at
  # most 40 (test_full_spectrum takes the rest).
  lw = min({18: n, 33: (2 * n) // 3, 48: max(2, n // 5)}[lat], 40)
  kw = dict(longitude_wavenumbers=lw, total_wavenumbers=lw + 1,
            longitude_nodes=2 * n, latitude_nodes=lat)
  og, g = osht.Grid(**kw), sh.Grid(**kw)
  x = ost.sht_modal_input(og, 3).astype(np.float64)
  ref = og.to_nodal(x)
  assert l2(g.to_nodal(x.astype(np.float32)), ref) < 2e-6
  z = ref.astype(np.float32).astype(np.float64)
  assert l2(g.to_modal(z.astype(np.float32)), og.to_modal(z)) < 2e-6


@pytest.mark.parametrize('n', [8, 48, 180])
def test_linear_truncation(n):
  kw = dict(longitude_wavenumbers=n, total_wavenumbers=n + 1,
            longitude_nodes=2 * n, latitude_nodes=n)
  og, g = osht.Grid(**kw), sh.Grid(**kw)
  x = ost.sht_modal_input(og, 2).astype(np.float64)
  ref = og.to_nodal(x)
  assert l2(g.to_nodal(x.astype(np.float32)), ref) < 2e-6
  z = ref.astype(np.float32).astype(np.float64)
  assert l2(g.to_modal(z.astype(np.float32)), og.to_modal(z)) < 2e-6


@pytest.mark.parametrize('name', ['T31', 'TL47', 'TL95', 'T106', 'TL159', 'TL179', 'T213'])
def test_named_grids_whose_longitudes_are_no_power_of_two(name):
  g = getattr(sh.Grid, name)()
  og = osht.Grid(longitude_wavenumbers=g.longitude_wavenumbers,
                 total_wavenumbers=g.total_wavenumbers, longitude_nodes=g.longitude_nodes,
                 latitude_nodes=g.latitude_nodes)
  x = ost.sht_modal_input(og, 2).astype(np.float64)
  ref = og.to_nodal(x)
  assert l2(g.to_nodal(x.astype(np.float32)), ref) < 2e-6
  z = ref.astype(np.float32).astype(np.float64)
  assert l2(g.to_modal(z.astype(np.float32)), og.to_modal(z)) < 2e-6


def phase_errors(n, lat, fields):
  """Relative L2 errors of the inverse and the forward longitude phase alone, at
  the widest truncation (lw = N) and on random rows of the full spectrum, against
  NumPy's FFT in 64 bits."""
  g = sh.Grid(longitude_wavenumbers=n, total_wavenumbers=n + 1, longitude_nodes=2 * n,
              latitude_nodes=lat)
  rng = np.random.default_rng(n)
  def run(phase, x, rows):
    d = torch.as_tensor(x, device='cuda')
    out = torch.full((fields, rows, lat), torch.nan, device='cuda')
    _lib.check(_lib.lib().dino_sht_phase(g.plan.handle, phase, sh.ptr(d), sh.ptr(out), fields,
                                         sh.stream_handle()))
    return out
  f = rng.standard_normal((fields, 2 * n - 1, lat)).astype(np.float32)
  f64 = f.astype(np.float64)
  spectrum = np.zeros((fields, n + 1, lat), complex)
  spectrum[:, 0] = f64[:, 0] / np.sqrt(2 * np.pi)
  spectrum[:, 1:n] = (f64[:, 1::2] - 1j * f64[:, 2::2]) / (2 * np.sqrt(np.pi))
  inverse = l2(run(1, f, 2 * n), np.fft.irfft(spectrum, n=2 * n, axis=1) * 2 * n)
  x = rng.standard_normal((fields, 2 * n, lat)).astype(np.float32)
  spectrum = np.fft.rfft(x.astype(np.float64), axis=1)
  ref = np.zeros((fields, 2 * n - 1, lat))
  ref[:, 0] = spectrum[:, 0].real / np.sqrt(2 * np.pi)
  ref[:, 1::2] = spectrum[:, 1:n].real / np.sqrt(np.pi)
  ref[:, 2::2] = -spectrum[:, 1:n].imag / np.sqrt(np.pi)
  weights = (g.plan.nodes[1] * 2 * np.pi / (2 * n)).astype(np.float32)
  return inverse, l2(run(2, x, 2 * n - 1), ref * weights)


@pytest.mark.parametrize('lat', [1, 2, 33, 48])
@pytest.mark.parametrize('n', LENGTHS)
def test_full_spectrum(n, lat):
  inverse, forward = phase_errors(n, lat, 3)
  bound = np.sqrt(np.log2(2 * n)) * 6e-8
  assert inverse < bound
  assert forward < bound


# Errors (1e-8) that a twiddle product of one rounded product and one FMA leaves,
# measured with one column a thread on the inputs of phase_errors.  Two rounded
# products leave 0.7 to 1.2 % more, another order of the same sums 0.1 % more or
# less, so the bound lies half a percent above.
FMA_ERRORS = {32: (9.2037, 9.2350), 64: (9.9177, 9.8483), 128: (10.4355, 10.4931),
              256: (10.8582, 10.9540), 512: (11.5894, 11.6117)}


@pytest.mark.parametrize('n', FMA_ERRORS)
def test_twiddle_products_round_once(n):
  inverse, forward = phase_errors(n, 48, 64 if n < 64 else 8)
  assert inverse < 1.005e-8 * FMA_ERRORS[n][0]
  assert forward < 1.005e-8 * FMA_ERRORS[n][1]
