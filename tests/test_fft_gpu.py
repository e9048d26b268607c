"""GPU longitude transforms at every real-FFT length and at tile remainders.

Every supported half length N = I / 2 (each radix schedule), with latitude
counts that fill no 16-column tile, leave an even remainder or are odd (the
scalar row path), at quadratic, linear (lw = N) and short truncations, and
odd field counts, against the FP64 oracle.  Bound: relative L2 2e-6, as the
other FP32 transform tests (FP32 Legendre sums 3e-7, FFT rounding below
log2(2560) * 6e-8 = 7e-7).
"""

import numpy as np
import pytest

from oracle import sht as osht
from oracle import states as ost

pytestmark = pytest.mark.gpu

from dinosaur_b200 import spherical_harmonic as sh  # noqa: E402

LENGTHS = (8, 16, 32, 48, 64, 96, 128, 160, 180, 256, 320, 512, 640, 1280)


def l2(a, b):
  a = a.double().cpu().numpy()
  return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize('lat', [18, 33, 48])
@pytest.mark.parametrize('n', LENGTHS)
def test_lengths(n, lat):
  # Longitude wavenumbers: up to the FFT's own limit lw = N on short rows.
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
