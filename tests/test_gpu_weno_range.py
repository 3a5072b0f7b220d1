"""GPU: WENO face values over the range of magnitudes that the square of a
smoothness indicator leaves: fields of 1e-300 to 1e75 in double precision and
of 1e-28 to 1e8 in single, the high sides of jumps included. (1 / B^2 needs
B^2 <= 1.8e308 and 3.4e38; B is at most 34 times the square of the largest
difference.) Beside a jump beyond that the candidates across it drop out.

Bounds as in tests/test_gpu_weno_jumps.py; for WENO3 beta_r = d^2 + eps is off
by 4 u of itself, a weight by 11 u, the weighted mean by 22 u and its sums by
some 10 u of the offsets: (40 size + 2 |v|) u."""

import numpy as np
import pytest
import torch

from tests import weno_reference as ref

pytestmark = pytest.mark.gpu
LINES, LENGTH = 1000, 12


@pytest.mark.parametrize('k', [3, 2])
@pytest.mark.parametrize('dtype,scale,ratio,noise', [
    (d, x, r, n) for d, xs in (
        (torch.float64, (1e-300, 1e-100, 1e-20, 1e-8, 1.0, 1e20, 1e62, 1e70,
                         1e73)),
        (torch.float32, (1e-28, 1e-8, 1.0, 1e4, 1e6)))
    for x in xs for r, n in ((1.0, 0.5), (1e2, 0.1), (1e2, 0.0))
] + [(torch.float64, 1.0, 1e80, 0.0), (torch.float64, 1e-20, 1e100, 0.0),
     (torch.float32, 1.0, 1e12, 0.0)])
def test_face_values_at_a_scale(dtype, scale, ratio, noise, k):
  from swirlc_b200.numerics import interpolation
  npd = np.float32 if dtype == torch.float32 else np.float64
  rng = np.random.default_rng(5)
  v = ref.jump_lines(rng, LINES, LENGTH, scale, ratio, noise, npd)
  neg, pos = interpolation.weno(
      torch.tensor(v.reshape(10, 100, LENGTH), device='cuda'), 'y', k)
  u = float(np.finfo(npd).eps) / 2
  face, factor = (ref.face, 450) if k == 3 else (ref.face3, 40)
  for side, got, first in (('right', neg, k), ('left', pos, k - 1)):
    got = got.cpu().numpy().reshape(LINES, LENGTH)
    for i in range(3, LENGTH - 2):
      s = [v[:, i - first + j] for j in range(2 * k - 1)]
      want, size = face(side, s)
      err = np.abs(got[:, i].astype(ref.LD) - want)
      tol = (factor * size + 2 * np.abs(s[k - 1].astype(ref.LD))) * u
      assert np.isfinite(got[:, i]).all()
      worst = (err / tol).max()
      assert worst <= 1, f'{side} face {i}: {float(worst):.3g} of the bound'
