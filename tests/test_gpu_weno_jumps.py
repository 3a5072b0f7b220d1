"""GPU: WENO5 face values beside a strong jump are as accurate, relative to the
low side's own values, as anywhere else.

Bound (u = unit roundoff). A difference is off by u of itself, the linear parts
a_r, b_r of an indicator by 4u and 8u of the larger difference E of its
candidate, B_r = 13/3 a_r^2 + b_r^2 + 4 eps by 133 u E^2 + 3 u B_r; B_r is at
least 1.3 E^2, so B_r is off by 105 u of itself and the weight 1 / B_r^2 by
215 u. A weighted mean of offsets then moves by at most 430 u, and its sums by
some 15 u more, of the mean `size` of the offsets; the cell value and the last
sum add 2 u of themselves: (450 size + 2 |v|) u."""

import numpy as np
import pytest
import torch

from tests import weno_reference as ref

pytestmark = pytest.mark.gpu
LINES, LENGTH = 150, 14


@pytest.mark.parametrize('dim', ['x', 'y', 'z'])
@pytest.mark.parametrize('low,ratio,noise', [
    (1.0, 1.0, 0.0), (1.0, 1.0, 0.3), (1.0, 1e2, 0.01), (0.01, 1e2, 0.1),
    (0.01, 1e5, 0.0), (0.01, 1e5, 0.1), (1e-5, 1e9, 0.1)])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
def test_face_values_beside_a_jump(dtype, low, ratio, noise, dim):
  from swirlc_b200.numerics import interpolation
  npd = np.float32 if dtype == torch.float32 else np.float64
  rng = np.random.default_rng(7)
  v = ref.jump_lines(rng, LINES, LENGTH, low, ratio, noise, npd)
  a = v.reshape(10, 15, LENGTH)  # [z][x][y]
  order = {'x': (0, 2, 1), 'y': (0, 1, 2), 'z': (2, 0, 1)}[dim]
  back = tuple(np.argsort(order))
  neg, pos = interpolation.weno(
      torch.tensor(np.ascontiguousarray(a.transpose(order)), device='cuda'),
      dim, 3)
  u = float(np.finfo(npd).eps) / 2
  for side, got, first in (('right', neg, 3), ('left', pos, 2)):
    got = got.cpu().numpy().transpose(back).reshape(LINES, LENGTH)
    for i in range(3, LENGTH - 2):
      s = [v[:, i - first + k] for k in range(5)]
      want, size = ref.face(side, s)
      err = np.abs(got[:, i].astype(ref.LD) - want)
      tol = (450 * size + 2 * np.abs(s[2].astype(ref.LD))) * u
      worst = (err / tol).max()
      assert worst <= 1, f'{side} face {i}: {float(worst):.3g} of the bound'
