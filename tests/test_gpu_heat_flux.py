"""GPU: the heat flux, whose temperatures differ little from cell to cell, is no
further off than correctly rounded quotients p / rho allow.

Bound (u = unit roundoff, k = cp nu (rho_a + rho_b) / (2 pr R h)): each quotient
is off by u of itself (1 % more for the last correction's own rounding), the
difference, the coefficient and the products by some 10 u of the result (12 in
single precision, where 1 / h is the hardware's and nu and h are rounded):
k u (1.01 (T_a + T_b) + 10 |T_b - T_a|) with T = p / rho."""

import numpy as np
import pytest
import torch

from swirlc_b200 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('contrast', [1e-6, 1e-2, 0.5])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
def test_heat_flux(dtype, contrast):
  from swirlc_b200.numerics import _pointwise
  from swirlc_b200.physics import constant
  rng = np.random.default_rng(4)
  shape, nu, pr = (24, 26, 28), 1e-2, 0.7
  h = {'dx': 1 / 26, 'dy': 0.037, 'dz': 0.3}

  class Cfg:
    dx, dy, dz = h['dx'], h['dy'], h['dz']

  npd, u, steps = ((np.float32, 2.0**-24, 12) if dtype == torch.float32 else
                   (np.float64, 2.0**-53, 10))
  rho = rng.uniform(0.5, 2.0, shape).astype(npd)
  p = (rho * (1.0 + contrast * rng.uniform(-1, 1, shape))).astype(npd)
  out = _pointwise.viscous_terms(
      nat.SWC_VISC_HEAT,
      {'rho': torch.tensor(rho, device='cuda'),
       'p': torch.tensor(p, device='cuda')}, Cfg, nu=nu, pr=pr)
  wide = np.longdouble
  r, t = rho.astype(wide), p.astype(wide) / rho.astype(wide)
  for axis, name, got in zip((1, 2, 0), ('dx', 'dy', 'dz'), out):
    cut = lambda f, s: np.take(f, range(*s), axis=axis)
    n = shape[axis]
    a, b = (0, n - 1), (1, n)
    k = (wide(constant.CP) * wide(nu) * (cut(r, a) + cut(r, b)) /
         (2 * wide(pr) * wide(constant.R) * wide(h[name])))
    want = -k * (cut(t, b) - cut(t, a))
    err = np.abs(cut(got.cpu().numpy(), b).astype(wide) - want)
    tol = k * u * (1.01 * (cut(t, a) + cut(t, b)) +
                   steps * np.abs(cut(t, b) - cut(t, a)))
    worst = (err / tol).max()
    assert worst <= 1, f'{name}: {float(worst):.3g} of the bound'
