"""GPU: the extended stage where a second tile begins along each edge of the
shapes that carry most variables (y by x: 8 x 16 in double precision, 16 x 24
in single), and WENO5 with scalars and a reference pressure together; one RK3
step against the oracle."""

import numpy as np
import pytest
import torch

from oracle import swirlc_oracle as orc
from tests import test_gpu_extensions as ext

pytestmark = pytest.mark.gpu

SCALARS = ('y', 'c', 'z2')


def _window(ns, nx, ny, nz):
  from swirlc_b200 import configs
  cfg, state = configs.kelvin_helmholtz(n=max(nx, ny, nz), nu=1e-3)
  hw = cfg['halo_width']
  for d, n in {'x': nx, 'y': ny, 'z': nz}.items():
    cfg.update({'n' + d: n, 'core_n' + d: n, d: cfg[d][:n]})
  state = {k: np.ascontiguousarray(
      v[:nz + 2 * hw, :nx + 2 * hw, :ny + 2 * hw]) for k, v in state.items()}
  return ext._with_scalars(cfg, state, SCALARS[:ns])


@pytest.mark.parametrize('ns,nx,ny,nz,dtype', [
    (3, 17, 9, 5, torch.float64), (3, 33, 23, 4, torch.float64),
    (3, 25, 17, 5, torch.float32), (3, 49, 15, 4, torch.float32)])
def test_scalars_beyond_the_first_tile(ns, nx, ny, nz, dtype):
  cfg, state = _window(ns, nx, ny, nz)
  ext._check(cfg, state, dtype)


@pytest.mark.parametrize('ns,nx,ny,nz,dtype', [
    (1, 17, 33, 5, torch.float32), (2, 25, 17, 6, torch.float32),
    (3, 33, 15, 4, torch.float32), (1, 17, 17, 5, torch.float64),
    (2, 18, 9, 5, torch.float64), (3, 33, 9, 4, torch.float64)])
def test_scalars_and_reference_pressure(ns, nx, ny, nz, dtype):
  cfg, state = _window(ns, nx, ny, nz)
  cfg = dict(cfg, numeric_flux_scheme='HLL')
  prim = orc.conservative_to_primitive(
      {k: np.asarray(state[k], np.float64) for k in orc.BASE_CONSERVATIVE})
  helper = {'p_ref': 0.9 * orc.pressure(prim, 0.0), 'rho_ref': prim['rho']}
  ext._check(cfg, state, dtype, helper)
