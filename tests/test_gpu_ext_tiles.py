"""GPU: the extended stage (transported scalars, reference states) at the
edges of its tiles: 16 cells along y, and 12, 16 or 24 along x depending on
how many variables the stage carries; one RK3 step against the oracle."""

import pytest
import torch

from tests import test_gpu_extensions as ext

pytestmark = pytest.mark.gpu

SCALARS = ('y', 'c', 'z2')


@pytest.mark.parametrize('ns,nx,ny,nz,dtype', [
    (1, 13, 17, 5, torch.float32), (2, 12, 16, 6, torch.float32),
    (2, 25, 15, 4, torch.float32), (3, 24, 33, 5, torch.float32),
    (3, 23, 4, 9, torch.float32), (1, 17, 9, 5, torch.float64),
    (2, 13, 17, 4, torch.float64), (3, 16, 8, 5, torch.float64)])
def test_scalars_on_ragged_tiles(ns, nx, ny, nz, dtype):
  import numpy as np
  from swirlc_b200 import configs
  cfg, state = configs.kelvin_helmholtz(n=max(nx, ny, nz), nu=1e-3)
  # A window of the cube: periodic in itself once its halos are refilled.
  hw = cfg['halo_width']
  sizes = {'x': nx, 'y': ny, 'z': nz}
  for d, n in sizes.items():
    cfg.update({'n' + d: n, 'core_n' + d: n, d: cfg[d][:n]})
  state = {k: np.ascontiguousarray(
      v[:nz + 2 * hw, :nx + 2 * hw, :ny + 2 * hw]) for k, v in state.items()}
  cfg, state = ext._with_scalars(cfg, state, SCALARS[:ns])
  ext._check(cfg, state, dtype)


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('ns,nx,ny,nz', [(0, 17, 15, 6), (1, 12, 33, 5),
                                         (3, 25, 16, 7)])
def test_reference_states_on_ragged_tiles(ns, nx, ny, nz, dtype):
  """float64: an input rounding (1e-16) moves the horizontal momentum, which
  is the remainder of the 1e5 Pa balance, by 2e-9 of itself; the bar allows
  some tens of those."""
  from swirlc_b200 import configs
  cfg, state = configs.buoyant_bubble(nx=nx, ny=ny, nz=nz)
  helper = configs.buoyant_bubble_reference_states(nx=nx, ny=ny, nz=nz)
  if ns:
    cfg, state = ext._with_scalars(cfg, state, SCALARS[:ns])
  ext._check(cfg, state, dtype, helper, tol64=1e-7)
