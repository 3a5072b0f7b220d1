"""The batched step says why it refuses the 8x32 tile."""

import pytest
import torch

from swirlc_b200 import _native as nat


def test_tile_8x32_of_double_precision_weno5():
  # The addresses are only compared; nothing is launched.
  lib = nat.load(require_cuda=False)
  scheme = nat.SwcScheme()
  scheme.dtype = nat.dtype_code(torch.float64)
  scheme.interp = nat.SWC_WENO5
  m = (nat.SwcBatchMember * 1)()
  g = m[0].grid
  g.nx, g.ny, g.nz, g.halo, g.sx, g.sz = 32, 8, 8, 3, 14, 14 * 38
  g.dx = g.dy = g.dz = 0.1
  for i in range(5):
    m[0].u[i] = 4096 * (1 + i)
  for i in range(10):
    m[0].work[i] = 4096 * (10 + i)
  m[0].clock, m[0].tile = 4096 * 30, 2
  before = nat.launch_count()
  with pytest.raises(NotImplementedError) as e:
    nat.check(lib.swc_batch_step(scheme, 3, 1, m, None))
  assert nat.launch_count() == before
  assert 'double-precision WENO5' in str(e.value)
  assert 'shared memory' not in str(e.value)
