"""A step that swc_rk_step refuses launches nothing: neither the fields nor the
clock, which the first fill of a step moves, are touched."""

import ctypes

import pytest
import torch

from swirlc_b200 import _native as nat

N, H = 8, 3
SHAPE = (N + 2 * H,) * 3


def _call(lib, u, work, clock, bad):
  """swc_rk_step's status for one fault; u, work, clock: addresses."""
  grid = nat.SwcGrid()
  grid.nx = grid.ny = grid.nz = N
  grid.halo, grid.sx, grid.sz = H, SHAPE[2], SHAPE[1] * SHAPE[2]
  grid.dx = grid.dy = grid.dz = 0.1
  scheme = nat.SwcScheme()
  scheme.dtype, scheme.riemann = nat.dtype_code(torch.float32), 1
  bcs = (nat.SwcFieldBC * 5)()
  order, work = 3, list(work)
  if bad == 'halo':
    grid.halo = 2
    grid.nx = grid.ny = grid.nz = N + 2
  elif bad == 'interp':
    scheme.interp = 7
  elif bad == 'riemann':
    scheme.riemann = 5
  elif bad == 'scalars':
    scheme.nscalars = 1
  elif bad == 'alias':
    work[0] = u[0]
  elif bad == 'alias_last':  # RK2's second stage: w1 -> u
    order, work[4] = 2, u[4]
  elif bad == 'alias_work':  # RK3's second stage: w1 -> w2
    work[7] = work[2]
  elif bad == 'bc':
    bcs[2].side[1][0].kind = 9
  before = nat.launch_count()
  rc = lib.swc_rk_step(grid, scheme, bcs, order, nat.addr_array(u),
                       nat.addr_array(work), clock, None)
  return rc, nat.launch_count() - before


FAULTS = {'halo': ValueError, 'interp': NotImplementedError,
          'riemann': ValueError, 'scalars': NotImplementedError,
          'alias': ValueError, 'alias_last': ValueError,
          'alias_work': ValueError, 'bc': NotImplementedError}


@pytest.mark.parametrize('bad', sorted(FAULTS))
def test_refused_before_any_launch(bad):
  # The addresses are only compared.
  lib = nat.load(require_cuda=False)
  rc, launches = _call(lib, [4096 * (1 + i) for i in range(5)],
                       [4096 * (11 + i) for i in range(10)], 4096 * 31, bad)
  with pytest.raises(FAULTS[bad]):
    nat.check(rc)
  assert launches == 0


@pytest.mark.gpu
@pytest.mark.parametrize('bad', sorted(FAULTS))
def test_refused_step_leaves_clock_and_fields(bad):
  lib = nat.load()
  u = [torch.full(SHAPE, 1.0 + i, device='cuda') for i in range(5)]
  work = [torch.zeros(SHAPE, device='cuda') for _ in range(10)]
  clock = torch.tensor([0.5, 1e-3, 0.2, 0.9, 0.0, 0.0], dtype=torch.float64,
                       device='cuda')
  before = [t.clone() for t in u] + [clock.clone()]
  rc, launches = _call(lib, [t.data_ptr() for t in u],
                       [t.data_ptr() for t in work], clock.data_ptr(), bad)
  torch.cuda.synchronize()
  assert rc != 0 and launches == 0
  for a, b in zip(u + [clock], before):
    assert torch.equal(a, b)
