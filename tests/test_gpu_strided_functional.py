"""GPU: the functional calls on fields that are windows of larger arrays
(SwcGrid strides beyond the padded extents) write the cells of their window
only, and the same values as on contiguous fields, where one pass fills the
halos and where conditions on primitives take copies and three passes."""

import numpy as np
import pytest
import torch

from tests.test_gpu_functional_calls import _setup

pytestmark = pytest.mark.gpu
GAP = 7.5  # what the surroundings hold


class _Windows:
  """n windows of a grid's shape, each with cells on all sides."""

  def __init__(self, n, shape, dtype):
    z, x, y = shape
    self.whole = [torch.full((z + 2, x + 3, y + 5), GAP, dtype=dtype,
                             device='cuda') for _ in range(n)]
    self.win = [w[1:z + 1, 2:x + 2, 3:y + 3] for w in self.whole]
    self.sx, self.sz = y + 5, (x + 3) * (y + 5)

  def untouched(self):
    for a, w in zip(self.whole, self.win):
      w.fill_(GAP)
      assert (a == GAP).all()


@pytest.mark.parametrize('kind,nx,ny,nz,dtype', [
    ('periodic', 18, 26, 5, torch.float32), ('bubble', 9, 34, 7, torch.float64),
    ('primitive', 17, 33, 4, torch.float32),
    ('primitive', 16, 5, 6, torch.float64)])
def test_windows_of_larger_arrays(kind, nx, ny, nz, dtype):
  from swirlc_b200 import _native as nat
  s, fields = _setup(kind, nx, ny, nz, dtype)
  lib, dt, nf = nat.load(), s.dt_tensor(1e-4), len(fields)
  u, out, work = (_Windows(n, s.shape, dtype) for n in (nf, nf, 2 * nf))
  for a, b in zip(u.win, fields):
    a.copy_(b)
  grid = nat.SwcGrid.from_buffer_copy(s.grid)
  grid.sx, grid.sz = u.sx, u.sz
  ptr = lambda w: nat.ptr_array(w.win)
  filled = [f.clone() for f in fields]
  s.fill_halos(filled)
  nat.check(lib.swc_halo_copy(grid, s.scheme.dtype, nf, ptr(u), ptr(out),
                              nat.ptr_array(work.win[:nf]), s.bcs, 0,
                              nat.stream_ptr()))
  inner = (slice(s.hw, -s.hw),) * 3
  for a, b, c in zip(out.win, filled, work.win):
    assert torch.equal(a, b)
    c[inner] = 0.0
    assert not c.any()
  out.untouched()
  nat.check(lib.swc_rhs(grid, s.scheme, s.bcs, None, ptr(u), ptr(out), ptr(work),
                        nat.stream_ptr()))
  for a, b in zip(out.win, s.rhs(fields)):
    assert torch.equal(a, b)
  for order, step in ((2, s.rk2), (3, s.rk3)):
    nat.check(lib.swc_rk_step_out(grid, s.scheme, s.bcs, None, order, ptr(u),
                                  ptr(out), ptr(work), dt.data_ptr(),
                                  nat.stream_ptr()))
    for a, b in zip(out.win, step(fields, 1e-4)):
      assert torch.equal(a, b), order
  for a, b in zip(u.win, fields):
    assert torch.equal(a, b)
  for w in (u, out, work):
    w.untouched()
