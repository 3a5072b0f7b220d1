"""GPU: the functional calls (swc_halo_copy, swc_rhs, swc_rk_step_out) give the
bits of their composition from copies, halo fills and stages, for every kind of
boundary condition, at the edges of the copy's blocks (32 cells along y, 8
rows of two cells along x), and leave the caller's fields as they are."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _setup(kind, nx, ny, nz, dtype):
  from swirlc_b200 import configs, engine
  from swirlc_b200.core import parameter
  from swirlc_b200.physics import physics_models
  if kind == 'bubble':  # Dirichlet layers and walls along z
    cfg, state = configs.buoyant_bubble(nx=nx, ny=ny, nz=nz)
  else:
    cfg, state = configs.sod(n=nx, ny=ny, nz=nz)  # Neumann along x
    cells = cfg['bc']['cell_averages']
    if kind == 'periodic':
      cells.update(configs._periodic())
    if kind == 'slope':  # Neumann increments differ between the fields
      for k, n in enumerate(cells):
        cells[n] = dict(cells[n], x={s: (cells[n]['x'][s][0], 1e-3 * (k + s))
                                     for s in (0, 1)})
    if kind == 'primitive':
      cells['u'] = cells.pop('rho_u')
  cfg = parameter.SwirlCParameters(dict(cfg, dt=1e-4))
  fields = [torch.tensor(state[n], dtype=dtype, device='cuda')
            for n in cfg.conservative_variable_names]
  return engine.Solver(cfg, physics_models.PhysicsModels(cfg),
                       fields[0].shape, dtype), fields


def _composed(s, fields, dt, order):
  from swirlc_b200 import _native as nat
  dtt = s.dt_tensor(dt)
  u0 = [f.clone() for f in fields]
  s.fill_halos(u0)
  if order == 0:
    out = s.new_fields(zero=True)
    s.stage(u0, None, out, nat.SWC_OUT_RHS)
    return out
  u1, u2 = s.new_fields(), s.new_fields()
  s.stage(u0, None, u1, nat.SWC_OUT_EULER, dt=dtt)
  s.fill_halos(u1)
  if order == 2:
    s.stage(u1, u0, u2, nat.SWC_OUT_AVERAGE, 0.5, 0.0, dt=dtt)
  else:
    s.stage(u1, u0, u2, nat.SWC_OUT_CONVEX, 0.75, 0.25, dt=dtt)
    s.fill_halos(u2)
    s.stage(u2, u0, u1, nat.SWC_OUT_CONVEX, 1 / 3, 2 / 3, dt=dtt)
    u1, u2 = u2, u1
  s.fill_halos(u2)
  return u2


@pytest.mark.parametrize('kind,nx,ny,nz,dtype', [
    ('periodic', 18, 26, 5, torch.float32), ('periodic', 19, 27, 4, torch.float64),
    ('neumann', 10, 4, 3, torch.float32), ('slope', 11, 25, 6, torch.float32),
    ('slope', 17, 5, 5, torch.float64), ('bubble', 9, 58, 7, torch.float32),
    ('bubble', 26, 3, 12, torch.float64), ('primitive', 10, 7, 4, torch.float32),
    ('neumann', 33, 2, 2, torch.float32)])
def test_functional_calls_equal_their_composition(kind, nx, ny, nz, dtype):
  from swirlc_b200 import _native as nat
  s, fields = _setup(kind, nx, ny, nz, dtype)
  keep = [f.clone() for f in fields]
  want = [f.clone() for f in fields]
  s.fill_halos(want)
  dst, clear = s.new_fields(), [torch.full_like(f, 5.0) for f in fields]
  nat.check(nat.load().swc_halo_copy(
      ctypes.byref(s.grid), s.scheme.dtype, len(fields), nat.ptr_array(fields),
      nat.ptr_array(dst), nat.ptr_array(clear), s.bcs, 0, nat.stream_ptr()))
  inner = (slice(s.hw, -s.hw),) * 3
  for a, b, c in zip(dst, want, clear):
    assert torch.equal(a, b)
    c[inner] = 0.0
    assert not c.any()
  dt = 1e-4
  calls = [(0, s.rhs), (2, lambda f: s.rk2(f, dt)), (3, lambda f: s.rk3(f, dt))]
  if min(nx, ny, nz) < s.hw:
    # A periodic dim narrower than the halo copies halo layers of the array
    # itself: of the caller's field in the first fill, but of an uninitialised
    # work state in a step's later ones.
    calls = calls[:1]
  for order, call in calls:
    for a, b in zip(call(fields), _composed(s, fields, dt, order)):
      assert torch.equal(a, b), order
  for a, b in zip(fields, keep):
    assert torch.equal(a, b)


def test_functional_calls_take_any_strides():
  s, fields = _setup('periodic', 12, 9, 6, torch.float32)
  turned = [f.permute(2, 0, 1).contiguous().permute(1, 2, 0) for f in fields]
  for a, b in zip(s.rk3(turned, 1e-4), s.rk3(fields, 1e-4)):
    assert torch.equal(a, b)


def test_clock_of_a_step_without_one_pass_fills():
  """The clock advances alike where the fills carry it and where conditions on
  a primitive take three passes and launches of its own."""
  from swirlc_b200 import engine
  for kind, scheme in (('neumann', 'rk3'), ('primitive', 'rk2')):
    s, fields = _setup(kind, 16, 8, 4, torch.float32)
    st = engine.Stepper(s, fields, cfl=0.3, t_end=1.0, scheme=scheme)
    limit = float(st.clock[2])
    st.step(1)
    c = st.clock.cpu().numpy()
    assert c[1] == 0.3 * limit and c[0] == c[1] and 0 < c[2] < 1e300
    assert st.steps_done() == 1
    first = c[2]
    st.step(1)
    c = st.clock.cpu().numpy()
    assert c[1] == 0.3 * first and np.isclose(c[0], 0.3 * (limit + first), rtol=1e-15)
