"""Reference states given as lists of z slices (the functional API's form) are
stacked into tensors of their own: these must live until the call that reads
them is issued, and the results must be those of the tensor form."""

import gc
import weakref

import pytest
import torch

from swirlc_b200 import _native as nat
from swirlc_b200 import engine
from swirlc_b200.common import utils

NZ, NX, NY = 8, 7, 7


def _host_solver():
  """A Solver's functional calls without a device."""
  s = object.__new__(engine.Solver)
  s.names = ['rho', 'rho_u', 'rho_v', 'rho_w', 'rho_e']
  s.shape, s.dtype, s.device = (NZ, NX, NY), torch.float32, 'cpu'
  s.ext, s.use_ext, s._layout = nat.SwcStageExt(), False, None
  s.grid, s.scheme, s._dt_cache = nat.SwcGrid(), nat.SwcScheme(), {}
  s.bcs = (nat.SwcFieldBC * 5)()
  return s


class _Lib:
  """Stands in for the library: looks at the reference states when called."""

  def __init__(self, stacked):
    self.stacked, self.calls = stacked, 0

  def _look(self, ext):
    gc.collect()
    alive = [r() for r in self.stacked]
    assert len(alive) == 2 and all(t is not None for t in alive)
    ext = getattr(ext, '_obj', ext)  # byref
    assert (ext.p_ref, ext.rho_ref) == tuple(t.data_ptr() for t in alive)
    self.calls += 1
    return 0

  def swc_rhs(self, grid, scheme, bcs, ext, *rest):
    return self._look(ext)

  def swc_rk_step_out(self, grid, scheme, bcs, ext, *rest):
    return self._look(ext)

  def swc_rk_stage_ext(self, grid, scheme, ext, *rest):
    return self._look(ext)


@pytest.mark.parametrize('call', ['rhs', 'rk2', 'rk3', 'stage'])
def test_stacked_reference_states_outlive_the_call(call, monkeypatch):
  s, stacked = _host_solver(), []

  def stack(self, helper, name):
    t = utils.as_tensor3d(helper[name])
    stacked.append(weakref.ref(t))
    return t
  lib = _Lib(stacked)
  monkeypatch.setattr(engine.Solver, '_helper_field', stack)
  monkeypatch.setattr(nat, 'load', lambda: lib)
  monkeypatch.setattr(nat, 'stream_ptr', lambda: 0)
  helper = {k: [torch.full((NX, NY), v) for _ in range(NZ)]
            for k, v in (('p_ref', 1.0), ('rho_ref', 2.0))}
  fields = [torch.ones(s.shape) for _ in s.names]
  if call == 'rhs':
    s.rhs(fields, helper)
  elif call == 'stage':
    s.stage(fields, None, [f.clone() for f in fields], nat.SWC_OUT_RHS,
            helper=helper)
  else:
    getattr(s, call)(fields, 1e-3, helper)
  assert lib.calls == 1


@pytest.mark.gpu
def test_slices_give_the_bits_of_the_tensors():
  from swirlc_b200 import configs
  from swirlc_b200.core import parameter
  from swirlc_b200.physics import physics_models
  nx, ny, nz = 40, 24, 20
  cfg, state = configs.buoyant_bubble(nx=nx, ny=ny, nz=nz)
  ref = configs.buoyant_bubble_reference_states(nx=nx, ny=ny, nz=nz)
  cfg = parameter.SwirlCParameters(dict(cfg, dt=1e-4))
  dev = lambda a: torch.tensor(a, dtype=torch.float32, device='cuda')
  fields = [dev(state[n]) for n in cfg.conservative_variable_names]
  s = engine.Solver(cfg, physics_models.PhysicsModels(cfg), fields[0].shape,
                    torch.float32)
  whole = {k: dev(v) for k, v in ref.items()}
  slices = {k: list(t.unbind(0)) for k, t in whole.items()}
  for call in (lambda h: s.rhs(fields, h), lambda h: s.rk2(fields, 1e-4, h),
               lambda h: s.rk3(fields, 1e-4, h)):
    for a, b in zip(call(slices), call(whole)):
      assert torch.equal(a, b)
  whole_loop = engine.Stepper(s, [f.clone() for f in fields], dt=1e-4,
                              helper=whole)
  slice_loop = engine.Stepper(s, [f.clone() for f in fields], dt=1e-4,
                              helper=slices)
  whole_loop.step(2)
  slice_loop.capture()
  slice_loop.step(2)
  for a, b in zip(slice_loop.u, whole_loop.u):
    assert torch.equal(a, b)
