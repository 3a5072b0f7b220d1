"""GPU: one stage's combination c0 u0 + c1 (uk + dt L) for weights and states
other than those of a Runge-Kutta step: u0 is read cell by cell, so it may be
any field, a million times larger than uk or a million times smaller.

Bound: with d = uk + dt L the sum is c0 u0 + c1 d (weights, dt, product, two
sums: 6 u of each term) or (c0 + c1) u0 + c1 ((uk - u0) + dt L), which the stage
may take where c1 |u0| is at most 2 c0 |u0|: at most 12 u of |c0 u0| + |c1 d|
with |d| taken as |uk| + |dt L|."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('u0_scale', [1e-6, 1.0, 1e6])
@pytest.mark.parametrize('c0,c1', [
    (0.0, 1.0), (1.0, 0.0), (0.75, 0.25), (1 / 3, 2 / 3), (0.1, 0.9),
    (1e-3, 1.0), (-0.5, 1.5), (2.0, -1.0)])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
def test_weighted_stage(dtype, c0, c1, u0_scale):
  from swirlc_b200 import _native as nat
  from swirlc_b200 import configs, engine
  from swirlc_b200.core import parameter
  from swirlc_b200.physics import physics_models
  cfg, state = configs.kelvin_helmholtz(n=16, nu=1e-3)
  cfg = parameter.SwirlCParameters(dict(cfg, dt=1e-3))
  uk = [torch.tensor(state[n], dtype=dtype, device='cuda')
        for n in cfg.conservative_variable_names]
  s = engine.Solver(cfg, physics_models.PhysicsModels(cfg), uk[0].shape, dtype)
  s.fill_halos(uk)
  rng = np.random.default_rng(2)
  u0 = [torch.tensor(u0_scale * rng.uniform(-1, 1, f.shape), device='cuda')
        .to(dtype) for f in uk]
  dt = 1e-3
  rhs, out = s.new_fields(), s.new_fields()
  s.stage(uk, None, rhs, nat.SWC_OUT_RHS)
  s.stage(uk, u0, out, nat.SWC_OUT_CONVEX, c0, c1, dt=s.dt_tensor(dt))
  u = float(torch.finfo(dtype).eps) / 2
  i = slice(s.hw, -s.hw)
  wide = lambda t: t.cpu().numpy()[i, i, i].astype(np.longdouble)
  for k, n in enumerate(cfg.conservative_variable_names):
    a, b, dl = wide(u0[k]), wide(uk[k]), np.longdouble(dt) * wide(rhs[k])
    want = np.longdouble(c0) * a + np.longdouble(c1) * (b + dl)
    tol = 12 * u * (abs(c0 * a) + abs(c1) * (abs(b) + abs(dl)))
    assert (np.abs(wide(out[k]) - want) <= tol).all(), n
