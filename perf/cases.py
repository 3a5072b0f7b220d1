"""Timed workloads of the framework, through its public entry points.

A case is a dict of plain values. `kind` names the call that is timed:

  step     core.simulation.Simulation.step on a state dict (functional step)
  loop     `steps` steps of an engine.Stepper, one step captured in a CUDA
           graph, with the device CFL clock: what core.driver runs
  rhs      the right-hand side returned by
           equations.compressible_navier_stokes.get_rhs_fn
  batch    one step of a batch.BatchStepper over many small grids
  adjoint  adjoint.simulate, a loss, and the gradients of the initial fields
           and of the viscosity

`flow` names the set-up: `shear` (periodic, developed shear layer), `tube`
(shock tube along x, outflow in x) and `bubble` (stratified atmosphere
between z walls under gravity, SI units).
"""

import math
from types import SimpleNamespace

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from swirlc_b200 import adjoint
from swirlc_b200 import batch
from swirlc_b200 import engine
from swirlc_b200.boundary import bc_types
from swirlc_b200.core import parameter
from swirlc_b200.core import simulation
from swirlc_b200.equations import compressible_navier_stokes as cns
from swirlc_b200.physics import physics_models

BC = bc_types.BoundaryCondition
NAMES = ['rho', 'rho_u', 'rho_v', 'rho_w', 'rho_e']
SCALARS = ['y', 'c', 'm']
HALO = 3
REPLICAS = np.array([[[0]]])
# Constants of the model (air, SI).
GAMMA, GRAV = 1.4, 9.81
RGAS = 8.314 / 0.029
CP = RGAS / (GAMMA - 1.0) + RGAS
P0, T0, LZ_BUBBLE = 1.0e5, 300.0, 1.0e3

DEFAULTS = {'kind': 'loop', 'flow': 'shear', 'nx': 64, 'ny': 64, 'nz': 64,
            'dtype': 'f32', 'interp': 'WENO_5', 'limiter': 'van_leer',
            'flux': 'HLLC', 'visc': True, 'scheme': 'rk3', 'steps': 1,
            'scalars': 0, 'helper': False, 'members': 0, 'every': 0}


def listed():
  return [
      # The smallest set-up of the framework, one functional step: latency,
      # launches and host work.
      dict(name='sod_256x8x8_step', kind='step', flow='tube', nx=256, ny=8,
           nz=8, visc=False),
      # The same tube in the time loop to its end time takes ~220 such steps;
      # ten of them, replayed from the graph.
      dict(name='sod_256x8x8_loop', kind='loop', flow='tube', nx=256, ny=8,
           nz=8, visc=False, steps=10),
      # A right-hand side on a small grid of odd sizes, as a user's own time
      # integrator calls it.
      dict(name='rhs_61x47x33', kind='rhs', nx=61, ny=47, nz=33, flux='HLL'),
      # The second-order integrator and the third-order scheme on a ragged
      # grid of middle size.
      dict(name='rk2_weno3_150x94x70', kind='step', nx=150, ny=94, nz=70,
           interp='WENO_3', flux='HLL', scheme='rk2'),
      # Shear layer at the size of the gradient runs, in the time loop.
      dict(name='kh_128_loop', kind='loop', nx=128, ny=128, nz=128, steps=2),
      # The headline benchmark.
      dict(name='kh_256_loop', kind='loop', nx=256, ny=256, nz=256),
      # Double precision: the runs that error figures are stated against.
      dict(name='kh_112_f64_loop', kind='loop', nx=112, ny=112, nz=112,
           dtype='f64'),
      # The largest configuration: buoyant bubble, MUSCL + HLL, gravity.
      dict(name='bubble_512x512x256_loop', kind='loop', flow='bubble', nx=512,
           ny=512, nz=256, interp='MUSCL', flux='HLL', visc=False),
      # The bubble with its hydrostatic reference states, functional step.
      dict(name='bubble_ref_128x128x96_step', kind='step', flow='bubble',
           nx=128, ny=128, nz=96, interp='MUSCL', flux='HLL', visc=False,
           helper=True),
      # Two transported scalars on a ragged grid.
      dict(name='scalars_100x84x72_step', kind='step', nx=100, ny=84, nz=72,
           scalars=2),
      # 64 quasi-1-D Riemann problems of uneven sizes advanced together.
      dict(name='riemann_batch_64', kind='batch', flow='tube', nx=4096, ny=32,
           nz=32, visc=False, members=64),
      # Gradient of a run: forward with checkpoints, loss, reverse sweep.
      dict(name='adjoint_96_4steps', kind='adjoint', nx=96, ny=96, nz=96,
           steps=4, every=2),
  ]


def draw(rng):
  """A case of the ranges that the listed ones stand for."""
  kind = rng.choice(['step', 'step', 'loop', 'loop', 'rhs', 'batch',
                     'adjoint'])
  c = {'kind': kind}
  if kind == 'batch':
    c.update(flow='tube', visc=False, members=int(2**rng.uniform(1, 6)),
             nx=int(2**rng.uniform(7, 12)), ny=rng.choice([8, 16, 32]))
    c['nz'] = c['ny']
    return c
  # A single-precision right-hand side or gradient of the bubble is rounding
  # of the hydrostatic balance: it is drawn in steps only.
  flow = rng.choice(['shear', 'shear', 'shear', 'tube', 'bubble'] if
                    kind in ('step', 'loop') else ['shear', 'shear', 'tube'] if
                    kind == 'rhs' else ['shear'])
  most = 20 if kind in ('adjoint', 'rhs') else 24
  size = 2**rng.uniform(12.5, most)
  side = size**(1 / 3)
  if flow == 'tube':
    n2 = int(2**rng.uniform(2.6, 5.2))
    c.update(nx=int(min(4096, max(48, size / 16 / n2**2))), ny=n2, nz=n2 + 1)
  else:
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    c.update(nx=max(8, int(side * a)), ny=max(8, int(side * b)),
             nz=max(8, int(side / a / b)))
  # Gradients through a limiter jump at every extremum of a rough field, where
  # rounding decides the side: those runs use WENO5.
  interp = rng.choice(['WENO_5'] if kind == 'adjoint' else
                      ['WENO_5', 'WENO_5', 'WENO_3', 'MUSCL'])
  c.update(flow=flow, interp=interp, flux=rng.choice(['HLLC', 'HLL']),
           limiter=rng.choice(['van_leer', 'mc', 'minmod']),
           visc=flow == 'shear' and rng.random() < 0.7,
           dtype='f64' if rng.random() < 0.2 else 'f32',
           scheme=rng.choice(['rk3', 'rk3', 'rk2']))
  if flow == 'bubble':
    # The helper states go with HLL: HLLC takes wave speeds from p - p_ref.
    c.update(interp='MUSCL', flux='HLL')
    c['helper'] = kind == 'step' and rng.random() < 0.5
  if kind == 'loop':
    c['steps'] = rng.randint(1, 3)
  if kind == 'step' and flow == 'shear':
    c['scalars'] = rng.choice([0, 0, 1, 2, 3])
  if kind == 'adjoint':
    c.update(steps=rng.randint(2, 5), every=rng.choice([0, 2]),
             scheme='rk3', dtype='f32')
  return c


def _full(case):
  return SimpleNamespace(**dict(DEFAULTS, **case))


def _members(c):
  """Sizes of a batch's members: uneven lengths and widths up to the case's."""
  r = np.random.default_rng(c.members * 100003 + c.nx)
  out = []
  for _ in range(c.members):
    nx = int(np.exp(r.uniform(np.log(64), np.log(c.nx))))
    nyz = int(r.choice([n for n in (4, 8, 16, 32) if n <= c.ny]))
    out.append((nx, nyz, nyz))
  return out


# ---------------------------------------------------------------- set-ups
def _centres(n, length):
  x = np.linspace(0.0, length, n + 1, dtype=np.float32)
  return (x[:-1] + 0.5 * np.diff(x)[0]).astype(np.float32)


def _lengths(c, nx, ny, nz):
  if c.flow == 'tube':
    return 1.0, ny / nx, nz / nx
  if c.flow == 'bubble':
    return LZ_BUBBLE * nx / nz, LZ_BUBBLE * ny / nz, LZ_BUBBLE
  return 1.0, 1.0, 1.0


def _mesh_z(z):
  """Cell centres along z with the solver's halo coordinates."""
  z = z.astype(np.float32)
  lo = (z[1] - z[0]) * np.linspace(-HALO, -1, HALO).astype(np.float32)
  hi = z[-1] + (z[-1] - z[-2]) * np.linspace(1, HALO, HALO).astype(np.float32)
  return np.concatenate([lo, z, hi]).astype(np.float64)


def _hydrostatic(z):
  p = P0 * np.exp(-GRAV * z / (RGAS * T0))
  return p / (RGAS * T0), p


def _setup(c, nx, ny, nz):
  """(configuration dict, boundary conditions per field as `exact` reads
  them: 'periodic', 'neumann' or [low layers, high layers])."""
  lx, ly, lz = _lengths(c, nx, ny, nz)
  x, y, z = _centres(nx, lx), _centres(ny, ly), _centres(nz, lz)
  scal = SCALARS[:c.scalars]
  names = NAMES + ['rho_' + s for s in scal]
  plain = {n: {'x': 'periodic', 'y': 'periodic', 'z': 'periodic'}
           for n in names}
  if c.flow == 'tube':
    for n in names:
      plain[n]['x'] = 'neumann'
  if c.flow == 'bubble':
    zm = _mesh_z(z)
    ends = (zm[:HALO], zm[nz + HALO:])
    for n in names:
      plain[n]['z'] = 'neumann'
    plain['rho_w']['z'] = [[0.0] * HALO] * 2
    plain['rho']['z'] = [[float(_hydrostatic(v)[0]) for v in e] for e in ends]
    plain['rho_e']['z'] = [
        [float(_hydrostatic(v)[1] / (GAMMA - 1.0) +
               _hydrostatic(v)[0] * GRAV * v) for v in e] for e in ends]

  def bc_of(b):
    if b == 'periodic':
      return {0: (BC.PERIODIC,), 1: (BC.PERIODIC,)}
    if b == 'neumann':
      return {0: (BC.NEUMANN, 0.0), 1: (BC.NEUMANN, 0.0)}
    return {s: (BC.DIRICHLET, 0.0 if not any(b[s]) else list(b[s]))
            for s in (0, 1)}

  cfg = {
      'cx': 1, 'cy': 1, 'cz': 1, 'halo_width': HALO, 'nx': nx, 'ny': ny,
      'nz': nz, 'core_nx': nx, 'core_ny': ny, 'core_nz': nz, 'lx': lx,
      'ly': ly, 'lz': lz, 'x': x, 'y': y, 'z': z,
      'dx': float(np.diff(x)[0]), 'dy': float(np.diff(y)[0]),
      'dz': float(np.diff(z)[0]), 'interpolation_scheme': c.interp,
      'muscl_limiter': c.limiter, 'numeric_flux_scheme': c.flux,
      'include_diffusion': c.visc, 'time_integration_scheme': c.scheme,
      'transport_parameters': {'nu': 1e-4, 'pr': 0.7},
      'conservative_variable_names': names,
      'primitive_variable_names': ['rho', 'u', 'v', 'w', 'e'] + scal,
      'bc': {'cell_averages': {n: {d: bc_of(b) for d, b in plain[n].items()}
                               for n in names}},
      'cfl': 0.2 if c.flow == 'bubble' else 0.5,
  }
  # A fixed step at which the functional steps run: sound speeds of about 2
  # (tube: 4), air in the bubble.
  h = min(cfg['dx'], cfg['dy'], cfg['dz'])
  cfg['dt'] = 0.2 * h / {'shear': 3.0, 'tube': 6.0, 'bubble': 360.0}[c.flow]
  if c.flow == 'bubble':
    cfg.update(g={'x': 0.0, 'y': 0.0, 'z': -1.0},
               source_functions=['gravity'])
  return cfg, plain


def _fields(c, cfg, rng, dtype, out=None):
  """Conserved fields [nz+2h, nx+2h, ny+2h] on the GPU."""
  g = torch.Generator(device='cuda').manual_seed(int(rng.integers(1 << 31)))
  kw = dict(device='cuda', dtype=torch.float32)

  def axis(v, view):
    d = float(v[1] - v[0])
    n = len(v)
    t = float(v[0]) + d * (torch.arange(-HALO, n + HALO, **kw))
    return t.view(view)

  z, x, y = (axis(cfg['z'], (-1, 1, 1)), axis(cfg['x'], (1, -1, 1)),
             axis(cfg['y'], (1, 1, -1)))
  lx, ly, lz = cfg['lx'], cfg['ly'], cfg['lz']

  def waves(amp, n=3):
    """Sum of a few separable periodic modes."""
    s = 0.0
    for _ in range(n):
      k = rng.integers(1, 4, 3)
      ph = rng.uniform(0, 2 * np.pi, 3)
      s = s + (amp / n * float(rng.uniform(0.5, 1.5))) * (
          torch.sin(2 * np.pi * int(k[0]) * x / lx + ph[0]) *
          torch.sin(2 * np.pi * int(k[1]) * y / ly + ph[1]) *
          torch.sin(2 * np.pi * int(k[2]) * z / lz + ph[2]))
    return s

  shape = (z.numel(), x.numel(), y.numel())

  def noise(amp):
    return amp * (2.0 * torch.rand(shape, generator=g, **kw) - 1.0)

  pe = 0.0
  if c.flow == 'shear':
    # Shear layers of u over y with a density contrast, rolled up by large
    # waves at Mach numbers around one, and small-scale noise.
    prof = torch.tanh(12.0 * (0.25 - torch.abs(y / ly - 0.5 + 0.03 *
                                               torch.sin(4 * np.pi * x / lx))))
    a, mean = 1.0, (0.0, 0.0, 0.0)
    if c.kind == 'adjoint':
      # Weaker, and carried by a mean flow: a gradient has jumps where a
      # contact speed changes sign (the upwind side of a face), and there any
      # rounding decides it.
      a, mean = 0.25, (0.6, 0.5, 0.4)
    rho = 1.5 + 0.5 * prof + waves(0.2) + noise(0.03)
    u = mean[0] + a * (0.8 * prof + waves(0.4)) + noise(0.03)
    v = mean[1] + a * waves(0.5) + noise(0.03)
    w = mean[2] + a * waves(0.5) + noise(0.03)
    p = 1.0 + waves(0.3) + noise(0.03)
  elif c.flow == 'tube':
    # Seeded left and right states, the diaphragm in the middle.
    s = (x < 0.5).float()
    lr = lambda a, b: s * float(rng.uniform(a, b)) + (1 - s) * float(
        rng.uniform(a, b))
    one = torch.ones(shape, **kw)
    rho, p = lr(0.2, 2.0) * one, lr(0.2, 8.0) * one
    u, v, w = lr(-0.8, 0.8) * one, lr(-0.5, 0.5) * one, lr(-0.5, 0.5) * one
  else:
    # Isothermal atmosphere with a warm bubble and a wind.
    zm = torch.as_tensor(_mesh_z(cfg['z']), device='cuda').view(-1, 1, 1)
    pe = GRAV * zm
    p = (P0 * torch.exp(-GRAV * zm / (RGAS * T0))).float()
    r2 = ((x - 0.5 * lx)**2 + (y - 0.5 * ly)**2 + (z - 0.3 * lz)**2)
    temp = T0 + 2.0 * torch.exp(-r2 / (0.2 * lz)**2) + waves(0.3)
    p = p * torch.ones_like(temp)
    rho = p / (RGAS * temp)
    u, v, w = 8.0 + waves(3.0), 5.0 + waves(3.0), waves(3.0)
  dst = out or [torch.empty(shape, device='cuda', dtype=dtype)
                for _ in NAMES]
  e = (p / ((GAMMA - 1.0) * rho)).to(torch.float64) + 0.5 * (
      u * u + v * v + w * w) + pe
  for d, val in zip(dst, (rho, rho * u, rho * v, rho * w, rho * e)):
    d.copy_(val)
  for k in range(c.scalars):
    phi = 0.5 + waves(0.4) + noise(0.02)
    dst.append((rho * phi).to(dtype).contiguous())
  return dst


def _references(cfg, shape, dtype):
  zm = torch.as_tensor(_mesh_z(cfg['z']), device='cuda').view(-1, 1, 1)
  p = P0 * torch.exp(-GRAV * zm / (RGAS * T0))
  return {'p_ref': p.to(dtype).expand(shape).contiguous(),
          'rho_ref': (p / (RGAS * T0)).to(dtype).expand(shape).contiguous()}


def _inputs(c, seed):
  """Everything `run` and `exact` start from: configuration, fields, helper
  states (and the batch's members)."""
  dtype = torch.float32 if c.dtype == 'f32' else torch.float64
  rng = np.random.default_rng(seed)
  if c.kind == 'batch':
    sizes = _members(c)
    cells = [math.prod(n + 2 * HALO for n in s) for s in sizes]
    flat = [torch.empty(sum(cells), device='cuda', dtype=dtype) for _ in NAMES]
    out, at = [], 0
    for (nx, ny, nz), n in zip(sizes, cells):
      cfg, plain = _setup(c, nx, ny, nz)
      shape = (nz + 2 * HALO, nx + 2 * HALO, ny + 2 * HALO)
      fields = [f[at:at + n].view(shape) for f in flat]
      _fields(c, cfg, rng, dtype, fields)
      out.append((cfg, plain, fields))
      at += n
    return out, flat
  cfg, plain = _setup(c, c.nx, c.ny, c.nz)
  fields = _fields(c, cfg, rng, dtype)
  helper = _references(cfg, fields[0].shape, dtype) if c.helper else {}
  return cfg, plain, fields, helper


def _observed(fields, seed):
  """What a run is compared with in data assimilation: every field, off by
  a tenth of its size."""
  g = torch.Generator(device='cuda').manual_seed(int(seed) + 77)
  out = []
  for f in fields:
    f = f.detach()
    out.append(f + 0.1 * f.square().mean().sqrt() * torch.randn(
        f.shape, generator=g, device='cuda', dtype=f.dtype))
  return out


def _misfit(fields, seen):
  inner = (slice(HALO, -HALO),) * 3
  return sum(0.5 * (f[inner] - o[inner]).square().sum()
             for f, o in zip(fields, seen))


def _dts(c, cfg):
  """Steps of a gradient run, well below the stability limit: over longer ones
  float32 rounding shows in the gradient itself (1e-4 of it in the weights'
  derivatives on smooth fields)."""
  return [0.05 * cfg['dt'] * (1.0 + 0.1 * i) for i in range(c.steps)]


# ------------------------------------------------------------------- runs
def prepare(case, seed):
  c = _full(case)
  st = SimpleNamespace(c=c)
  if c.kind == 'batch':
    members, st.flat = _inputs(c, seed)
    st.stepper = batch.BatchStepper(
        [(cfg, dict(zip(NAMES, fields))) for cfg, _, fields in members],
        st.flat[0].dtype, c.scheme)
    st.stepper.capture(c.steps)
    return st
  user_cfg, _, fields, helper = _inputs(c, seed)
  cfg = parameter.SwirlCParameters(user_cfg)
  pm = physics_models.PhysicsModels(cfg)
  st.names = list(cfg.conservative_variable_names)
  st.states, st.helper = dict(zip(st.names, fields)), helper
  if c.kind == 'step':
    st.sim = simulation.Simulation(None, cfg)
  elif c.kind == 'rhs':
    st.rhs = cns.get_rhs_fn(REPLICAS, cfg, pm)
  else:
    solver = engine.Solver(cfg, pm, fields[0].shape, fields[0].dtype)
    if c.kind == 'loop':
      st.stepper = engine.Stepper(solver, fields, cfl=cfg.cfl,
                                  scheme=c.scheme)
      st.stepper.capture()
    else:
      st.solver, st.dts = solver, _dts(c, user_cfg)
      st.runner = adjoint.RunAdjoint(solver, c.every, c.scheme, c.steps)
      st.fields = [f.requires_grad_() for f in fields]
      st.seen = _observed(fields, seed)
      st.nu = torch.tensor(1e-4, dtype=torch.float64, device='cuda',
                           requires_grad=True)
  return st


def run(state):
  c = state.c
  if c.kind == 'step':
    return state.sim.step(0, REPLICAS, 0, state.states, state.helper)
  if c.kind == 'rhs':
    return state.rhs(0, state.states, state.helper)
  if c.kind == 'loop':
    state.stepper.step(c.steps)
    return state.states
  if c.kind == 'batch':
    state.stepper.step(c.steps)
    return state.flat
  out = adjoint.simulate(state.runner, state.fields, state.dts, state.nu)
  loss = _misfit(out, state.seen)
  grads = torch.autograd.grad(loss, state.fields + [state.nu])
  # The viscosity's gradient in the precision of the fields it comes from.
  return {'fields': list(grads[:-1]), 'nu': grads[-1].to(torch.float32)}


def work(case):
  """Each step reads and writes every field once (its stages follow one
  another only through neighbouring cells, its step size through the whole
  grid); operations as the scheme needs them at the least."""
  c = _full(case)
  sizes = _members(c) if c.kind == 'batch' else [(c.nx, c.ny, c.nz)]
  cells = sum(math.prod(s) for s in sizes)
  nf = 5 + c.scalars
  esz = 4 if c.dtype == 'f32' else 8
  recon = {'WENO_5': 60, 'WENO_3': 24, 'MUSCL': 8}[c.interp]
  face = (nf + 2 + c.helper) * recon + 110 + (70 if c.visc else 0)
  stage = cells * (3 * face + 10 * nf + 25)
  stages = c.steps * (1 if c.kind == 'rhs' else 3 if c.scheme == 'rk3' else 2)
  moved = c.steps * cells * esz * (2 * nf + 2 * c.helper)
  if c.kind == 'adjoint':
    # The reverse of a step reads its state and the cotangents and writes the
    # cotangents; it costs about three times the forward operations.
    return {'bytes': moved + c.steps * cells * esz * 3 * nf,
            'flops': 4 * stages * stage}
  return {'bytes': moved, 'flops': stages * stage}


# ------------------------------------------- the same results in 64 bits
_AX = {'x': 1, 'y': 2, 'z': 0}


def _fill(f, bcs):
  """Halo fill of one field along x, y, z (a new tensor)."""
  h = HALO
  for d in ('x', 'y', 'z'):
    ax, b = _AX[d], bcs[d]
    n = f.shape[ax] - 2 * h
    mid = f.narrow(ax, h, n)
    if b == 'periodic':
      lo, hi = f.narrow(ax, n, h), f.narrow(ax, h, h)
    elif b == 'neumann':
      rep = [h if a == ax else 1 for a in range(3)]
      lo, hi = f.narrow(ax, h, 1).repeat(rep), f.narrow(ax, h + n - 1,
                                                         1).repeat(rep)
    else:
      view = [h if a == ax else 1 for a in range(3)]
      like = f.narrow(ax, 0, h)
      lo, hi = (torch.tensor(v, dtype=f.dtype, device=f.device).view(view)
                .expand_as(like) for v in b)
    f = torch.cat([lo, mid, hi], ax)
  return f


def _weno(v, ax, n, lo, k):
  """Both face values of the `n` cells from `lo` along `ax`: (right, left)."""
  s = lambda o: v.narrow(ax, lo + o, n)
  if k == 3:
    a, b, c, d, e = s(-2), s(-1), s(0), s(1), s(2)
    beta = [13 / 12 * (c - 2 * d + e)**2 + 0.25 * (3 * c - 4 * d + e)**2,
            13 / 12 * (b - 2 * c + d)**2 + 0.25 * (b - d)**2,
            13 / 12 * (a - 2 * b + c)**2 + 0.25 * (a - 4 * b + 3 * c)**2]
    qr = [(2 * c + 5 * d - e) / 6, (-b + 5 * c + 2 * d) / 6,
          (2 * a - 7 * b + 11 * c) / 6]
    ql = [(11 * c - 7 * d + 2 * e) / 6, (2 * b + 5 * c - d) / 6,
          (-a + 5 * b + 2 * c) / 6]
    dr = [0.3, 0.6, 0.1]
  else:
    b, c, d = s(-1), s(0), s(1)
    beta = [(d - c)**2, (c - b)**2]
    qr, ql = [(c + d) / 2, (3 * c - b) / 2], [(3 * c - d) / 2, (b + c) / 2]
    dr = [2 / 3, 1 / 3]
  iw = [(1e-6 + x)**-2 for x in beta]

  def side(q, dd):
    al = [w * i for w, i in zip(dd, iw)]
    return sum(x * y for x, y in zip(al, q)) / sum(al)

  return side(qr, dr), side(ql, dr[::-1])


def _muscl(v, ax, n, lo, limiter):
  s = lambda o: v.narrow(ax, lo + o, n)
  dp, dm = s(1) - s(0), s(0) - s(-1)
  zero = torch.zeros_like(dp)
  same = dp * dm > 0
  r = torch.where(same, dm, zero) / torch.where(same, dp,
                                                torch.ones_like(dp))
  if limiter == 'van_leer':
    phi = 2 * r / (1 + r)
  elif limiter == 'mc':
    phi = torch.clamp(torch.minimum(2 * r, 0.5 * (1 + r)), max=2.0)
  else:
    phi = torch.clamp(r, max=1.0)
  half = 0.5 * phi * dp
  return s(0) + half, s(0) - half


def _speeds(l, r, pl, pr, pe):
  """HLL wave speeds from Roe averages (rotated frame: u[0] is normal)."""
  cl, cr = torch.sqrt(GAMMA * pl / l.r), torch.sqrt(GAMMA * pr / r.r)
  a, b = torch.sqrt(l.r), torch.sqrt(r.r)
  inv = 1 / (a + b)
  u = [(a * x + b * y) * inv for x, y in zip(l.u, r.u)]
  hs = (a * l.h + b * r.h) * inv - 0.5 * sum(x * x for x in u) - pe
  c = torch.sqrt((GAMMA - 1.0) * hs)
  return (torch.minimum(l.u[0] - cl, u[0] - c),
          torch.maximum(r.u[0] + cr, u[0] + c))


def _physical(q, p_mom):
  m = q.r * q.u[0]
  return [m, m * q.u[0] + p_mom, m * q.u[1], m * q.u[2],
          m * (q.e + q.p / q.r)] + [m * s for s in q.s]


def _riemann(c, l, r, pdl, pdr, pe):
  """Flux in the rotated frame: rho, normal, two tangential, energy, scalars."""
  zero = torch.zeros_like(l.r)
  if c.flux == 'HLL':
    sl, sr = _speeds(l, r, l.p, r.p, pe)
    ds = sr - sl
    t1 = (torch.minimum(sr, zero) - torch.minimum(sl, zero)) / ds
    t3 = (sr * sl.abs() - sl * sr.abs()) / (2 * ds)
    cons = lambda q: [q.r] + [q.r * s for s in q.u + [q.e] + q.s]
    return [t1 * b + (1 - t1) * a - t3 * (ub - ua) for a, b, ua, ub in zip(
        _physical(l, pdl), _physical(r, pdr), cons(l), cons(r))]
  sl, sr = _speeds(l, r, pdl, pdr, pe)
  num = (pdr - pdl + l.r * l.u[0] * (sl - l.u[0]) -
         r.r * r.u[0] * (sr - r.u[0]))
  sm = num / (l.r * (sl - l.u[0]) - r.r * (sr - r.u[0]))
  sm = torch.where(sm.abs() < 1e-6, zero, sm)

  def star(q, s, f, pd):
    rat, dv = s / (s - sm), sm - q.u[0]
    return [f[0] + q.r * dv * rat,
            f[1] + q.r * s * ((s - q.u[0]) / (s - sm) * sm - q.u[0]),
            f[2] + q.r * dv * q.u[1] * rat, f[3] + q.r * dv * q.u[2] * rat,
            f[4] + q.r * rat * dv * (q.e + pd / q.r + (s - q.u[0]) * sm)
            ] + [f[5 + k] + q.r * dv * v * rat for k, v in enumerate(q.s)]

  fl, fr = _physical(l, pdl), _physical(r, pdr)
  return [torch.where(sl >= 0, a, torch.where(
      sm >= 0, b, torch.where(sr >= 0, d, e))) for a, b, d, e in zip(
          fl, star(l, sl, fl, pdl), star(r, sr, fr, pdr), fr)]


def _viscous(prim, d, h, nu):
  """Viscous flux on the faces normal to dim d: three momenta, energy."""
  ax = [_AX[k] for k in 'xyz']

  def at(q, cell, **shift):
    """q on the cells left (0) or right (1) of every face, shifted."""
    for k in range(3):
      n = q.shape[ax[k]] - 2 * HALO
      q = (q.narrow(ax[k], HALO - 1 + cell, n + 1) if k == d else
           q.narrow(ax[k], HALO + shift.get('xyz'[k], 0), n))
    return q

  def central(q, cell, k):
    s = 'xyz'[k]
    return (at(q, cell, **{s: 1}) - at(q, cell, **{s: -1})) / (2 * h[k])

  rho, vel, p = prim[0], prim[1:4], prim[5]
  both = lambda f: 0.5 * (f(0) + f(1))
  bwd = lambda q: (at(q, 1) - at(q, 0)) / h[d]
  own = [bwd(vel[k]) if k == d else both(lambda s, k=k: central(vel[k], s, k))
         for k in range(3)]
  rf = both(lambda s: at(rho, s))
  tau = []
  for k in range(3):
    s = (own[d] - sum(own) / 3 if k == d else
         0.5 * (bwd(vel[k]) + both(lambda s, k=k: central(vel[d], s, k))))
    tau.append(2 * rf * nu * s)
  q = -both(lambda s: CP / 0.7 * nu * at(rho, s)) * bwd(p / (rho * RGAS))
  work_ = sum(both(lambda s, k=k: at(vel[k], s)) * tau[k] for k in range(3))
  return [-t for t in tau] + [q - work_]


def _faces(c, cfg, prim, pe, d, nu):
  """Total flux on the faces normal to dim d, in (x, y, z) momentum order."""
  ax = _AX['xyz'[d]]
  cut = []
  for q in prim:
    for k in range(3):
      if k != d:
        a = _AX['xyz'[k]]
        q = q.narrow(a, HALO, q.shape[a] - 2 * HALO)
    cut.append(q)
  n = cut[0].shape[ax] - 2 * HALO
  if c.interp == 'MUSCL':
    both = [_muscl(q, ax, n + 2, HALO - 1, c.limiter) for q in cut]
  else:
    both = [_weno(q, ax, n + 2, HALO - 1, 3 if c.interp == 'WENO_5' else 2)
            for q in cut]
  t1, t2 = (1 if d == 0 else 0), (1 if d == 2 else 2)

  def state(side):
    v = [b[0].narrow(ax, 0, n + 1) if side == 0 else b[1].narrow(ax, 1, n + 1)
         for b in both]
    ns = c.scalars
    q = SimpleNamespace(r=v[0], u=[v[1 + d], v[1 + t1], v[1 + t2]], e=v[4],
                        p=v[5], h=v[6], s=v[7:7 + ns])
    return q, (v[7 + ns] if c.helper else q.p)

  (l, pdl), (r, pdr) = state(0), state(1)
  if c.flow == 'bubble':
    pe = pe.narrow(0, HALO, n + 1 if d == 2 else pe.shape[0] - 2 * HALO)
  f = _riemann(c, l, r, pdl, pdr, pe)
  out = [f[0], None, None, None, f[4]] + f[5:]
  out[1 + d], out[1 + t1], out[1 + t2] = f[1], f[2], f[3]
  if c.visc:
    v = _viscous(prim, d, (cfg['dx'], cfg['dy'], cfg['dz']), nu)
    for k in range(4):
      out[1 + k] = out[1 + k] + v[k]
  return out


def _rhs64(c, cfg, u, helper, nu):
  """Right-hand side on the interior for halo-filled 64-bit fields."""
  rho = u[0]
  vel = [m / rho for m in u[1:4]]
  e = u[4] / rho
  pe = 0.0
  if c.flow == 'bubble':
    pe = GRAV * torch.as_tensor(_mesh_z(cfg['z']), device=rho.device).view(
        -1, 1, 1)
  p = (GAMMA - 1.0) * rho * (e - 0.5 * sum(v * v for v in vel) - pe)
  prim = [rho] + vel + [e, p, e + p / rho] + [s / rho for s in u[5:]]
  if c.helper:
    # Zero in the halo layers, as the exchange of the helper variable sets.
    pd = torch.zeros_like(p)
    inner = (slice(HALO, -HALO),) * 3
    pd[inner] = (p - helper['p_ref'].double())[inner]
    prim.append(pd)
  inner = (slice(HALO, -HALO),) * 3
  out = [torch.zeros_like(f[inner]) for f in u]
  if c.flow == 'bubble':
    dr = rho - helper['rho_ref'].double() if c.helper else rho
    out[3] = out[3] - GRAV * dr[inner]
  for d, h in enumerate((cfg['dx'], cfg['dy'], cfg['dz'])):
    if torch.is_grad_enabled():
      f = checkpoint(_faces, c, cfg, prim, pe, d, nu, use_reentrant=False)
    else:
      f = _faces(c, cfg, prim, pe, d, nu)
    ax = _AX['xyz'[d]]
    for k, q in enumerate(f):
      n = q.shape[ax] - 1
      out[k] = out[k] - (q.narrow(ax, 1, n) - q.narrow(ax, 0, n)) / h
  return out


def _cfl64(cfg, c, u):
  inner = (slice(HALO, -HALO),) * 3
  r, a, b, w, e = (f[inner] for f in u[:5])
  pe = 0.0
  if c.flow == 'bubble':
    pe = GRAV * torch.as_tensor(_mesh_z(cfg['z']), device=r.device)[
        HALO:-HALO].view(-1, 1, 1)
  v = [a / r, b / r, w / r]
  p = (GAMMA - 1.0) * (e - 0.5 * r * sum(x * x for x in v) - r * pe)
  s = torch.sqrt(GAMMA * p / r)
  return cfg['cfl'] * min(float((h / (x.abs() + s)).min()) for x, h in zip(
      v, (cfg['dx'], cfg['dy'], cfg['dz'])))


def _pad(f, interior):
  """`f` with its interior replaced."""
  inner = (slice(HALO, -HALO),) * 3
  g = f.clone()
  g[inner] = interior
  return g


def _step64(c, cfg, plain, u, dt, helper, nu):
  """One step: (halo-filled input, interiors of the result)."""
  inner = (slice(HALO, -HALO),) * 3
  names = list(plain)
  filled = [_fill(f, plain[n]) for n, f in zip(names, u)]
  i0 = [f[inner] for f in filled]

  def euler(a):
    return [f[inner] + dt * l for f, l in zip(a, _rhs64(c, cfg, a, helper,
                                                        nu))]

  def again(i):
    return [_fill(_pad(f, x), plain[n]) for n, f, x in zip(names, filled, i)]

  i1 = euler(filled)
  if c.scheme == 'rk2':
    return filled, [0.5 * (a + b) for a, b in zip(i0, euler(again(i1)))]
  i2 = [0.75 * a + 0.25 * b for a, b in zip(i0, euler(again(i1)))]
  return filled, [a / 3 + 2 * b / 3 for a, b in zip(i0, euler(again(i2)))]


def _loop64(c, cfg, plain, u, steps):
  """In-place steps: the halos hold what the last step's fill put there."""
  dt = _cfl64(cfg, c, u)
  for _ in range(steps):
    filled, i = _step64(c, cfg, plain, u, dt, {}, 1e-4)
    u = [_pad(f, x) for f, x in zip(filled, i)]
    dt = _cfl64(cfg, c, u)
  return u


def exact(case, seed):
  c = _full(case)
  if c.kind == 'batch':
    with torch.no_grad():
      members, _ = _inputs(c, seed)
      res = [_loop64(c, cfg, plain, [f.double() for f in fields], c.steps)
             for cfg, plain, fields in members]
    return [torch.cat([m[k].reshape(-1) for m in res]) for k in range(5)]
  cfg, plain, fields, helper = _inputs(c, seed)
  names = list(plain)
  u = [f.double() for f in fields]
  if c.kind == 'adjoint':
    u = [f.requires_grad_() for f in u]
    nu = torch.tensor(1e-4, dtype=torch.float64, device='cuda',
                      requires_grad=True)
    s = u
    for dt in _dts(c, cfg):
      filled, i = _step64(c, cfg, plain, s, dt, helper, nu)
      s = [_pad(f, x) for f, x in zip(filled, i)]
    loss = _misfit(s, [f.double() for f in _observed(fields, seed)])
    grads = torch.autograd.grad(loss, u + [nu], allow_unused=True)
    return {'fields': list(grads[:-1]), 'nu':
            torch.zeros(()) if grads[-1] is None else grads[-1]}
  with torch.no_grad():
    if c.kind == 'loop':
      return dict(zip(names, _loop64(c, cfg, plain, u, c.steps)))
    if c.kind == 'rhs':
      filled = [_fill(f, plain[n]) for n, f in zip(names, u)]
      out = _rhs64(c, cfg, filled, helper, 1e-4)
      return {n: _pad(torch.zeros_like(f), x) for n, f, x in zip(
          names, filled, out)}
    filled, i = _step64(c, cfg, plain, u, cfg['dt'], helper, 1e-4)
    return {n: _fill(_pad(f, x), plain[n]) for n, f, x in zip(names, filled,
                                                               i)}
