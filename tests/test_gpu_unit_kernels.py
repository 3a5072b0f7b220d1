"""GPU: device functions by themselves (tests/native/unit_kernels.cu), against
extended precision."""

import ctypes
import os

import numpy as np
import pytest
import torch

from tests import weno_reference as ref

pytestmark = pytest.mark.gpu
LIB = os.path.join(os.path.dirname(__file__), 'native', 'libunit_kernels.so')


@pytest.fixture(scope='module')
def lib():
  return ctypes.CDLL(LIB)


def _ptr(t):
  return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize('low,ratio,noise', [
    (1.0, 1.0, 0.0), (1.0, 1.0, 0.3), (1.0, 2.0, 0.01), (1.0, 1e2, 0.01),
    (0.01, 1e2, 0.1), (0.01, 1e5, 0.0), (0.01, 1e5, 0.1), (1e-5, 1e9, 0.1)])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
def test_weno5_reverse_beside_a_jump(lib, dtype, low, ratio, noise):
  """Bound, with the forward's figures (tests/test_gpu_weno_jumps.py): the
  normalised weights are off by 430 u of themselves, the mean offset by 450 u of
  its size, 1 / B_r by 105 u and the linear parts a_r, b_r by 8 u of their
  size; sums and the products of these add some 15 u: 1000 u of the size of
  each cell's cotangent."""
  npd = np.float32 if dtype == torch.float32 else np.float64
  rng = np.random.default_rng(11)
  n = 20000
  v = np.ascontiguousarray(
      ref.jump_lines(rng, n, 5, low, ratio, noise, npd).T)
  rb, lb = (rng.normal(size=n).astype(npd) for _ in range(2))
  dv, drb, dlb = (torch.tensor(a, device='cuda') for a in (v, rb, lb))
  out = torch.empty_like(dv)
  torch.cuda.synchronize()
  assert lib.unit_weno5_vjp(n, int(dtype == torch.float64), _ptr(dv),
                            _ptr(drb), _ptr(dlb), _ptr(out)) == 0
  torch.cuda.synchronize()
  want, size = ref.vjp(v, rb, lb)
  u = float(np.finfo(npd).eps) / 2
  got = out.cpu().numpy().astype(ref.LD)
  for k in range(5):
    worst = (np.abs(got[k] - want[k]) / (1000 * u * size[k])).max()
    assert worst <= 1, f'cell {k}: {float(worst):.3g} of the bound'


def test_rcp_normal_within_one_unit(lib):
  """The reciprocal of the WENO denominators in double precision is within one
  unit in the last place of 1 / a wherever a and 1 / a are normal: random
  mantissas over all exponents, values next to powers of two, and the range of
  the denominators (weights up to 4, factors 2 to 12)."""
  rng = np.random.default_rng(3)
  n = 400000
  a = np.ldexp(rng.uniform(1, 2, n), rng.integers(-1022, 1022, n))
  powers = np.ldexp(1.0, np.arange(-1021, 1022))
  near = np.concatenate([powers + j * np.spacing(powers) for j in range(4)] +
                        [powers - j * np.spacing(powers) / 2
                         for j in range(1, 4)])
  ends = np.array([np.finfo(np.float64).tiny, 2.0**1022])
  a = np.concatenate([a, near, ends, rng.uniform(1, 80, n)])
  a *= np.where(rng.integers(0, 2, a.size) == 1, 1.0, -1.0)
  da = torch.tensor(a, device='cuda')
  out = torch.empty_like(da)
  torch.cuda.synchronize()
  assert lib.unit_rcp_normal(a.size, _ptr(da), _ptr(out)) == 0
  torch.cuda.synchronize()
  want = 1.0 / a
  off = np.abs(out.cpu().numpy().view(np.int64) - want.view(np.int64))
  assert off.max() <= 1, (off.max(), a[off.argmax()])
