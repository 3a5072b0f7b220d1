"""WENO5 of the reference prototype (demo/swirl_c_prototype.ipynb `weno5`,
cell 4) on the five cells v[0..4] around v[2], as written there, in extended
precision, with the size each rounding error can have.

Both face values are a weighted mean of three candidates; `size` arrays bound
the terms a value is summed from by absolute values of its own differences, so
that size times the unit roundoff is an error relative to what lies next to the
face and not to a jump elsewhere in the stencil: a candidate across a jump J
has a weight of about J^-4 and J times that is nothing."""

import numpy as np

LD = np.longdouble
_Q = {'right': ((0, 0, 2, 5, -1), (0, -1, 5, 2, 0), (2, -7, 11, 0, 0)),
      'left': ((0, 0, 11, -7, 2), (0, 2, 5, -1, 0), (-1, 5, 2, 0, 0))}
_D = {'right': (3, 6, 1), 'left': (1, 6, 3)}
_A = ((0, 0, 1, -2, 1), (0, 1, -2, 1, 0), (1, -2, 1, 0, 0))
_B = ((0, 0, 3, -4, 1), (0, 1, 0, -1, 0), (1, -4, 3, 0, 0))


def _dot(c, v):
  return sum(LD(k) * x for k, x in zip(c, v) if k)


def _parts(v):
  """Indicators beta_r + eps, their linear parts and the candidates' sizes
  (sums of the absolute differences of a candidate's cells)."""
  v = [np.asarray(x).astype(LD) for x in v]
  d = [abs(v[k + 1] - v[k]) for k in range(4)]
  a, b = [_dot(c, v) for c in _A], [_dot(c, v) for c in _B]
  beta = [LD(13) / 12 * x * x + y * y / 4 + LD(1) / 10**6 for x, y in zip(a, b)]
  return v, a, b, beta, [d[2] + d[3], d[1] + d[2], d[0] + d[1]]


def _mean(side, v, beta, reach):
  """Normalised weights, candidate offsets from v[2], their mean, and the
  candidates' and the mean's sizes: an offset is at most 5/6 of `reach`."""
  w = [LD(k) / x**2 for k, x in zip(_D[side], beta)]
  om = [x / (w[0] + w[1] + w[2]) for x in w]
  q = [_dot(c, v) / 6 - v[2] for c in _Q[side]]
  size = [LD(5) / 6 * x for x in reach]
  return (om, q, sum(o * x for o, x in zip(om, q)), size,
          sum(o * x for o, x in zip(om, size)))


def face(side, v):
  """(value, size of its offset from v[2])."""
  v, _, _, beta, reach = _parts(v)
  _, _, mean, _, size = _mean(side, v, beta, reach)
  return v[2] + mean, size


def face3(side, v):
  """The same of WENO3 (k = 2) on the three cells around v[1]."""
  v = [np.asarray(x).astype(LD) for x in v]
  d0, dm = v[2] - v[1], v[1] - v[0]
  w = [LD(k) / (d * d + LD(1) / 10**6)**2
       for k, d in zip((2, 1) if side == 'right' else (1, 2), (d0, dm))]
  om = [x / (w[0] + w[1]) for x in w]
  off = (om[0] * d0 + om[1] * dm) / 2
  return (v[1] + (off if side == 'right' else -off),
          (om[0] * abs(d0) + om[1] * abs(dm)) / 2)


def vjp(v, right_bar, left_bar):
  """Cotangents of the five cells for those of the two face values, and the
  size of each."""
  v, a, b, beta, reach = _parts(v)
  out = [LD(0) * v[0] for _ in range(5)]
  size = [LD(0) * v[0] for _ in range(5)]
  for side, bar in (('right', right_bar), ('left', left_bar)):
    bar = np.asarray(bar).astype(LD)
    om, q, mean, qs, ms = _mean(side, v, beta, reach)
    for r in range(3):
      # d mean = sum om_r dq_r + om_r (q_r - mean) d ln(1 / beta_r^2).
      f = om[r] * (q[r] - mean) * (-2 / beta[r])
      fs = om[r] * (qs[r] + ms) * (2 / beta[r])
      for k in range(5):
        c = LD(_Q[side][r][k]) / 6
        out[k] = out[k] + bar * (om[r] * c + f * (
            LD(13) / 6 * a[r] * _A[r][k] + b[r] * _B[r][k] / 2))
        size[k] = size[k] + abs(bar) * (om[r] * abs(c) + fs * reach[r] * (
            LD(13) / 6 * abs(_A[r][k]) + LD(3) / 2 * abs(_B[r][k])))
  return out, size


def jump_lines(rng, lines, length, low, ratio, noise, dtype):
  """[lines, length] values: `low` with one jump to `low * ratio` (up or down,
  anywhere along the line), each cell disturbed by up to `noise` of itself."""
  at = rng.integers(1, length, (lines, 1))
  up = rng.integers(0, 2, (lines, 1)) == 1
  v = np.where((np.arange(length) >= at) == up, low * ratio, low)
  return (v * (1.0 + noise * rng.uniform(-1, 1, v.shape))).astype(dtype)
