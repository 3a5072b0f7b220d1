// Reverse of the WENO5 cell reconstruction (recon_cell<0>, swc_physics.cuh).
#pragma once

#include "swc_physics.cuh"

namespace swc {

// On one or two variables (the lanes of O): both face values of the cell v[2]
// from v[0..4] = v[c-2 .. c+2], which share the smoothness indicators;
// vb[k] += d right/dv[k] * rb + d left/dv[k] * lb. With the forward's
// differences e and f, B_r = 13/3 a_r^2 + b_r^2 + 4 eps, w_r = 1/B_r^2 and the
// candidates' offsets R_r, L_r (times 6) of weno5_side_v, a face value is
// v0 +- c / 6 with c = sum alpha_r R_r / sum alpha_r, alpha = (w0, 2 w1, w2/3)
// on the right and (w0/3, 2 w1, w2) on the left. For g = cotangent / (6 sum
// alpha) of a face the offsets' cotangents are g alpha_r and the weights' g
// (R_r - c) times alpha_r / w_r; the differences' cotangents move onto the
// cells last. Each R_r - c is what candidate r itself adds, so a jump next to
// the cell enters with that candidate's weight only (written in third
// differences, terms of the size of the jump cancelled: 3e-2 of the cotangents
// of cells of 0.01 beside 1000 in single precision). 114 products and sums
// and 5 reciprocals per cell, against 150 with the candidates of each face
// spelled out.
template <class O>
__device__ __forceinline__ void weno5_cell_vjp_v(const typename O::V* v,
                                                 typename O::V rb,
                                                 typename O::V lb,
                                                 typename O::V* vb) {
  using S = typename O::S;
  using V = typename O::V;
  auto k = [](double c) -> V { return O::splat(S(c)); };
  const V e0 = O::sub(v[1], v[0]), e1 = O::sub(v[2], v[1]);
  const V e2 = O::sub(v[3], v[2]), e3 = O::sub(v[4], v[3]);
  // a_2, a_1, a_0 of the candidates r = 2, 1, 0.
  const V f0 = O::sub(e1, e0), f1 = O::sub(e2, e1), f2 = O::sub(e3, e2);
  const V c0 = O::mul(k(13.0 / 3.0), f0), c1 = O::mul(k(13.0 / 3.0), f1);
  const V c2 = O::mul(k(13.0 / 3.0), f2);
  const V b0 = O::fma(k(-3), e2, e3), b1 = O::add(e2, e1);
  const V b2 = O::fma(k(-3), e1, e0);
  const V eps = k(4e-6);
  const V i0 = O::rcp(O::fma(c2, f2, O::fma(b0, b0, eps)));
  const V i1 = O::rcp(O::fma(c1, f1, O::fma(b1, b1, eps)));
  const V i2 = O::rcp(O::fma(c0, f0, O::fma(b2, b2, eps)));
  const V w0 = O::mul(i0, i0), w1 = O::mul(i1, i1), w2 = O::mul(i2, i2);
  const V m1 = O::mul(k(2), w1);
  const V u0 = O::mul(k(1.0 / 3.0), w0), u2 = O::mul(k(1.0 / 3.0), w2);
  const V r0 = O::sub(O::mul(k(4), e2), e3), r1 = O::fma(k(2), e2, e1);
  const V r2 = O::fma(k(5), e1, O::mul(k(-2), e0));
  const V l2 = O::sub(O::mul(k(4), e1), e0), l1 = O::fma(k(2), e1, e2);
  const V l0 = O::fma(k(5), e2, O::mul(k(-2), e3));
  const V dr = O::rcp(O::add(O::add(w0, m1), u2));
  const V dl = O::rcp(O::add(O::add(w2, m1), u0));
  const V cr = O::mul(O::fma(u2, r2, O::fma(m1, r1, O::mul(w0, r0))), dr);
  const V cl = O::mul(O::fma(u0, l0, O::fma(m1, l1, O::mul(w2, l2))), dl);
  const V gr = O::mul(O::mul(k(1.0 / 6.0), rb), dr);
  const V gl = O::mul(O::mul(k(-1.0 / 6.0), lb), dl);
  // Cotangents of the weights (of w1 halved), then x_r = 2 dB_r = -4 w_r / B_r
  // dw_r.
  const V y0 = O::fma(O::mul(k(1.0 / 3.0), gl), O::sub(l0, cl),
                      O::mul(gr, O::sub(r0, cr)));
  const V y1 = O::fma(gl, O::sub(l1, cl), O::mul(gr, O::sub(r1, cr)));
  const V y2 = O::fma(O::mul(k(1.0 / 3.0), gr), O::sub(r2, cr),
                      O::mul(gl, O::sub(l2, cl)));
  const V x0 = O::mul(O::mul(k(-4), O::mul(w0, i0)), y0);
  const V x1 = O::mul(O::mul(k(-8), O::mul(w1, i1)), y1);
  const V x2 = O::mul(O::mul(k(-4), O::mul(w2, i2)), y2);
  // Cotangents of the second differences, of the b_r and of the offsets, then
  // of the first differences.
  const V g0 = O::mul(c0, x2), g1 = O::mul(c1, x1), g2 = O::mul(c2, x0);
  const V z0 = O::mul(b0, x0), z1 = O::mul(b1, x1), z2 = O::mul(b2, x2);
  const V p0 = O::mul(gr, w0), p1 = O::mul(gr, m1), p2 = O::mul(gr, u2);
  const V q0 = O::mul(gl, u0), q1 = O::mul(gl, m1), q2 = O::mul(gl, w2);
  const V d0 = O::fma(k(-2), p2, O::sub(O::sub(z2, g0), q2));
  const V d1 = O::add(
      O::fma(k(4), q2, O::fma(k(2), q1, O::fma(k(5), p2, p1))),
      O::add(O::fma(k(-3), z2, z1), O::sub(g0, g1)));
  const V d2 = O::add(
      O::fma(k(4), p0, O::fma(k(2), p1, O::fma(k(5), q0, q1))),
      O::add(O::fma(k(-3), z0, z1), O::sub(g1, g2)));
  const V d3 = O::fma(k(-2), q0, O::sub(O::add(z0, g2), p0));
  vb[0] = O::sub(vb[0], d0);
  vb[1] = O::add(vb[1], O::sub(d0, d1));
  vb[2] = O::add(vb[2], O::add(O::add(rb, lb), O::sub(d1, d2)));
  vb[3] = O::add(vb[3], O::sub(d2, d3));
  vb[4] = O::add(vb[4], d3);
}

}  // namespace swc
