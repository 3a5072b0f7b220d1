// Device-side physics of the Swirl-C compressible RHS, shared by the fused
// stage kernel and the unit-level kernels.
//
// Each function states the reference lines it follows (paths relative to the
// swirl_c project root). Arithmetic runs in T (float or double).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace swc {

// physics/constant.py:17-41. Python doubles rounded once to T, as TF does
// when it mixes a Python float with a float32 tensor.
template <typename T>
struct K {
  static constexpr double kGamma = 1.4;
  static constexpr double kR = 8.314 / 0.029;
  static constexpr double kCv = kR / (kGamma - 1.0);
  static constexpr double kCp = kCv + kR;
  static constexpr double kG = 9.81;
  __device__ static constexpr T gamma() { return T(kGamma); }
  __device__ static constexpr T gm1() { return T(kGamma - 1.0); }
  __device__ static constexpr T r_gas() { return T(kR); }
  __device__ static constexpr T cp() { return T(kCp); }
  __device__ static constexpr T grav() { return T(kG); }
};

template <typename T>
__device__ __forceinline__ T dnn(T x, T y) {  // tf.math.divide_no_nan
  return y == T(0) ? T(0) : x / y;
}
// Single precision is built with -use_fast_math: 1/x is the hardware
// reciprocal approximation (<= 1 ulp) and x/y the 2-ulp division.
__device__ __forceinline__ float rcp_(float x) { return 1.0f / x; }
__device__ __forceinline__ double rcp_(double x) { return 1.0 / x; }
__device__ __forceinline__ float sqrt_(float x) { return sqrtf(x); }
__device__ __forceinline__ double sqrt_(double x) { return sqrt(x); }
__device__ __forceinline__ float min_(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ double min_(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ float max_(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double max_(double a, double b) { return fmax(a, b); }
__device__ __forceinline__ float abs_(float a) { return fabsf(a); }
__device__ __forceinline__ double abs_(double a) { return fabs(a); }
// Finite test on the exponent bits (unaffected by fast-math flags).
__device__ __forceinline__ bool finite_(float a) {
  return (__float_as_uint(a) & 0x7f800000u) != 0x7f800000u;
}
__device__ __forceinline__ bool finite_(double a) {
  return (static_cast<unsigned long long>(__double_as_longlong(a)) &
          0x7ff0000000000000ull) != 0x7ff0000000000000ull;
}
// CFL limit of one cell as it enters the min-reduction: delta_d/(|u_d|+c),
// or 0 when rho, p or rho_e is not finite or the limit itself is NaN
// (p/rho < 0). 0 is never a limit of a finite state, so a reduced minimum of
// 0 reports a non-finite or unphysical state to the host
// (swc_clock_status).
template <typename T>
__device__ __forceinline__ double cfl_limit_or_flag(T rho, T p, T rhoe, T l) {
  const bool ok = finite_(rho) && finite_(p) && finite_(rhoe) && (l == l);
  return ok ? double(l) : 0.0;
}

// 1/a of a normal, finite a whose reciprocal is normal too: the hardware's
// starting value x (relative error below 2^-19) and one step of Householder's
// third-order iteration, x (1 + r + r^2) with r = 1 - a x, whose remainder r^3
// is below 2^-57. About half the instructions of the correctly rounded quotient
// and no branch; the result is within one unit in the last place of it (tested
// over every exponent).
__device__ __forceinline__ double rcp_normal(double a) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(a));
  const double r = __fma_rn(-a, x, 1.0);
  return __fma_rn(__fma_rn(r, r, r), x, x);
}
// w_r = 1/b_r^2 up to a common factor, for positive b_r, without reciprocals:
// w_0 = (b_1 b_2 s)^2 and so on. The power of two s brings the largest product
// to [1, 2), so that no weight that counts leaves the normal range, however
// large or small the b_r. b_r above 2^511, whose squares overflow, count as
// 2^511. A step of KH 112^3: 1238 us; with one reciprocal per b_r 1281;
// with a fixed scale, whose products leave the normal range for fields below
// 1e-8 and above 1e62, 1193.
__device__ __forceinline__ double limit_511(double b) {
  const int hi = __double2hiint(b);
  return __hiloint2double(hi < 0x5fe00000 ? hi : 0x5fe00000, __double2loint(b));
}
// 2^-e for a product p = 2^e f, 1 <= f < 2, given by its upper word.
__device__ __forceinline__ double unit_scale(int hi) {
  return __hiloint2double(0x7fe00000 - (hi & 0x7ff00000), 0);
}
__device__ __forceinline__ void inv_squares(double b0, double b1, double b2,
                                            double& w0, double& w1,
                                            double& w2) {
  b0 = limit_511(b0);
  b1 = limit_511(b1);
  b2 = limit_511(b2);
  const double p0 = __dmul_rn(b1, b2), p1 = __dmul_rn(b0, b2);
  const double p2 = __dmul_rn(b0, b1);
  const double s = unit_scale(max(max(__double2hiint(p0), __double2hiint(p1)),
                                  __double2hiint(p2)));
  const double q0 = __dmul_rn(p0, s), q1 = __dmul_rn(p1, s);
  const double q2 = __dmul_rn(p2, s);
  w0 = __dmul_rn(q0, q0);
  w1 = __dmul_rn(q1, q1);
  w2 = __dmul_rn(q2, q2);
}
__device__ __forceinline__ void inv_squares(double b0, double b1, double& w0,
                                            double& w1) {
  b0 = limit_511(b0);
  b1 = limit_511(b1);
  const double s = unit_scale(max(__double2hiint(b0), __double2hiint(b1)));
  const double q0 = __dmul_rn(b1, s), q1 = __dmul_rn(b0, s);
  w0 = __dmul_rn(q0, q0);
  w1 = __dmul_rn(q1, q1);
}

// ---------------------------------------------------------------------------
// Lane-generic arithmetic of the fused stage. Face reconstruction
// applies the same formulas to every variable on the same stencil cells, so
// two variables share one instruction stream: Two<float> runs them as
// Blackwell f32x2 instructions (FFMA2 / FADD2 / FMUL2 issue both lanes in one
// slot), Two<double> as two scalar lanes, One<T> is a single variable. Every
// product and sum is rounded as written (no contraction), so a value comes
// out bit for bit the same whichever lane count, call site or form (face
// pair or cell-centred) computes it. Reciprocals run per lane.
// ---------------------------------------------------------------------------
template <typename T>
struct One;
template <>
struct One<float> {
  using S = float;
  using V = float;
  static __device__ __forceinline__ V splat(float a) { return a; }
  static __device__ __forceinline__ V fma(V a, V b, V c) { return __fmaf_rn(a, b, c); }
  static __device__ __forceinline__ V mul(V a, V b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ V add(V a, V b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ V rcp(V a) { return 1.0f / a; }
  // 1/a for a normal, nonzero, finite a.
  static __device__ __forceinline__ V rcpn(V a) { return 1.0f / a; }
  // a / b as a times the reciprocal of b (what the fast-math quotient is).
  static __device__ __forceinline__ V div(V a, V b) { return __fmul_rn(a, 1.0f / b); }
  // a / b with rb = rcp(b) at hand: the product a rb is off by 2 units of
  // roundoff and more; its remainder, exact in an FMA, leaves one.
  static __device__ __forceinline__ V quot(V a, V b, V rb) {
    const V q = __fmul_rn(a, rb);
    return __fmaf_rn(__fmaf_rn(-q, b, a), rb, q);
  }
  // x where p > 0, else 0.
  static __device__ __forceinline__ V sel_pos(V p, V x) { return p > 0.0f ? x : 0.0f; }
  template <class F>
  static __device__ __forceinline__ V map3(F f, V a, V b, V c) { return f(a, b, c); }
};
template <>
struct One<double> {
  using S = double;
  using V = double;
  static __device__ __forceinline__ V splat(double a) { return a; }
  static __device__ __forceinline__ V fma(V a, V b, V c) { return __fma_rn(a, b, c); }
  static __device__ __forceinline__ V mul(V a, V b) { return __dmul_rn(a, b); }
  static __device__ __forceinline__ V add(V a, V b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return __dsub_rn(a, b); }
  static __device__ __forceinline__ V rcp(V a) { return 1.0 / a; }
  static __device__ __forceinline__ V rcpn(V a) { return rcp_normal(a); }
  static __device__ __forceinline__ V div(V a, V b) { return __ddiv_rn(a, b); }
  static __device__ __forceinline__ V quot(V a, V b, V rb) {
    const V q = __dmul_rn(a, rb);
    return __fma_rn(__fma_rn(-q, b, a), rb, q);
  }
  static __device__ __forceinline__ V sel_pos(V p, V x) { return p > 0.0 ? x : 0.0; }
  template <class F>
  static __device__ __forceinline__ V map3(F f, V a, V b, V c) { return f(a, b, c); }
};
template <typename T>
struct Two;
template <>
struct Two<float> {
  using S = float;
  using V = float2;
  static __device__ __forceinline__ V mk(float a, float b) { return make_float2(a, b); }
  static __device__ __forceinline__ V splat(float a) { return make_float2(a, a); }
  static __device__ __forceinline__ V fma(V a, V b, V c) { return __ffma2_rn(a, b, c); }
  static __device__ __forceinline__ V mul(V a, V b) { return __fmul2_rn(a, b); }
  static __device__ __forceinline__ V add(V a, V b) { return __fadd2_rn(a, b); }
  // a - b, rounded once (b * -1 is exact).
  static __device__ __forceinline__ V sub(V a, V b) { return __ffma2_rn(b, splat(-1.0f), a); }
  static __device__ __forceinline__ V rcp(V a) { return make_float2(1.0f / a.x, 1.0f / a.y); }
  static __device__ __forceinline__ V rcpn(V a) { return rcp(a); }
  static __device__ __forceinline__ V div(V a, V b) { return __fmul2_rn(a, rcp(b)); }
  static __device__ __forceinline__ V sel_pos(V p, V x) {
    return make_float2(p.x > 0.0f ? x.x : 0.0f, p.y > 0.0f ? x.y : 0.0f);
  }
  template <class F>
  static __device__ __forceinline__ V map3(F f, V a, V b, V c) {
    return make_float2(f(a.x, b.x, c.x), f(a.y, b.y, c.y));
  }
};
template <>
struct Two<double> {
  using S = double;
  using V = double2;
  static __device__ __forceinline__ V mk(double a, double b) { return make_double2(a, b); }
  static __device__ __forceinline__ V splat(double a) { return make_double2(a, a); }
  static __device__ __forceinline__ V fma(V a, V b, V c) {
    return make_double2(__fma_rn(a.x, b.x, c.x), __fma_rn(a.y, b.y, c.y));
  }
  static __device__ __forceinline__ V mul(V a, V b) {
    return make_double2(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y));
  }
  static __device__ __forceinline__ V add(V a, V b) {
    return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y));
  }
  static __device__ __forceinline__ V sub(V a, V b) {
    return make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y));
  }
  static __device__ __forceinline__ V rcp(V a) { return make_double2(1.0 / a.x, 1.0 / a.y); }
  static __device__ __forceinline__ V rcpn(V a) {
    return make_double2(rcp_normal(a.x), rcp_normal(a.y));
  }
  static __device__ __forceinline__ V div(V a, V b) {
    return make_double2(__ddiv_rn(a.x, b.x), __ddiv_rn(a.y, b.y));
  }
  static __device__ __forceinline__ V sel_pos(V p, V x) {
    return make_double2(p.x > 0.0 ? x.x : 0.0, p.y > 0.0 ? x.y : 0.0);
  }
  template <class F>
  static __device__ __forceinline__ V map3(F f, V a, V b, V c) {
    return make_double2(f(a.x, b.x, c.x), f(a.y, b.y, c.y));
  }
};

// Primitive state at a face or a cell: rho, (u, v, w), e, p, h.
template <typename T>
struct Prim {
  T r;
  T u[3];
  T e, p, h;
};

// Cell primitives from conserved values (utils.py:145-183 multiplies by the
// reciprocal of rho) and p, h (generic.py:27-87, 356-388).
// p / rho = (gamma - 1) e_int, so h needs no division of its own.
template <typename T>
__device__ __forceinline__ void cons_to_prim(T rho, T ru, T rv, T rw, T re,
                                             T pe, T& u, T& v, T& w, T& e,
                                             T& p, T& h) {
  using O = One<T>;
  const T inv = O::rcp(rho);
  u = O::mul(inv, ru);
  v = O::mul(inv, rv);
  w = O::mul(inv, rw);
  e = O::mul(inv, re);
  const T q2 = O::fma(w, w, O::fma(v, v, O::mul(u, u)));
  const T eint = O::sub(O::fma(T(-0.5), q2, e), pe);
  p = O::mul(O::mul(K<T>::gm1(), rho), eint);
  h = O::fma(K<T>::gm1(), eint, e);
}

// ---------------------------------------------------------------------------
// Face reconstruction. A stencil s[0 .. LO+RI-1] holds the cell values
// v[i-LO .. i+RI-1] around face i-1/2; neg comes from the left cell i-1,
// pos from the right cell i (compressible_navier_stokes.py:597-615).
// WENO-JS weights alpha_r = d_r / (eps + beta_r)^2 with eps = 1e-6 and the
// candidate polynomials of the reference prototype
// (demo/swirl_c_prototype.ipynb `weno5`, cell 4).
// ---------------------------------------------------------------------------
template <int SCHEME>
struct Stencil;

template <>
struct Stencil<0> {  // WENO5
  static constexpr int LO = 3, RI = 3;
};
template <>
struct Stencil<1> {  // WENO3
  static constexpr int LO = 2, RI = 2;
};
template <>
struct Stencil<2> {  // MUSCL
  static constexpr int LO = 2, RI = 2;
};
template <>
struct Stencil<3> {  // NODE (identity)
  static constexpr int LO = 0, RI = 1;
};

// MUSCL slope of cell c for the monotonized-central (1) and minmod (2)
// limiters: phi(r) * dp with r = dnn(dm, dp); or (limiter 3) the reference
// prototype's slope (demo/swirl_c_prototype.ipynb `muscl`, cell 4): minmod
// of the central difference (v[c+1] - v[c-1]) / 4, the forward and the
// backward difference, i.e. the smallest magnitude of the three where all
// three have the same sign, else 0. The van Leer limiter (0) is formed lane
// by lane in muscl_slope_v.
template <typename T>
__device__ __forceinline__ T muscl_slope(T vm1, T v0, T vp1, int limiter) {
  T dp = vp1 - v0, dm = v0 - vm1;
  if (limiter == 3) {
    const T c2 = (vp1 - vm1) * T(0.25);
    const T m = min_(min_(abs_(c2), abs_(dp)), abs_(dm));
    const bool up = c2 > T(0) && dp > T(0) && dm > T(0);
    const bool down = c2 < T(0) && dp < T(0) && dm < T(0);
    return up ? m : (down ? -m : T(0));
  }
  T r = dnn(dm, dp);
  T phi;
  if (limiter == 1) {  // monotonized central
    phi = max_(T(0), min_(min_(T(2) * r, T(0.5) * (T(1) + r)), T(2)));
  } else {  // minmod
    phi = max_(T(0), min_(r, T(1)));
  }
  return phi * dp;
}

// ---------------------------------------------------------------------------
// Cell-centred reconstruction: both face values of one cell c from its
// stencil s[0 .. CL+CR] = v[c-CL .. c+CR]. `right` is the neg value of face
// c+1/2, `left` the pos value of face c-1/2. For WENO the smoothness
// indicators and the reciprocals 1/(eps+beta_r)^2 are shared by both sides.
// NODE keeps the identity mock's convention (face i-1/2 takes v[i] on both
// sides), i.e. right(c) = v[c+1], left(c) = v[c].
// ---------------------------------------------------------------------------
template <int SCHEME>
struct CellStencil;
template <>
struct CellStencil<0> {
  static constexpr int CL = 2, CR = 2;
};
template <>
struct CellStencil<1> {
  static constexpr int CL = 1, CR = 1;
};
template <>
struct CellStencil<2> {
  static constexpr int CL = 1, CR = 1;
};
template <>
struct CellStencil<3> {
  static constexpr int CL = 0, CR = 1;
};

// WENO5-JS on the cell stencil v[c-2..c+2]: alpha_r = d_r / (eps + beta_r)^2
// with eps = 1e-6, the smoothness indicators
// beta_r = 13/12 a_r^2 + 1/4 b_r^2 and the candidate polynomials q_r of the
// reference prototype's `weno5`; the value is sum alpha_r q_r / sum alpha_r.
// It is evaluated as v0 plus the weighted mean of the candidates' offsets
// q_r - v0, each written in the first differences e_k = v[k+1] - v[k] of its
// own three cells (dm2, dm1, d0, d1 around the cell; weights
// w_r = 1/beta_r^2 up to a common factor; d = (0.3, 0.6, 0.1) and mirrored):
//   right (c+1/2): v0 + (w0 (4 d0 - d1) + 2 w1 (dm1 + 2 d0)
//                        + w2 (5 dm1 - 2 dm2) / 3) / (6 w0 + 12 w1 + 2 w2)
//   left  (c-1/2): v0 - (w2 (4 dm1 - dm2) + 2 w1 (d0 + 2 dm1)
//                        + w0 (5 d0 - 2 d1) / 3) / (2 w0 + 12 w1 + 6 w2)
// A candidate whose cells hold a jump J enters with J times its weight of
// about J^-4 only, so a face value is accurate to a few units in the last
// place of what lies on its own side. (The shorter form of a central candidate
// and a correction in third differences has two terms of size J that cancel:
// 2e-4 of a low side of 0.01 beside 1000 in single precision.) A uniform
// field comes out unrounded. The differences are shared: by the two faces of
// a cell and, in the face form, by the two cells.
// B_r = 4 (beta_r + eps) = 13/3 a_r^2 + (b_r^2 + 4 eps), so eps folds into an
// FMA; a_r is the second difference e_hi - e_lo of candidate r's three cells,
// b_r = e_hi - 3 e_lo (r = 0), e_lo + e_hi (r = 1), e_lo - 3 e_hi (r = 2) up
// to sign.
// w_r = 1/B_r^2: by the hardware reciprocal in single precision, up to a common
// factor in double (inv_squares). Jumps reach up to 2e9 and 1e76.
template <class O>
struct Weno5Tri {  // second difference a of three cells and 13/3 a
  typename O::V a, ca;
};
template <class O>
__device__ __forceinline__ Weno5Tri<O> weno5_tri(typename O::V e_lo,
                                                 typename O::V e_hi) {
  using S = typename O::S;
  const typename O::V a = O::sub(e_hi, e_lo);
  return {a, O::mul(O::splat(S(13.0 / 3.0)), a)};
}
// 4 (beta + eps) = 13/3 a^2 + (b^2 + 4 eps).
template <class O>
__device__ __forceinline__ typename O::V weno5_b4(const Weno5Tri<O>& t,
                                                  typename O::V b) {
  using S = typename O::S;
  return O::fma(t.ca, t.a, O::fma(b, b, O::splat(S(4e-6))));
}
template <class O>
struct Weno5W {
  typename O::V w0, w1, w2;
};
// Cell with the differences dm2 = v[c-1]-v[c-2], dm1 = v[c]-v[c-1],
// d0 = v[c+1]-v[c], d1 = v[c+2]-v[c+1] and the second differences
// t2 = (dm2, dm1), t1 = (dm1, d0), t0 = (d0, d1).
template <class O>
__device__ __forceinline__ Weno5W<O> weno5_weights(
    const Weno5Tri<O>& t2, const Weno5Tri<O>& t1, const Weno5Tri<O>& t0,
    typename O::V dm2, typename O::V dm1, typename O::V d0,
    typename O::V d1) {
  using S = typename O::S;
  using V = typename O::V;
  const V m3 = O::splat(S(-3));
  const V b0 = weno5_b4<O>(t0, O::fma(m3, d0, d1));
  const V b1 = weno5_b4<O>(t1, O::add(d0, dm1));
  const V b2 = weno5_b4<O>(t2, O::fma(m3, dm1, dm2));
  Weno5W<O> w;
  if constexpr (std::is_same<V, double>::value) {
    inv_squares(b0, b1, b2, w.w0, w.w1, w.w2);
  } else if constexpr (std::is_same<V, double2>::value) {
    inv_squares(b0.x, b1.x, b2.x, w.w0.x, w.w1.x, w.w2.x);
    inv_squares(b0.y, b1.y, b2.y, w.w0.y, w.w1.y, w.w2.y);
  } else {
    w = {O::rcp(O::mul(b0, b0)), O::rcp(O::mul(b1, b1)),
         O::rcp(O::mul(b2, b2))};
  }
  return w;
}
// The face value on one side of a cell: wn, wf are the weights of the
// candidates that reach farthest towards the face and away from it; dn, dn1
// (df, df1) the first and second of the differences on those two sides.
// RIGHT: w0, w2, d0, d1, dm1, dm2; left: w2, w0, dm1, dm2, d0, d1. The mean
// offset is formed with both signs turned on the right (FMAs of two lanes
// have no negated operand).
template <class O, bool RIGHT>
__device__ __forceinline__ typename O::V weno5_side_v(
    typename O::V wn, typename O::V w1, typename O::V wf, typename O::V v0,
    typename O::V dn, typename O::V dn1, typename O::V df,
    typename O::V df1) {
  using S = typename O::S;
  using V = typename O::V;
  const V on = O::fma(O::splat(S(-4)), dn, dn1);
  const V o1 = O::fma(O::splat(S(2)), dn, df);
  const V of = O::fma(O::splat(S(-2.5)), df, df1);
  const V m1 = O::mul(O::splat(S(-2)), w1);
  const V mf = O::mul(O::splat(S(2.0 / 3.0)), wf);
  const V num = O::fma(mf, of, O::fma(m1, o1, O::mul(wn, on)));
  const S s = RIGHT ? S(-1) : S(1);
  const V den = O::fma(O::splat(s * S(2)), wf,
                       O::fma(O::splat(s * S(12)), w1,
                              O::mul(O::splat(s * S(6)), wn)));
  return O::fma(num, O::rcpn(den), v0);
}
template <class O>
__device__ __forceinline__ typename O::V weno5_right_v(
    const Weno5W<O>& w, typename O::V v0, typename O::V dm2,
    typename O::V dm1, typename O::V d0, typename O::V d1) {
  return weno5_side_v<O, true>(w.w0, w.w1, w.w2, v0, d0, d1, dm1, dm2);
}
template <class O>
__device__ __forceinline__ typename O::V weno5_left_v(
    const Weno5W<O>& w, typename O::V v0, typename O::V dm2,
    typename O::V dm1, typename O::V d0, typename O::V d1) {
  return weno5_side_v<O, false>(w.w2, w.w1, w.w0, v0, dm1, dm2, d0, d1);
}

// WENO3 (k = 2) on v[c-1..c+1], d0 = v[c+1]-v[c], dm = v[c]-v[c-1]: weights
// w_r = 1/(eps + beta_r)^2 up to a common factor with beta = (d0^2, dm^2);
// right face (d = (2/3, 1/3), candidates v0 + d0/2 and v0 + dm/2):
// v0 + (w0 d0 + w1 dm / 2) / (2 w0 + w1); left face (d mirrored, candidates
// v0 - d0/2 and v0 - dm/2): v0 - (w0 d0 / 2 + w1 dm) / (w0 + 2 w1).
template <class O>
__device__ __forceinline__ void weno3_weights(typename O::V d0,
                                              typename O::V dm,
                                              typename O::V& w0,
                                              typename O::V& w1) {
  using S = typename O::S;
  using V = typename O::V;
  const V eps = O::splat(S(1e-6));
  const V b0 = O::fma(d0, d0, eps), b1 = O::fma(dm, dm, eps);
  if constexpr (std::is_same<V, double>::value) {
    inv_squares(b0, b1, w0, w1);
  } else if constexpr (std::is_same<V, double2>::value) {
    inv_squares(b0.x, b1.x, w0.x, w1.x);
    inv_squares(b0.y, b1.y, w0.y, w1.y);
  } else {
    w0 = O::rcp(O::mul(b0, b0));
    w1 = O::rcp(O::mul(b1, b1));
  }
}
template <class O>
__device__ __forceinline__ typename O::V weno3_side_v(
    typename O::V w0, typename O::V w1, typename O::V v0, typename O::V d0,
    typename O::V dm, bool right) {
  using S = typename O::S;
  using V = typename O::V;
  const V a = O::mul(w0, d0), b = O::mul(w1, dm);
  const V half = O::splat(S(0.5));
  // The left denominator is negated (the correction is subtracted).
  const V num = right ? O::fma(half, b, a) : O::fma(half, a, b);
  const V den = right ? O::fma(O::splat(S(2)), w0, w1)
                      : O::fma(O::splat(S(-2)), w1, O::mul(O::splat(S(-1)), w0));
  return O::fma(num, O::rcpn(den), v0);
}

// MUSCL slopes per lane (muscl_slope).
template <class O>
__device__ __forceinline__ typename O::V muscl_slope_v(typename O::V vm1,
                                                       typename O::V v0,
                                                       typename O::V vp1,
                                                       int limiter) {
  using S = typename O::S;
  if (limiter == 0) {
    // van Leer: phi(r) dp = (r + |r|) / (1 + |r|) dp with r = dm / dp is, in
    // exact arithmetic, the harmonic mean 2 dm dp / (dm + dp) where dm and
    // dp have the same sign (dm dp > 0) and 0 elsewhere (dp = 0 or dm = 0
    // included, as divide_no_nan gives r = 0 there). It is formed as
    // 2 dm * (dp / (dm + dp)): one quotient instead of two, no ratio r and
    // no product that can overflow (dp / (dm + dp) lies in (0, 1]), so
    // extreme ratios beside subnormal values (double precision keeps them)
    // need no special case; every lane op is a paired one where O pairs.
    const typename O::V dp = O::sub(vp1, v0), dm = O::sub(v0, vm1);
    const typename O::V q = O::div(dp, O::add(dm, dp));
    return O::sel_pos(O::mul(dm, dp), O::mul(O::add(dm, dm), q));
  }
  return O::map3([limiter](S a, S b, S c) { return muscl_slope(a, b, c, limiter); },
                 vm1, v0, vp1);
}

// Face i-1/2 from s[k] = v[i-LO+k] (Stencil<SCHEME>): neg from cell i-1
// (its right face), pos from cell i (its left face).
template <int SCHEME, class O>
__device__ __forceinline__ void recon_face(const typename O::V* s, int limiter,
                                           typename O::V& neg,
                                           typename O::V& pos) {
  using S = typename O::S;
  using V = typename O::V;
  if constexpr (SCHEME == 0) {
    // Cells i-1 (s[0..4]) and i (s[1..5]) share the differences e1..e3 and the
    // second differences f1, f2.
    V e[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) e[k] = O::sub(s[k + 1], s[k]);
    Weno5Tri<O> f[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) f[k] = weno5_tri<O>(e[k], e[k + 1]);
    neg = weno5_right_v<O>(
        weno5_weights<O>(f[0], f[1], f[2], e[0], e[1], e[2], e[3]), s[2],
        e[0], e[1], e[2], e[3]);
    pos = weno5_left_v<O>(
        weno5_weights<O>(f[1], f[2], f[3], e[1], e[2], e[3], e[4]), s[3],
        e[1], e[2], e[3], e[4]);
  } else if constexpr (SCHEME == 1) {
    V w0, w1;
    const V d0 = O::sub(s[1], s[0]), d1 = O::sub(s[2], s[1]),
            d2 = O::sub(s[3], s[2]);
    weno3_weights<O>(d1, d0, w0, w1);
    neg = weno3_side_v<O>(w0, w1, s[1], d1, d0, true);
    weno3_weights<O>(d2, d1, w0, w1);
    pos = weno3_side_v<O>(w0, w1, s[2], d2, d1, false);
  } else if constexpr (SCHEME == 2) {
    neg = O::fma(O::splat(S(0.5)), muscl_slope_v<O>(s[0], s[1], s[2], limiter), s[1]);
    pos = O::fma(O::splat(S(-0.5)), muscl_slope_v<O>(s[1], s[2], s[3], limiter), s[2]);
  } else {
    neg = s[0];
    pos = s[0];
  }
}

// Both faces of cell c from s[k] = v[c-CL+k] (CellStencil<SCHEME>): `left`
// is the pos value of face c-1/2, `right` the neg value of face c+1/2, bit
// for bit what recon_face gives for them.
template <int SCHEME, class O>
__device__ __forceinline__ void recon_cell(const typename O::V* s, int limiter,
                                           typename O::V& left,
                                           typename O::V& right) {
  using S = typename O::S;
  using V = typename O::V;
  if constexpr (SCHEME == 0) {
    V e[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) e[k] = O::sub(s[k + 1], s[k]);
    Weno5Tri<O> f[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) f[k] = weno5_tri<O>(e[k], e[k + 1]);
    const Weno5W<O> w =
        weno5_weights<O>(f[0], f[1], f[2], e[0], e[1], e[2], e[3]);
    right = weno5_right_v<O>(w, s[2], e[0], e[1], e[2], e[3]);
    left = weno5_left_v<O>(w, s[2], e[0], e[1], e[2], e[3]);
  } else if constexpr (SCHEME == 1) {
    V w0, w1;
    const V dm = O::sub(s[1], s[0]), d0 = O::sub(s[2], s[1]);
    weno3_weights<O>(d0, dm, w0, w1);
    right = weno3_side_v<O>(w0, w1, s[1], d0, dm, true);
    left = weno3_side_v<O>(w0, w1, s[1], d0, dm, false);
  } else if constexpr (SCHEME == 2) {
    const typename O::V sl = muscl_slope_v<O>(s[0], s[1], s[2], limiter);
    right = O::fma(O::splat(S(0.5)), sl, s[1]);
    left = O::fma(O::splat(S(-0.5)), sl, s[1]);
  } else {
    left = s[0];
    right = s[1];
  }
}

// ---------------------------------------------------------------------------
// Riemann solvers.
// ---------------------------------------------------------------------------
// Every product and sum below is rounded as written (One<T>), so a flux has
// the same bits in every kernel and on every axis, whatever is inlined
// around it. Quotients by the densities are products with their reciprocals,
// formed once per face state.

// Roe-averaged wave-speed estimates (hll.py:178-283): c = sqrt(gamma p/rho)
// per side, Roe averages with sqrt(rho) weights and reciprocal_no_nan,
// c~ from the sensible enthalpy with the potential energy pe of the cell at
// the face index (generic.py:144-148, 391-423). pl, pr: the pressures of the
// two sides; il, ir: 1/rho.
template <typename T, int D>
__device__ __forceinline__ void hll_speeds(const Prim<T>& l, const Prim<T>& r,
                                           T pl, T pr, T il, T ir, T pe,
                                           T& s_l, T& s_r) {
  using O = One<T>;
  const T c_l = sqrt_(O::mul(O::mul(K<T>::gamma(), pl), il));
  const T c_r = sqrt_(O::mul(O::mul(K<T>::gamma(), pr), ir));
  const T rl = sqrt_(l.r), rr = sqrt_(r.r);
  const T den = O::add(rl, rr);
  const T inv = den == T(0) ? T(0) : O::rcp(den);
  // Separate products, so mirror-image states give exactly u~ = 0
  // (hll.py:243-261).
  T ru[3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
    ru[i] = O::mul(O::add(O::mul(rl, l.u[i]), O::mul(rr, r.u[i])), inv);
  const T rh = O::mul(O::add(O::mul(rl, l.h), O::mul(rr, r.h)), inv);
  constexpr int A = (D + 1) % 3, B = (D + 2) % 3;
  const T q2 = O::fma(ru[B], ru[B], O::fma(ru[A], ru[A], O::mul(ru[D], ru[D])));
  const T hs = O::sub(O::fma(T(-0.5), q2, rh), pe);
  const T rc = sqrt_(O::mul(K<T>::gm1(), hs));
  s_l = min_(O::sub(l.u[D], c_l), O::sub(ru[D], rc));
  s_r = max_(O::add(r.u[D], c_r), O::add(ru[D], rc));
}

// HLLC contact speed (hllc.py:328-341), zeroed when |s_m| < 1e-6.
template <typename T, int D>
__device__ __forceinline__ T hllc_contact(const Prim<T>& l, const Prim<T>& r,
                                          T pl, T pr, T s_l, T s_r) {
  using O = One<T>;
  const T vl = l.u[D], vr = r.u[D];
  const T al = O::mul(l.r, O::sub(s_l, vl)), ar = O::mul(r.r, O::sub(s_r, vr));
  const T num = O::add(O::sub(pr, pl), O::sub(O::mul(al, vl), O::mul(ar, vr)));
  const T den = O::sub(al, ar);
  const T s_m = den == T(0) ? T(0) : O::div(num, den);
  return abs_(s_m) < T(1e-6) ? T(0) : s_m;
}

// Flux across a face normal to D and those of NS transported scalars with
// face values phl / phr (generic branches: compressible_navier_stokes.py:
// 419-427, hll.py:159-170, hllc.py:182-192). The physical flux
// (compressible_navier_stokes.py:338-427) is, with the mass flux m = rho*u_D:
// m; m*u_i (+ p_d when i == D); m*(e + p/rho) with the full p; m*phi. pdl /
// pdr is p_dyn = p - p_ref where the helper state is present (:378), else p.
//
// RIEMANN 0, HLL (hll.py:107-170): F = t1 F_R + t2 F_L - t3 (U_R - U_L), wave
// speeds from the full pressure.
// RIEMANN 1, HLLC (hllc.py:105-257): wave speeds and star states from p_d
// (hllc.py:109-120). The four-way select of hllc.py:229-243 picks one side
// and whether its star flux applies; only that flux is formed. With
// K = rho (s_m - u_D) s_k / (s_k - s_m) the star flux is the physical one
// plus K (1, s_k, u_t1, u_t2, e + p_d/rho + (s_k - u_D) s_m): the reference's
// rho s_k ((s_k - u_D)/(s_k - s_m) s_m - u_D) is K s_k.
template <int RIEMANN, typename T, int D, int NS>
__device__ __forceinline__ void face_flux(const Prim<T>& l, const Prim<T>& r,
                                          T pdl, T pdr, T pe, const T* phl,
                                          const T* phr, T* f, T* fs) {
  using O = One<T>;
  const T il = O::rcp(l.r), ir = O::rcp(r.r);
  constexpr int A = (D + 1) % 3, B = (D + 2) % 3;
  T s_l, s_r;
  if constexpr (RIEMANN == 0) {
    hll_speeds<T, D>(l, r, l.p, r.p, il, ir, pe, s_l, s_r);
    const T ds = O::sub(s_r, s_l);
    const T rds = ds == T(0) ? T(0) : O::rcp(ds);
    const T t1 = O::mul(O::sub(min_(s_r, T(0)), min_(s_l, T(0))), rds);
    const T t2 = O::sub(T(1), t1);
    const T n3 = O::mul(O::sub(O::mul(s_l, abs_(s_r)), O::mul(s_r, abs_(s_l))),
                        O::mul(T(0.5), rds));  // -t3
    const T ml = O::mul(l.r, l.u[D]), mr = O::mul(r.r, r.u[D]);
    auto mix = [&](T fl, T fr, T ul, T ur) -> T {
      return O::fma(t1, fr, O::fma(t2, fl, O::mul(n3, O::sub(ur, ul))));
    };
    f[0] = mix(ml, mr, l.r, r.r);
    f[1 + D] = mix(O::fma(ml, l.u[D], pdl), O::fma(mr, r.u[D], pdr), ml, mr);
    f[1 + A] = mix(O::mul(ml, l.u[A]), O::mul(mr, r.u[A]), O::mul(l.r, l.u[A]),
                   O::mul(r.r, r.u[A]));
    f[1 + B] = mix(O::mul(ml, l.u[B]), O::mul(mr, r.u[B]), O::mul(l.r, l.u[B]),
                   O::mul(r.r, r.u[B]));
    f[4] = mix(O::mul(ml, O::fma(l.p, il, l.e)), O::mul(mr, O::fma(r.p, ir, r.e)),
               O::mul(l.r, l.e), O::mul(r.r, r.e));
#pragma unroll
    for (int k = 0; k < NS; ++k)
      fs[k] = mix(O::mul(ml, phl[k]), O::mul(mr, phr[k]), O::mul(l.r, phl[k]),
                  O::mul(r.r, phr[k]));
  } else {
    hll_speeds<T, D>(l, r, pdl, pdr, il, ir, pe, s_l, s_r);
    const T s_m = hllc_contact<T, D>(l, r, pdl, pdr, s_l, s_r);
    const bool c1 = s_l >= T(0);
    const bool c2 = (s_l <= T(0)) && (s_m >= T(0));
    const bool c3 = (s_m <= T(0)) && (s_r >= T(0));
    const bool left = c1 || c2;
    const bool star = !c1 && (c2 || c3);
    const T rk = left ? l.r : r.r, ik = left ? il : ir;
    const T v = left ? l.u[D] : r.u[D];
    const T ua = left ? l.u[A] : r.u[A], ub = left ? l.u[B] : r.u[B];
    const T e = left ? l.e : r.e, p = left ? l.p : r.p;
    const T pd = left ? pdl : pdr;
    const T s_k = left ? s_l : s_r;
    const T m = O::mul(rk, v);
    const T g = O::sub(s_k, s_m);
    const T rat = g == T(0) ? T(0) : O::div(s_k, g);
    // Selected, not multiplied by 0: outside the star region the speeds may
    // be infinite or NaN.
    const T kk = star ? O::mul(O::mul(rk, O::sub(s_m, v)), rat) : T(0);
    const T sk = star ? s_k : T(0);
    const T y = star ? O::mul(O::sub(s_k, v), s_m) : T(0);
    f[0] = O::add(m, kk);
    f[1 + D] = O::fma(kk, sk, O::fma(m, v, pd));
    f[1 + A] = O::mul(f[0], ua);
    f[1 + B] = O::mul(f[0], ub);
    f[4] = O::fma(m, O::fma(p, ik, e),
                  O::mul(kk, O::add(O::fma(pd, ik, e), y)));
#pragma unroll
    for (int k = 0; k < NS; ++k)
      fs[k] = O::mul(f[0], left ? phl[k] : phr[k]);
  }
}

// ---------------------------------------------------------------------------
// Viscous flux on the face between cells a (i-1) and b (i)
// (compressible_navier_stokes.py:618-707; diffusion.py:33-109;
// fluid.py:31-111), in the frame rotated so that the face normal is axis 0.
// g11, g10: central differences along t1 of the t1 and the normal velocity,
// averaged over the two cells; g22, g20: the same along t2. rh = 1/h of the
// normal axis; kq = cp / (2 Pr R). Returns the momentum fluxes -tau_c0 and
// the energy flux q_0 - u_f . tau_.0 in f[0..3].
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void viscous_flux(T ra, T rb, const T* ua,
                                             const T* ub, T pa, T pb, T g11,
                                             T g10, T g22, T g20, T rh, T nu,
                                             T kq, T* f) {
  using O = One<T>;
  T bd[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) bd[c] = O::mul(O::sub(ub[c], ua[c]), rh);
  const T div = O::add(O::add(bd[0], g11), g22);
  const T mu2 = O::mul(nu, O::add(ra, rb));  // 2 nu rho_f
  const T mu = O::mul(T(0.5), mu2);
  const T tau[3] = {O::mul(mu2, O::fma(T(-1.0 / 3.0), div, bd[0])),
                    O::mul(mu, O::add(bd[1], g10)),
                    O::mul(mu, O::add(bd[2], g20))};
  // Temperatures (times R) differ little from cell to cell: what their
  // quotients are off by is most of the heat flux's error.
  const T dt = O::sub(O::quot(pb, rb, O::rcp(rb)), O::quot(pa, ra, O::rcp(ra)));
  const T q = O::mul(O::mul(O::mul(kq, mu2), dt), rh);  // -q_0
  const T d2 = O::fma(
      O::add(ua[2], ub[2]), tau[2],
      O::fma(O::add(ua[1], ub[1]), tau[1],
             O::mul(O::add(ua[0], ub[0]), tau[0])));  // 2 u_f . tau
#pragma unroll
  for (int c = 0; c < 3; ++c) f[c] = -tau[c];
  f[3] = -O::fma(T(0.5), d2, q);
}
// cp / (2 Pr R) of viscous_flux (T = p / (rho R), kappa = cp nu rho / Pr).
template <typename T>
__device__ __forceinline__ T heat_coefficient(double pr) {
  return T(0.5 * K<T>::kCp / (pr * K<T>::kR));
}

}  // namespace swc
