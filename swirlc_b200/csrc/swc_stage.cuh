// Fused RK stage kernel: halo-filled conserved state -> primitives -> face
// reconstruction -> Riemann (+ viscous) flux -> divergence + source -> stage
// combination, one pass over the grid per RK stage.
//
// Reference path replaced: the rhs of get_rhs_fn
// (compressible_navier_stokes.py:68-268) evaluated inside rk3.integrate /
// rk2.integrate (rk3.py:87-120, rk2.py:69-86).
//
// Work decomposition (2.5-D plane marching). A CTA owns a TY x TX column of
// cells in the (y, x) plane and marches along z over `zseg` planes. A ring
// of RING planes of primitives (with an in-plane halo HR) lives in shared
// memory; each step computes every y- and x-face of the centre plane into
// shared memory and the z-face above each column in registers (the face
// below is carried from the previous step), converts the next plane, which
// arrived in its ring slot meanwhile, and after the step's one barrier forms
// the divergence and the stage update of the centre plane. Each face flux is
// computed exactly once per CTA. x and y faces reconstruct both face states
// from the face's stencil; z faces take them from cell-centred
// reconstructions of the column's cells, one per cell, whose upper-face
// value is carried up the column. The primitives are reconstructed two at a
// time (f32x2 lanes) and stored two at a time: one 8-byte shared-memory load
// (16 in double precision) brings both lanes of a stencil cell into a
// register pair. Everything up to the stage update is explicitly rounded.
#pragma once

#include <type_traits>

#include "swc_physics.cuh"
#include "swirlc_b200.h"

// Members per batched launch (the member table is a launch parameter).
#define SWC_BATCH_CHUNK 64

namespace swc {

struct StageArgs {
  int nx, ny, nz, halo;
  long long sx, sz;
  double dx, dy, dz;
  const void* uk[SWC_MAX_FIELDS];
  const void* u0[SWC_MAX_FIELDS];
  void* uout[SWC_MAX_FIELDS];
  int mode;
  // SWC_OUT_CONVEX forms c0 u0 + c1 ((uk - u0) + dt L): for the caller's
  // w0 u0 + w1 (uk + dt L) c0 is w0 + w1 (stage_weights). The change is rounded
  // at its own size and the result once, and 1/3 and 2/3 rounded to 32 bits,
  // which add up to 1 + 3e-8, do not scale the state: the error of a gradient
  // with respect to the fields against 64 bits fell from 4.5e-6 to 2.3e-6.
  double c0, c1;
  const double* dt;
  double* dtmin_out;
  const void* pe[3];
  int has_pe;
  int limiter;
  double nu, pr;
  int gravity_mask;
  double g[3];
  int zseg;
  // Where halo cells along x, y, z are read: as stored, or from the interior
  // cell they copy (periodic for every field, or Neumann of slope 0 for every
  // field): a stage whose input needs no fill before it.
  int halo_from[3];
};
enum { kHaloStored, kHaloWrapped, kHaloClamped };
// mode, c0 and c1 of a stage of the caller's mode and weights; the average
// w0 (u0 + uk + dt L) is the combination with both weights w0.
inline void stage_weights(StageArgs& a, int mode, double w0, double w1) {
  const double second = mode == SWC_OUT_AVERAGE ? w0 : w1;
  a.mode = mode == SWC_OUT_AVERAGE ? SWC_OUT_CONVEX : mode;
  a.c0 = w0 + second;
  a.c1 = second;
}

// Padded coordinate a halo cell c of a dim of n cells is read from.
__device__ __forceinline__ int halo_source(int c, int n, int h, int from) {
  if (from == kHaloStored || (c >= h && c < n + h)) return c;
  if (from == kHaloWrapped) return c < h ? c + n : c - n;
  return c < h ? h : n + h - 1;
}

__device__ __forceinline__ void atomic_min_pos(double* addr, double v) {
  // Non-negative doubles order like their bit patterns.
  atomicMin(reinterpret_cast<unsigned long long*>(addr),
            static_cast<unsigned long long>(__double_as_longlong(v)));
}

template <int SCHEME, bool VISC>
struct Geom {
  static constexpr int LO = Stencil<SCHEME>::LO;
  static constexpr int RI = Stencil<SCHEME>::RI;
  static constexpr int NW = LO + RI;
  // Cell-centred stencil v[c-CL .. c+CR] (z faces).
  static constexpr int CL = CellStencil<SCHEME>::CL;
  static constexpr int CR = CellStencil<SCHEME>::CR;
  static constexpr int CW = CL + CR + 1;
  static constexpr int cmax(int a, int b) { return a > b ? a : b; }
  static constexpr int NOFF = cmax(NW, CW);
  static constexpr int HR = cmax(cmax(LO, RI - 1), VISC ? 1 : 0);
  // Planes below / above the centre plane zc held in the ring: the cell
  // above (zc+1) is reconstructed along z while zc is processed, and the
  // first pass of a segment also reconstructs its own plane.
  static constexpr int ZLO = cmax(cmax(cmax(LO - 1, CL), VISC ? 1 : 0), 0);
  static constexpr int ZHI = cmax(cmax(cmax(RI, CR + 1), VISC ? 1 : 0), 1);
  // The next plane is converted while the faces of plane zc are still being
  // read, into the slot of plane zc-ZLO-SPARE. The faces read plane zc, the
  // planes from zc+1-CL up (the z reconstruction of cell zc+1) and, viscous,
  // zc-1 (tangential differences), so that slot is free when ZLO >= 1,
  // ZLO >= CL and, viscous, ZLO >= 2; otherwise one spare slot is added
  // (not loaded by the warm-up, so the halo depth the arrays need does not
  // change).
  static constexpr int SPARE =
      (ZLO >= 1 && ZLO >= CL && (!VISC || ZLO >= 2)) ? 0 : 1;
  static constexpr int RING = ZLO + 1 + ZHI + SPARE;
  // Halo layers the stored arrays need.
  static constexpr int NEED = cmax(HR, cmax(ZLO + 1, ZHI));
};

// Shared-memory layout. NS transported scalars and (HELP) the p_dyn helper
// add reconstructed variables to the 7 primitives. A ring slot holds the
// variables (rho, e), (u, v), (w, p), (h, x0), (x1, x2) .. as arrays of pairs
// and, when their number is odd, the last one alone; x0, x1 .. are the
// scalars, then p_dyn. An incoming plane is copied straight into the pair
// positions of its slot (rho_u where u goes, p_ref where p_dyn goes) and
// converted in place, each cell by the thread that copied it.
template <typename T, int SCHEME, bool VISC, int TY, int TX, int NS = 0,
          bool HELP = false>
struct Layout {
  using G = Geom<SCHEME, VISC>;
  static constexpr int NV = 7 + NS + (HELP ? 1 : 0);  // ring variables
  static constexpr int NP = NV / 2;                   // pairs
  static constexpr int NF = 5 + NS;                   // flux components
  static constexpr int PW = TY + 2 * G::HR;
  static constexpr int PH = TX + 2 * G::HR;
  static constexpr int PS = PW * PH;
  static constexpr int NT = TX * TY;
  static constexpr int PER = (PS + NT - 1) / NT;  // plane cells per thread
  static constexpr int SLOT = (NV * PS + 3) / 4 * 4;  // 16-byte multiple
  static constexpr int RING_ELEMS = G::RING * SLOT;
  // x- and y-face fluxes, two buffers each (planes alternate), so that
  // threads may start the next plane's faces while others still form the
  // update of this one. The z-face flux stays in the registers of the
  // thread that computes and uses it. Components as (rho, rho_e),
  // (rho_u, rho_v), (rho_w, scalar 0) .. pairs and the last one alone.
  static constexpr int NFP = NF / 2;
  static constexpr int NY = TX * (TY + 1), NX = (TX + 1) * TY;
  static constexpr int FY_ELEMS = (NF * NY + 3) / 4 * 4;
  static constexpr int FX_ELEMS = (NF * NX + 3) / 4 * 4;
  static constexpr size_t SMEM =
      sizeof(T) * (size_t)(RING_ELEMS + 2 * (FY_ELEMS + FX_ELEMS));
  // Offset in a ring slot of variable q (in the order rho, e, u, v, w, p, h,
  // x0 ..) of plane cell 0, and the step from one cell to the next.
  __host__ __device__ static constexpr int var_off(int q) {
    return q / 2 < NP ? (q / 2) * 2 * PS + (q & 1) : 2 * NP * PS;
  }
  __host__ __device__ static constexpr int var_step(int q) {
    return q / 2 < NP ? 2 : 1;
  }
};

// 4- or 8-byte asynchronous global->shared copy (LDGSTS), cached in L1 so
// the centre-plane reload of the stage update hits on chip.
template <typename T>
__device__ __forceinline__ void cp_async(T* smem, const T* gmem) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  if constexpr (sizeof(T) == 4) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s),
                 "l"(gmem));
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s),
                 "l"(gmem));
  }
}
// Hint that the line holding *p will be read soon (no register is used;
// callers pass only addresses they will load).
__device__ __forceinline__ void prefetch_l1(const void* p) {
  asm volatile("prefetch.global.L1 [%0];\n" ::"l"(p));
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::);
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// One CTA's work: the TY x TX column at (y0, x0), z segment zb of `a`.
// The potential energy (PE), NS scalars, HELP (p_ref/rho_ref) and EXT (face
// and flux overrides from `ext` on the grid's boundary faces) are compiled in
// only where asked for.
template <typename T, int SCHEME, int RIEMANN, bool VISC, int TY, int TX,
          bool PE = true, int NS = 0, bool HELP = false, bool EXT = false>
__device__ __forceinline__ void stage_body(const StageArgs& a,
                                           const SwcStageExt* ext, const int y0,
                                           const int x0, const int zb) {
  using G = Geom<SCHEME, VISC>;
  using L = Layout<T, SCHEME, VISC, TY, TX, NS, HELP>;
  using O1 = One<T>;
  using O2 = Two<T>;
  using V2 = typename O2::V;
  constexpr int NV = L::NV, NP = L::NP, NF = L::NF, NFP = L::NFP;
  constexpr int LO = G::LO, NW = G::NW, HR = G::HR, ZLO = G::ZLO,
                ZHI = G::ZHI, RING = G::RING, SPARE = G::SPARE, CL = G::CL,
                CW = G::CW;
  constexpr int PW = L::PW, PS = L::PS, NT = L::NT, PER = L::PER;
  constexpr int SLOT = L::SLOT;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* const ring = reinterpret_cast<T*>(smem_raw);
  T* const fy0 = ring + L::RING_ELEMS;
  T* const fx0 = fy0 + 2 * L::FY_ELEMS;

  const int tid = threadIdx.x;
  // Cell of this thread. For TY = 16 a warp covers two rows ROWGAP apart, so
  // that the two half-warps of a 4-byte access to a plane (row pitch PW)
  // hit disjoint banks: ROWGAP * PW = 16 (mod 32) words with 8 rows for
  // PW = 22 and 4 rows for PW = 20. (8-byte accesses are served half a warp
  // at a time.)
  int ty, tx;
  if constexpr (TY == 16 && TX % 16 == 0) {
    constexpr int ROWGAP = PW % 8 == 4 ? 4 : 8;
    const int w = tid >> 5, lane = tid & 31;
    ty = lane & 15;
    tx = (w / ROWGAP) * 2 * ROWGAP + w % ROWGAP + (lane >> 4) * ROWGAP;
  } else {
    ty = tid % TY;
    tx = tid / TY;
  }
  const int z0 = zb * a.zseg;
  const int z1 = min(z0 + a.zseg, a.nz);
  const int h = a.halo;
  const int nxa = a.nx + 2 * h, nya = a.ny + 2 * h;
  const long long sx = a.sx, sz = a.sz;

  const T* __restrict__ pex = static_cast<const T*>(a.pe[0]);
  const T* __restrict__ pey = static_cast<const T*>(a.pe[1]);
  const T* __restrict__ pez = static_cast<const T*>(a.pe[2]);
  // Potential energy of cell (xa, ya) of a plane with z part `az`. Gravity
  // along z alone, the usual case, costs one load per plane.
  const bool pe_xy = PE && (pex || pey);
  auto az_at = [&](int za) -> T { return PE && pez ? pez[za] : T(0); };
  auto pe_of = [&](int xa, int ya, T az) -> T {
    if (!pe_xy) return PE ? -az : T(0);
    const T ax = pex ? pex[xa] : T(0);
    const T ay = pey ? pey[ya] : T(0);
    return O1::sub(O1::sub(-ax, ay), az);
  };

  const T dx = T(a.dx), dy = T(a.dy), dz = T(a.dz);
  // Reciprocals of the launch-constant spacings.
  const T rdx = rcp_(dx), rdy = rcp_(dy), rdz = rcp_(dz);
  const T nu = T(a.nu);
  const T kq = VISC ? heat_coefficient<T>(a.pr) : T(0);

  // Pair j, or variable q, of plane cell `pos` in the slot at `s`.
  auto P2 = [&](const T* s, int j, int pos) -> V2 {
    return reinterpret_cast<const V2*>(s)[j * PS + pos];
  };
  auto V1 = [&](const T* s, int q, int pos) -> T {
    return s[L::var_off(q) + L::var_step(q) * pos];
  };

  // Plane cells this thread copies and converts: idx = tid + k*NT, at
  // element goff[k] of a plane (negative: none).
  // (32 bits: a field whose plane has 2^31 elements does not fit the device.)
  int goff[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int idx = tid + k * NT;
    const int px = idx / PW, py = idx - px * PW;
    const int xa = x0 - HR + px + h, ya = y0 - HR + py + h;
    goff[k] = (idx < PS && xa < nxa && ya < nya)
                  ? (int)(halo_source(xa, a.nx, h, a.halo_from[0]) * sx) +
                        halo_source(ya, a.ny, h, a.halo_from[1])
                  : -1;
  }
  auto issue_plane = [&](int z, int slot) {
    const long long zo =
        (long long)halo_source(z + h, a.nz, h, a.halo_from[2]) * sz;
    T* const s = ring + slot * SLOT;
#pragma unroll
    for (int v = 0; v < 5 + NS + (HELP ? 1 : 0); ++v) {
      // rho, rho_u, rho_v, rho_w, rho_e, scalars, p_ref.
      constexpr int kVar[5] = {0, 2, 3, 4, 1};
      const int q = v < 5 ? kVar[v < 5 ? v : 0] : 7 + (v - 5);
      const T* src;
      if (HELP && v == 5 + NS) src = static_cast<const T*>(ext->p_ref);
      else src = static_cast<const T*>(a.uk[v]);
      src += zo;
#pragma unroll
      for (int k = 0; k < PER; ++k)
        if (goff[k] >= 0)
          cp_async(s + L::var_off(q) + L::var_step(q) * (tid + k * NT),
                   src + goff[k]);
    }
    cp_async_commit();
  };
  // Converts this thread's cells of plane z in place.
  auto convert_plane = [&](int z, int slot) {
    T* const s = ring + slot * SLOT;
    const T az = az_at(z + h);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int idx = tid + k * NT;
      if (idx >= PS) break;
      const bool ok = goff[k] >= 0;
      V2 re = P2(s, 0, idx), uv = P2(s, 1, idx), wp = P2(s, 2, idx);
      if (!ok) {
        re = O2::splat(T(1));
        uv = wp = O2::splat(T(0));
      }
      T pe = PE ? -az : T(0);
      if (pe_xy && ok) {
        const int px = idx / PW, py = idx - px * PW;
        pe = pe_of(x0 - HR + px + h, y0 - HR + py + h, az);
      }
      T u, vv, w, e, p, hh;
      cons_to_prim(re.x, uv.x, uv.y, wp.x, re.y, pe, u, vv, w, e, p, hh);
      V2* const d = reinterpret_cast<V2*>(s) + idx;
      d[0] = O2::mk(re.x, e);
      d[PS] = O2::mk(u, vv);
      d[2 * PS] = O2::mk(w, p);
      if constexpr (NS > 0 || HELP) {
        const T inv = O1::rcp(re.x);
#pragma unroll
        for (int q = 0; q < NS; ++q) {
          T& x = s[L::var_off(7 + q) + L::var_step(7 + q) * idx];
          x = ok ? O1::mul(inv, x) : T(0);
        }
        if constexpr (HELP) {
          // p_dyn = p - p_ref, zero in the halo layers beyond the grid's
          // boundary (exchange_halos with DIRICHLET 0 on all sides).
          const int px = idx / PW, py = idx - px * PW;
          const int xa = x0 - HR + px + h, ya = y0 - HR + py + h, za = z + h;
          const bool out =
              (xa < h && ext->boundary[0][0]) ||
              (xa >= a.nx + h && ext->boundary[0][1]) ||
              (ya < h && ext->boundary[1][0]) ||
              (ya >= a.ny + h && ext->boundary[1][1]) ||
              (za < h && ext->boundary[2][0]) ||
              (za >= a.nz + h && ext->boundary[2][1]);
          T& x = s[L::var_off(7 + NS) + L::var_step(7 + NS) * idx];
          x = (ok && !out) ? O1::sub(p, x) : T(0);
        }
      }
      s[L::var_off(6) + L::var_step(6) * idx] = hh;
    }
  };
  const int zfirst = z0 - ZLO - 1;
  // Ring slot of plane zc + d (-ZLO-1 <= d <= ZHI+2) from that of plane zc.
  auto near_slot = [&](int slot, int d) {
    int q = slot + d;
    if (d < 0) q = q < 0 ? q + RING : q;
    else q = q >= RING ? q - RING : q;
    return q;
  };
  static_assert(ZLO + 1 <= RING && ZHI + 2 <= RING, "near_slot range");

  constexpr int NSA = NS > 0 ? NS : 1;
  // Face values of every variable: the pairs and the last one alone.
  struct Faces {
    V2 q[NP];
    T o;
  };
  auto state = [&](const Faces& f, int n, Prim<T>& s, T* ph, T& pd) {
    // Normal n, tangential t1, t2 in the rotated frame: x:(x,y,z),
    // y:(y,x,z), z:(z,x,y).
    const T u = f.q[1].x, v = f.q[1].y, w = f.q[2].x;
    s.r = f.q[0].x;
    s.e = f.q[0].y;
    s.p = f.q[2].y;
    s.u[0] = n == 2 ? w : (n == 0 ? u : v);
    s.u[1] = n == 0 ? v : u;
    s.u[2] = n == 2 ? v : w;
    auto var = [&](int q) -> T {
      return q / 2 < NP ? ((q & 1) ? f.q[q / 2 < NP ? q / 2 : 0].y
                                   : f.q[q / 2 < NP ? q / 2 : 0].x)
                        : f.o;
    };
    s.h = var(6);
#pragma unroll
    for (int k = 0; k < NS; ++k) ph[k] = var(7 + k);
    pd = HELP ? var(7 + NS) : s.p;
  };

  // Face BCs on both face states (boundary.py:247-337): a primitive is set
  // directly, a conservative one divided by the face density. Flux BCs of
  // one type (boundary.py:89-183). dn: face normal; bside: -1, or the side
  // (0 low, 1 high) of the grid boundary the face lies on; pidx: its index
  // in a face plane [A][B].
  auto plane_val = [&](const SwcOverride& o, long long pidx) -> T {
    return o.plane ? static_cast<const T*>(o.plane)[pidx] : T(o.value);
  };
  auto face_bc = [&](int dn, int bside, long long pidx, Prim<T>& l,
                     Prim<T>& r, T* phl, T* phr) {
    const int t1 = dn == 0 ? 1 : 0;
    const int n = ext->nface[dn][bside];
    for (int i = 0; i < n; ++i) {
      const SwcOverride& o = ext->face[dn][bside][i];
      const T val = plane_val(o, pidx);
      const bool cons = o.mode == SWC_FACE_CONSERVATIVE;
      const T vl = cons ? dnn(val, l.r) : val;
      const T vr = cons ? dnn(val, r.r) : val;
      const int c = o.var - 1;
      const int rr = c == dn ? 0 : (c == t1 ? 1 : 2);
#pragma unroll
      for (int q = 0; q < 3; ++q)
        if (o.var >= 1 && o.var <= 3 && q == rr) {
          l.u[q] = vl;
          r.u[q] = vr;
        }
      if (o.var == 4) {
        l.e = vl;
        r.e = vr;
      }
#pragma unroll
      for (int q = 0; q < NS; ++q)
        if (o.var == 5 + q) {
          phl[q] = vl;
          phr[q] = vr;
        }
    }
  };
  auto flux_bc = [&](int dn, int bside, long long pidx, int type, T* fb) {
    const int n = ext->nflux[dn][bside];
    for (int i = 0; i < n; ++i) {
      const SwcOverride& o = ext->flux[dn][bside][i];
      if (o.mode != type) continue;
      const T val = plane_val(o, pidx);
#pragma unroll
      for (int v = 0; v < NF; ++v)
        if (o.var == v) fb[v] = val;
    }
  };
  // Total flux (x, y, z momentum order, then scalars) from the face states
  // and the viscous flux v (rotated, VISC only).
  auto flux = [&](int dn, const Faces& lo, const Faces& hi, T pe, const T* v,
                  int bside, long long pidx, T* f) {
    Prim<T> l, r;
    T phl[NSA], phr[NSA], pdl, pdr, g[5], gs[NSA];
    state(lo, dn, l, phl, pdl);
    state(hi, dn, r, phr, pdr);
    if constexpr (EXT)
      if (bside >= 0) face_bc(dn, bside, pidx, l, r, phl, phr);
    if constexpr (!HELP) {
      pdl = l.p;
      pdr = r.p;
    }
    face_flux<RIEMANN, T, 0, NS>(l, r, pdl, pdr, pe, phl, phr, g, gs);
    auto rot = [&](T n, T a1, T a2, T* out) {
      out[1] = dn == 0 ? n : a1;
      out[2] = dn == 1 ? n : (dn == 0 ? a1 : a2);
      out[3] = dn == 2 ? n : a2;
    };
    if constexpr (EXT) {
      f[0] = g[0];
      rot(g[1], g[2], g[3], f);
      f[4] = g[4];
#pragma unroll
      for (int k = 0; k < NS; ++k) f[5 + k] = gs[k];
      if (bside >= 0) flux_bc(dn, bside, pidx, SWC_FLUX_CONVECTIVE, f);
      T fv[NF];
#pragma unroll
      for (int k = 0; k < NF; ++k) fv[k] = T(0);
      if constexpr (VISC) {
        rot(v[0], v[1], v[2], fv);
        fv[4] = v[3];
        if (bside >= 0) flux_bc(dn, bside, pidx, SWC_FLUX_DIFFUSIVE, fv);
      }
#pragma unroll
      for (int k = 0; k < NF; ++k) f[k] = O1::add(f[k], fv[k]);
      if (bside >= 0) flux_bc(dn, bside, pidx, SWC_FLUX_TOTAL, f);
    } else {
      if constexpr (VISC) {
#pragma unroll
        for (int k = 0; k < 4; ++k) g[1 + k] = O1::add(g[1 + k], v[k]);
      }
      f[0] = g[0];
      rot(g[1], g[2], g[3], f);
      f[4] = g[4];
#pragma unroll
      for (int k = 0; k < NS; ++k) f[5 + k] = gs[k];
    }
  };
  // Grid-boundary side of the face normal to `dn` stored at index i of n
  // (face i-1/2: i = 0 is the low boundary, i = n the high one,
  // boundary.py:140-183).
  auto side_of = [&](int dn, int i, int n) -> int {
    int b = -1;
    if constexpr (EXT) {
      if (i == 0 && ext->boundary[dn][0]) b = 0;
      if (i == n && ext->boundary[dn][1]) b = 1;
    }
    return b;
  };

  // MUSCL: one branch on the limiter per face, not per variable, with the
  // van Leer slope (paired lanes, no branch) compiled on its own.
  auto by_limiter = [&](auto recon) {
    if (SCHEME == 2 && a.limiter == SWC_LIM_VAN_LEER) recon(SWC_LIM_VAN_LEER);
    else recon(a.limiter);
  };

  // Flux buffers of the plane in progress, and this thread's z-face flux.
  T* fx = fx0;
  T* fy = fy0;
  T fzr[NF];
  T azc = T(0), azu = az_at(z0 - 1 + h);  // az of planes zc and zc+1
  // x (isx) or y face at row fxx, column fyy of plane zc, in slot sc, into
  // the flux buffers; only the stencil's stride and the order of u and v
  // differ between the axes.
  auto face_xy = [&](bool isx, int zc, int sc, int fxx, int fyy) {
    const int dn = isx ? 0 : 1;
    const int pos = (HR + fxx) * PW + HR + fyy;
    const int st = isx ? PW : 1;
    const T* const s = ring + sc * SLOT;
    T fv[4];
    if constexpr (VISC) {
      // Cells a = i-1, b = i; t1 is the other in-plane axis, t2 is z.
      const int s1 = isx ? 1 : PW;
      const int pa = pos - st, pb = pos;
      const T r1 = O1::mul(T(0.25), isx ? rdy : rdx);
      const T r2 = O1::mul(T(0.25), rdz);
      const V2 d1 = O2::add(O2::sub(P2(s, 1, pa + s1), P2(s, 1, pa - s1)),
                            O2::sub(P2(s, 1, pb + s1), P2(s, 1, pb - s1)));
      const T* const su = ring + near_slot(sc, 1) * SLOT;
      const T* const sd = ring + near_slot(sc, -1) * SLOT;
      const int vn = (isx ? L::var_off(2) : L::var_off(3));
      auto dz4 = [&](int off) -> T {
        return O1::add(O1::sub(su[off + 2 * pa], sd[off + 2 * pa]),
                       O1::sub(su[off + 2 * pb], sd[off + 2 * pb]));
      };
      const T g11 = O1::mul(isx ? d1.y : d1.x, r1);
      const T g10 = O1::mul(isx ? d1.x : d1.y, r1);
      const T g22 = O1::mul(dz4(L::var_off(4)), r2);
      const T g20 = O1::mul(dz4(vn), r2);
      const V2 ua2 = P2(s, 1, pa), ub2 = P2(s, 1, pb);
      const V2 wa = P2(s, 2, pa), wb = P2(s, 2, pb);
      const T ua[3] = {isx ? ua2.x : ua2.y, isx ? ua2.y : ua2.x, wa.x};
      const T ub[3] = {isx ? ub2.x : ub2.y, isx ? ub2.y : ub2.x, wb.x};
      viscous_flux<T>(V1(s, 0, pa), V1(s, 0, pb), ua, ub, wa.y, wb.y, g11, g10,
                      g22, g20, isx ? rdx : rdy, nu, kq, fv);
    }
    Faces lo, hi;
    by_limiter([&](int limiter) {
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        V2 sv[NW];
#pragma unroll
        for (int k = 0; k < NW; ++k) sv[k] = P2(s, j, pos + (k - LO) * st);
        recon_face<SCHEME, O2>(sv, limiter, lo.q[j], hi.q[j]);
      }
      if constexpr (NV & 1) {
        T sv[NW];
#pragma unroll
        for (int k = 0; k < NW; ++k) sv[k] = V1(s, NV - 1, pos + (k - LO) * st);
        recon_face<SCHEME, O1>(sv, limiter, lo.o, hi.o);
      }
    });
    const T pe = pe_of(x0 + fxx + h, y0 + fyy + h, azc);
    int bside = -1;
    long long pidx = 0;
    if constexpr (EXT) {
      bside = isx ? side_of(0, x0 + fxx, a.nx) : side_of(1, y0 + fyy, a.ny);
      pidx = isx ? (long long)(zc + h) * nya + (y0 + fyy + h)
                 : (long long)(zc + h) * nxa + (x0 + fxx + h);
    }
    T f[NF];
    flux(dn, lo, hi, pe, fv, bside, pidx, f);
    T* const buf = isx ? fx : fy;
    const int n = isx ? L::NX : L::NY;
    const int p = isx ? fxx * TY + fyy : fxx * (TY + 1) + fyy;
    V2* const b2 = reinterpret_cast<V2*>(buf) + p;
    b2[0] = O2::mk(f[0], f[4]);
    b2[n] = O2::mk(f[1], f[2]);
#pragma unroll
    for (int j = 2; j < NFP; ++j) {
      const int c = 2 * j;  // components (3, 5), (6, 7)
      b2[j * n] = O2::mk(c == 4 ? f[3] : f[c], f[c + 1 < NF ? c + 1 : 0]);
    }
    if constexpr (NF & 1) buf[2 * NFP * n + p] = f[NF == 5 ? 3 : NF - 1];
  };
  // z-face above plane zc (slot sc), into fzr. The cell above it (zc+1) is
  // reconstructed along z: its lower-face value is this face's upper state,
  // its upper-face value the next face's lower state, carried in zq.
  Faces zq;
  auto recon_z = [&](const int* sl, int pos, Faces& lo, Faces& hi) {
    by_limiter([&](int limiter) {
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        V2 sv[CW];
#pragma unroll
        for (int k = 0; k < CW; ++k) sv[k] = P2(ring + sl[k], j, pos);
        recon_cell<SCHEME, O2>(sv, limiter, lo.q[j], hi.q[j]);
      }
      if constexpr (NV & 1) {
        T sv[CW];
#pragma unroll
        for (int k = 0; k < CW; ++k) sv[k] = V1(ring + sl[k], NV - 1, pos);
        recon_cell<SCHEME, O1>(sv, limiter, lo.o, hi.o);
      }
    });
  };
  auto face_z = [&](int zc, int sc) {
    const int pos = (HR + tx) * PW + HR + ty;
    T fv[4];
    if constexpr (VISC) {
      const T* const sa = ring + sc * SLOT;
      const T* const sb = ring + near_slot(sc, 1) * SLOT;
      const T r1 = O1::mul(T(0.25), rdx), r2 = O1::mul(T(0.25), rdy);
      auto diff = [&](int q, int st) -> T {
        return O1::add(O1::sub(V1(sa, q, pos + st), V1(sa, q, pos - st)),
                       O1::sub(V1(sb, q, pos + st), V1(sb, q, pos - st)));
      };
      const T g11 = O1::mul(diff(2, PW), r1), g10 = O1::mul(diff(4, PW), r1);
      const T g22 = O1::mul(diff(3, 1), r2), g20 = O1::mul(diff(4, 1), r2);
      const V2 ua2 = P2(sa, 1, pos), ub2 = P2(sb, 1, pos);
      const V2 wa = P2(sa, 2, pos), wb = P2(sb, 2, pos);
      const T ua[3] = {wa.x, ua2.x, ua2.y}, ub[3] = {wb.x, ub2.x, ub2.y};
      viscous_flux<T>(V1(sa, 0, pos), V1(sb, 0, pos), ua, ub, wa.y, wb.y, g11,
                      g10, g22, g20, rdz, nu, kq, fv);
    }
    int sl[CW];
#pragma unroll
    for (int k = 0; k < CW; ++k) sl[k] = near_slot(sc, 1 - CL + k) * SLOT;
    Faces lo, up;
    recon_z(sl, pos, lo, up);
    const T pe = pe_of(x0 + tx + h, y0 + ty + h, azu);
    flux(2, zq, lo, pe, fv, side_of(2, zc + 1, a.nz),
         (long long)(x0 + tx + h) * nya + (y0 + ty + h), fzr);
    zq = up;
  };

  // Constants of the update, in shared memory: read once per plane after the
  // barrier, they hold no registers while the faces are computed.
  __shared__ T upd[6];
  if (tid == 0) {
    upd[0] = -rdx;
    upd[1] = -rdy;
    upd[2] = -rdz;
    upd[3] = T(a.dt ? *a.dt : 0.0);
    upd[4] = T(a.c0);
    upd[5] = T(a.c1);
  }

  // ---- warm-up: planes zfirst .. z0+ZHI-1, all copies in flight at once
  // (the ring of the loop's first pass, zc = z0-1, which only computes the
  // z-face below the segment, so that every face of every segment comes from
  // the same code: results do not depend on where segments start).
  for (int i = 0; i < RING - SPARE; ++i) issue_plane(zfirst + i, i);
  cp_async_wait_all();
  for (int i = 0; i < RING - SPARE; ++i) convert_plane(zfirst + i, i);
  __syncthreads();
  const bool own = (x0 + tx < a.nx) && (y0 + ty < a.ny);
  T flo[NF];

  T dtmin_local = T(__longlong_as_double(0x7ff0000000000000ll));  // infinity
  const int xa_c = x0 + tx + h, ya_c = y0 + ty + h;

  // Per plane every owner computes three faces of its cell (z above, y and
  // x below); TY + TX threads also compute the tile's high x-row and high
  // y-column faces; owners of the last interior cell of a partial tile add
  // the face beyond it. The boundary block starts at a warp that moves on
  // from plane to plane (and from tile to tile), so its extra pass falls on
  // every SM sub-partition in turn instead of always on the last warp's.
  static_assert(TY + TX <= NT, "boundary faces need TY + TX threads");
  static_assert(NT % 32 == 0, "whole warps");
  constexpr int NWARP = NT / 32;
  const int tile_rot = x0 / TX + y0 / TY;
  int bkind = -1, bx = 0, by = 0;
  auto boundary_faces = [&](int zc) {
    int wb = tid - ((zc - z0 + tile_rot) % NWARP) * 32;
    if (wb < 0) wb += NT;
    bkind = -1;
    if (wb < TY + TX) {
      if (wb < TY) { bkind = 0; bx = TX; by = wb; }
      else { bkind = 1; bx = wb - TY; by = TY; }
      if (bkind == 0 && !(x0 + TX <= a.nx && y0 + by < a.ny)) bkind = -1;
      if (bkind == 1 && !(y0 + TY <= a.ny && x0 + bx < a.nx)) bkind = -1;
    }
  };
  const bool ex_x = own && (x0 + tx + 1 == a.nx) && (tx + 1 < TX);
  const bool ex_y = own && (y0 + ty + 1 == a.ny) && (ty + 1 < TY);

  // One barrier per plane: faces of plane zc (x and y into flux buffer
  // zc & 1, z into registers), then the in-place conversion of plane
  // zc+ZHI+1 in a slot no face of plane zc reads, the barrier, and the update
  // of plane zc, which reads no ring slot. A thread may start the faces of
  // plane zc+1 while others still update plane zc: they write the other flux
  // buffer, and buffer zc & 1 is next written after the following barrier.
  // The copy of plane zc+ZHI+2 starts after that barrier, into the slot of
  // plane zc+1-ZLO-SPARE: the faces of plane zc were its last readers.
  int sc = ZLO;  // slot of plane zc
  for (int zc = z0 - 1; zc < z1; ++zc, sc = near_slot(sc, 1)) {
    const bool pre = zc < z0;  // only the z-face below the segment
    azc = azu;
    azu = az_at(zc + 1 + h);
    fx = fx0 + ((zc - z0 + 1) & 1) * L::FX_ELEMS;
    fy = fy0 + ((zc - z0 + 1) & 1) * L::FY_ELEMS;
    if (pre) {
      if (own) {
        // Upper-face value of cell z0-1: the lower state of the segment's
        // first z face.
        int sl[CW];
#pragma unroll
        for (int k = 0; k < CW; ++k) sl[k] = near_slot(sc, -CL + k) * SLOT;
        Faces lf;
        recon_z(sl, (HR + tx) * PW + HR + ty, lf, zq);
      }
      // The first pass reads plane zc-CL, whose slot the next plane may
      // take: every thread has read it before the copy starts.
      __syncthreads();
      if (zc + 1 < z1) issue_plane(zc + ZHI + 1, near_slot(sc, ZHI + 1));
    } else {
      boundary_faces(zc);
    }
    if (own) face_z(zc, sc);
    if (own && !pre) {
      // Inlined for each axis: strides and rotations are constants there,
      // which takes a tenth of the instructions out (KH 256^3 4.80 -> 4.60 ms
      // per step). The extra faces below mix both axes in one warp and share
      // a third copy.
      face_xy(false, zc, sc, tx, ty);
      face_xy(true, zc, sc, tx, ty);
    }
    const int nxy = pre ? 0 : (bkind >= 0) + ex_x + ex_y;
#pragma unroll 1
    for (int j = 0; j < nxy; ++j) {
      bool isx;
      int fxx = tx, fyy = ty;
      if (bkind >= 0 && j == 0) {
        isx = bkind == 0; fxx = bx; fyy = by;
      } else {
        isx = ex_x && j == (bkind >= 0);
        if (isx) fxx = tx + 1;
        else fyy = ty + 1;
      }
      face_xy(isx, zc, sc, fxx, fyy);
    }
    // The cell's density for the gravity source, read while plane zc's
    // slot is certain to hold it (before the barrier).
    const T rho_cell = (a.gravity_mask && own && !pre)
                           ? V1(ring + sc * SLOT, 0, (HR + tx) * PW + HR + ty)
                           : T(0);
    // The update's own-cell reads start here: the conversion and the barrier
    // hide their latency.
    const long long o = (zc + h) * sz + (long long)xa_c * sx + ya_c;
    T ukc[NF], u0c[NF];
    if (own && !pre) {
#pragma unroll
      for (int v = 0; v < NF; ++v) {
        ukc[v] = __ldg(static_cast<const T*>(a.uk[v]) + o);
        u0c[v] = a.mode == SWC_OUT_CONVEX
                     ? __ldg(static_cast<const T*>(a.u0[v]) + o)
                     : T(0);
      }
    }
    if (zc + 1 < z1) {
      cp_async_wait_all();
      convert_plane(zc + ZHI + 1, near_slot(sc, ZHI + 1));
    }
    __syncthreads();
    if (zc + 2 < z1) issue_plane(zc + ZHI + 2, near_slot(sc, ZHI + 2));
    if (pre) {
      if (own) {
#pragma unroll
        for (int v = 0; v < NF; ++v) flo[v] = fzr[v];
      }
      continue;
    }

    // ---- divergence, source and stage combination.
    if (own) {
      T src[5] = {T(0), T(0), T(0), T(0), T(0)};
      if (a.gravity_mask) {
        // Buoyancy acts on rho, or on rho - rho_ref with helper states.
        T rho_c = rho_cell;
        if constexpr (HELP)
          rho_c = rho_c - __ldg(static_cast<const T*>(ext->rho_ref) + o);
#pragma unroll
        for (int d = 0; d < 3; ++d)
          if (a.gravity_mask & (1 << d))
            src[1 + d] = rho_c * K<T>::grav() * T(a.g[d]);
      }
      // Flux components as the buffers hold them: (0, 4), (1, 2), (3, 5),
      // (6, 7) pairs and the last one alone.
      const int px = tx * TY + ty, py = tx * (TY + 1) + ty;
      const T mdx = upd[0], mdy = upd[1], mdz = upd[2], dt = upd[3],
              c0 = upd[4], c1 = upd[5];
      T out[NF];
      auto one = [&](auto o_tag, auto ddx, auto ddy, auto fhi, auto fl,
                     auto rhs, auto uk, auto u0) {
        using O = decltype(o_tag);
        rhs = O::fma(ddx, O::splat(mdx), rhs);
        rhs = O::fma(ddy, O::splat(mdy), rhs);
        rhs = O::fma(O::sub(fhi, fl), O::splat(mdz), rhs);
        if (a.mode == SWC_OUT_RHS) return rhs;
        if (a.mode == SWC_OUT_EULER) return O::fma(rhs, O::splat(dt), uk);
        return O::fma(O::fma(rhs, O::splat(dt), O::sub(uk, u0)), O::splat(c1),
                      O::mul(u0, O::splat(c0)));
      };
#pragma unroll
      for (int j = 0; j < NFP; ++j) {
        const V2* const bx2 = reinterpret_cast<const V2*>(fx) + px + j * L::NX;
        const V2* const by2 = reinterpret_cast<const V2*>(fy) + py + j * L::NY;
        constexpr int kA[4] = {0, 1, 3, 6}, kB[4] = {4, 2, 5, 7};
        const int p = kA[j], q = kB[j];
        const V2 r = one(O2{}, O2::sub(bx2[TY], bx2[0]), O2::sub(by2[1], by2[0]),
                         O2::mk(fzr[p], fzr[q]), O2::mk(flo[p], flo[q]),
                         O2::mk(p < 5 ? src[p] : T(0), q < 5 ? src[q] : T(0)),
                         O2::mk(ukc[p], ukc[q]), O2::mk(u0c[p], u0c[q]));
        out[p] = r.x;
        out[q] = r.y;
      }
      if constexpr (NF & 1) {
        constexpr int p = NF == 5 ? 3 : NF - 1;
        const T* const bx1 = fx + 2 * NFP * L::NX + px;
        const T* const by1 = fy + 2 * NFP * L::NY + py;
        out[p] = one(O1{}, O1::sub(bx1[TY], bx1[0]), O1::sub(by1[1], by1[0]),
                     fzr[p], flo[p], p < 5 ? src[p] : T(0), ukc[p], u0c[p]);
      }
#pragma unroll
      for (int v = 0; v < NF; ++v) flo[v] = fzr[v];
#pragma unroll
      for (int v = 0; v < NF; ++v) static_cast<T*>(a.uout[v])[o] = out[v];
      if (a.dtmin_out) {
        T u, v, w, e, p, hh;
        cons_to_prim(out[0], out[1], out[2], out[3], out[4],
                     pe_of(xa_c, ya_c, azc), u, v, w, e, p, hh);
        T c = sqrt_(K<T>::gamma() * p / out[0]);
        T l = min_(min_(dx / (abs_(u) + c), dy / (abs_(v) + c)),
                   dz / (abs_(w) + c));
        dtmin_local =
            min_(dtmin_local, T(cfl_limit_or_flag(out[0], p, out[4], l)));
      }
    }
  }

  if (a.dtmin_out) {
    // Block min of the CFL limits, then one atomic per CTA.
    __shared__ double red[32];
    double m = fmin(double(dtmin_local), 1e300);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
      m = fmin(m, __shfl_xor_sync(0xffffffffu, m, off));
    if ((tid & 31) == 0) red[tid >> 5] = m;
    __syncthreads();
    if (tid < 32) {
      m = (tid < NT / 32) ? red[tid] : 1e300;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
        m = fmin(m, __shfl_xor_sync(0xffffffffu, m, off));
      if (tid == 0 && m < 1e300) atomic_min_pos(a.dtmin_out, m);
    }
  }
}

// Resident CTAs per SM the register budget is set for: the inviscid MUSCL
// stage in single precision is light enough (shared memory 70 KB) for three.
template <typename T, int SCHEME, bool VISC>
constexpr int stage_min_blocks() {
  return sizeof(T) == 4 ? ((SCHEME == 2 && !VISC) ? 3 : 2) : 1;
}

template <typename T, int SCHEME, int RIEMANN, bool VISC, int TY, int TX,
          bool PE>
__global__ void __launch_bounds__(TY* TX, (stage_min_blocks<T, SCHEME, VISC>()))
    stage_kernel(const StageArgs a) {
  stage_body<T, SCHEME, RIEMANN, VISC, TY, TX, PE>(
      a, nullptr, blockIdx.x * TY, blockIdx.y * TX, blockIdx.z);
}

// Tile and resident CTAs per SM of an extended stage, whose ring is larger by
// the scalars and p_dyn: the first of these that shared memory holds (228 KB
// per SM, 1 KB of it reserved per CTA). Two CTAs hide each other's barriers
// and four to six more warps hide latency: with one 16 x 16 CTA (8 warps) the
// issue slots were 27 % busy.
//   single precision: 2 x (16 x 16), 2 x (16 x 12), 1 x (16 x 24)
//   double precision: 1 x (16 x 16), 1 x (16 x 12), 1 x (8 x 16)
// EXT (face and flux overrides, few and small in practice) keeps one CTA and
// its registers.
struct ExtTile {
  int ty, tx, ctas;
};
template <typename T, int SCHEME, bool VISC, int NS, bool HELP, bool EXT>
constexpr ExtTile ext_tile() {
  constexpr size_t kSm = 228 * 1024, kCta = 1024 + 512;  // + static shared
  constexpr size_t s16 = Layout<T, SCHEME, VISC, 16, 16, NS, HELP>::SMEM + kCta;
  constexpr size_t s12 = Layout<T, SCHEME, VISC, 16, 12, NS, HELP>::SMEM + kCta;
  constexpr size_t s24 = Layout<T, SCHEME, VISC, 16, 24, NS, HELP>::SMEM + kCta;
  if (sizeof(T) == 4) {
    if (EXT) return {16, 16, 1};
    if (2 * s16 <= kSm) return {16, 16, 2};
    if (2 * s12 <= kSm) return {16, 12, 2};
    if (s24 <= kSm) return {16, 24, 1};
    return {16, 16, 1};
  }
  if (s16 <= kSm) return {16, 16, 1};
  if (s12 <= kSm) return {16, 12, 1};
  return {8, 16, 1};
}

// Extended stage: NS transported scalars, HELP reference states, EXT face and
// flux overrides on the grid boundary.
template <typename T, int SCHEME, int RIEMANN, bool VISC, int TY, int TX,
          int CTAS, int NS, bool HELP, bool EXT>
__global__ void __launch_bounds__(TY* TX, CTAS)
    stage_kernel_ext(const StageArgs a, const SwcStageExt e) {
  stage_body<T, SCHEME, RIEMANN, VISC, TY, TX, true, NS, HELP, EXT>(
      a, &e, blockIdx.x * TY, blockIdx.y * TX, blockIdx.z);
}

// Batched stage: the CTAs of up to SWC_BATCH_CHUNK independent grids in one
// launch. CTA t belongs to the member m with pre[m] <= t < pre[m+1]; its
// tiles are numbered y fastest, then x, then z segment. The member table
// travels in the launch parameters, so the launch needs no device memory
// of its own and is captured whole by a CUDA graph.
struct StageBatch {
  int n;
  int pre[SWC_BATCH_CHUNK + 1];
  StageArgs m[SWC_BATCH_CHUNK];
};

template <typename T, int SCHEME, int RIEMANN, bool VISC, int TY, int TX,
          bool PE>
__global__ void __launch_bounds__(TY* TX, sizeof(T) == 4 ? 2 : 1)
    stage_batch_kernel(const StageBatch b) {
  const int t = blockIdx.x;
  int lo = 0, hi = b.n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (b.pre[mid] <= t) lo = mid;
    else hi = mid;
  }
  // The member's record, copied to shared memory once per CTA, is read at
  // fixed addresses (no register holds a per-member offset).
  static_assert(sizeof(StageArgs) % 8 == 0, "StageArgs is copied as words");
  __shared__ StageArgs sa;
  {
    const long long* src = reinterpret_cast<const long long*>(&b.m[lo]);
    long long* dst = reinterpret_cast<long long*>(&sa);
    for (int i = threadIdx.x; i < (int)(sizeof(StageArgs) / 8); i += blockDim.x)
      dst[i] = src[i];
  }
  __syncthreads();
  const int local = t - b.pre[lo];
  const int nby = (sa.ny + TY - 1) / TY, nbx = (sa.nx + TX - 1) / TX;
  const int by = local % nby, rest = local / nby;
  stage_body<T, SCHEME, RIEMANN, VISC, TY, TX, PE>(
      sa, nullptr, by * TY, (rest % nbx) * TX, rest / nbx);
}

}  // namespace swc
