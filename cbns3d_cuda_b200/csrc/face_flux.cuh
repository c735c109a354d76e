// face_flux.cuh - numerical flux through one grid face: characteristic-wise
// WENO5-JS reconstruction in the Roe-averaged eigenbasis of the two adjacent
// nodes, followed by the local Lax-Friedrichs flux.
//
// Restates, per face, the arithmetic of the reference's
//   rec_riemann_{xi,eta,zeta}_kernel  src/rec_riemann_kernel.cu:15-247
//   calc_eigenvectors_roe             src/calc_eigenvectors_roe.cu:13-152
//   rec_weno5 / weno5                 src/weno.cu:13-120
//   lf_flux                           src/lf_flux.cu:13-80
// with the same basis construction (tangent (0,nz,-ny) unless its norm is
// below 1e-8), the same WENO5-JS weights (eps = 1e-6 inside beta, before
// squaring), the same Cartesian wave-speed bound of the LF dissipation, and the
// same use of the node primitives for the Roe average.  The algebra is
// reorganised for the GPU (all of it is exact rearrangement, so results agree to
// rounding):
//   * WENO5 in differences: a reconstructed value is the centre node's value
//     plus a combination of the five first differences g1..g5 of the stencil,
//     and the smoothness indicators are quadratic in the same differences.  The
//     projection is linear, so the five differences of the conservative states
//     are projected (not the six states, nor ten), and the projected-back
//     correction is added to the centre node's conservative state, which is
//     never projected.  The differences of neighbouring states carry less
//     rounding than combinations of the states themselves;
//   * the two sides share the four second differences of a field, whose squares
//     enter three indicators each; the indicators are kept times 4 (and times
//     the projection's scale squared), which the weights cancel;
//   * the left eigenvectors are applied through their structure
//     (w0,w2 = A +- B, w1 = f0 - 2A, w3,w4 = tangential momenta) and the right
//     eigenvectors likewise, instead of 5x5 matrix products; the second
//     tangent is the cross product of the unit normal and the first;
//   * an FP64 WENO5 value takes one reciprocal (weights scaled by the product of
//     the squared indicators);
//   * the Lax-Friedrichs flux is formed from the reconstructed conservative
//     values, each side's collected into one coefficient ((q_n +- ws)/2).
// About 690 FP64 instructions per face (projecting the states, with each side's
// indicators and IEEE divisions and roots, took about 1,150).  Every operation
// is an explicit fused multiply-add, multiply or add, so each compilation of
// the flux (stage kernels, their batched forms, the WENO5-face pass) rounds
// alike.  Bound by the FP64 pipe (FP64) and by issue (FP32).  Measured, one
// launch each: FP64 stage 2 on 256x256x128 2.19 -> 1.86 ms, FP32 stage 2 on
// 193x161x129 0.645 -> 0.480 ms, the WENO5-face pass of a 256x256x128 hybrid
// step 0.208 -> 0.171 ms; the error of a right-hand side against 80-bit
// arithmetic falls by 1.1 to 3 times (density and energy of a vortex 6.5e-15
// and 7.7e-14 -> 3.9e-15 and 4.3e-14 in FP64, 2.9e-6 and 3.6e-5 -> 2.1e-6 and
// 2.3e-5 with the FP32 flux).
//
// Reciprocals and square roots: FP32 uses the approximate hardware forms (PTX
// rcp.approx.ftz / rsqrt.approx.ftz / sqrt.approx.ftz, within 2 ulp): the FP32
// flux carries ~1e-7 relative error anyway.  FP64 starts from the hardware's
// 20-bit approximations and takes one third-order Householder iteration
// (A. S. Householder, The Numerical Treatment of a Single Nonlinear Equation,
// 1970), three and five fused operations, which leaves at most 1 unit in the
// last place (reciprocal) or 2 (roots) where the library's correctly rounded
// forms cost several times as much; the flux is no further from 80-bit
// arithmetic for it (above).  Values stored or compared outside the flux (the
// primitives, the spectral radius) use the correctly rounded forms.
// R is the arithmetic type (double for the plain path, float for the split path).
#pragma once

#include <cuda_runtime.h>

namespace cbns {

template <typename R>
struct FluxConsts {
  R gamma, gam1, gam1_inv;
};

// one rounding each, never contracted
__device__ __forceinline__ double fm(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fm(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double ml(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float ml(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double ad(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float ad(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double sb(double a, double b) { return __dadd_rn(a, -b); }
__device__ __forceinline__ float sb(float a, float b) { return __fadd_rn(a, -b); }

// Two faces at once: each operation one packed FP32 instruction (two
// correctly rounded results), half the instructions to issue.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 mk(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void halves(F2 x, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ F2 fm(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 ml(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 ad(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 sb(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}

// The element type of R, and a constant of type R.
template <typename R>
struct Elem {
  using T = R;
  static constexpr bool pair = false;
};
template <>
struct Elem<F2> {
  using T = float;
  static constexpr bool pair = true;
};
template <typename R>
__device__ __forceinline__ R cst(double x) {
  if constexpr (Elem<R>::pair) return mk((float)x, (float)x);
  else return (R)x;
}
// a*b - c, -x and 2a - b: the sign costs a packed operation, a scalar one nothing
template <typename R>
__device__ __forceinline__ R fms(R a, R b, R c) {
  if constexpr (Elem<R>::pair) return sb(ml(a, b), c);
  else return fm(a, b, -c);
}
template <typename R>
__device__ __forceinline__ R neg(R x) {
  if constexpr (Elem<R>::pair) return ml(x, cst<R>(-1.0));
  else return -x;
}
template <typename R>
__device__ __forceinline__ R twice_less(R a, R b) {
  if constexpr (Elem<R>::pair) return sb(ad(a, a), b);
  else return fm(R(2), a, -b);
}

// 1/x.  FP64: r(1 + e + e^2) with e = 1 - x r, r the 20-bit approximation (error e^3 ~ 2^-60).
__device__ __forceinline__ double rcp_(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fm(-x, r, 1.0);
  return fm(r, fm(e, e, e), r);
}
__device__ __forceinline__ float rcp_(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// 1/sqrt(x).  FP64: y(1 + e/2 + 3e^2/8) with e = 1 - x y^2.
__device__ __forceinline__ double rsqrt_(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fm(ml(-x, y), y, 1.0);
  return fm(ml(y, e), fm(0.375, e, 0.5), y);
}
__device__ __forceinline__ float rsqrt_(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// sqrt(x); FP64: x rsqrt(x), 0 at 0
__device__ __forceinline__ double sqrt_(double x) { return x == 0.0 ? x : ml(x, rsqrt_(x)); }
__device__ __forceinline__ float sqrt_(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The same half by half for two faces; |u| + c, max and c|x| (fmax drops a NaN).
template <typename F>
__device__ __forceinline__ F2 each(F2 x, const F& f) {
  float a, b;
  halves(x, a, b);
  return mk(f(a), f(b));
}
template <typename F>
__device__ __forceinline__ F2 each(F2 x, F2 y, const F& f) {
  float a, b, c, d;
  halves(x, a, b);
  halves(y, c, d);
  return mk(f(a, c), f(b, d));
}
__device__ __forceinline__ F2 rcp_(F2 x) {
  return each(x, [](float a) { return rcp_(a); });
}
__device__ __forceinline__ F2 rsqrt_(F2 x) {
  return each(x, [](float a) { return rsqrt_(a); });
}
__device__ __forceinline__ F2 sqrt_(F2 x) {
  return each(x, [](float a) { return sqrt_(a); });
}
template <typename T>
__device__ __forceinline__ T abs_add(T u, T c) {
  return ad(fabs(u), c);
}
__device__ __forceinline__ F2 abs_add(F2 u, F2 c) {
  return each(u, c, [](float a, float b) { return ad(fabsf(a), b); });
}
template <typename T>
__device__ __forceinline__ T max_(T a, T b) {
  return fmax(a, b);
}
__device__ __forceinline__ F2 max_(F2 a, F2 b) {
  return each(a, b, [](float x, float y) { return fmaxf(x, y); });
}
template <typename T>
__device__ __forceinline__ T half_abs(T x) {
  return ml(T(0.5), fabs(x));
}
__device__ __forceinline__ F2 half_abs(F2 x) {
  return each(x, [](float a) { return ml(0.5f, fabsf(a)); });
}

// Scale of the differences WENO5 works on: in FP32 the indicators and the squares
// of their reciprocals stay in range for differences up to 1e10 (eps enters at
// 4e-9); FP64 takes the 1/6 of the candidate values here.
template <typename R>
struct WenoScale {
  static constexpr bool d = sizeof(typename Elem<R>::T) == 8;
  static constexpr double s = d ? 1.0 / 6.0 : 1.0 / 32.0;  // of the projected differences
  static constexpr double post = d ? 1.0 : 32.0 / 6.0;     // of the correction
};

// WENO5-JS of one field from its differences g1..g5 (scaled): the correction
// to the centre value of the low side (stencil points 0..4, centre 2) and
// minus that of the high side (points 5..1, centre 3), before WenoScale::post.
// eps4 = 4 eps scale^2.
template <typename R>
__device__ __forceinline__ void weno5_pair(R g1, R g2, R g3, R g4, R g5, R eps4, R* lo, R* mhi) {
  const R c = cst<R>(13.0 / 3.0), two = cst<R>(2.0);
  const R d1 = sb(g2, g1), d2 = sb(g3, g2), d3 = sb(g3, g4), d4 = sb(g4, g5);  // d3, d4 negated
  const R t1 = fm(ml(c, d1), d1, eps4), t2 = fm(ml(c, d2), d2, eps4);
  const R t3 = fm(ml(c, d3), d3, eps4), t4 = fm(ml(c, d4), d4, eps4);
  auto side = [](R e1, R e2, R e3, R t1, R t2, R t3, R gn, R gc, R* out) {
    // gn, gc: the difference next to the far pair and the one across the face
    const R s1 = fm(e1, e1, t1), s2 = fm(e2, e2, t2), s3 = fm(e3, e3, t3);
    // the weights' square roots, up to a common factor.  FP64: one reciprocal in
    // all.  FP32: one per indicator -- products of two indicators, squared, leave
    // the range from differences of 2e5 on; scaling them back into it took
    // longer (split 193x161x129, 40 steps: 66.0 ms with the bare products, 69.8
    // scaled, 67.9 with the reciprocals).
    R p1, p2, p3;
    if constexpr (sizeof(typename Elem<R>::T) == 4) {
      p1 = rcp_(s1);
      p2 = rcp_(s2);
      p3 = rcp_(s3);
    } else {
      p1 = ml(s2, s3);
      p2 = ml(s1, s3);
      p3 = ml(s1, s2);
    }
    const R u1 = ml(p1, p1), u2 = ml(cst<R>(6.0), ml(p2, p2)), u3 = ml(cst<R>(3.0), ml(p3, p3));
    const R q1 = twice_less(e1, gn), q2 = ad(e2, gc), q3 = ad(e3, gc);
    const R n = fm(u3, q3, fm(u2, q2, ml(u1, q1)));
    *out = ml(n, rcp_(ad(u3, ad(u2, u1))));
  };
  side(fm(two, g2, d1), ad(g2, g3), fm(two, g3, d3), t1, t2, t3, g2, g3, lo);
  side(fm(two, g4, d4), ad(g3, g4), fm(two, g3, d2), t4, t3, t2, g4, g3, mhi);
}

// Local Lax-Friedrichs flux from the two reconstructed conservative states
// (the reference's lf_flux with R = the high side H, L = the low side): the
// component-wise Cartesian wave-speed bound, flux = (F_L + F_H - ws (U_H -
// U_L)) / 2.
template <typename R>
__device__ __forceinline__ void lf_flux(const R L[5], const R H[5], R nx, R ny, R nz,
                                        const FluxConsts<typename Elem<R>::T>& C, R out[5]) {
  R pL, hL, sLx, sLy, sLz, pH, hH, sHx, sHy, sHz;  // pressure, q_n / 2, |u_i| + c
  const R half = cst<R>(0.5), gam1 = cst<R>(C.gam1), gamma = cst<R>(C.gamma);
  auto side = [&](const R q[5], R& p, R& h, R& sx, R& sy, R& sz) {
    const R i = rcp_(q[0]);
    const R u = ml(q[1], i), v = ml(q[2], i), w = ml(q[3], i);
    p = ml(gam1, fm(cst<R>(-0.5), fm(q[3], w, fm(q[2], v, ml(q[1], u))), q[4]));
    const R c = sqrt_(ml(ml(gamma, p), i));
    h = ml(half, fm(w, nz, fm(v, ny, ml(u, nx))));
    sx = abs_add(u, c);
    sy = abs_add(v, c);
    sz = abs_add(w, c);
  };
  side(L, pL, hL, sLx, sLy, sLz);
  side(H, pH, hH, sHx, sHy, sHz);
  const R ws = half_abs(fm(max_(sHz, sLz), nz, fm(max_(sHy, sLy), ny, ml(max_(sHx, sLx), nx))));
  const R a = ad(hL, ws), b = sb(hH, ws), hp = ml(half, ad(pL, pH));
  out[0] = fm(H[0], b, ml(L[0], a));
  out[1] = fm(hp, nx, fm(H[1], b, ml(L[1], a)));
  out[2] = fm(hp, ny, fm(H[2], b, ml(L[2], a)));
  out[3] = fm(hp, nz, fm(H[3], b, ml(L[3], a)));
  out[4] = fm(pH, hH, fm(pL, hL, fm(H[4], b, ml(L[4], a))));
}

// First unit tangent l of the face normal n, yz = ny^2 + nz^2.
template <typename R>
__device__ __forceinline__ void tangent(R nx, R ny, R nz, R yz, R& lx, R& ly, R& lz) {
  if (yz > R(1.0e-16)) {
    const R il = rsqrt_(yz);
    lx = R(0);
    ly = ml(nz, il);
    lz = ml(-ny, il);
  } else {
    const R il = rsqrt_(fm(nz, nz, ml(nx, nx)));
    lx = ml(-nz, il);
    ly = R(0);
    lz = ml(nx, il);
  }
}
__device__ __forceinline__ void tangent(F2 nx, F2 ny, F2 nz, F2 yz, F2& lx, F2& ly, F2& lz) {
  float x0, x1, y0, y1, z0, z1, s0, s1, a0, a1, b0, b1, c0, c1;
  halves(nx, x0, x1);
  halves(ny, y0, y1);
  halves(nz, z0, z1);
  halves(yz, s0, s1);
  tangent(x0, y0, z0, s0, a0, b0, c0);
  tangent(x1, y1, z1, s1, a1, b1, c1);
  lx = mk(a0, a1);
  ly = mk(b0, b1);
  lz = mk(c0, c1);
}

// Flux through the face between stencil points 2 (node a) and 3 (node b).
// ld(p, n) returns conservative variable n at stencil point p (p = 0..5 are the
// nodes a-2 .. b+2 along the face normal).  (nx,ny,nz) is the face area vector
// 0.5*(J grad(xi)|_a + J grad(xi)|_b).  out[0..4] receives the flux.
template <typename R, typename LD>
__device__ __forceinline__ void face_flux(const LD& ld, R nx, R ny, R nz, const FluxConsts<typename Elem<R>::T>& C,
                                          R out[5]) {
  const R half = cst<R>(0.5);
  // orthonormal basis (n, l, m): u, l, m = u x l
  R ux, uy, uz, lx, ly, lz;
  {
    const R yz = fm(nz, nz, ml(ny, ny));
    const R in = rsqrt_(fm(nx, nx, yz));
    ux = ml(nx, in);
    uy = ml(ny, in);
    uz = ml(nz, in);
    tangent(nx, ny, nz, yz, lx, ly, lz);
  }
  const R mx = fms(uy, lz, ml(uz, ly)), my = fms(uz, lx, ml(ux, lz)), mz = fms(ux, ly, ml(uy, lx));

  // Roe averages of the node primitives at a and b (the reference reads them
  // from the primitive arrays, which hold exactly these values on every node a
  // face touches)
  R uu, vv, ww, H, hq, c, ic, qn, ql, qm;
  {
    const R gam1 = cst<R>(C.gam1);
    auto node = [&](int p, R& i, R& u, R& v, R& w, R& h) {
      i = rcp_(ld(p, 0));
      u = ml(ld(p, 1), i);
      v = ml(ld(p, 2), i);
      w = ml(ld(p, 3), i);
      const R E = ld(p, 4), k = fm(ld(p, 3), w, fm(ld(p, 2), v, ml(ld(p, 1), u)));
      h = ml(fm(gam1, fm(cst<R>(-0.5), k, E), E), i);
    };
    R ia, ua, va, wa, Ha, ib, ub, vb, wb, Hb;
    node(2, ia, ua, va, wa, Ha);
    node(3, ib, ub, vb, wb, Hb);
    const R sr = sqrt_(ml(ld(3, 0), ia));
    const R is = rcp_(ad(cst<R>(1.0), sr));
    uu = ml(fm(sr, ub, ua), is);
    vv = ml(fm(sr, vb, va), is);
    ww = ml(fm(sr, wb, wa), is);
    H = ml(fm(sr, Hb, Ha), is);
    hq = ml(half, fm(ww, ww, fm(vv, vv, ml(uu, uu))));
    const R c2 = ml(gam1, sb(H, hq));
    ic = rsqrt_(c2);
    c = ml(c2, ic);
    qn = fm(ww, uz, fm(vv, uy, ml(uu, ux)));
    ql = fm(ww, lz, fm(vv, ly, ml(uu, lx)));
    qm = fm(ww, mz, fm(vv, my, ml(uu, mx)));
  }

  // characteristic projection of the five differences and WENO5 per field, in
  // two groups (acoustic and entropy fields, which share A and B; shear
  // fields), which keeps at most 15 projected values live
  constexpr double S = WenoScale<R>::s, P = WenoScale<R>::post;
  R wl[5], wh[5];
  {
    R W[3][5];
    {
      const R K = ml(cst<R>(S * (double)C.gam1), ml(ic, ic));  // 2 S (gamma-1)/(2 c^2)
      const R nK = neg(K);
      const R a0 = ml(K, hq), a1 = ml(nK, uu), a2 = ml(nK, vv), a3 = ml(nK, ww);
      const R nh = ml(cst<R>(-0.5 * S), ic);
      const R b0 = neg(ml(nh, qn)), b1 = ml(nh, ux), b2 = ml(nh, uy), b3 = ml(nh, uz);
#pragma unroll
      for (int p = 0; p < 5; ++p) {
        const R g0 = sb(ld(p + 1, 0), ld(p, 0)), g1 = sb(ld(p + 1, 1), ld(p, 1)), g2 = sb(ld(p + 1, 2), ld(p, 2)),
                g3 = sb(ld(p + 1, 3), ld(p, 3)), g4 = sb(ld(p + 1, 4), ld(p, 4));
        const R A = fm(a3, g3, fm(a2, g2, fm(a1, g1, fm(a0, g0, ml(K, g4)))));  // 2 A
        const R B = fm(b3, g3, fm(b2, g2, fm(b1, g1, ml(b0, g0))));
        W[0][p] = fm(half, A, B);
        W[1][p] = fms(cst<R>(S), g0, A);
        if constexpr (Elem<R>::pair) W[2][p] = sb(A, W[0][p]);
        else W[2][p] = fms(half, A, B);
      }
    }
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      weno5_pair(W[s][0], W[s][1], W[s][2], W[s][3], W[s][4], cst<R>(4.0e-6 * S * S), &wl[s], &wh[s]);
      if constexpr (P == 1.0) {
        wh[s] = neg(wh[s]);
      } else {
        wl[s] = ml(cst<R>(P), wl[s]);
        wh[s] = ml(cst<R>(-P), wh[s]);
      }
    }
  }
  {
    // FP64: unscaled here, the corrections scaled (4 products instead of 8)
    constexpr double T = P == 1.0 ? 1.0 : S, Q = P == 1.0 ? S : P;
    R W[2][5];
    const R sc = cst<R>(T), nsc = cst<R>(-T);
    const R l1 = ml(sc, lx), l2 = ml(sc, ly), l3 = ml(sc, lz), l0 = ml(nsc, ql);
    const R m1 = ml(sc, mx), m2 = ml(sc, my), m3 = ml(sc, mz), m0 = ml(nsc, qm);
#pragma unroll
    for (int p = 0; p < 5; ++p) {
      const R g0 = sb(ld(p + 1, 0), ld(p, 0)), g1 = sb(ld(p + 1, 1), ld(p, 1)), g2 = sb(ld(p + 1, 2), ld(p, 2)),
              g3 = sb(ld(p + 1, 3), ld(p, 3));
      W[0][p] = fm(l3, g3, fm(l2, g2, fm(l1, g1, ml(l0, g0))));
      W[1][p] = fm(m3, g3, fm(m2, g2, fm(m1, g1, ml(m0, g0))));
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      weno5_pair(W[s][0], W[s][1], W[s][2], W[s][3], W[s][4], cst<R>(4.0e-6 * T * T), &wl[3 + s], &wh[3 + s]);
      wl[3 + s] = ml(cst<R>(Q), wl[3 + s]);
      wh[3 + s] = ml(cst<R>(-Q), wh[3 + s]);
    }
  }

  // the corrections back to conservative variables, added to the centre nodes
  R L[5], Hs[5];
  auto back = [&](int p, const R* w, R* q) {
    const R s = ad(w[0], w[2]), d = ml(sb(w[2], w[0]), c), r = ad(s, w[1]);
    q[0] = ad(ld(p, 0), r);
    q[1] = fm(mx, w[4], fm(lx, w[3], fm(ux, d, fm(uu, r, ld(p, 1)))));
    q[2] = fm(my, w[4], fm(ly, w[3], fm(uy, d, fm(vv, r, ld(p, 2)))));
    q[3] = fm(mz, w[4], fm(lz, w[3], fm(uz, d, fm(ww, r, ld(p, 3)))));
    q[4] = fm(qm, w[4], fm(ql, w[3], fm(hq, w[1], fm(qn, d, fm(H, s, ld(p, 4))))));
  };
  back(2, wl, L);
  back(3, wh, Hs);
  lf_flux<R>(L, Hs, nx, ny, nz, C, out);
}

// Flux through the same face with the linear upwind-biased 5th-order
// reconstruction of each conservative variable (the WENO5 candidate values
// combined with the ideal weights 0.1/0.6/0.3: (2a - 13b + 47c + 27d - 3e)/60).
// With ideal weights the characteristic projection cancels (it is linear and
// the same for every stencil point), so this equals characteristic WENO5
// wherever the nonlinear weights sit at their linear values -- the faces the
// learned sensor sends here.  Same Lax-Friedrichs flux as face_flux.
template <typename R, typename LD>
__device__ __forceinline__ void face_flux_linear(const LD& ld, R nx, R ny, R nz,
                                                 const FluxConsts<typename Elem<R>::T>& C, R out[5]) {
  const R k60 = cst<R>(1.0 / 60.0), c2 = cst<R>(2.0), c13 = cst<R>(-13.0), c47 = cst<R>(47.0), c27 = cst<R>(27.0),
          c3 = cst<R>(-3.0);
  R ql[5], qh[5];
#pragma unroll
  for (int n = 0; n < 5; ++n) {
    const R f0 = ld(0, n), f1 = ld(1, n), f2 = ld(2, n), f3 = ld(3, n), f4 = ld(4, n), f5 = ld(5, n);
    ql[n] = ml(fm(c3, f4, fm(c27, f3, fm(c47, f2, fm(c13, f1, ml(c2, f0))))), k60);
    qh[n] = ml(fm(c3, f1, fm(c27, f2, fm(c47, f3, fm(c13, f4, ml(c2, f5))))), k60);
  }
  lf_flux<R>(ql, qh, nx, ny, nz, C, out);
}

}  // namespace cbns
