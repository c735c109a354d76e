// sigma.cuh - the spectral radius of a node (src/time_step_kernel.cu:13-96) and
// a cheap FP32 bound above it.
//
// dt needs the largest FP64 spectral radius of the grid, and evaluating it at
// every node (about 70 FP64 operations with four square roots) costs stage 3 a
// tenth of its time in FP64 (1829 -> 1707 us on 256x256x128) and a fifth in the
// hybrid (584 -> 458).  Most nodes are far below the largest value already found,
// so a node is evaluated in FP64 only if its FP32 bound reaches it, or if its
// squared sound speed is not safely positive in FP32 (the FP64 value may be a
// NaN, which must end the run): the result is the same to the bit.
#pragma once

#include "cbns_common.cuh"
#include "face_flux.cuh"

namespace cbns {

__device__ __forceinline__ float abs_(float x) { return fabsf(x); }
__device__ __forceinline__ F2 abs_(F2 x) {
  return each(x, [](float a) { return fabsf(a); });
}

__device__ __forceinline__ float min_(float x, float y) { return fminf(x, y); }
__device__ __forceinline__ F2 min_(F2 x, F2 y) {
  return each(x, y, [](float a, float b) { return fminf(a, b); });
}

// An upper bound of the spectral radius of a node (or two): q its state, A its
// area vectors J*grad(xi|eta|zeta), iJ = 1/J, all rounded to FP32.  The
// pressure E - rho u^2/2 carries rounding of E's size, so 1e-6 of E is added to
// it; |u.A| carries rounding of |u||A|'s size, so 1e-6 (|u|+|v|+|w|) is added to
// the sound speed; the remaining 40 roundings are covered by the factor 1 +
// 2e-5.  small: the least of the |A|^2 (below 1e-30 a square root flushes to zero
// and the bound holds nothing) and of c^2 less 2.5e-6 gamma (gamma-1) |E|/rho.
// The padded pressure exceeds the FP64 one by at most 1.7e-6 of E ((gamma-1)
// aside), so a node whose FP64 pressure is not positive has a negative small;
// an ordinary node comes near that only above Mach 1000.
template <typename R>
__device__ __forceinline__ R sigma_bound(const R q[5], const R A[9], R iJ, float gamma, float gam1, R& small) {
  const R i = rcp_(q[0]);
  const R u = ml(q[1], i), v = ml(q[2], i), w = ml(q[3], i);
  const R k = fm(q[3], w, fm(q[2], v, ml(q[1], u)));
  const R p = ml(cst<R>(gam1), fm(cst<R>(-0.5), k, ml(cst<R>(1.0 + 1.0e-6), q[4])));
  const R c2 = ml(ml(cst<R>(gamma), p), i);
  const R c = fm(cst<R>(1.0e-6), ad(abs_(u), ad(abs_(v), abs_(w))), sqrt_(c2));
  small = fm(cst<R>(-2.5e-6 * gamma * gam1), abs_(ml(q[4], i)), c2);
  R s = cst<R>(0.0);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const R x = A[3 * d], y = A[3 * d + 1], z = A[3 * d + 2];
    const R nn = fm(z, z, fm(y, y, ml(x, x)));
    small = min_(small, nn);
    s = ad(s, fm(c, sqrt_(nn), abs_(fm(w, z, fm(v, y, ml(u, x))))));
  }
  return ml(s, ml(abs_(iJ), cst<R>(1.0 + 2.0e-5)));
}

// Whether a node with bound b may reach `found`, a spectral radius already met
// (a lower bound of the maximum).  NaN: yes.
__device__ __forceinline__ bool sigma_reaches(float b, float small, float found) {
  return !(b < found) || !(small > 1.0e-30f);
}

// The spectral radius in FP64, correctly rounded divisions and roots and explicit
// roundings: every kernel gives the same.
__device__ __forceinline__ double sigma_exact(const double q[5], const double A[9], double iJ, double gamma,
                                              double gam1) {
  const double r = q[0], ir = __drcp_rn(r);
  const double uu = __dmul_rn(q[1], ir), vv = __dmul_rn(q[2], ir), ww = __dmul_rn(q[3], ir);
  const double k = __fma_rn(ww, ww, __fma_rn(vv, vv, __dmul_rn(uu, uu)));
  const double pp = __dmul_rn(gam1, __fma_rn(-__dmul_rn(0.5, r), k, q[4]));
  const double cs = __dsqrt_rn(__ddiv_rn(__dmul_rn(gamma, pp), r));
  double s = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {  // grad(xi|eta|zeta) = A / J
    const double x = __dmul_rn(A[3 * d], iJ), y = __dmul_rn(A[3 * d + 1], iJ), z = __dmul_rn(A[3 * d + 2], iJ);
    const double un = __fma_rn(ww, z, __fma_rn(vv, y, __dmul_rn(uu, x)));
    const double nn = __fma_rn(z, z, __fma_rn(y, y, __dmul_rn(x, x)));
    s = __dadd_rn(s, __dadd_rn(fabs(un), __dmul_rn(cs, __dsqrt_rn(nn))));
  }
  return s;
}

// The largest spectral radius a CTA (or an earlier one) has met, as an FP32
// value not above it, in shared memory: positive floats order like their bits.
__device__ __forceinline__ float sigma_start(const StepState* st) {
  const unsigned long long b = *(const volatile unsigned long long*)&st->sigma_bits;
  const double s = __longlong_as_double((long long)b);
  return s == s ? __double2float_rd(s) : 0.f;
}
__device__ __forceinline__ void sigma_found(int* best, double s) {
  if (s == s) atomicMax(best, __float_as_int(__double2float_rd(s)));
}

}  // namespace cbns
