// Device physics of the WENO-FD hot path, templated on the arithmetic type.
//
// With T = double and the translation unit built with -fmad=false, every
// expression below rounds exactly like the reference compiled without FMA
// contraction: operands are combined in the reference's evaluation order
// (C++ left-to-right), divisions and square roots are IEEE correctly rounded,
// and common subexpressions are shared only where the reference computes the
// identical operation on identical operands.  Citations are to files of
// infinity-07/FD-WENO-EulerEquation.
#pragma once

#include "approx.cuh"
#include "int_f64.cuh"
#include "wenofd_internal.h"

namespace wenofd {
namespace dev {

__device__ __forceinline__ double tsqrt(double x) { return sqrt(x); }
// FP32: the units of the FP32 forms are compiled with -prec-sqrt=false, so
// this is the hardware approximation there (about 1 ulp).
__device__ __forceinline__ float tsqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double tabs(double x) { return fabs(x); }
__device__ __forceinline__ float tabs(float x) { return fabsf(x); }

// Division.  FP64: IEEE '/'.  FP32 form: __fdividef, reciprocal times
// numerator (about 2 ulp; the FP32 form is not bitwise and does not need
// IEEE rounding).
__device__ __forceinline__ double tdiv(double a, double b) { return a / b; }
__device__ __forceinline__ float tdiv(float a, float b) { return __fdividef(a, b); }

// Pressure from conserved variables (utils/equations.hpp:108-112):
// p = (gamma - 1) * (E - 0.5 * rho * (u*u + v*v)), u = U1/U0, v = U2/U0.
template <typename T>
__device__ __forceinline__ void primitives(T gamma, const T U[4], T &u, T &v, T &p) {
  u = tdiv(U[1], U[0]);
  v = tdiv(U[2], U[0]);
  p = (gamma - T(1.0)) * (U[3] - T(0.5) * U[0] * (u * u + v * v));
}

// fluxSplitX / fluxSplitY (utils/equations.hpp:365-393) with getPhyFluxX/Y
// (105-134) and getMaxEigenValueX/Y (149-171): pointwise Lax-Friedrichs,
// F+- = 0.5 * (F +- (|u_n| + c) U).
template <typename T, int DIR>
__device__ __forceinline__ void flux_split(T gamma, const T U[4], T fm[4], T fp[4]) {
  T u, v, p;
  primitives(gamma, U, u, v, p);
  const T rho = U[0], E = U[3];
  T F[4];
  if (DIR == 0) {
    F[0] = rho * u;
    F[1] = rho * u * u + p;
    F[2] = rho * u * v;
    F[3] = (E + p) * u;
  } else {
    F[0] = rho * v;
    F[1] = rho * u * v;
    F[2] = rho * v * v + p;
    F[3] = (E + p) * v;
  }
  const T c = tsqrt(tdiv(gamma * p, rho));
  const T ws = (DIR == 0 ? tabs(u) : tabs(v)) + c;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    fm[r] = T(0.5) * (F[r] - ws * U[r]);
    fp[r] = T(0.5) * (F[r] + ws * U[r]);
  }
}

// Packed FP32 pairs: Blackwell issues two FP32 adds, multiplies or FMAs of a
// float2 as one instruction (round-to-nearest each, as the scalar forms).
// The FP32 forms run independent chains on pairs: the (x, y) and (z, w)
// halves of a node's float4 (stage_f32.cuh), and the two sides of a
// characteristic field's reconstruction (weno2 below).
__device__ __forceinline__ float2 lo2(const float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float4 join2(const float2 a, const float2 b) { return make_float4(a.x, a.y, b.x, b.y); }
__device__ __forceinline__ float2 splat2(float a) { return make_float2(a, a); }
// a - b, exactly as the scalar subtraction rounds it
__device__ __forceinline__ float2 sub2(const float2 a, const float2 b) { return __ffma2_rn(b, splat2(-1.0f), a); }

// ---------------------------------------------------------------- WENO

// Smoothness indicators shared by all four schemes (include/Utility.hpp
// 427-437, 465-475): beta = 13/12 t1^2 + 1/4 t2^2 evaluated as
// ((13/12*t1)*t1) + ((1/4*t2)*t2).
template <typename T>
__device__ __forceinline__ void betas(T a, T b, T c, T d, T e, T &bm, T &b0, T &bp) {
  const T c1312 = T(13.0 / 12.0), c14 = T(0.25);
  T t1 = (a - T(2.0) * b + c);
  T t2 = (a - T(4.0) * b + T(3.0) * c);
  bm = c1312 * t1 * t1 + c14 * t2 * t2;
  t1 = (b - T(2.0) * c + d);
  t2 = (b - d);
  b0 = c1312 * t1 * t1 + c14 * t2 * t2;
  t1 = (c - T(2.0) * d + e);
  t2 = (T(3.0) * c - T(4.0) * d + e);
  bp = c1312 * t1 * t1 + c14 * t2 * t2;
}

// Candidate values p0..p2 at x_{i+1/2} (include/Utility.hpp:499-501).
template <typename T>
__device__ __forceinline__ T combine(T w0, T w1, T w2, T a, T b, T c, T d, T e) {
  const T c13 = T(1.0 / 3.0), c16 = T(1.0 / 6.0), c56 = T(5.0 / 6.0), c76 = T(7.0 / 6.0), c116 = T(11.0 / 6.0);
  const T p0 = c13 * a - c76 * b + c116 * c;
  const T p1 = -c16 * b + c56 * c + c13 * d;
  const T p2 = c13 * c + c56 * d - c16 * e;
  return w0 * p0 + w1 * p1 + w2 * p2;
}

// WENO-JS, include/Utility.hpp:415-456 (eps = 1e-6).
template <typename T>
__device__ __forceinline__ T weno_js(T a, T b, T c, T d, T e) {
  T b0, b1, b2;
  betas(a, b, c, d, e, b0, b1, b2);
  const T eps = T(1.0e-6);
  T w0 = tdiv(T(0.1), ((eps + b0) * (eps + b0)));
  T w1 = tdiv(T(0.6), ((eps + b1) * (eps + b1)));
  T w2 = tdiv(T(0.3), ((eps + b2) * (eps + b2)));
  const T sum = w0 + w1 + w2;
  w0 = tdiv(w0, sum);
  w1 = tdiv(w1, sum);
  w2 = tdiv(w2, sum);
  return combine(w0, w1, w2, a, b, c, d, e);
}

// WENO-Z, include/Utility.hpp:457-504 (eps = 1e-20).
//
// FP64: the weight products are taken left to right, tau*inv*tau*inv, as in
// the reference (lines 489-491), with no guard.  FP32: (tau/(beta+1e-20))^2
// overflows where a stencil is exactly flat (beta = 0) next to a jump, so the
// ratio r is capped at 1e18 before squaring (r^2 <= 1e36 stays finite); a
// weight that large already makes its stencil's normalised weight 1 to FP32
// precision, so the cap changes nothing else.
template <typename T>
__device__ __forceinline__ void wenoz_weights(T a, T b, T c, T d, T e, T &w0, T &w1, T &w2) {
  T bm, b0, bp;
  betas(a, b, c, d, e, bm, b0, bp);
  const T eps = T(1.0e-20);
  const T ibm = tdiv(T(1.0), (bm + eps));
  const T ib0 = tdiv(T(1.0), (b0 + eps));
  const T ibp = tdiv(T(1.0), (bp + eps));
  const T tau = tabs(bm - bp);
  if constexpr (sizeof(T) == 4) {
    const T rm = fminf(tau * ibm, 1.0e18f), r0 = fminf(tau * ib0, 1.0e18f), rp = fminf(tau * ibp, 1.0e18f);
    w0 = T(0.1) * (T(1.0) + rm * rm);
    w1 = T(0.6) * (T(1.0) + r0 * r0);
    w2 = T(0.3) * (T(1.0) + rp * rp);
  } else {
    w0 = T(0.1) * (T(1.0) + (tau * ibm * tau * ibm));
    w1 = T(0.6) * (T(1.0) + (tau * ib0 * tau * ib0));
    w2 = T(0.3) * (T(1.0) + (tau * ibp * tau * ibp));
  }
  const T ws = w0 + w1 + w2;
  w0 = tdiv(w0, ws);
  w1 = tdiv(w1, ws);
  w2 = tdiv(w2, ws);
}

template <typename T>
__device__ __forceinline__ T weno_z(T a, T b, T c, T d, T e) {
  T w0, w1, w2;
  wenoz_weights(a, b, c, d, e, w0, w1, w2);
  return combine(w0, w1, w2, a, b, c, d, e);
}

// pow(x, 2) of the reference's ZP/ZPI weights is evaluated as x*x, the
// correctly rounded square.  glibc's pow(x, 2) differs from it by one ulp on
// about 0.1% of inputs, so WENO-ZP/ZPI agree with the reference to rounding
// rather than bit for bit (WENO-JS and WENO-Z have no pow).
template <typename T> __device__ __forceinline__ T sq(T x) { return x * x; }

// FP32 ZP/ZPI: eps = 1e-40 is subnormal in FP32 and the weight ratios can
// exceed the FP32 range, so the FP32 form divides with IEEE '/' (subnormal
// safe) and caps each ratio term at 1e18 before it is squared or summed.
template <typename T> __device__ __forceinline__ T zdiv(T a, T b) { return tdiv(a, b); }
template <> __device__ __forceinline__ float zdiv<float>(float a, float b) { return fminf(a / b, 1.0e18f); }

// WENO-ZP, include/Utility.hpp:505-558 (eps = 1e-40; lambda = pow(dx, 2/3)).
template <typename T>
__device__ __forceinline__ T weno_zp(T a, T b, T c, T d, T e, T lambda) {
  T bm, b0, bp;
  betas(a, b, c, d, e, bm, b0, bp);
  const T tau = tabs(bm - bp);
  const T eps = T(1.0e-40);
  T w0 = T(0.1) * (T(1) + sq(zdiv((tau + eps), (bm + eps))) + zdiv(lambda * (bm + eps), (tau + eps)));
  T w1 = T(0.6) * (T(1) + sq(zdiv((tau + eps), (b0 + eps))) + zdiv(lambda * (b0 + eps), (tau + eps)));
  T w2 = T(0.3) * (T(1) + sq(zdiv((tau + eps), (bp + eps))) + zdiv(lambda * (bp + eps), (tau + eps)));
  const T sum = w0 + w1 + w2;
  w0 = tdiv(w0, sum);
  w1 = tdiv(w1, sum);
  w2 = tdiv(w2, sum);
  return combine(w0, w1, w2, a, b, c, d, e);
}

// WENO-ZPI, include/Utility.hpp:559-615 (lambda = 3.3, eps = 1e-40).
template <typename T>
__device__ __forceinline__ T weno_zpi(T a, T b, T c, T d, T e) {
  T bm, b0, bp;
  betas(a, b, c, d, e, bm, b0, bp);
  const T tau = tabs(bm - bp);
  const T lambda = T(3.3);
  const T mx_in = (b0 < bp) ? bp : b0;  // std::max(beta, betap)
  const T bmax = (bm < mx_in) ? mx_in : bm;
  const T mn_in = (bp < b0) ? bp : b0;  // std::min(beta, betap)
  const T bmin = (mn_in < bm) ? mn_in : bm;
  const T alpha = T(1) - zdiv(bmin, (bmax + T(1e-40)));
  const T eps = T(1.0e-40);
  T w0 = T(0.1) * (T(1) + sq(zdiv(tau, (bm + eps))) + zdiv(lambda * alpha * (bm), (bmax + eps)));
  T w1 = T(0.6) * (T(1) + sq(zdiv(tau, (b0 + eps))) + zdiv(lambda * alpha * (b0), (bmax + eps)));
  T w2 = T(0.3) * (T(1) + sq(zdiv(tau, (bp + eps))) + zdiv(lambda * alpha * (bp), (bmax + eps)));
  const T sum = w0 + w1 + w2;
  w0 = tdiv(w0, sum);
  w1 = tdiv(w1, sum);
  w2 = tdiv(w2, sum);
  return combine(w0, w1, w2, a, b, c, d, e);
}

// CWENOFD::useWENO (src/WENOFD.cpp:823-848), scheme fixed at compile time.
template <typename T, int SCHEME>
__device__ __forceinline__ T weno(T a, T b, T c, T d, T e, T zp_lambda) {
  if (SCHEME == kWenoJS) return weno_js(a, b, c, d, e);
  if (SCHEME == kWenoZ) return weno_z(a, b, c, d, e);
  if (SCHEME == kWenoZP) return weno_zp(a, b, c, d, e, zp_lambda);
  return weno_zpi(a, b, c, d, e);
}

// FP32 WENO-JS / WENO-Z on two stencils at once, used for the + and - sides of
// one characteristic field: the arithmetic runs on packed pairs (38 of them),
// the reciprocals and the caps per element.  Written for the FMA pipe, which
// bounds the FP32 form, on the stencil's differences d1..d4:
//   4 beta_k + 4 eps = B_k = 13/3 s_k^2 + (t_k^2 + 4 eps), s the second
//   differences and t = (d1 - 3 d2, d2 + d3, d4 - 3 d3);
//   ratios tau/beta from tau = B_0 - B_2 (squared, so unsigned), capped at 1e15
//   before squaring (a larger weight already makes its stencil's normalised
//   weight 1 to FP32 precision, and products with it stay finite);
//   the result c + sum alpha_k P_k / (6 sum alpha_k) with the candidates' 6 (p_k
//   - c) = (5 d2 - 2 d1, d2 + 2 d3, 4 d3 - d4), which also cancels less than the
//   candidates themselves.
// Explicitly rounded operations: every unit computes the same bits.
// The reciprocals, and the roots of the face's eigenvectors, are the bare
// hardware approximations (approx.cuh; B_k is never zero): with the division
// intrinsic's handling of subnormals one reconstruction takes 104 instructions
// instead of 65.
__device__ __forceinline__ float2 rcp2(float2 x) { return make_float2(rcp_ftz(x.x), rcp_ftz(x.y)); }

template <int SCHEME>
__device__ __forceinline__ float2 weno2(float2 a, float2 b, float2 c, float2 d, float2 e) {
  static_assert(SCHEME == kWenoJS || SCHEME == kWenoZ, "packed WENO-JS and WENO-Z only");
  const float2 d1 = sub2(b, a), d2 = sub2(c, b), d3 = sub2(d, c), d4 = sub2(e, d);
  const float2 s0 = sub2(d2, d1), s1 = sub2(d3, d2), s2 = sub2(d4, d3);
  const float2 m3 = splat2(-3.0f);
  const float2 t0 = __ffma2_rn(m3, d2, d1), t1 = __fadd2_rn(d2, d3), t2 = __ffma2_rn(m3, d3, d4);
  const float2 eps = splat2(SCHEME == kWenoZ ? 4.0e-20f : 4.0e-6f), c133 = splat2(float(13.0 / 3.0));
  const float2 B0 = __ffma2_rn(c133, __fmul2_rn(s0, s0), __ffma2_rn(t0, t0, eps));
  const float2 B1 = __ffma2_rn(c133, __fmul2_rn(s1, s1), __ffma2_rn(t1, t1, eps));
  const float2 B2 = __ffma2_rn(c133, __fmul2_rn(s2, s2), __ffma2_rn(t2, t2, eps));
  float2 r0 = rcp2(B0), r1 = rcp2(B1), r2 = rcp2(B2);
  float2 w0, w1, w2;  // alpha_0, -alpha_1, alpha_2, times 10
  if constexpr (SCHEME == kWenoZ) {
    const float2 tau = sub2(B0, B2);
    auto cap = [](float2 x) { return make_float2(fminf(fabsf(x.x), 1.0e15f), fminf(fabsf(x.y), 1.0e15f)); };
    r0 = cap(__fmul2_rn(tau, r0));
    r1 = cap(__fmul2_rn(tau, r1));
    r2 = cap(__fmul2_rn(tau, r2));
    w0 = __ffma2_rn(r0, r0, splat2(1.0f));
    w1 = __ffma2_rn(__fmul2_rn(splat2(-6.0f), r1), r1, splat2(-6.0f));
    w2 = __ffma2_rn(__fmul2_rn(splat2(3.0f), r2), r2, splat2(3.0f));
  } else {
    w0 = __fmul2_rn(r0, r0);
    w1 = __fmul2_rn(__fmul2_rn(splat2(-6.0f), r1), r1);
    w2 = __fmul2_rn(__fmul2_rn(splat2(3.0f), r2), r2);
  }
  const float2 isum = rcp2(sub2(__fadd2_rn(w0, w2), w1));
  const float2 q0 = __ffma2_rn(splat2(2.0f), t0, d2), q1 = __ffma2_rn(splat2(2.0f), d3, d2), q2 = sub2(t2, d3);
  const float2 num = __ffma2_rn(w1, q1, __ffma2_rn(w2, q2, __fmul2_rn(w0, q0)));
  return __ffma2_rn(__fmul2_rn(num, isum), splat2(float(-1.0 / 6.0)), c);
}

// The two sides of one characteristic field at a face: the + side on F+
// stencil values p0..p4, the - side on F- values mirrored (m4..m0), summed.
// FP64 evaluates them one after the other as the reference does; FP32
// WENO-JS and WENO-Z evaluate both at once on packed pairs.
template <typename T, int SCHEME>
__device__ __forceinline__ T weno_sides(const T vp[5], const T vm[5], T zp_lambda) {
  if constexpr (sizeof(T) == 4 && (SCHEME == kWenoJS || SCHEME == kWenoZ)) {
    const float2 r = weno2<SCHEME>(make_float2(vp[0], vm[4]), make_float2(vp[1], vm[3]), make_float2(vp[2], vm[2]),
                                   make_float2(vp[3], vm[1]), make_float2(vp[4], vm[0]));
    return r.x + r.y;
  } else {
    const T hp = weno<T, SCHEME>(vp[0], vp[1], vp[2], vp[3], vp[4], zp_lambda);
    const T hm = weno<T, SCHEME>(vm[4], vm[3], vm[2], vm[1], vm[0], zp_lambda);
    return hp + hm;
  }
}

// ------------------------------------------------------- one face flux

// Characteristic WENO flux at one face (src/WENOFD.cpp:526-643 in x,
// 668-791 in y): average state of the two nodes, L and R of the x- or
// y-Jacobian there (utils/equations.hpp:174-299), five projected F+ (nodes
// face-3..face+1) and five F- (face-2..face+2), one WENO per characteristic
// field and side (minus side mirrored), back-projection.  L and R are built
// from one set of (u, v, p, c, B1, B2, H): the reference recomputes them per
// matrix from the same inputs, which gives identical values.
//
// fp(s, r) / fm(s, r): component r of F+ at node face-3+s and of F- at node
// face-2+s, s = 0..4.
template <typename T>
struct StridedStencil {  // SoA: nodes `ss` elements apart, components `cs` apart
  const T *p;
  int ss, cs;
  __device__ __forceinline__ T operator()(int s, int r) const { return p[s * ss + r * cs]; }
};
template <typename T, int DIR, int SCHEME, typename St>
__device__ __forceinline__ void face_flux_st(T gamma, T zp_lambda, const T um[4], const T u0[4], const St &fp,
                                             const St &fm, T out[4]) {
  T ave[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) ave[r] = T(0.5) * (um[r] + u0[r]);
  T u, v, p;
  primitives(gamma, ave, u, v, p);
  const T rho = ave[0], E = ave[3];
  const T c = tsqrt(tdiv(gamma * p, rho));
  const T B1 = tdiv((gamma - T(1)), (c * c));
  const T B2 = B1 * (u * u + v * v) * T(0.5);
  const T H = tdiv((E + p), rho);
  const T ic = tdiv(T(1.0), c);
  const T nc = tdiv(DIR == 0 ? u : v, c);  // u/c in x, v/c in y
  const T B1u = B1 * u, B1v = B1 * v;

  T vh[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    T l0, l1, l2, l3;  // row k of the left eigenvector matrix
    if (DIR == 0) {
      if (k == 0) { l0 = (B2 + nc) * T(0.5); l1 = -(B1u + ic) * T(0.5); l2 = -(B1v) * T(0.5); l3 = B1 * T(0.5); }
      if (k == 1) { l0 = v; l1 = T(0); l2 = T(-1); l3 = T(0); }
      if (k == 2) { l0 = (T(1) - B2); l1 = B1u; l2 = B1v; l3 = -B1; }
      if (k == 3) { l0 = (B2 - nc) * T(0.5); l1 = -(B1u - ic) * T(0.5); l2 = -B1v * T(0.5); l3 = B1 * T(0.5); }
    } else {
      if (k == 0) { l0 = (B2 + nc) * T(0.5); l1 = -(B1u) * T(0.5); l2 = -(B1v + ic) * T(0.5); l3 = B1 * T(0.5); }
      if (k == 1) { l0 = -u; l1 = T(1); l2 = T(0); l3 = T(0); }
      if (k == 2) { l0 = T(1) - B2; l1 = B1u; l2 = B1v; l3 = -B1; }
      if (k == 3) { l0 = (B2 - nc) * T(0.5); l1 = -(B1u) * T(0.5); l2 = -(B1v - ic) * T(0.5); l3 = B1 * T(0.5); }
    }
    T vp[5], vm[5];
#pragma unroll
    for (int s = 0; s < 5; ++s) {
      T x = l0 * fp(s, 0);
      x += l1 * fp(s, 1);
      x += l2 * fp(s, 2);
      x += l3 * fp(s, 3);
      vp[s] = x;
      T y = l0 * fm(s, 0);
      y += l1 * fm(s, 1);
      y += l2 * fm(s, 2);
      y += l3 * fm(s, 3);
      vm[s] = y;
    }
    vh[k] = weno_sides<T, SCHEME>(vp, vm, zp_lambda);
  }

  // R * vh, rows in the reference's order (utils/equations.hpp:239-299).
  const T q2 = (u * u + v * v) * T(0.5);
  T R[4][4];
  if (DIR == 0) {
    R[0][0] = T(1);      R[0][1] = T(0);  R[0][2] = T(1); R[0][3] = T(1);
    R[1][0] = u - c;     R[1][1] = T(0);  R[1][2] = u;    R[1][3] = u + c;
    R[2][0] = v;         R[2][1] = T(-1); R[2][2] = v;    R[2][3] = v;
    R[3][0] = H - c * u; R[3][1] = -v;    R[3][2] = q2;   R[3][3] = H + c * u;
  } else {
    R[0][0] = T(1);      R[0][1] = T(0);  R[0][2] = T(1); R[0][3] = T(1);
    R[1][0] = u;         R[1][1] = T(1);  R[1][2] = u;    R[1][3] = u;
    R[2][0] = v - c;     R[2][1] = T(0);  R[2][2] = v;    R[2][3] = v + c;
    R[3][0] = H - c * v; R[3][1] = u;     R[3][2] = q2;   R[3][3] = H + c * v;
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    T f = R[r][0] * vh[0];
    f += R[r][1] * vh[1];
    f += R[r][2] * vh[2];
    f += R[r][3] * vh[3];
    out[r] = f;
  }
}

// ------------------------------------------------- FP32 face and split
//
// The FP32 forms' face flux and split, in as few FMA-pipe operations as the
// scheme needs (the FMA pipe and issue bound the FP32 form) and with explicitly
// rounded operations, so that the per-solve and batched kernels agree bit for
// bit.

// Quantities of the x- (DIR 0) or y-Jacobian at a face's average state: normal
// and tangential velocity, (u^2 + v^2)/2, sound speed and its inverse, enthalpy,
// (gamma - 1)/(2 c^2).
struct Eigen32 {
  float un, ut, k2, c, ic, H, b;
};
template <int DIR>
__device__ __forceinline__ Eigen32 eigen32(float gamma, const float4 um, const float4 u0) {
  const float g1 = __fadd_rn(gamma, -1.0f);
  const float ir = rcp_ftz(__fadd_rn(um.x, u0.x));  // halves of the sums cancel in quotients
  const float u = __fmul_rn(__fadd_rn(um.y, u0.y), ir), v = __fmul_rn(__fadd_rn(um.z, u0.z), ir);
  const float e = __fmul_rn(__fadd_rn(um.w, u0.w), ir);  // E / rho
  Eigen32 q;
  q.k2 = __fmul_rn(0.5f, __fmaf_rn(u, u, __fmul_rn(v, v)));
  const float h = __fmul_rn(g1, __fadd_rn(e, -q.k2));  // p / rho
  const float c2 = __fmul_rn(gamma, h);
  // one Newton step on the hardware's 1/c: L and R are inverses to rounding
  const float y = rsqrt_ftz(c2);
  q.ic = __fmaf_rn(__fmul_rn(0.5f, y), __fmaf_rn(__fmul_rn(-c2, y), y, 1.0f), y);
  q.c = __fmul_rn(c2, q.ic);
  q.H = __fadd_rn(e, h);
  q.b = __fmul_rn(__fmul_rn(0.5f, g1), __fmul_rn(q.ic, q.ic));
  q.un = DIR == 0 ? u : v;
  q.ut = DIR == 0 ? v : u;
  return q;
}

// Characteristic flux at a face (face_flux_st) from float4 nodes P, M (F+ at
// face-3.., F- at face-2.., `ss` apart).  Rows 0 and 3 of L are Q + D and Q - D
// with Q = (B1/2)((u^2+v^2)/2 f0 - u f1 - v f2 + f3) and D = (un f0 - fn)/(2c),
// row 2 is f0 - 2 Q: 10 operations a node instead of 16.  In y row 1 of L and
// column 1 of R change sign together.
template <int DIR, int SCHEME>
__device__ __forceinline__ float4 face_flux_f32(float gamma, float zpl, const float4 um, const float4 u0,
                                                const float4 *P, const float4 *M, int ss) {
  const Eigen32 g = eigen32<DIR>(gamma, um, u0);
  const float q0 = __fmul_rn(g.b, g.k2), qn = -__fmul_rn(g.b, g.un), qt = -__fmul_rn(g.b, g.ut);
  const float dn = __fmul_rn(-0.5f, g.ic), d0 = -__fmul_rn(dn, g.un);
  float vp[4][5], vm[4][5];
  auto project = [&](const float4 f, float &x0, float &x1, float &x2, float &x3) {
    const float fn = DIR == 0 ? f.y : f.z, ft = DIR == 0 ? f.z : f.y;
    const float Q = __fmaf_rn(g.b, f.w, __fmaf_rn(qt, ft, __fmaf_rn(qn, fn, __fmul_rn(q0, f.x))));
    const float D = __fmaf_rn(dn, fn, __fmul_rn(d0, f.x));
    x0 = __fadd_rn(Q, D);
    x1 = __fmaf_rn(g.ut, f.x, -ft);
    x2 = __fmaf_rn(-2.0f, Q, f.x);
    x3 = __fadd_rn(Q, -D);
  };
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    project(P[s * ss], vp[0][s], vp[1][s], vp[2][s], vp[3][s]);
    project(M[s * ss], vm[0][s], vm[1][s], vm[2][s], vm[3][s]);
  }
  float h[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) h[k] = weno_sides<float, SCHEME>(vp[k], vm[k], zpl);
  const float S = __fadd_rn(h[0], h[3]), cD = __fmul_rn(g.c, __fadd_rn(h[3], -h[0]));
  const float o0 = __fadd_rn(S, h[2]);
  const float on = __fmaf_rn(g.un, o0, cD), ot = __fmaf_rn(g.ut, o0, -h[1]);
  const float o3 =
      __fmaf_rn(g.k2, h[2], __fmaf_rn(-g.ut, h[1], __fmaf_rn(g.un, cD, __fmul_rn(g.H, S))));
  return DIR == 0 ? make_float4(o0, on, ot, o3) : make_float4(o0, ot, on, o3);
}

// Pointwise Lax-Friedrichs split of one node in direction DIR: halves of the
// physical flux -+ half the wave speed times U.
template <int DIR>
__device__ __forceinline__ void split4(float gamma, const float4 q, float4 &fm, float4 &fp) {
  const float ir = rcp_ftz(q.x);
  const float u = __fmul_rn(q.y, ir), v = __fmul_rn(q.z, ir);
  const float g1 = __fadd_rn(gamma, -1.0f);
  const float p = __fmul_rn(g1, __fmaf_rn(-0.5f, __fmaf_rn(q.y, u, __fmul_rn(q.z, v)), q.w));
  const float mn = DIR == 0 ? q.y : q.z, mt = DIR == 0 ? q.z : q.y, un = DIR == 0 ? u : v;
  const float c = sqrt_ftz(__fmul_rn(__fmul_rn(gamma, p), ir));
  const float hu = __fmul_rn(0.5f, un), hw = __fmul_rn(0.5f, __fadd_rn(fabsf(un), c));
  const float f0 = __fmul_rn(0.5f, mn), fn = __fmaf_rn(mn, hu, __fmul_rn(0.5f, p)), ft = __fmul_rn(mt, hu);
  const float f3 = __fmul_rn(__fadd_rn(q.w, p), hu);
  const float2 F01 = make_float2(f0, DIR == 0 ? fn : ft), F23 = make_float2(DIR == 0 ? ft : fn, f3);
  const float2 mws = splat2(-hw), pws = splat2(hw);
  fm = join2(__ffma2_rn(mws, lo2(q), F01), __ffma2_rn(mws, hi2(q), F23));
  fp = join2(__ffma2_rn(pws, lo2(q), F01), __ffma2_rn(pws, hi2(q), F23));
}

// ------------------------------------ FP64 on the FP64 and integer pipes
//
// The FP64 parity tile's flux split, reconstruction and face flux, bit for bit
// flux_split, weno and face_flux_st on the values they take: sums and
// FMAs stay on the FP64 pipe, products, reciprocals and quotients run on the
// integer pipes (int_f64.cuh).  Fewer operations as well, each change exact:
//  - a product by a power of two is exact, so a - 2b, the sum with
//    (1/4 t2) t2 = 1/4 (t2 t2), 0.5 (F -+ P) and the like are one FMA;
//  - quotients by one divisor share its reciprocal;
//  - entries of L and R that are 0 or +-1 cost nothing (the reference adds
//    their products, which can only change the sign of a zero; no zero's sign
//    reaches the state, since rhs starts at +0);
//  - rows 0, 2 and 3 of L share the products B1 u_n f_n, B1 u_t f_t and B1 f_3
//    (times 1 or +-1/2).
// Values outside the integer forms' domain (huge, tiny, infinite or NaN; far
// from any flow) take the plain functions above.

// One WENO-JS or WENO-Z reconstruction.  Out of line: some 1,500 instructions,
// called eight times per face from both sweeps.
// Stencil values are zeros or at least 2^-200, so differences are zeros or at
// least 2^-253 and the indicators zeros or at least 2^-506; below 2^75, so no
// product overflows.  tau/beta may be tiny: its square is taken flushing
// subnormals to zero, which 1 + square rounds away.
template <int SCHEME>
__device__ __noinline__ double weno_plain(double a, double b, double c, double d, double e, double zp_lambda) {
  return weno<double, SCHEME>(a, b, c, d, e, zp_lambda);
}
template <int SCHEME>
__device__ __noinline__ double weno_int(double a, double b, double c, double d, double e) {
  if (!(in_range<-200, 75>(a) && in_range<-200, 75>(b) && in_range<-200, 75>(c) && in_range<-200, 75>(d) &&
        in_range<-200, 75>(e)))
    return weno_plain<SCHEME>(a, b, c, d, e, 0.0);
  const double c1312 = 13.0 / 12.0;
  const double c3 = int_mul(3.0, c);
  double t1 = fma(-2.0, b, a) + c, t2 = fma(-4.0, b, a) + c3;
  const double bm = fma(0.25, int_mul(t2, t2), int_mul(int_mul(c1312, t1), t1));
  t1 = fma(-2.0, c, b) + d;
  t2 = b - d;
  const double b0 = fma(0.25, int_mul(t2, t2), int_mul(int_mul(c1312, t1), t1));
  t1 = fma(-2.0, d, c) + e;
  t2 = fma(-4.0, d, c3) + e;
  const double bp = fma(0.25, int_mul(t2, t2), int_mul(int_mul(c1312, t1), t1));
  double w0, w1, w2;
  if constexpr (SCHEME == kWenoZ) {
    const double tau = fabs(bm - bp);
    auto weight = [tau](double linear, double beta) {
      const double ib = IntDivisor(beta + 1.0e-20).reciprocal();
      const double r = int_mul_ftz(int_mul_ftz(int_mul(tau, ib), tau), ib);
      return int_mul(linear, 1.0 + r);
    };
    w0 = weight(0.1, bm);
    w1 = weight(0.6, b0);
    w2 = weight(0.3, bp);
  } else {
    auto weight = [](double linear, double beta) {
      const double x = 1.0e-6 + beta;
      return IntDivisor(int_mul(x, x)).quotient(linear);
    };
    w0 = weight(0.1, bm);
    w1 = weight(0.6, b0);
    w2 = weight(0.3, bp);
  }
  const IntDivisor by_sum(w0 + w1 + w2);
  w0 = by_sum.quotient(w0);
  w1 = by_sum.quotient(w1);
  w2 = by_sum.quotient(w2);
  const double c13 = 1.0 / 3.0, c16 = 1.0 / 6.0, c56 = 5.0 / 6.0, c76 = 7.0 / 6.0, c116 = 11.0 / 6.0;
  const double p0 = int_mul(c13, a) - int_mul(c76, b) + int_mul(c116, c);
  const double p1 = int_mul(c56, c) - int_mul(c16, b) + int_mul(c13, d);
  const double p2 = int_mul(c13, c) + int_mul(c56, d) - int_mul(c16, e);
  return int_mul(w0, p0) + int_mul(w1, p1) + int_mul(w2, p2);
}

// Conserved variables whose primitives the integer forms take: density and
// energy in [2^-60, 2^60), momenta zeros or [2^-200, 2^60).
__device__ __forceinline__ bool state_in_range(double rho, double mu, double mv, double E) {
  return positive_in_range<-60, 60>(rho) && in_range<-200, 60>(mu) && in_range<-200, 60>(mv) &&
         positive_in_range<-60, 60>(E);
}

// flux_split in direction dir (0: x, 1: y).  False: a value outside the range
// of the face fluxes' integer forms (the split fluxes are right either way).
__device__ __forceinline__ bool flux_split_f64(int dir, double gamma, const double U[4], double fm[4], double fp[4]) {
  const double rho = U[0], E = U[3];
  bool ok = state_in_range(rho, U[1], U[2], E);
  if (ok) {
    const IntDivisor by_rho(rho);
    const double u = by_rho.quotient(U[1]), v = by_rho.quotient(U[2]);
    const double p = int_mul(gamma - 1.0, fma(-0.5, int_mul(rho, int_mul(u, u) + int_mul(v, v)), E));
    ok = positive_in_range<-60, 60>(p);
    if (ok) {
      const double un = dir == 0 ? u : v;  // normal velocity
      double F[4];
      F[0] = int_mul(rho, un);
      const double a = int_mul(F[0], un) + p;
      // rho u v in the reference's order: (rho u) v
      const double b = int_mul(dir == 0 ? F[0] : int_mul(rho, u), v);
      F[1] = dir == 0 ? a : b;
      F[2] = dir == 0 ? b : a;
      F[3] = int_mul(E + p, un);
      const double ws = fabs(un) + int_sqrt(by_rho.quotient(int_mul(gamma, p)));
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const double P = int_mul(ws, U[r]), h = int_half(F[r]);
        fm[r] = fma(-0.5, P, h);
        fp[r] = fma(0.5, P, h);
        ok = ok && in_range<-200, 70>(fm[r]) && in_range<-200, 70>(fp[r]);
      }
      return ok;
    }
  }
  if (dir == 0) flux_split<double, 0>(gamma, U, fm, fp);
  else flux_split<double, 1>(gamma, U, fm, fp);
  return false;
}

// The face flux (face_flux_st) in direction dir.  fp / fm point at F+ of node
// face-3 and F- of node face-2, component 0; stencil nodes `ss` elements apart,
// components `cs` apart.  False: a value left the integer forms' domain and
// `out` is not set.  One body for both directions: the normal and tangential
// components change places, and the reference's row 1 of L and column 1 of R
// change sign together in y, which changes no result.
// pair: two adjacent lanes share the face (the even lane takes the + side, the
// odd one the - side; all 32 lanes of the warp call it); both return it whole.
template <int SCHEME>
__device__ __forceinline__ bool face_flux_f64(int dir, bool pair, double gamma, double zp_lambda, const double um[4],
                                              const double u0[4], const double *fp, const double *fm, int ss, int cs,
                                              double out[4]) {
  const double rho = int_half(um[0] + u0[0]), E = int_half(um[3] + u0[3]);
  const double mu = int_half(um[1] + u0[1]), mv = int_half(um[2] + u0[2]);
  bool ok = state_in_range(rho, mu, mv, E);
  const IntDivisor by_rho(rho);
  const double u = by_rho.quotient(mu), v = by_rho.quotient(mv);
  const double K = int_mul(u, u) + int_mul(v, v);
  const double p = int_mul(gamma - 1.0, fma(-0.5, int_mul(rho, K), E));
  ok = ok && positive_in_range<-60, 60>(p);
  const double c = int_sqrt(by_rho.quotient(int_mul(gamma, p)));
  const double H = by_rho.quotient(E + p);
  const double un = dir == 0 ? u : v, ut = dir == 0 ? v : u;  // normal and tangential velocity
  const IntDivisor by_c(c);
  const double ic = by_c.reciprocal(), nc = by_c.quotient(un);
  const double B1 = IntDivisor(int_mul(c, c)).quotient(gamma - 1.0);
  const double B2 = int_half(int_mul(B1, K)), B1n = int_mul(B1, un), B1t = int_mul(B1, ut);
  // column 0 and the normal momentum's of rows 0 and 3, column 0 of row 2; the
  // tangential momentum's are -1/2 B1t in rows 0 and 3
  const double l00 = int_half(B2 + nc), l30 = int_half(B2 - nc), l20 = 1.0 - B2;
  const double l0n = -int_half(B1n + ic), l3n = -int_half(B1n - ic);
  const int cn = dir == 0 ? cs : 2 * cs, ct = dir == 0 ? 2 * cs : cs;

  double vh[4] = {0.0, 0.0, 0.0, 0.0};
  const int lane_side = int(threadIdx.x) & 1;
#pragma unroll 1
  for (int side = pair ? lane_side : 0; ok && side < (pair ? lane_side + 1 : 2); ++side) {
    // the - side is mirrored: from its last node down
    const double *f = side == 0 ? fp : fm + 4 * ss;
    const int step = side == 0 ? ss : -ss;
    double x[4][5] = {};  // (the first four shifts move what no node has set yet)
#pragma unroll 1
    for (int q = 0; q < 5; ++q, f += step) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) x[k][j] = x[k][j + 1];
      const double f0 = f[0], fn = f[cn], ft = f[ct], f3 = f[3 * cs];
      const double Pn = int_mul(B1n, fn), Pt = int_mul(B1t, ft), P3 = int_mul(B1, f3);
      const double a0 = int_mul(l00, f0), b0 = int_mul(l0n, fn), a3 = int_mul(l30, f0), b3 = int_mul(l3n, fn);
      const double a2 = int_mul(l20, f0);
      // the momenta's terms in the order x, y
      x[0][4] = fma(0.5, P3, dir == 0 ? fma(-0.5, Pt, a0 + b0) : fma(-0.5, Pt, a0) + b0);
      x[1][4] = int_mul(ut, f0) - ft;
      x[2][4] = (a2 + (dir == 0 ? Pn : Pt)) + (dir == 0 ? Pt : Pn) - P3;
      x[3][4] = fma(0.5, P3, dir == 0 ? fma(-0.5, Pt, a3 + b3) : fma(-0.5, Pt, a3) + b3);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if constexpr (SCHEME == kWenoJS || SCHEME == kWenoZ)
        vh[k] += weno_int<SCHEME>(x[k][0], x[k][1], x[k][2], x[k][3], x[k][4]);
      else
        vh[k] += weno_plain<SCHEME>(x[k][0], x[k][1], x[k][2], x[k][3], x[k][4], zp_lambda);
    }
  }
  if (pair) {  // warp-uniform
#pragma unroll
    for (int k = 0; k < 4; ++k) vh[k] += __shfl_xor_sync(0xffffffffu, vh[k], 1);
  }
  ok = ok && in_range<-400, 200>(vh[0]) && in_range<-400, 200>(vh[1]) && in_range<-400, 200>(vh[2]) &&
       in_range<-400, 200>(vh[3]);

  // R * vh, rows in the reference's order (utils/equations.hpp:239-299)
  const double q2 = int_half(K), cun = int_mul(c, un);
  out[0] = (vh[0] + vh[2]) + vh[3];
  const double on = int_mul(un - c, vh[0]) + int_mul(un, vh[2]) + int_mul(un + c, vh[3]);
  const double ot = int_mul(ut, vh[0]) - vh[1] + int_mul(ut, vh[2]) + int_mul(ut, vh[3]);
  out[1] = dir == 0 ? on : ot;
  out[2] = dir == 0 ? ot : on;
  out[3] = int_mul(H - cun, vh[0]) - int_mul(ut, vh[1]) + int_mul(q2, vh[2]) + int_mul(H + cun, vh[3]);
  return ok;
}

// face_flux_st out of line, for faces outside the integer forms' domain.
struct Flux4 {
  double v[4];
};
template <int DIR, int SCHEME>
__device__ __noinline__ Flux4 face_flux_plain(double gamma, double zp_lambda, double um0, double um1, double um2,
                                              double um3, double u00, double u01, double u02, double u03,
                                              const double *fp, const double *fm, int ss, int cs) {
  const double um[4] = {um0, um1, um2, um3}, u0[4] = {u00, u01, u02, u03};
  Flux4 o;
  face_flux_st<double, DIR, SCHEME>(gamma, zp_lambda, um, u0, StridedStencil<double>{fp, ss, cs},
                                    StridedStencil<double>{fm, ss, cs}, o.v);
  return o;
}

}  // namespace dev
}  // namespace wenofd
