// air_math.cuh -- per-face / per-node arithmetic of the calorically-perfect-air RHS, written once and
// instantiated for T = double (plain FP64 path) and T = float (mixed path).  The expressions are
// algebraically those of the reference source they cite, in forms of their own (differences of points, shared
// quotients, products in place of divisions); parity with the reference, 1e-12, is what the tests check.  On a
// rectilinear block (rectilinear() in host.h) the terms of the off-diagonal metric entries, rounding there, are
// left out on purpose.
#pragma once

#include <cuda_runtime.h>

namespace ostc {

constexpr double kGamma = 1.4;
constexpr double kRuD = 8314.462618;
constexpr double kMwD = 28.9647;

template <typename T> __device__ __forceinline__ T tsqrt(T x);
template <> __device__ __forceinline__ double tsqrt<double>(double x) { return sqrt(x); }
template <> __device__ __forceinline__ float tsqrt<float>(float x) { return sqrtf(x); }
// 1 / sqrt(x), from which the callers form sqrt(x) = x / sqrt(x) and 1 / x = (1 / sqrt(x))^2.  FP32:
// one reciprocal square root stands in for a square root and a division.  FP64 keeps the correctly
// rounded square root and division: with the reciprocal square root the FP64 sweeps ran 3 % faster,
// but the multi-block reference fixtures moved from inside the 1e-12 parity bar to 1.1-1.8e-12.
template <typename T> __device__ __forceinline__ T trsqrt(T x);
template <> __device__ __forceinline__ double trsqrt<double>(double x) { return 1.0 / sqrt(x); }
template <> __device__ __forceinline__ float trsqrt<float>(float x) { return rsqrtf(x); }
template <typename T> __device__ __forceinline__ T tabs(T x);
template <> __device__ __forceinline__ double tabs<double>(double x) { return fabs(x); }
template <> __device__ __forceinline__ float tabs<float>(float x) { return fabsf(x); }
template <typename T> __device__ __forceinline__ T tmin(T a, T b);
template <> __device__ __forceinline__ double tmin<double>(double a, double b) { return fmin(a, b); }
template <> __device__ __forceinline__ float tmin<float>(float a, float b) { return fminf(a, b); }
template <typename T> __device__ __forceinline__ T tmax(T a, T b);
template <> __device__ __forceinline__ double tmax<double>(double a, double b) { return fmax(a, b); }
template <> __device__ __forceinline__ float tmax<float>(float a, float b) { return fmaxf(a, b); }

// Sutherland viscosity (Transport.cu:6-9); always FP64 (it feeds the FP64 state path).
__device__ __forceinline__ double sutherland(double t) {
  return 1.7894e-5 * pow(t / 288.16, 1.5) * (288.16 + 110) / (t + 110);
}

// ------------------------------------------------------------------ axis-aligned metrics
//
// AX: the component of the metric row k that a sweep of a rectilinear block carries (DevBlock::rect: the
// off-diagonal metric entries are zero); -1: all three.  The other two terms of every product with k are
// zeros then and are left out.
template <int AX, typename T>
__device__ __forceinline__ T kdot(const T *k, const T *v) {
  if constexpr (AX < 0) return k[0] * v[0] + k[1] * v[1] + k[2] * v[2];
  else return k[AX] * v[AX];
}
// a + b k[q]
template <int AX, typename T>
__device__ __forceinline__ T kadd(T a, T b, const T *k, int q) {
  if constexpr (AX < 0) return a + b * k[q];
  else return q == AX ? a + b * k[AX] : a;
}

// ------------------------------------------------------------------ characteristic WENO-Z

// Convex WENO-Z combination sum_k a_k q_k / sum_k a_k with a_k = d_k (1 + tau / D_k) and
// D_k = (eps + beta_k)^2 (AWENO.cu:193-197, 245-251), sum_k d_k = 1; the q_k are the candidates'
// distances from one stencil point and lin their linear combination sum_k d_k q_k.
// FP64: multiplying numerator and denominator by prod_k D_k leaves one division per combination
// instead of one per weight (products of up to four D_k stay far inside the FP64 range), and the two
// sides of a face share one division (finish).  With e_k = d_k prod_{i != k} D_i the sums are
// prod D lin + tau sum e_k q_k over prod D + tau sum e_k.
// FP32: products of D_k can underflow, so each weight keeps its own fast division.  The
// reference's WENO7 indicator beta2 (AWENO.cu:236-238, 263-265) is neither shift-invariant nor
// positive semi-definite, so eps + beta2 can pass through zero; in FP32 its square can underflow to
// 0, so D_k is floored at 1e-30 (the weight is then ~1e30 times the linear weight: that stencil is
// selected, as in FP64).
template <typename T> struct WenoComb;
template <> struct WenoComb<double> {
  // numerator and denominator of the combination
  static __device__ __forceinline__ void c3(const double *d, const double *D, double tau, const double *q, double lin,
                                            double &num, double &den) {
    const double e0 = d[0] * (D[1] * D[2]), a = D[0] * D[2], e1 = d[1] * a, e2 = d[2] * (D[0] * D[1]);
    const double P = a * D[1];
    num = P * lin + tau * (e0 * q[0] + e1 * q[1] + e2 * q[2]);
    den = P + tau * (e0 + e1 + e2);
  }
  static __device__ __forceinline__ void c4(const double *d, const double *D, double tau, const double *q, double lin,
                                            double &num, double &den) {
    const double a = D[0] * D[1], b = D[2] * D[3], P = a * b;
    const double e0 = d[0] * (D[1] * b), e1 = d[1] * (D[0] * b), e2 = d[2] * (D[3] * a), e3 = d[3] * (D[2] * a);
    num = P * lin + tau * (e0 * q[0] + e1 * q[1] + e2 * q[2] + e3 * q[3]);
    den = P + tau * (e0 + e1 + e2 + e3);
  }
  // the two sides' quotients from one division: a denominator is a sum of products of up to four
  // (eps + beta)^2 factors, so the product of two stays inside the FP64 range
  static __device__ __forceinline__ void finish(double nm, double dm, double np, double dp, double &vm, double &vp) {
    const double q = 1.0 / (dm * dp);
    vm = nm * dp * q;
    vp = np * dm * q;
  }
};
template <> struct WenoComb<float> {
  template <int N>
  static __device__ __forceinline__ void comb(const float *d, const float *D, float tau, const float *q, float &num,
                                              float &den) {
    num = den = 0.f;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const float a = d[k] + d[k] * __fdividef(tau, fmaxf(D[k], 1e-30f));
      num += a * q[k];
      den += a;
    }
  }
  static __device__ __forceinline__ void c3(const float *d, const float *D, float tau, const float *q, float, float &num,
                                            float &den) {
    comb<3>(d, D, tau, q, num, den);
  }
  static __device__ __forceinline__ void c4(const float *d, const float *D, float tau, const float *q, float, float &num,
                                            float &den) {
    comb<4>(d, D, tau, q, num, den);
  }
  static __device__ __forceinline__ void finish(float nm, float dm, float np, float dp, float &vm, float &vp) {
    vm = __fdividef(nm, dm);
    vp = __fdividef(np, dp);
  }
};

// Characteristic WENO5-Z interpolation of one field, v its values at the 6 points i-2..i+3, at i+1/2
// (AWENO.cu:156-210).  Smoothness indicators and candidate interpolants are the
// reference's, written with the differences of consecutive points (which the stencils and the two sides
// share) and, the candidates, as distances from point i: fewer operations, and none of the digits of the
// field's level is lost.  (AWENO7 + HLLC at 512 x 256 x 128, three sweeps a stage: FP64 10.1 -> 8.9 ms, FP32 at
// 385 x 257 x 129 4.3 -> 3.7 ms.)
template <typename T>
__device__ __forceinline__ void weno5(const T *v, T &vminus, T &vplus) {
  const T d0 = v[1] - v[0], d1 = v[2] - v[1], d2 = v[3] - v[2], d3 = v[4] - v[3], d4 = v[5] - v[4];
  const T eps = T(1e-6), o8 = T(0.125);
  // 13/12 of the squared second differences
  T s0 = d1 - d0, s1 = d2 - d1, s2 = d3 - d2, s3 = d4 - d3;
  s0 = T(13.0 / 12) * s0 * s0;
  s1 = T(13.0 / 12) * s1 * s1;
  s2 = T(13.0 / 12) * s2 * s2;
  s3 = T(13.0 / 12) * s3 * s3;
  auto quarter = [](T x) { return T(0.25) * x * x; };
  const T q1 = o8 * (d1 + T(3) * d2), q2 = o8 * (T(5) * d2 - d3);
  T nm, dm, np, dp;
  {
    const T w[3] = {T(1.0 / 16), T(5.0 / 8), T(5.0 / 16)};
    const T q3[3] = {o8 * (T(7) * d1 - T(3) * d0), q1, q2};
    const T b0 = s0 + quarter(T(3) * d1 - d0), b1 = s1 + quarter(d1 + d2), b2 = s2 + quarter(T(3) * d2 - d3);
    const T D[3] = {(eps + b0) * (eps + b0), (eps + b1) * (eps + b1), (eps + b2) * (eps + b2)};
    WenoComb<T>::c3(w, D, (b0 - b2) * (b0 - b2), q3, w[0] * q3[0] + w[1] * q3[1] + w[2] * q3[2], nm, dm);
  }
  {
    const T w[3] = {T(5.0 / 16), T(5.0 / 8), T(1.0 / 16)};
    const T q3[3] = {q1, q2, d2 - o8 * (T(7) * d3 - T(3) * d4)};
    const T b0 = s1 + quarter(T(3) * d2 - d1), b1 = s2 + quarter(d2 + d3), b2 = s3 + quarter(T(3) * d3 - d4);
    const T D[3] = {(eps + b0) * (eps + b0), (eps + b1) * (eps + b1), (eps + b2) * (eps + b2)};
    WenoComb<T>::c3(w, D, (b0 - b2) * (b0 - b2), q3, w[0] * q3[0] + w[1] * q3[1] + w[2] * q3[2], np, dp);
  }
  WenoComb<T>::finish(nm, dm, np, dp, vminus, vplus);
  vminus += v[2];
  vplus += v[2];
}

// a (A a + B b + C c) + b (D b + E c) + F c^2
template <typename T>
__device__ __forceinline__ T weno_quad(T a, T b, T c, double A, double B, double C, double D, double E, double F) {
  const double k = 1.0 / 2880;
  return a * (T(k * A) * a + T(k * B) * b + T(k * C) * c) + b * (T(k * D) * b + T(k * E) * c) + T(k * F) * c * c;
}

// Smoothness indicators of the WENO7-Z interpolation (AWENO.cu:230-242, 257-269) of one side, from its
// points' differences d[0..5] (d[i] = v[i+1] - v[i]) and the points v2, v3.  b0, b1 and b3 are quadratic
// forms of the differences (9 operations each; 22 from the points).  b2 as the reference writes it has
// -30414 v2 v3 + 6649 v3^2 where the symmetric form has -30414 v3 v4 + 6649 v4^2, which leaves terms in
// the points themselves.
template <typename T>
__device__ __forceinline__ void weno7_betas(const T *d, T v2, T v3, T &b0, T &b1, T &b2, T &b3) {
  const double k = 1.0 / 2880;
  b0 = weno_quad<T>(d[3], d[4], d[5], 25729, -63436, 22778, 45076, -33916, 6649);
  b1 = weno_quad<T>(d[2], d[3], d[4], 6649, -17116, 5978, 17236, -13036, 3169);
  b2 = d[1] * (T(k * 3169) * d[1] + T(k * -13036) * d[2] + T(k * 5978) * d[3]) +
       d[2] * (T(k * 17236) * d[2] + T(k * 30414) * v3) + T(k * 17116) * d[3] * v2;
  b3 = weno_quad<T>(d[0], d[1], d[2], 6649, -33916, 22778, 45076, -63436, 25729);
}

// Characteristic WENO7-Z interpolation from the 8 points i-3..i+4 (AWENO.cu:212-280), in differences as
// weno5; the candidates are distances from point i.
template <typename T>
__device__ __forceinline__ void weno7(const T *v, T &vminus, T &vplus) {
  T d[7];
#pragma unroll
  for (int s = 0; s < 7; ++s) d[s] = v[s + 1] - v[s];
  const T eps = T(1e-6), o16 = T(0.0625);
  const T qb = o16 * (T(5) * d[3] + T(4) * d[2] - d[1]), qc = o16 * (d[2] + T(8) * d[3] - d[4]),
          qd = o16 * (T(11) * d[3] - T(4) * d[4] + d[5]);
  T nm, dm, np, dp;
  {
    const T w[4] = {T(7.0 / 64), T(35.0 / 64), T(21.0 / 64), T(1.0 / 64)};
    const T q4[4] = {qd, qc, qb, o16 * (T(19) * d[2] - T(16) * d[1] + T(5) * d[0])};
    T b0, b1, b2, b3;
    weno7_betas<T>(d, v[2], v[3], b0, b1, b2, b3);
    const T tau = (b3 + T(5) * (b2 - b1)) - b0;
    const T D[4] = {(eps + b0) * (eps + b0), (eps + b1) * (eps + b1), (eps + b2) * (eps + b2), (eps + b3) * (eps + b3)};
    WenoComb<T>::c4(w, D, tau * tau, q4, w[0] * q4[0] + w[1] * q4[1] + w[2] * q4[2] + w[3] * q4[3], nm, dm);
  }
  {
    const T w[4] = {T(1.0 / 64), T(21.0 / 64), T(35.0 / 64), T(7.0 / 64)};
    const T q4[4] = {d[3] - o16 * (T(19) * d[4] - T(16) * d[5] + T(5) * d[6]), qd, qc, qb};
    T b0, b1, b2, b3;
    weno7_betas<T>(d + 1, v[3], v[4], b0, b1, b2, b3);
    const T tau = (b3 + T(5) * (b2 - b1)) - b0;
    const T D[4] = {(eps + b0) * (eps + b0), (eps + b1) * (eps + b1), (eps + b2) * (eps + b2), (eps + b3) * (eps + b3)};
    WenoComb<T>::c4(w, D, tau * tau, q4, w[0] * q4[0] + w[1] * q4[1] + w[2] * q4[2] + w[3] * q4[3], np, dp);
  }
  WenoComb<T>::finish(nm, dm, np, dp, vminus, vplus);
  vminus += v[3];
  vplus += v[3];
}

template <int NG, typename T>
__device__ __forceinline__ void weno(const T *v, T &vminus, T &vplus) {
  if constexpr (NG == 3) weno5<T>(v, vminus, vplus);
  else weno7<T>(v, vminus, vplus);
}

// One characteristic field: the products of the row Lr of the left eigenvector matrix with the stencil's
// conservative variables q(s, v), interpolated.
template <int NG, typename T, class Q>
__device__ __forceinline__ void weno_char(const T *Lr, const Q &q, T &vminus, T &vplus) {
  T v[2 * NG];
#pragma unroll
  for (int s = 0; s < 2 * NG; ++s) {
    T acc = T(0);
#pragma unroll
    for (int j = 0; j < 5; ++j) acc += Lr[j] * q(s, j);
    v[s] = acc;
  }
  weno<NG, T>(v, vminus, vplus);
}

// AWENO_interpolation<Air> (AWENO.cu:15-154).  NG = 3 (WENO5) or 4 (WENO7); q(s, v) for
// s in [0, 2*NG) is point i-NG+1+s, v = 0..4 conservative variables, v = 5 pressure.
// mt0/mt1: metric row of the sweep direction at i and i+1.  pl/pr: rho,u,v,w,p,rhoE.
// The left eigenvector matrix is built one row per characteristic field and the right one column
// by column, so only one row/column is live at a time; the reference's divisions by cm2, cm,
// gradK and rho are replaced by multiplications with their reciprocals.  The back projection
// accumulates field by field in the reference's summation order.
// AX >= 0 (axis-aligned normal k = +-e_AX): the two acoustic fields and the entropy field share one
// product X = alpha rho - (gamma - 1)(u . m - rhoE) per point (A = X / (2 c^2), B = (u rho - m)_n / (2 c):
// A + B, A - B and rho - 2 A), and each shear field is (m_t - u_t rho) / c: 15 operations a point instead
// of 25 (the signs k of the shear and entropy fields cancel between their rows and columns).
template <int NG, typename T, int AX, class Q>
__device__ __forceinline__ void aweno_interp(const Q &q, const T *mt0, const T *mt1, T *pl, T *pr) {
  constexpr int cl = NG - 1, cr = NG;
  const T gm1 = T(kGamma - 1), igm1 = T(1.0 / (kGamma - 1));
  const T l0 = q(cl, 0), r0 = q(cr, 0);
  const T rsl = trsqrt(l0), rsr = trsqrt(r0);
  const T sl = l0 * rsl, sr = r0 * rsr;
  const T isum = T(1) / (sl + sr);
  const T rlc = sl * isum, rrc = sr * isum;
  const T il0 = rsl * rsl, ir0 = rsr * rsr;
  const T um = rlc * q(cl, 1) * il0 + rrc * q(cr, 1) * ir0;
  const T vm = rlc * q(cl, 2) * il0 + rrc * q(cr, 2) * ir0;
  const T wm = rlc * q(cl, 3) * il0 + rrc * q(cr, 3) * ir0;
  const T ekm = T(0.5) * (um * um + vm * vm + wm * wm);
  const T hl = (q(cl, 4) + q(cl, 5)) * il0;
  const T hr = (q(cr, 4) + q(cr, 5)) * ir0;
  const T hm = rlc * hl + rrc * hr;
  const T cm2 = gm1 * (hm - ekm);
  const T icm = trsqrt(cm2);
  const T cm = cm2 * icm, icm2 = icm * icm;
  const T alpha = gm1 * ekm;
  const T h2 = T(0.5) * icm2;
  T ql[5] = {T(0), T(0), T(0), T(0), T(0)}, qr[5] = {T(0), T(0), T(0), T(0), T(0)};
  if constexpr (AX >= 0) {
    constexpr int n = 1 + AX, t1 = 1 + (AX + 1) % 3, t2 = 1 + (AX + 2) % 3;
    const T vel[4] = {T(0), um, vm, wm};
    const T k = mt0[AX] + mt1[AX] < T(0) ? T(-1) : T(1), kc = k * cm;
    T a[2 * NG], bq[2 * NG], v[2 * NG];
#pragma unroll
    for (int s = 0; s < 2 * NG; ++s) {
      const T r = q(s, 0), m = q(s, n);
      T X = alpha * r + gm1 * q(s, 4);
      X -= gm1 * (vel[n] * m + vel[t1] * q(s, t1) + vel[t2] * q(s, t2));
      a[s] = h2 * X;
      bq[s] = (h2 * kc) * (vel[n] * r - m);
    }
    T vmi, vpl;
#pragma unroll
    for (int l = 0; l < 5; ++l) {
      if (l == 0 || l == 4) {
        const T sg = l == 0 ? T(-1) : T(1);
#pragma unroll
        for (int s = 0; s < 2 * NG; ++s) v[s] = l == 0 ? a[s] + bq[s] : a[s] - bq[s];
        weno<NG, T>(v, vmi, vpl);
        const T rn = vel[n] + sg * kc, re = hm + sg * kc * vel[n];
        ql[0] += vmi;
        qr[0] += vpl;
        ql[n] += rn * vmi;
        qr[n] += rn * vpl;
        ql[t1] += vel[t1] * vmi;
        qr[t1] += vel[t1] * vpl;
        ql[t2] += vel[t2] * vmi;
        qr[t2] += vel[t2] * vpl;
        ql[4] += re * vmi;
        qr[4] += re * vpl;
      } else if (l == n) {
#pragma unroll
        for (int s = 0; s < 2 * NG; ++s) v[s] = q(s, 0) - T(2) * a[s];
        weno<NG, T>(v, vmi, vpl);
        ql[0] += vmi;
        qr[0] += vpl;
#pragma unroll
        for (int m = 1; m < 4; ++m) {
          ql[m] += vel[m] * vmi;
          qr[m] += vel[m] * vpl;
        }
        ql[4] += ekm * vmi;
        qr[4] += ekm * vpl;
      } else {
#pragma unroll
        for (int s = 0; s < 2 * NG; ++s) v[s] = icm * (q(s, l) - vel[l] * q(s, 0));
        weno<NG, T>(v, vmi, vpl);
        ql[l] += cm * vmi;
        qr[l] += cm * vpl;
        const T re = vel[l] * cm;
        ql[4] += re * vmi;
        qr[4] += re * vpl;
      }
    }
  } else {
  T kx = T(0.5) * (mt0[0] + mt1[0]);
  T ky = T(0.5) * (mt0[1] + mt1[1]);
  T kz = T(0.5) * (mt0[2] + mt1[2]);
  const T igk = trsqrt(kx * kx + ky * ky + kz * kz);
  kx *= igk;
  ky *= igk;
  kz *= igk;
  const T Uk = kx * um + ky * vm + kz * wm;
#pragma unroll
  for (int l = 0; l < 5; ++l) {
    T Lr[5], Rc[5];
    if (l == 0) {
      Lr[0] = (alpha + Uk * cm) * h2;
      Lr[1] = -(gm1 * um + kx * cm) * h2;
      Lr[2] = -(gm1 * vm + ky * cm) * h2;
      Lr[3] = -(gm1 * wm + kz * cm) * h2;
      Lr[4] = gm1 * h2;
      Rc[0] = T(1); Rc[1] = um - kx * cm; Rc[2] = vm - ky * cm; Rc[3] = wm - kz * cm; Rc[4] = hm - Uk * cm;
    } else if (l == 1) {
      Lr[0] = kx * (T(1) - alpha * icm2) - (kz * vm - ky * wm) * icm;
      Lr[1] = kx * gm1 * um * icm2;
      Lr[2] = (kx * gm1 * vm + kz * cm) * icm2;
      Lr[3] = (kx * gm1 * wm - ky * cm) * icm2;
      Lr[4] = -kx * gm1 * icm2;
      Rc[0] = kx; Rc[1] = kx * um; Rc[2] = kx * vm + kz * cm; Rc[3] = kx * wm - ky * cm;
      Rc[4] = kx * alpha * igm1 + (kz * vm - ky * wm) * cm;
    } else if (l == 2) {
      Lr[0] = ky * (T(1) - alpha * icm2) - (kx * wm - kz * um) * icm;
      Lr[1] = (ky * gm1 * um - kz * cm) * icm2;
      Lr[2] = ky * gm1 * vm * icm2;
      Lr[3] = (ky * gm1 * wm + kx * cm) * icm2;
      Lr[4] = -ky * gm1 * icm2;
      Rc[0] = ky; Rc[1] = ky * um - kz * cm; Rc[2] = ky * vm; Rc[3] = ky * wm + kx * cm;
      Rc[4] = ky * alpha * igm1 + (kx * wm - kz * um) * cm;
    } else if (l == 3) {
      Lr[0] = kz * (T(1) - alpha * icm2) - (ky * um - kx * vm) * icm;
      Lr[1] = (kz * gm1 * um + ky * cm) * icm2;
      Lr[2] = (kz * gm1 * vm - kx * cm) * icm2;
      Lr[3] = kz * gm1 * wm * icm2;
      Lr[4] = -kz * gm1 * icm2;
      Rc[0] = kz; Rc[1] = kz * um + ky * cm; Rc[2] = kz * vm - kx * cm; Rc[3] = kz * wm;
      Rc[4] = kz * alpha * igm1 + (ky * um - kx * vm) * cm;
    } else {
      Lr[0] = (alpha - Uk * cm) * h2;
      Lr[1] = -(gm1 * um - kx * cm) * h2;
      Lr[2] = -(gm1 * vm - ky * cm) * h2;
      Lr[3] = -(gm1 * wm - kz * cm) * h2;
      Lr[4] = gm1 * h2;
      Rc[0] = T(1); Rc[1] = um + kx * cm; Rc[2] = vm + ky * cm; Rc[3] = wm + kz * cm; Rc[4] = hm + Uk * cm;
    }
    T vmi, vpl;
    weno_char<NG, T>(Lr, q, vmi, vpl);
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      ql[m] += Rc[m] * vmi;
      qr[m] += Rc[m] * vpl;
    }
  }
  }
  const T iqq = T(1) / (ql[0] * qr[0]);
  const T iql = qr[0] * iqq, iqr = ql[0] * iqq;
  pl[0] = ql[0];
  pl[1] = ql[1] * iql;
  pl[2] = ql[2] * iql;
  pl[3] = ql[3] * iql;
  pl[4] = gm1 * (ql[4] - T(0.5) * (pl[1] * pl[1] + pl[2] * pl[2] + pl[3] * pl[3]) * ql[0]);
  pl[5] = ql[4];
  pr[0] = qr[0];
  pr[1] = qr[1] * iqr;
  pr[2] = qr[2] * iqr;
  pr[3] = qr[3] * iqr;
  pr[4] = gm1 * (qr[4] - T(0.5) * (pr[1] * pr[1] + pr[2] * pr[2] + pr[3] * pr[3]) * qr[0]);
  pr[5] = qr[4];
}

// ------------------------------------------------------------------ Riemann solvers

// riemannSolver_ausmPlus<Air> (RiemannSolver.cuh:9-96); divisions by the face-normal magnitude,
// sound speed and densities go through reciprocals.
template <typename T, int AX = -1>
__device__ __forceinline__ void ausm_plus(const T *pl, const T *pr, const T *mt0, const T *mt1, T j0, T j1, T *fc) {
  T k[3];
#pragma unroll
  for (int q = 0; q < 3; ++q)
    if (AX < 0 || q == AX) k[q] = T(0.5) * (j0 * mt0[q] + j1 * mt1[q]);
  const T k2s = kdot<AX>(k, k);
  const T igkj = trsqrt(k2s);
  const T gkj = k2s * igkj;
  const T ul = kdot<AX>(k, pl + 1) * igkj;
  const T ur = kdot<AX>(k, pr + 1) * igkj;
  const T p_l = pl[4], p_r = pr[4], rho_l = pl[0], rho_r = pr[0];
  const T gam = T(kGamma);
  const T irl = T(1) / rho_l, irr = T(1) / rho_r;
  const T c = T(0.5) * (tsqrt(gam * p_l * irl) + tsqrt(gam * p_r * irr));
  const T ic = T(1) / c;
  const T mach_l = ul * ic, mach_r = ur * ic;
  T mlp, mrn, plp, prn;
  const T alpha = T(3 / 16.0);
  if (tabs(mach_l) > T(1)) {
    mlp = T(0.5) * (mach_l + tabs(mach_l));
    plp = mach_l > T(0) ? T(1) : T(0);
  } else {
    const T a = (mach_l + T(1)) * (mach_l + T(1)) * T(0.25);
    const T b = (mach_l * mach_l - T(1)) * (mach_l * mach_l - T(1));
    mlp = a + T(0.125) * b;
    plp = a * (T(2) - mach_l) + alpha * mach_l * b;
  }
  if (tabs(mach_r) > T(1)) {
    mrn = T(0.5) * (mach_r - tabs(mach_r));
    prn = mach_r < T(0) ? T(1) : T(0);
  } else {
    const T a = (mach_r - T(1)) * (mach_r - T(1)) * T(0.25);
    const T b = (mach_r * mach_r - T(1)) * (mach_r * mach_r - T(1));
    mrn = -a - T(0.125) * b;
    prn = a * (T(2) + mach_r) - alpha * mach_r * b;
  }
  const T p_coeff = plp * p_l + prn * p_r;
  const T m_half = mlp + mrn;
  const T mach_pos = T(0.5) * (m_half + tabs(m_half));
  const T mach_neg = T(0.5) * (m_half - tabs(m_half));
  const T mass_flux = c * (rho_l * mach_pos + rho_r * mach_neg);
  const T coeff = mass_flux * gkj;
  const bool left = mass_flux >= T(0);
  const T *s = left ? pl : pr;
  fc[0] = coeff;
#pragma unroll
  for (int q = 0; q < 3; ++q) fc[1 + q] = kadd<AX>(coeff * s[1 + q], p_coeff, k, q);
  fc[4] = coeff * (s[5] + s[4]) * (left ? irl : irr);
}

// riemannSolver_hllc<Air> (RiemannSolver.cuh:98-230), with shared reciprocals.
template <typename T, int AX = -1>
__device__ __forceinline__ void hllc(const T *pl, const T *pr, const T *mt0, const T *mt1, T j0, T j1, T *fc) {
  const T gam = T(kGamma);
  const T rsl = trsqrt(pl[0]), rsr = trsqrt(pr[0]);
  const T sql = pl[0] * rsl, sqr = pr[0] * rsr;
  const T isq = T(1) / (sql + sqr);
  const T rl_c = sql * isq;
  const T rr_c = sqr * isq;
  const T ut = pl[1] * rl_c + pr[1] * rr_c;
  const T vt = pl[2] * rl_c + pr[2] * rr_c;
  const T wt = pl[3] * rl_c + pr[3] * rr_c;
  const T irl = rsl * rsl, irr = rsr * rsr;
  const T hl = (pl[5] + pl[4]) * irl;
  const T hr = (pr[5] + pr[4]) * irr;
  const T ht = hl * rl_c + hr * rr_c;
  const T ekt = T(0.5) * (ut * ut + vt * vt + wt * wt);
  const T ct = tsqrt((gam - T(1)) * (ht - ekt));
  T k[3];
#pragma unroll
  for (int q = 0; q < 3; ++q)
    if (AX < 0 || q == AX) k[q] = T(0.5) * (mt0[q] + mt1[q]);
  const T k2s = kdot<AX>(k, k);
  const T igk = trsqrt(k2s);
  const T gradK = k2s * igk;
  const T vt3[3] = {ut, vt, wt};
  const T Ubar = kdot<AX>(k, vt3) * igk;
  const T jac = T(0.5) * (j0 + j1);
  const T Ul = kdot<AX>(k, pl + 1);
  const T Ur = kdot<AX>(k, pr + 1);
  const T unl = Ul * igk, unr = Ur * igk;
  const T cl = tsqrt(gam * pl[4] * irl);
  const T sl = tmin(unl - cl, Ubar - ct);
  if (sl >= T(0)) {
    const T rU = pl[0] * Ul;
    fc[0] = jac * rU;
#pragma unroll
    for (int q = 0; q < 3; ++q) fc[1 + q] = jac * kadd<AX>(rU * pl[1 + q], pl[4], k, q);
    fc[4] = jac * ((pl[5] + pl[4]) * Ul);
    return;
  }
  const T cr = tsqrt(gam * pr[4] * irr);
  const T sr = tmax(unr + cr, Ubar + ct);
  if (sr < T(0)) {
    const T rU = pr[0] * Ur;
    fc[0] = jac * rU;
#pragma unroll
    for (int q = 0; q < 3; ++q) fc[1 + q] = jac * kadd<AX>(rU * pr[1 + q], pr[4], k, q);
    fc[4] = jac * ((pr[5] + pr[4]) * Ur);
    return;
  }
  const T sm = ((pr[0] * Ur * (sr - unr) - pl[0] * Ul * (sl - unl)) * igk + pl[4] - pr[4]) /
               (pr[0] * (sr - unr) - pl[0] * (sl - unl));
  const T pm = pl[0] * (sl - unl) * (sm - unl) + pl[4];
  const bool left = sm >= T(0);
  const T *q = left ? pl : pr;
  const T sk = left ? sl : sr, Uk = left ? Ul : Ur, irk = left ? irl : irr;
  const T pc = T(1) / (sk - sm);
  const T Q = jac * pc * sm * (sk * gradK - Uk) * q[0];
  fc[0] = Q;
  const T dP = (sk * pm - sm * q[4]) * pc * jac;
#pragma unroll
  for (int c = 0; c < 3; ++c) fc[1 + c] = kadd<AX>(Q * q[1 + c], dP, k, c);
  fc[4] = Q * q[5] * irk + pc * jac * (sk * pm * sm * gradK - sm * q[4] * Uk);
}

// riemannSolver_laxFriedrich<Air> (RiemannSolver.cuh:420-460): face-averaged metric, the larger
// spectral radius of the two sides.
template <typename T, int AX = -1>
__device__ __forceinline__ void lax_friedrichs(const T *pl, const T *pr, const T *mt0, const T *mt1, T j0, T j1,
                                               T *fc) {
  T k[3];
#pragma unroll
  for (int q = 0; q < 3; ++q)
    if (AX < 0 || q == AX) k[q] = T(0.5) * (mt0[q] + mt1[q]);
  const T gradK = tsqrt(kdot<AX>(k, k));
  const T Ukl = kdot<AX>(k, pl + 1);
  const T Ukr = kdot<AX>(k, pr + 1);
  const T cl = tsqrt(T(kGamma) * pl[4] / pl[0]);
  const T cr = tsqrt(T(kGamma) * pr[4] / pr[0]);
  const T sr = tmax(tabs(Ukl) + cl * gradK, tabs(Ukr) + cr * gradK);
  const T hj = T(0.25) * (j0 + j1);
  const T rUl = pl[0] * Ukl, rUr = pr[0] * Ukr;
  fc[0] = (rUl + rUr - sr * (pr[0] - pl[0])) * hj;
#pragma unroll
  for (int q = 0; q < 3; ++q)
    fc[1 + q] = (kadd<AX>(rUl * pl[1 + q] + rUr * pr[1 + q], pl[4] + pr[4], k, q) -
                 sr * (pr[1 + q] * pr[0] - pl[1 + q] * pl[0])) * hj;
  fc[4] = ((pl[5] + pl[4]) * Ukl + (pr[5] + pr[4]) * Ukr - sr * (pr[5] - pl[5])) * hj;
}

// Harten entropy-fix threshold of one node (compute_entropy_fix_delta<Air>, InviscidScheme.cu:417-456):
// factor * (|U| + |V| (+ |W|) + c * mean |grad xi|).  m: the 9 metric entries of the node, b: rho..p.
template <typename T>
__device__ __forceinline__ T entropy_fix_delta(const T *m, const T *b, T factor, bool dim3) {
  const T U = tabs(b[1] * m[0] + b[2] * m[1] + b[3] * m[2]);
  const T V = tabs(b[1] * m[3] + b[2] * m[4] + b[3] * m[5]);
  const T W = tabs(b[1] * m[6] + b[2] * m[7] + b[3] * m[8]);
  const T kx = tsqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
  const T ky = tsqrt(m[3] * m[3] + m[4] * m[4] + m[5] * m[5]);
  const T kz = tsqrt(m[6] * m[6] + m[7] * m[7] + m[8] * m[8]);
  const T c = tsqrt(T(kGamma) * b[4] / b[0]);
  if (!dim3) return factor * (U + V + c * T(0.5) * (kx + ky));
  return factor * (U + V + W + c * (kx + ky + kz) / T(3));
}

// riemannSolver_Roe<Air> (RiemannSolver.cuh:279-417): the half sum of the two sides' physical fluxes
// (each with its own node's metric and Jacobian, compute_half_sum_left_right_flux :232-277) plus
// the Roe dissipation with Harten's entropy fix on |lambda| below the face-averaged threshold.
template <typename T>
__device__ __forceinline__ void roe(const T *pl, const T *pr, const T *mt0, const T *mt1, T j0, T j1, T d0, T d1,
                                    T *fc) {
  {
    const T jx = j0 * mt0[0], jy = j0 * mt0[1], jz = j0 * mt0[2];
    const T Uk = pl[1] * jx + pl[2] * jy + pl[3] * jz;
    const T co = Uk * pl[0];
    fc[0] = T(0.5) * co;
    fc[1] = T(0.5) * (co * pl[1] + pl[4] * jx);
    fc[2] = T(0.5) * (co * pl[2] + pl[4] * jy);
    fc[3] = T(0.5) * (co * pl[3] + pl[4] * jz);
    fc[4] = T(0.5) * Uk * (pl[4] + pl[5]);
  }
  {
    const T jx = j1 * mt1[0], jy = j1 * mt1[1], jz = j1 * mt1[2];
    const T Uk = pr[1] * jx + pr[2] * jy + pr[3] * jz;
    const T co = Uk * pr[0];
    fc[0] += T(0.5) * co;
    fc[1] += T(0.5) * (co * pr[1] + pr[4] * jx);
    fc[2] += T(0.5) * (co * pr[2] + pr[4] * jy);
    fc[3] += T(0.5) * (co * pr[3] + pr[4] * jz);
    fc[4] += T(0.5) * Uk * (pr[4] + pr[5]);
  }
  const T dl = tsqrt(pl[0]), dr = tsqrt(pr[0]);
  const T inv = T(1) / (dl + dr);
  const T u = (dl * pl[1] + dr * pr[1]) * inv;
  const T v = (dl * pl[2] + dr * pr[2]) * inv;
  const T w = (dl * pl[3] + dr * pr[3]) * inv;
  const T ek = T(0.5) * (u * u + v * v + w * w);
  const T hl = (pl[5] + pl[4]) / pl[0];
  const T hr = (pr[5] + pr[4]) / pr[0];
  const T h = (dl * hl + dr * hr) * inv;
  const T gm1 = T(kGamma - 1);
  const T c = tsqrt(gm1 * (h - ek));
  T kx = T(0.5) * (mt0[0] + mt1[0]);
  T ky = T(0.5) * (mt0[1] + mt1[1]);
  T kz = T(0.5) * (mt0[2] + mt1[2]);
  const T gradK = tsqrt(kx * kx + ky * ky + kz * kz);
  T Uk = kx * u + ky * v + kz * w;
  T ch[3] = {Uk - gradK * c, Uk, Uk + gradK * c};
  const T da = T(0.5) * (d0 + d1);
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    ch[n] = tabs(ch[n]);
    if (ch[n] < da) ch[n] = T(0.5) * (ch[n] * ch[n] / da + da);
  }
  const T igk = T(1) / gradK;
  kx *= igk;
  ky *= igk;
  kz *= igk;
  Uk *= igk;
  const T ja = T(0.5) * (j0 + j1);
  const T q0 = ja * (pr[0] - pl[0]);
  const T q1 = ja * (pr[0] * pr[1] - pl[0] * pl[1]);
  const T q2 = ja * (pr[0] * pr[2] - pl[0] * pl[2]);
  const T q3 = ja * (pr[0] * pr[3] - pl[0] * pl[3]);
  const T q4 = ja * (pr[5] - pl[5]);
  const T ic = T(1) / c;
  T c1 = gm1 * (ek * q0 - u * q1 - v * q2 - w * q3 + q4) * ic * ic;
  T c2 = (kx * q1 + ky * q2 + kz * q3 - Uk * q0) * ic;
  const T c3 = q0 - c1;
  const T L0 = T(0.5) * (c1 - c2);
  const T L1 = kx * c3 - ((kz * v - ky * w) * q0 - kz * q2 + ky * q3) * ic;
  const T L2 = ky * c3 - ((kx * w - kz * u) * q0 - kx * q3 + kz * q1) * ic;
  const T L3 = kz * c3 - ((ky * u - kx * v) * q0 - ky * q1 + kx * q2) * ic;
  const T L4 = T(0.5) * (c1 + c2);
  const T b0 = -ch[0] * L0, b1 = -ch[1] * L1, b2 = -ch[1] * L2, b3 = -ch[1] * L3, b4 = -ch[2] * L4;
  const T c0 = kx * b1 + ky * b2 + kz * b3;
  c1 = c0 + b0 + b4;
  c2 = c * (b4 - b0);
  fc[0] += T(0.5) * c1;
  fc[1] += T(0.5) * (u * c1 + kx * c2 - c * (kz * b2 - ky * b3));
  fc[2] += T(0.5) * (v * c1 + ky * c2 - c * (kx * b3 - kz * b1));
  fc[3] += T(0.5) * (w * c1 + kz * c2 - c * (ky * b1 - kx * b2));
  fc[4] += T(0.5) * (h * c1 + Uk * c2 - c * c * c0 / gm1 +
                     c * ((kz * v - ky * w) * b1 + (kx * w - kz * u) * b2 + (ky * u - kx * v) * b3));
}

// ------------------------------------------------------------------ primitive reconstruction

// minmod with the reference's sign convention sgn(0) = +1 (Limiter.cuh:13-16, gxl_lib/Math.hpp:13-15).
template <typename T>
__device__ __forceinline__ T minmod(T a, T b) {
  const T sa = a < T(0) ? T(-1) : T(1), sb = b < T(0) ? T(-1) : T(1);
  return T(0.5) * (sa + sb) * tmin(tabs(a), tabs(b));
}

// Left/right primitive states at i+1/2 from nodes i-1, i, i+1, i+2 (v(m, l), m = -1..2), then the total
// energy of each side (reconstruction<Air>, InviscidScheme.cu:163-215; first_order_reconstruct,
// MUSCL_reconstruct (kappa = 1/3), NND2_reconstruct, Reconstruction.cu:5-45).
template <typename T, class V>
__device__ __forceinline__ void pv_reconstruct(const V &v, int recon, T *pl, T *pr) {
#pragma unroll
  for (int l = 0; l < 5; ++l) {
    const T a = v(0, l), bq = v(1, l);
    if (recon == 2 || recon == 3) {
      const T di = a - v(-1, l), di1 = bq - a, di2 = v(2, l) - bq;
      if (recon == 2) {
        const T k1 = T(1) - T(1.0 / 3.0), k2 = T(1) + T(1.0 / 3.0);
        pl[l] = a + T(0.25) * (k1 * minmod(di, di1) + k2 * minmod(di1, di));
        pr[l] = bq - T(0.25) * (k1 * minmod(di2, di1) + k2 * minmod(di1, di2));
      } else {
        pl[l] = a + T(0.5) * minmod(di, di1);
        pr[l] = bq - T(0.5) * minmod(di1, di2);
      }
    } else {
      pl[l] = a;
      pr[l] = bq;
    }
  }
  const T el = T(0.5) * (pl[1] * pl[1] + pl[2] * pl[2] + pl[3] * pl[3]);
  const T er = T(0.5) * (pr[1] * pr[1] + pr[2] * pr[2] + pr[3] * pr[3]);
  pl[5] = el * pl[0] + pl[4] / T(kGamma - 1);
  pr[5] = er * pr[0] + pr[4] / T(kGamma - 1);
}

// Whole AWENO face flux: interpolation then the selected Riemann solver (InviscidScheme.cu:333-345).
template <int NG, int RS, typename T, int AX = -1, class Q>
__device__ __forceinline__ void aweno_face_flux(const Q &q, const T *mt0, const T *mt1, T j0, T j1, T *fc) {
  T pl[6], pr[6];
  aweno_interp<NG, T, AX>(q, mt0, mt1, pl, pr);
  if constexpr (RS == 4) {
    hllc<T, AX>(pl, pr, mt0, mt1, j0, j1, fc);
  } else if constexpr (RS == 1) {
    lax_friedrichs<T, AX>(pl, pr, mt0, mt1, j0, j1, fc);
  } else {
    ausm_plus<T, AX>(pl, pr, mt0, mt1, j0, j1, fc);
  }
}

// Physical flux of one node for the central-difference correction (AWENO.cu:307-321).
// b: rho,u,v,w,p (bv 0..4); e: rho*E (cv 4); k: metric row of the sweep direction.
template <typename T, int AX = -1>
__device__ __forceinline__ void node_flux(const T *b, T e, const T *k, T jac, T *f) {
  const T Uk = kdot<AX>(k, b + 1);
  const T rhoUk = b[0] * Uk;
  f[0] = rhoUk * jac;
#pragma unroll
  for (int q = 0; q < 3; ++q) f[1 + q] = jac * kadd<AX>(rhoUk * b[1 + q], b[4], k, q);
  f[4] = jac * Uk * (e + b[4]);
}

// Central correction coefficients (AWENO.cu:327-350): dq += sum_m c_m (f(i+m) - f(i-m)), evaluated
// from the outermost pair inwards as the reference writes it.
template <int NG, typename T, class F>
__device__ __forceinline__ T cds_correction(const F &f, int l) {
  if constexpr (NG == 3) {
    const T c1 = T(-19.0 / 3840), c2 = T(13.0 / 320), c3 = T(-17.0 / 256);
    return c1 * (f(3, l) - f(-3, l)) + c2 * (f(2, l) - f(-2, l)) + c3 * (f(1, l) - f(-1, l));
  } else {
    const T c4 = T(-81.0 / 71680), c3 = T(1261.0 / 107520), c2 = T(-289.0 / 5120), c1 = T(421.0 / 5120);
    return c4 * (f(4, l) - f(-4, l)) + c3 * (f(3, l) - f(-3, l)) + c2 * (f(2, l) - f(-2, l)) +
           c1 * (f(1, l) - f(-1, l));
  }
}

}  // namespace ostc
