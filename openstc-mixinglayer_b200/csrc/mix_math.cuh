// mix_math.cuh -- device arithmetic of the multi-component (species = 1) path: NASA-7 thermodynamics,
// mixture transport, the temperature Newton iteration, finite-rate chemistry and the flux-split
// characteristic WENO7-Z face flux.  The species and reaction tables sit in constant memory: every
// thread of a warp reads the same coefficient at the same time, which the constant cache broadcasts.
#pragma once

#include "air_math.cuh"

namespace ostc {

constexpr int kMS = 16;  // species capacity of the device tables
constexpr int kMR = 64;  // reaction capacity
constexpr int kMol = 4, kNet = 6;  // molecules a side and species of a reaction in the lists of MixTables
constexpr double kPatmD = 101325.0;

// Species count as a compile-time constant: NS > 0 instantiates for exactly NS species (arrays in
// registers, loops unrolled); NS = 0 is the generic build that reads the count from the tables.
template <int NS> struct Spec {
  static constexpr int A = NS > 0 ? NS : kMS;  // array extent
};
#define OSTC_NS (NS > 0 ? NS : c_mix.ns)

template <typename T> __device__ __forceinline__ T tpow(T x, T y);
template <> __device__ __forceinline__ double tpow<double>(double x, double y) { return pow(x, y); }
template <> __device__ __forceinline__ float tpow<float>(float x, float y) { return powf(x, y); }
}  // namespace ostc
#include "dual.cuh"
namespace ostc {

struct MixTables {
  int ns, nr;
  int use_gibbs;  // some reaction takes kb from the equilibrium constant (backward_reaction_rate's n_gibbs)
  double weno_eps_scale, v_ref;
  double mw[kMS], imw[kMS], ru_mw[kMS], t_low[kMS], t_mid[kMS];
  double low[kMS][7], high[kMS][7];
  // the polynomials' integrals below / above t_mid: h / Ru T's a1/2, a2/3, a3/4, a4/5 and the Gibbs
  // energy's a1/2, a2/6, a3/12, a4/20, so that no evaluation divides
  double hint[2][kMS][4], gint[2][kMS][4];
  double lj_potent_inv[kMS], vis_coeff[kMS];
  double wj_div_wi_1_4[kMS][kMS], sqrt_wiwj_8[kMS][kMS], binary_diff[kMS][kMS], kb_over_eps[kMS][kMS];
  // collision integrals c T*^-0.145 + (T* + 0.5)^-2 at T* = T lj_potent_inv or T kb_over_eps: the constants'
  // powers lj_pow = 1.147 lj_potent_inv^-0.145 and, over the binary diffusion coefficient, kbe_pow =
  // kb_over_eps^-0.145 / D and inv_diff = 1 / D, so that a node takes one power of T for all of them
  double lj_pow[kMS], kbe_pow[kMS][kMS], inv_diff[kMS][kMS];
  int label[kMR], rev_type[kMR], order[kMR];
  signed char stoi_f[kMR][kMS], stoi_b[kMR][kMS];
  // the same by molecules: species of every forward / backward molecule of a reaction (kMol at most) and
  // its net coefficients by species (kNet at most); listed = 0 if some reaction has more
  int listed;
  signed char n_f[kMR], n_b[kMR], n_net[kMR], mol_f[kMR][kMol], mol_b[kMR][kMol], net[kMR][kNet];
  double nu[kMR][kNet];
  double A[kMR], b[kMR], Ea[kMR], A2[kMR], b2[kMR], Ea2[kMR], third_body[kMR][kMS];
  double troe_alpha[kMR], troe_t3[kMR], troe_t1[kMR], troe_t2[kMR];
};

// the tables of the bound context (one translation unit includes this header)
__constant__ MixTables c_mix;

// One species of compute_enthalpy_and_cp (Thermo.cu:136-192): h_i and cp_i in J/kg, cp frozen and h
// extrapolated linearly below t_low.  Horner form on the integrated coefficients of the tables: 10
// multiply-adds where the powers, products and quotients of the written form took about 45 operations,
// a division by 3 among them.
template <typename T = double>
__device__ __forceinline__ void mix_h_cp_one(int i, T t, T &h, T &cp) {
  const T tl = (T)c_mix.t_low[i];
  const T tt = t < tl ? tl : t;
  const int hi = tt < (T)c_mix.t_mid[i] ? 0 : 1;
  const double *a = hi ? c_mix.high[i] : c_mix.low[i];
  const double *q = c_mix.hint[hi][i];
  cp = ((((T)a[4] * tt + (T)a[3]) * tt + (T)a[2]) * tt + (T)a[1]) * tt + (T)a[0];
  h = ((((T)q[3] * tt + (T)q[2]) * tt + (T)q[1]) * tt + (T)q[0]) * tt + (T)a[0];
  h = h * tt + (T)a[5];
  h = cp * (t - tt) + h;
  h = h * (T)c_mix.ru_mw[i];
  cp = cp * (T)c_mix.ru_mw[i];
}

// compute_enthalpy_and_cp (Thermo.cu:136-192) of every species.  Either output may be null
// (compute_enthalpy / compute_cp).
template <int NS, typename T = double>
__device__ __forceinline__ void mix_h_cp(T t, T *h, T *cp) {
#pragma unroll
  for (int i = 0; i < OSTC_NS; ++i) {
    T hh, cc;
    mix_h_cp_one<T>(i, t, hh, cc);
    if (h) h[i] = hh;
    if (cp) cp[i] = cc;
  }
}

// compute_gibbs_div_rt (Thermo.cu:194-210), evaluated at t_low below it
template <int NS, typename T = double>
__device__ __forceinline__ void mix_gibbs_rt(T t, T *g) {
  const T ti = 1 / t, lt = log(t);
#pragma unroll
  for (int i = 0; i < OSTC_NS; ++i) {
    if (t < c_mix.t_low[i]) {
      const double tt = c_mix.t_low[i];
      const double *a = c_mix.low[i], *q = c_mix.gint[0][i];
      g[i] = a[0] * (1.0 - log(tt)) - tt * (q[0] + tt * (q[1] + tt * (q[2] + tt * q[3]))) + a[5] / tt - a[6];
    } else {
      const int hi = t < c_mix.t_mid[i] ? 0 : 1;
      const double *a = hi ? c_mix.high[i] : c_mix.low[i];
      const double *q = c_mix.gint[hi][i];
      g[i] = a[0] * (1.0 - lt) - t * (q[0] + t * (q[1] + t * (q[2] + t * q[3]))) + a[5] * ti - a[6];
    }
  }
}

// a / x and b / y.  FP64 takes one division for both (x y stays in range for the callers' factors, squares
// of reduced temperatures and the like); FP32 two fast ones.
__device__ __forceinline__ void div2(double a, double x, double b, double y, double &ax, double &by) {
  const double q = 1.0 / (x * y);
  ax = a * (y * q);
  by = b * (x * q);
}
__device__ __forceinline__ void div2(float a, float x, float b, float y, float &ax, float &by) {
  ax = __fdividef(a, x);
  by = __fdividef(b, y);
}

// Node properties of update_physical_properties<mixture> (FieldOperation.cuh:116-134) with
// compute_transport_property (Transport.cu:43-136): cp, gamma, acoustic speed, Wilke viscosity,
// Eucken-type conductivity and mixture-averaged rho*D_k (outputs written through the pointers).
// Bound by its divisions, powers and square roots, so their number is what the form minimises: one log
// and one exp a node (T^-0.145; the constants' powers are in the tables), one reciprocal square root a
// species (both square roots of the viscosities' ratios), one division for the two quotients of a
// species' viscosity and conductivity, and one for the (T* + 0.5)^2 of two species pairs - about 50
// where the written form takes 45 exponentials and 200 divisions for 9 species.  192 x 96 x 48: FP64 0.60 ->
// 0.31 ms a sweep; 257 x 129 x 65 in FP32 0.90 -> 0.61 ms.
template <int NS, typename T = double>
__device__ __forceinline__ void mix_properties(T rho, T p, T t, const T *y, T &gamma, T &acoustic, T &mu, T &cond,
                                               T *rhod) {
  const int ns = OSTC_NS;
  T cp[Spec<NS>::A];
  mix_h_cp<NS, T>(t, nullptr, cp);
  T mw = 0, cpt = 0, cvt = 0;
  for (int l = 0; l < ns; ++l) {
    mw += y[l] * (T)c_mix.imw[l];
    cpt += y[l] * cp[l];
    cvt += y[l] * (cp[l] - (T)c_mix.ru_mw[l]);
  }
  const T smw = mw;
  mw = 1 / mw;
  gamma = cpt / cvt;
  acoustic = tsqrt(gamma * T(kRuD) * t * smw);
  T X[Spec<NS>::A], vis[Spec<NS>::A], svis[Spec<NS>::A], isvis[Spec<NS>::A];
  const T st = tsqrt(t), tp = exp(T(-0.145) * log(t));
#pragma unroll
  for (int l = 0; l < ns; ++l) {
    X[l] = y[l] * mw * (T)c_mix.imw[l];
    // vis = coeff sqrt(T) / (lj_pow T^-0.145 + (T* + 0.5)^-2)
    const T a = t * (T)c_mix.lj_potent_inv[l] + T(0.5), a2 = a * a;
    vis[l] = (T)c_mix.vis_coeff[l] * st * a2 / ((T)c_mix.lj_pow[l] * tp * a2 + T(1));
    isvis[l] = rsqrt(vis[l]);
    svis[l] = vis[l] * isvis[l];
  }
  T visc = 0, cd = 0;
#pragma unroll
  for (int m = 0; m < ns; ++m) {
    T vt = 0;
#pragma unroll
    for (int n = 0; n < ns; ++n) {
      T pf = 1;
      if (m != n) {
        const T num = T(1) + svis[m] * isvis[n] * (T)c_mix.wj_div_wi_1_4[m][n];
        pf = num * num * (T)c_mix.sqrt_wiwj_8[m][n];
      }
      vt += pf * X[n];
    }
    const T ct = T(1.065) * vt - T(0.065) * X[m];
    const T vx = vis[m] * X[m];
    T a, c;
    div2(vx, vt, vx * (cp[m] + T(1.25) * (T)c_mix.ru_mw[m]), ct, a, c);
    visc += a;
    cd += c;
  }
  mu = visc;
  cond = cd;
  // mixture-averaged diffusion with the binary coefficients D_ln = coeff T^1.5 / (p Omega_D(T*)).
  // D_ln is symmetric in (l, n) (its tables are), so each pair is evaluated once and added to both
  // species' sums; w = T^1.5 / (p D_ln), two pairs sharing a division.
  const T eps = T(1e-12);
  T num[Spec<NS>::A], den[Spec<NS>::A];
  for (int l = 0; l < ns; ++l) num[l] = den[l] = 0;
  auto pair = [&](int l, int n, T q) {  // q = (T* + 0.5)^-2 / D
    const T w = tp * (T)c_mix.kbe_pow[l][n] + q;
    num[l] += (X[n] + eps) * (T)c_mix.mw[n];
    den[l] += (X[n] + eps) * w;
    num[n] += (X[l] + eps) * (T)c_mix.mw[l];
    den[n] += (X[l] + eps) * w;
  };
  auto sq = [&](int l, int n) -> T {
    const T a = t * (T)c_mix.kb_over_eps[l][n] + T(0.5);
    return a * a;
  };
#pragma unroll
  for (int l = 0; l < ns; ++l) {
#pragma unroll
    for (int n = l + 1; n < ns; n += 2) {
      T q0, q1;
      if (n + 1 < ns) {
        div2((T)c_mix.inv_diff[l][n], sq(l, n), (T)c_mix.inv_diff[l][n + 1], sq(l, n + 1), q0, q1);
        pair(l, n, q0);
        pair(l, n + 1, q1);
      } else {
        pair(l, n, (T)c_mix.inv_diff[l][n] / sq(l, n));
      }
    }
  }
  const T rs = rho * smw * (t * st / p);
#pragma unroll
  for (int l = 0; l < ns; ++l) rhod[l] = rs * num[l] / den[l];
}

// compute_temperature_and_pressure (FieldOperation.cu:3-40): Newton on e(T) starting from t, relative
// tolerance 1e-3, at most 1000 iterations.  Returns T; p = rho R T through pout.
template <int NS, typename T = double>
__device__ __forceinline__ T mix_temperature(T rho, T e, T t, const T *y, T &pout) {
  const int ns = OSTC_NS;
  T mw = 0;
  for (int l = 0; l < ns; ++l) mw += y[l] * c_mix.imw[l];
  mw = 1 / mw;
  const T gc = kRuD / mw;
  T err = 1.0;
  int iter = 0;
  T h[Spec<NS>::A], cp[Spec<NS>::A];
  while (err > 1e-3 && iter++ < 1000) {
    mix_h_cp<NS, T>(t, h, cp);
    T cpt = 0.0, hm = 0.0;
    for (int l = 0; l < ns; ++l) {
      cpt += cp[l] * y[l];
      hm += h[l] * y[l];
    }
    const T t1 = t - (hm - gc * t - e) / (cpt - gc);
    err = fabs(1 - t1 / t);
    t = t1;
  }
  pout = rho * t * gc;
  return t;
}

// A T^b exp(-Ea/T) (arrhenius, FiniteRateChem.cu:104-106) as A exp(b ln T - Ea/T): one exp per
// rate with ln T and 1/T formed once per node (the argument's rounding, ~1e-16 of |Ea/T| <= ~60,
// is the only difference from pow * exp)
__device__ __forceinline__ double arrhenius(double lt, double ti, double A, double b, double Ea) {
  return A * exp(fma(b, lt, -Ea * ti));
}

// x^n for the small integer reaction orders of the equilibrium constant, pow beyond |n| = 2
template <typename T>
__device__ __forceinline__ T ipow(T x, int n) {
  switch (n) {
    case 0: return T(1.0);
    case 1: return x;
    case -1: return 1.0 / x;
    case 2: return x * x;
    case -2: return 1.0 / (x * x);
    default: return pow(x, (double)n);
  }
}

__device__ __forceinline__ double texp10(double x) { return exp10(x); }
__device__ __forceinline__ Dual texp10(const Dual &x) { return pow(10.0, x); }

// Forward rate constant of reaction r (forward_reaction_rate, FiniteRateChem.cu:60-102) at T (with ln T,
// 1/T) and the third-body concentration sum cc.
template <typename T>
__device__ __forceinline__ T reaction_kf(int r, T t, T lt, T ti, T cc) {
  const int ty = c_mix.label[r];
  T kf = arrhenius(lt, ti, c_mix.A[r], c_mix.b[r], c_mix.Ea[r]);
  if (ty == 3) {
    kf += arrhenius(lt, ti, c_mix.A2[r], c_mix.b2[r], c_mix.Ea2[r]);
  } else if (ty == 4) {
    kf *= cc;
  } else if (ty > 4) {
    const T klow = arrhenius(lt, ti, c_mix.A2[r], c_mix.b2[r], c_mix.Ea2[r]);
    const T pr = klow * cc / kf;
    T F = 1.0;
    if (ty > 5) {
      T fc = (1 - c_mix.troe_alpha[r]) * exp(-t / c_mix.troe_t3[r]) +
                  c_mix.troe_alpha[r] * exp(-t / c_mix.troe_t1[r]);
      if (ty == 7) fc += exp(-c_mix.troe_t2[r] / t);
      const T lfc = log10(fc);
      const T cq = -0.4 - 0.67 * lfc, nq = 0.75 - 1.27 * lfc;
      const T lpr = log10(pr);
      const T tmp = (lpr + cq) / (nq - 0.14 * (lpr + cq));
      F = texp10(lfc / (1.0 + tmp * tmp));
    }
    kf = kf * pr / (1.0 + pr) * F;
  }
  return kf;
}

// Backward rate constant (backward_reaction_rate, FiniteRateChem.cu:104-150), dg = sum (nu_b - nu_f) g / (Ru T)
// where the equilibrium constant is used.  Irreversible: 0; the equilibrium constant for every other type
// but 2 when any reaction needs it (it also overwrites REV coefficients); else the REV Arrhenius
// coefficients (times the third-body sum for type 4).
template <typename T>
__device__ __forceinline__ T reaction_kb(int r, T lt, T ti, T cc, T kf, T dg) {
  const int ty = c_mix.label[r];
  if (ty == 0) return T(0.0);
  if (ty != 2 && c_mix.use_gibbs) {
    // kf / (temp_t^order exp(-dg)), temp_t = p_atm / (Ru T) 1e-3
    const T q = kf * exp(dg), temp_t = (kPatmD / kRuD * 1e-3) * ti;
    switch (c_mix.order[r]) {
      case 0: return q;
      case -1: return q * temp_t;
      case 1: return q / temp_t;
      default: return q / ipow(temp_t, c_mix.order[r]);
    }
  }
  if (c_mix.rev_type[r] == 1) {
    const T kb = arrhenius(lt, ti, c_mix.A2[r], c_mix.b2[r], c_mix.Ea2[r]);
    return ty == 4 ? kb * cc : kb;
  }
  return T(0.0);
}

// Both rate constants of reaction r; g: g_k / (Ru T) of every species.
template <int NS, typename T>
__device__ __forceinline__ void reaction_rates(int r, T t, T lt, T ti, T cc, const T *g, T &kf_out, T &kb_out) {
  const T kf = reaction_kf<T>(r, t, lt, ti, cc);
  T dg = 0;
  if (c_mix.use_gibbs && c_mix.label[r] != 0 && c_mix.label[r] != 2)
    for (int l = 0; l < OSTC_NS; ++l) dg += g[l] * (double)(c_mix.stoi_b[r][l] - c_mix.stoi_f[r][l]);
  kf_out = kf;
  kb_out = reaction_kb<T>(r, lt, ti, cc, kf, dg);
}

// The species arrays of one thread in shared memory: element e of `threads` interleaved columns, so that
// a reaction can address its species by list (a register array cannot be indexed) and consecutive threads
// stay on consecutive words.
struct ChemColumn {
  double *base;
  int threads;
  __device__ __forceinline__ double &operator()(int e) const { return base[(long long)e * threads]; }
};
// columns: concentrations, Gibbs energies, rates (ns each), and with the Jacobian ns x ns
__host__ __device__ constexpr int chem_columns(int ns, bool jac) { return 3 * ns + (jac ? ns * ns : 0); }

// finite_rate_chemistry (FiniteRateChem.cu:7-58, rates :60-195) over the reaction lists: omega_k in kg/(m^3 s)
// into om(k), and with JAC the Jacobian of compute_chem_src_jacobian (:197-217) into jc(m ns + n), in 1/s.
// Per reaction the sums run over its own species instead of all of them; the rates of a species add its
// net coefficient times q1 - q2 per reaction (the reference adds creation and destruction apart).
template <int NS, bool JAC>
__device__ __forceinline__ void mix_chemistry_listed(double rho, double t, const double *y, ChemColumn c, ChemColumn g,
                                                     ChemColumn om, ChemColumn jc) {
  const int ns = OSTC_NS, nr = c_mix.nr;
  const double lt = log(t), ti = 1.0 / t;
  for (int l = 0; l < ns; ++l) {
    c(l) = rho * y[l] * c_mix.imw[l] * 1e-3;
    om(l) = 0.0;
  }
  if (c_mix.use_gibbs) {
    double gr[Spec<NS>::A];
    mix_gibbs_rt<NS, double>(t, gr);
    for (int l = 0; l < ns; ++l) g(l) = gr[l];
  }
  if (JAC)
    for (int e = 0; e < ns * ns; ++e) jc(e) = 0.0;
#pragma unroll 1
  for (int r = 0; r < nr; ++r) {
    double cc = 0;
    if (c_mix.label[r] >= 4)
      for (int l = 0; l < ns; ++l) cc += c(l) * c_mix.third_body[r][l];
    const int nf = c_mix.n_f[r], nb = c_mix.n_b[r], nn = c_mix.n_net[r];
    double dg = 0;
    if (c_mix.use_gibbs)
      for (int e = 0; e < nn; ++e) dg += c_mix.nu[r][e] * g(c_mix.net[r][e]);
    double q1 = reaction_kf<double>(r, t, lt, ti, cc);
    double q2 = reaction_kb<double>(r, lt, ti, cc, q1, dg);
    for (int e = 0; e < nf; ++e) q1 *= c(c_mix.mol_f[r][e]);
    for (int e = 0; e < nb; ++e) q2 *= c(c_mix.mol_b[r][e]);
    const double q = q1 - q2;
    for (int e = 0; e < nn; ++e) {
      const int m = c_mix.net[r][e];
      const double nu = c_mix.nu[r][e];
      om(m) += nu * q;
      if (JAC) {
        for (int a = 0; a < nf; ++a) jc(m * ns + c_mix.mol_f[r][a]) += nu * q1;
        for (int a = 0; a < nb; ++a) jc(m * ns + c_mix.mol_b[r][a]) -= nu * q2;
      }
    }
  }
  for (int l = 0; l < ns; ++l) om(l) = om(l) * (c_mix.mw[l] * 1e+3);
  if (JAC) {
    for (int n = 0; n < ns; ++n) {
      const bool live = y[n] > 1e-25;
      const double inv = live ? 1.0 / (rho * y[n]) : 0.0;
      for (int m = 0; m < ns; ++m) jc(m * ns + n) = c_mix.mw[m] * (live ? jc(m * ns + n) * inv : 0.0) * 1e+3;
    }
  }
}

// finite_rate_chemistry (FiniteRateChem.cu:7-58, rates :60-195): omega_k in kg/(m^3 s) at one node.
// With jac non-null also the chemical source Jacobian of compute_chem_src_jacobian
// (FiniteRateChem.cu:197-217), [ns][ns] row-major, in 1/s; with omega_d non-null the destruction
// rates omega_d,k of chemical_source (:179-195), kg/(m^3 s).
template <int NS, typename T = double>
__device__ __forceinline__ void mix_chemistry(T rho, T t, const T *y, T *omega, T *jac = nullptr,
                                              T *omega_d = nullptr) {
  const int ns = OSTC_NS, nr = c_mix.nr;
  const T lt = log(t), ti = 1.0 / t;
  T c[Spec<NS>::A];
  for (int l = 0; l < ns; ++l) c[l] = rho * y[l] * c_mix.imw[l] * 1e-3;
  T g[Spec<NS>::A];
  if (c_mix.use_gibbs) mix_gibbs_rt<NS, T>(t, g);
  for (int l = 0; l < ns; ++l) omega[l] = 0;
  T cre[Spec<NS>::A], des[Spec<NS>::A];
  for (int l = 0; l < ns; ++l) cre[l] = des[l] = 0;
  for (int r = 0; r < nr; ++r) {
    const int ty = c_mix.label[r];
    T cc = 0;
    if (ty >= 4)
      for (int l = 0; l < ns; ++l) cc += c[l] * c_mix.third_body[r][l];
    T kf, kb;
    reaction_rates<NS, T>(r, t, lt, ti, cc, g, kf, kb);
    // concentration products: integer powers as products (pow(c, 1) = c, pow(c, 2) = c*c to within
    // the rounding of pow itself), pow only for higher orders
    T q1 = 1.0, q2 = ty != 0 ? 1.0 : 0.0;
#pragma unroll
    for (int l = 0; l < ns; ++l) {
      const int nf = c_mix.stoi_f[r][l];
      if (nf == 1) q1 *= c[l];
      else if (nf == 2) q1 *= c[l] * c[l];
      else if (nf) q1 *= pow(c[l], (double)nf);
    }
    if (ty != 0) {
#pragma unroll
      for (int l = 0; l < ns; ++l) {
        const int nb = c_mix.stoi_b[r][l];
        if (nb == 1) q2 *= c[l];
        else if (nb == 2) q2 *= c[l] * c[l];
        else if (nb) q2 *= pow(c[l], (double)nb);
      }
    }
    q1 *= kf;
    if (ty != 0) q2 *= kb;
    if (jac) {
      // sum over reactions in order, per (m, n): (nu_b,m - nu_f,m)(nu_f,n q1 - nu_b,n q2)
#pragma unroll
      for (int m = 0; m < ns; ++m) {
        const int dm = c_mix.stoi_b[r][m] - c_mix.stoi_f[r][m];
        if (dm == 0) continue;
#pragma unroll
        for (int n = 0; n < ns; ++n)
          jac[m * ns + n] += dm * (c_mix.stoi_f[r][n] * q1 - c_mix.stoi_b[r][n] * q2);
      }
    }
    for (int l = 0; l < ns; ++l) {
      cre[l] += q2 * c_mix.stoi_f[r][l] + q1 * c_mix.stoi_b[r][l];
      des[l] += q1 * c_mix.stoi_f[r][l] + q2 * c_mix.stoi_b[r][l];
    }
  }
  for (int l = 0; l < ns; ++l) omega[l] = cre[l] * (c_mix.mw[l] * 1e+3) - des[l] * (c_mix.mw[l] * 1e+3);
  if (omega_d)
    for (int l = 0; l < ns; ++l) omega_d[l] = des[l] * (c_mix.mw[l] * 1e+3);
  if (jac) {
#pragma unroll
    for (int n = 0; n < ns; ++n) {
      const bool live = y[n] > 1e-25;
      const T inv = live ? 1.0 / (rho * y[n]) : 0.0;
#pragma unroll
      for (int m = 0; m < ns; ++m) jac[m * ns + n] = c_mix.mw[m] * (live ? jac[m * ns + n] * inv : 0.0) * 1e+3;
    }
  }
}

// solve_chem_system (FiniteRateChem.cu:302-357) on columns: LU with partial pivoting of the ns x ns matrix
// a in place, right-hand side x solved in place.  The pivot search and the row exchange index the matrix
// by a value of their own per thread, which registers cannot; the row at hand is held in registers.
template <int NS>
__device__ __forceinline__ void mix_lu_solve_columns(ChemColumn a, ChemColumn x) {
  const int dim = OSTC_NS;
#pragma unroll 1
  for (int n = 0; n < dim; ++n) {
    int ik = n;
    double best = fabs(a(n * dim + n));
    for (int m = n + 1; m < dim; ++m) {
      const double v = fabs(a(m * dim + n));
      if (v > best) {
        best = v;
        ik = m;
      }
    }
    double row[Spec<NS>::A];
    for (int t = 0; t < dim; ++t) {
      row[t] = a(ik * dim + t);
      if (ik != n) a(ik * dim + t) = a(n * dim + t);
      a(n * dim + t) = row[t];
    }
    const double xn = x(ik);
    if (ik != n) x(ik) = x(n);
    x(n) = xn;
    const double ip = 1.0 / a(n * dim + n);
    for (int m = n + 1; m < dim; ++m) {
      const double f = a(m * dim + n) * ip;
      for (int t = 0; t < dim; ++t)
        if (t > n) a(m * dim + t) -= f * row[t];
      x(m) -= f * xn;
    }
  }
#pragma unroll 1
  for (int m = dim - 1; m >= 0; --m) {
    double v = x(m);
    for (int t = m + 1; t < dim; ++t) v -= a(m * dim + t) * x(t);
    x(m) = v / a(m * dim + m);
  }
}

// solve_chem_system (FiniteRateChem.cu:302-357): column-pivoted LU of the ns x ns matrix lhs in place,
// then forward / back substitution of b (length ns) in place.
template <int NS>
__device__ __forceinline__ void mix_lu_solve(double *lhs, double *b) {
  const int dim = OSTC_NS;
  int ipiv[Spec<NS>::A];
  for (int n = 0; n < dim; ++n) {
    int ik = n;
    for (int m = n; m < dim; ++m) {
      for (int t = 0; t < n; ++t) lhs[m * dim + n] -= lhs[m * dim + t] * lhs[t * dim + n];
      if (fabs(lhs[m * dim + n]) > fabs(lhs[ik * dim + n])) ik = m;
    }
    ipiv[n] = ik;
    if (ik != n)
      for (int t = 0; t < dim; ++t) {
        const double mid = lhs[ik * dim + t];
        lhs[ik * dim + t] = lhs[n * dim + t];
        lhs[n * dim + t] = mid;
      }
    for (int p = n + 1; p < dim; ++p)
      for (int t = 0; t < n; ++t) lhs[n * dim + p] -= lhs[n * dim + t] * lhs[t * dim + p];
    for (int m = n + 1; m < dim; ++m) lhs[m * dim + n] /= lhs[n * dim + n];
  }
  for (int m = 0; m < dim; ++m) {
    const int t = ipiv[m];
    if (t != m) {
      const double mid = b[t];
      b[t] = b[m];
      b[m] = mid;
    }
  }
  for (int m = 1; m < dim; ++m)
    for (int t = 0; t < m; ++t) b[m] -= lhs[m * dim + t] * b[t];
  b[dim - 1] /= lhs[dim * dim - 1];
  for (int m = dim - 2; m >= 0; --m) {
    for (int t = m + 1; t < dim; ++t) b[m] -= lhs[m * dim + t] * b[t];
    b[m] /= lhs[m * dim + m];
  }
}

// ---------------------------------------------------------------- flux-split WENO7 (71 / 72)

template <typename T>
__device__ __forceinline__ T fvs_beta7(T s1, T s2, T s3) {
  return s1 * (s1 + T(1.0 / 12) * s3) + T(13.0 / 12.0) * s2 * s2 + T(1043.0 / 960) * s3 * s3;
}

// 1 / (eps + beta_k) of the four Z weights: from one division where the product of the four stays in range (on
// a smooth stencil, an eps above 1e-75), else each takes its own.
__device__ __forceinline__ void fvs_inverses(double eps, const double *b, double *r) {
  const double g0 = eps + b[0], g1 = eps + b[1], g2 = eps + b[2], g3 = eps + b[3];
  const double p01 = g0 * g1, p23 = g2 * g3, p = p01 * p23;
  if (p > 1e-300 && p < 1e300) {
    const double q = 1.0 / p, q01 = p23 * q, q23 = p01 * q;
    r[0] = g1 * q01;
    r[1] = g0 * q01;
    r[2] = g3 * q23;
    r[3] = g2 * q23;
  } else {
    r[0] = 1.0 / g0;
    r[1] = 1.0 / g1;
    r[2] = 1.0 / g2;
    r[3] = 1.0 / g3;
  }
}

// tau / D_k of the four Z weights, D_k = (eps + beta_k)^2.  FP32: four fast divisions, D_k floored at 1e-30 so that
// a smooth stencil (beta = 0, where the scaled eps underflows) gives the linear weights instead of 0/0.
__device__ __forceinline__ void fvs_ratios(double tau, double eps, const double *b, double *r) {
  fvs_inverses(eps, b, r);
#pragma unroll
  for (int k = 0; k < 4; ++k) r[k] = tau * (r[k] * r[k]);
}
__device__ __forceinline__ void fvs_ratios(float tau, float eps, const float *b, float *r) {
#pragma unroll
  for (int k = 0; k < 4; ++k) r[k] = __fdividef(tau, fmaxf((eps + b[k]) * (eps + b[k]), 1e-30f));
}

// One side of the flux-split WENO7-Z (WENO.cu:1619-1693), its points v0..v6 upwind first: the face value
// is v3 + num / den.  The reference's derivatives s1, s2, s3 of each substencil and its interpolants are
// written with the first, second and third differences the substencils share: s1 = d + e/2 + t/3 and
// alike (the coefficients are those of WENO.cu:1626-1655 term by term), and the interpolant of every
// substencil is v3 + s1/2 + s2/12.  That takes 50 operations for the four indicators and interpolants
// instead of 110 from the points, and its differences lose no digits to the points' size.
template <typename T>
__device__ __forceinline__ void fvs_side(T v0, T v1, T v2, T v3, T v4, T v5, T v6, T eps, T &num, T &den) {
  const T d2 = v3 - v2, d3 = v4 - v3;
  const T e0 = (v2 - v1) - (v1 - v0), e1 = d2 - (v2 - v1), e2 = d3 - d2, e3 = (v5 - v4) - d3;
  const T e4 = (v6 - v5) - (v5 - v4);
  const T t0 = e1 - e0, t1 = e2 - e1, t2 = e3 - e2, t3 = e4 - e3;
  const T mid = d2 + T(0.5) * e2;
  const T s1[4] = {d2 + (T(0.5) * e1 + T(1.0 / 3) * t0), mid - T(1.0 / 6) * t1, mid - T(1.0 / 6) * t2,
                   d3 - (T(0.5) * e3 - T(1.0 / 3) * t3)};
  const T s2[4] = {e1 + t0, e2, e2, e3 - t3};
  const T s3[4] = {t0, t1, t2, t3};
  const T c[4] = {T(1.0 / 35), T(12.0 / 35), T(18.0 / 35), T(4.0 / 35)};
  T b[4], r[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) b[k] = fvs_beta7(s1[k], s2[k], s3[k]);
  fvs_ratios((b[0] - b[3]) * (b[0] - b[3]), eps, b, r);
  num = T(0);
  den = T(0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const T a = c[k] + c[k] * r[k];
    num += a * (T(0.5) * s1[k] + T(1.0 / 12) * s2[k]);
    den += a;
  }
}

// Both sides of the flux-split WENO7-Z: f+ + f-, the - side mirrored.  FP64 forms the two quotients with
// one division by the product of the two weight sums, which are at most tau / eps^2, ~1e80 with the epsilon of a
// reference state.  EPS0: no reference state, epsilon 0; a substencil of vanishing fluxes (a mass fraction of 1e-50
// beside one of 1e-3) then has a weight of 1e190 and each side takes its own division.
template <typename T, bool EPS0 = false>
__device__ __forceinline__ T fvs_weno7_core(const T *vp, const T *vm, T eps) {
  T np, dp, nm, dm;
  fvs_side(vp[0], vp[1], vp[2], vp[3], vp[4], vp[5], vp[6], eps, np, dp);
  fvs_side(vm[6], vm[5], vm[4], vm[3], vm[2], vm[1], vm[0], eps, nm, dm);
  if constexpr (sizeof(T) == 8) return vp[3] + vm[3] + (EPS0 ? np / dp + nm / dm : (np * dm + nm * dp) / (dp * dm));
  else return vp[3] + vm[3] + (__fdividef(np, dp) + __fdividef(nm, dm));
}

template <bool EPS0 = false>
__device__ __forceinline__ double fvs_weno7(const double *vp, const double *vm, double eps) {
  return fvs_weno7_core<double, EPS0>(vp, vm, eps);
}

// FP32 form.  beta ~ v^2 and tau ~ v^4, so the split fluxes of a minor species (|v| ~ 1e-11) or the
// energy flux of a coarse grid (|v| ~ 1e10) leave the FP32 range although the weights themselves
// (tau / (eps + beta)^2, scale-free as eps -> 0) are O(1).  The stencil is therefore scaled by the
// power of two 2^-E below its largest magnitude (exact), eps by 2^-2E, and the face value scaled back.
template <bool EPS0 = false>
__device__ __forceinline__ float fvs_weno7(const float *vp, const float *vm, double eps) {
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < 7; ++i) m = fmaxf(m, fmaxf(fabsf(vp[i]), fabsf(vm[i])));
  if (!(m > 0.f)) {  // all zero: the face value is 0 (or NaN, carried through)
    float z = 0.f;
#pragma unroll
    for (int i = 0; i < 7; ++i) z += vp[i] + vm[i];
    return z;
  }
  int ex = (__float_as_int(m) >> 23) & 0xff;  // biased exponent of m
  ex = ex < 1 ? 1 : (ex > 253 ? 253 : ex);
  const float inv = __int_as_float((254 - ex) << 23);  // 2^(127 - ex)
  const float scale = __int_as_float(ex << 23);        // 2^(ex - 127)
  float sp[7], sm[7];
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    sp[i] = vp[i] * inv;
    sm[i] = vm[i] * inv;
  }
  const double id = (double)inv;
  const float e = (float)(eps * id * id);
  return fvs_weno7_core<float>(sp, sm, e) * scale;
}

}  // namespace ostc
