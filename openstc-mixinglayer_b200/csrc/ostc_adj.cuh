// ostc_adj.cuh -- vector-Jacobian product of the multi-component right-hand side (ostc_rhs_vjp):
// cv_bar = (d dq / d cv)^T dq_bar at the current state, for the flux-split WENO7 sweeps (71 / 72),
// the mixture viscous sweeps, the finite-rate chemistry source, the mixture transport properties, the
// equation of state and the periodic / outflow ghost fills.  The reference has no adjoint; this is
// the discrete adjoint of the forward kernels in ostc_mix.cuh, term by term:
//   1. face sweeps (hand-written reverse): dq_bar -> adjoints of the node quantities they read
//      (cv, p, acoustic speed; u, v, w, T, Y, mu, lambda, rho*D), accumulated per padded node;
//   2. chemistry and transport properties (node-local, hand-written; Dual evaluations only of fall-off rates
//      and, for mechanisms that do not fit the reaction lists, of every rate): -> adjoints of rho, p, T, Y;
//   3. equation of state reverse (rho, u, v, w, p, T, Y as functions of cv, T through the
//      implicit energy relation) -> cv adjoint per padded node;
//   4. ghost fills in reverse order: a ghost's cv adjoint is added to the node it was copied from.
// Accumulation into the node planes uses atomicAdd, so results are reproducible to rounding, not bitwise.
#pragma once

#include "ostc_mix.cuh"

namespace ostc {

// Node adjoint planes (padded layout of the state): cv[nv], p, c (acoustic speed), rho, vel[3], T,
// Y[ns], mu, lam (conductivity), rhod[ns].
struct DevAdj {
  double *cv, *p, *c, *rho, *vel, *T, *Y, *mu, *lam, *rhod;
};

// One side of the flux-split WENO7-Z (fvs_side) and its gradient: v[0..6] upwind first; returns the side's
// face value and sets g[j] = af d(value) / d v[j].  In the differences fvs_side shares; the third
// smoothness indicator reuses the second stencil's second difference, as the forward function does.
__device__ __forceinline__ double weno7_side_bwd(const double *v, double eps, double af, double *g) {
  const double c[4] = {1.0 / 35, 12.0 / 35, 18.0 / 35, 4.0 / 35};
  const double d2 = v[3] - v[2], d3 = v[4] - v[3];
  const double e0 = (v[2] - v[1]) - (v[1] - v[0]), e1 = d2 - (v[2] - v[1]), e2 = d3 - d2, e3 = (v[5] - v[4]) - d3;
  const double e4 = (v[6] - v[5]) - (v[5] - v[4]);
  const double t0 = e1 - e0, t1 = e2 - e1, t2 = e3 - e2, t3 = e4 - e3;
  const double mid = d2 + 0.5 * e2;
  const double s1[4] = {d2 + (0.5 * e1 + (1.0 / 3) * t0), mid - (1.0 / 6) * t1, mid - (1.0 / 6) * t2,
                        d3 - (0.5 * e3 - (1.0 / 3) * t3)};
  const double s2[4] = {e1 + t0, e2, e2, e3 - t3};
  const double s3[4] = {t0, t1, t2, t3};
  double b[4], id[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) b[k] = fvs_beta7(s1[k], s2[k], s3[k]);
  fvs_inverses(eps, b, id);
  const double db = b[0] - b[3], tau = db * db;
  double a[4], q[4], S = 0, num = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    a[k] = c[k] + c[k] * tau * (id[k] * id[k]);
    q[k] = 0.5 * s1[k] + (1.0 / 12) * s2[k];
    S += a[k];
    num += a[k] * q[k];
  }
  const double iS = 1.0 / S, f = num * iS, w = af * iS;
  double a1[4], a2[4], a3[4], ab[4], aq[4], atau = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    aq[k] = w * a[k];
    const double aa = w * (q[k] - f) * c[k] * (id[k] * id[k]);
    atau += aa;
    ab[k] = -2.0 * aa * tau * id[k];
  }
  ab[0] += 2.0 * atau * db;
  ab[3] -= 2.0 * atau * db;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    a1[k] = ab[k] * (2 * s1[k] + (1.0 / 12) * s3[k]) + 0.5 * aq[k];
    a2[k] = ab[k] * (26.0 / 12.0) * s2[k] + (1.0 / 12) * aq[k];
    a3[k] = ab[k] * (2 * (1043.0 / 960) * s3[k] + (1.0 / 12) * s1[k]);
  }
  const double am = a1[1] + a1[2];
  const double h0 = (1.0 / 3) * a1[0] + a2[0] + a3[0], h1 = a3[1] - (1.0 / 6) * a1[1], h2 = a3[2] - (1.0 / 6) * a1[2],
               h3 = (1.0 / 3) * a1[3] - a2[3] + a3[3];  // of the third differences
  const double k0 = -h0, k1 = 0.5 * a1[0] + a2[0] + h0 - h1, k2 = 0.5 * am + a2[1] + a2[2] + h1 - h2,
               k3 = a2[3] - 0.5 * a1[3] + h2 - h3, k4 = h3;  // of the second differences
  const double l0 = -k0, l1 = k0 - k1, l2 = a1[0] + am + k1 - k2, l3 = a1[3] + k2 - k3, l4 = k3 - k4, l5 = k4;  // first
  g[0] = -l0;
  g[1] = l0 - l1;
  g[2] = l1 - l2;
  g[3] = af + l2 - l3;
  g[4] = l3 - l4;
  g[5] = l4 - l5;
  g[6] = l5;
  return v[3] + f;
}

// Reverse of the node's split fluxes F+- = J/2 (Uk Q + p grad k (+ p Uk in energy) +- l0 Q),
// Uk = (Q1 kx + Q2 ky + Q3 kz) / Q0, l0 = |Uk| + c |grad k| (compute_flux, WENO.cu:697-720):
// sets aQ[nv], ap, ac; the adjoints aFp, aFm of F+- are strided by `step`.
template <int NS>
__device__ __forceinline__ void fvs_node_bwd(const double *Q, double pk, double c, double k0m, double k1m, double k2m,
                                             double jac, const double *aFp, const double *aFm, int step, double *aQ,
                                             double &ap, double &ac) {
  const int nv = 5 + OSTC_NS;
  const double Uk = (Q[1] * k0m + Q[2] * k1m + Q[3] * k2m) / Q[0];
  const double kn = sqrt(k0m * k0m + k1m * k1m + k2m * k2m);
  const double l0 = fabs(Uk) + c * kn;
  const double hj = 0.5 * jac;
  double aUk = 0, al0 = 0;
  const double km[3] = {k0m, k1m, k2m};
  ap = ac = 0;
  for (int q = 0; q < nv; ++q) {
    const double fp = aFp[q * step], fm = aFm[q * step], S = fp + fm, D = fp - fm;
    aQ[q] = hj * (Uk * S + l0 * D);
    aUk += hj * Q[q] * S;
    al0 += hj * Q[q] * D;
    if (q >= 1 && q <= 3) ap += hj * km[q - 1] * S;
    if (q == 4) {
      ap += hj * Uk * S;
      aUk += hj * pk * S;
    }
  }
  aUk += al0 * (Uk > 0 ? 1.0 : (Uk < 0 ? -1.0 : 0.0));
  ac += al0 * kn;
  const double iq0 = 1.0 / Q[0];
  aQ[1] += aUk * k0m * iq0;
  aQ[2] += aUk * k1m * iq0;
  aQ[3] += aUk * k2m * iq0;
  aQ[0] -= aUk * Uk * iq0;
}

// d cp_i / dT of the NASA-7 polynomials (0 below t_low, where cp is frozen)
__device__ __forceinline__ double mix_dcp_dt_one(int i, double t) {
  if (t < c_mix.t_low[i]) return 0.0;
  const double *a = t < c_mix.t_mid[i] ? c_mix.low[i] : c_mix.high[i];
  return (a[1] + t * (2 * a[2] + t * (3 * a[3] + t * 4 * a[4]))) * c_mix.ru_mw[i];
}
template <int NS>
__device__ __forceinline__ void mix_dcp_dt(double t, double *dcp) {
#pragma unroll
  for (int i = 0; i < OSTC_NS; ++i) dcp[i] = mix_dcp_dt_one(i, t);
}

// Left-eigenvector row l (0..4) of the Roe-averaged mixture eigensystem (WENO.cu:822-898) as the
// forward sweep forms it: L[0..4] on the five flow components and cs, the factor of the species part.
__device__ __forceinline__ void fvs_lrow(int l, double alpha, double Ukb, double cm, double c2i, double gm1, double um,
                                         double vm, double wm, double kx, double ky, double kz, double *L, double &cs) {
  cs = 0.5;
  if (l == 0) {
    L[0] = (alpha + Ukb * cm) * c2i * 0.5;
    L[1] = -(gm1 * um + kx * cm) * c2i * 0.5;
    L[2] = -(gm1 * vm + ky * cm) * c2i * 0.5;
    L[3] = -(gm1 * wm + kz * cm) * c2i * 0.5;
    L[4] = gm1 * c2i * 0.5;
  } else if (l == 1) {
    cs = -kx;
    L[0] = kx * (1 - alpha * c2i) - (kz * vm - ky * wm) / cm;
    L[1] = kx * gm1 * um * c2i;
    L[2] = (kx * gm1 * vm + kz * cm) * c2i;
    L[3] = (kx * gm1 * wm - ky * cm) * c2i;
    L[4] = -kx * gm1 * c2i;
  } else if (l == 2) {
    cs = -ky;
    L[0] = ky * (1 - alpha * c2i) - (kx * wm - kz * um) / cm;
    L[1] = (ky * gm1 * um - kz * cm) * c2i;
    L[2] = ky * gm1 * vm * c2i;
    L[3] = (ky * gm1 * wm + kx * cm) * c2i;
    L[4] = -ky * gm1 * c2i;
  } else if (l == 3) {
    cs = -kz;
    L[0] = kz * (1 - alpha * c2i) - (ky * um - kx * vm) / cm;
    L[1] = (kz * gm1 * um + ky * cm) * c2i;
    L[2] = (kz * gm1 * vm - kx * cm) * c2i;
    L[3] = kz * gm1 * wm * c2i;
    L[4] = -kz * gm1 * c2i;
  } else {
    L[0] = (alpha - Ukb * cm) * c2i * 0.5;
    L[1] = -(gm1 * um - kx * cm) * c2i * 0.5;
    L[2] = -(gm1 * vm - ky * cm) * c2i * 0.5;
    L[3] = -(gm1 * wm - kz * cm) * c2i * 0.5;
    L[4] = gm1 * c2i * 0.5;
  }
}

// Adjoint of the Roe-state symbols that the rows of fvs_lrow read, given AL = adjoint of L[0..4]
struct RoeBar {
  double alpha, Ukb, cm, c2i, gm1, um, vm, wm;
};
__device__ __forceinline__ void fvs_lrow_bwd(int l, const double *AL, double alpha, double Ukb, double cm, double c2i,
                                             double gm1, double um, double vm, double wm, double kx, double ky,
                                             double kz, RoeBar &r) {
  const double V[3] = {um, vm, wm}, k[3] = {kx, ky, kz};
  double aV[3] = {0, 0, 0};
  if (l == 0 || l == 4) {
    const double sg = l == 0 ? 1.0 : -1.0;
    r.alpha += AL[0] * c2i * 0.5;
    r.Ukb += sg * AL[0] * cm * c2i * 0.5;
    r.cm += sg * AL[0] * Ukb * c2i * 0.5;
    r.c2i += AL[0] * (alpha + sg * Ukb * cm) * 0.5;
    for (int q = 0; q < 3; ++q) {
      const double a = AL[q + 1];
      r.gm1 -= a * V[q] * c2i * 0.5;
      aV[q] -= a * gm1 * c2i * 0.5;
      r.cm -= sg * a * k[q] * c2i * 0.5;
      r.c2i -= a * (gm1 * V[q] + sg * k[q] * cm) * 0.5;
    }
    r.gm1 += AL[4] * c2i * 0.5;
    r.c2i += AL[4] * gm1 * 0.5;
  } else {
    const int d = l - 1;
    const double kd = k[d];
    // E[d][q]: coefficient of cm in L[q + 1] (antisymmetric, from the rows above)
    const double E[3][3] = {{0.0, kz, -ky}, {-kz, 0.0, kx}, {ky, -kx, 0.0}};
    r.alpha -= AL[0] * kd * c2i;
    r.c2i -= AL[0] * kd * alpha;
    // L0's cross term -X/cm, X = (kz vm - ky wm, kx wm - kz um, ky um - kx vm)[d]
    const double X = d == 0 ? kz * vm - ky * wm : (d == 1 ? kx * wm - kz * um : ky * um - kx * vm);
    r.cm += AL[0] * X / (cm * cm);
    const double aX = -AL[0] / cm;
    if (d == 0) {
      aV[1] += kz * aX;
      aV[2] -= ky * aX;
    } else if (d == 1) {
      aV[2] += kx * aX;
      aV[0] -= kz * aX;
    } else {
      aV[0] += ky * aX;
      aV[1] -= kx * aX;
    }
    for (int q = 0; q < 3; ++q) {
      const double a = AL[q + 1];
      r.gm1 += a * kd * V[q] * c2i;
      aV[q] += a * kd * gm1 * c2i;
      r.cm += a * E[d][q] * c2i;
      r.c2i += a * (kd * gm1 * V[q] + E[d][q] * cm);
    }
    r.gm1 -= AL[4] * kd * c2i;
    r.c2i -= AL[4] * kd * gm1;
  }
  r.um += aV[0];
  r.vm += aV[1];
  r.wm += aV[2];
}

template <int DIR>
__host__ __device__ constexpr size_t adj_fvs_smem_bytes(int nv) {
  // F+, F- (recomputed) and their adjoints per staged node; per thread alpha_l of L and its adjoint, and the
  // adjoint of the Roe-averaged mass fraction, per species
  return ((size_t)FvsTile<DIR>::NST * FvsTile<DIR>::TXL * 4 * nv +
          (size_t)FvsTile<DIR>::TD * FvsTile<DIR>::TXL * 3 * (nv - 5)) * sizeof(double);
}

// Reverse of k_fvs: the tile recomputes the staged split fluxes, every face thread turns its face
// adjoint (from dq_bar of the nodes this tile owns) into adjoints of the staged split fluxes and of the
// Roe-averaged face state, and after a barrier every staged node maps its split-flux adjoints back to cv,
// p and c and adds them to the node planes.
// A face adds to the 7 staged nodes of each side's stencil, which its neighbours' faces add to as well.
// FP64 atomics on shared memory are compare-and-swap loops, and 728 of them a face were most of this
// kernel's time; instead the threads of the block step through the stencil together (scatter below): at
// step m every face adds to the node m places along, a different one each, with a barrier between the
// steps.  The flow rows reach the species' split fluxes with one factor alpha_l times a sum W[m] over the
// rows, and the species fields reach the density's with a sum Z[m], so those go out once per side.  One
// pass over the fields: the WENO reverse returns the face value too, which the adjoints of R need.
// 96 x 64 x 48, 9 species: 0.95 / 0.89 / 0.94 ms (x / y / z); with FP64 shared-memory atomics 2.4-2.6 ms each.
template <int DIR, int NS>
__global__ void __launch_bounds__(FvsTile<DIR>::TD * FvsTile<DIR>::TXL, 2) k_adj_fvs(DevBlock b, DevState s,
                                                                                      const double *__restrict__ dqb,
                                                                                      int nv, int scheme, DevAdj A) {
  constexpr int TXL = FvsTile<DIR>::TXL, TD = FvsTile<DIR>::TD, NST = FvsTile<DIR>::NST, NN = NST * TXL, NT = TD * TXL;
  extern __shared__ __align__(16) unsigned char adj_smem[];
  if (NS > 0) nv = 5 + NS;
  const int ns = OSTC_NS;
  double *Fp = reinterpret_cast<double *>(adj_smem);  // [nv][NST][TXL]
  double *Fm = Fp + NN * nv;
  double *aFp = Fm + NN * nv;
  double *aFm = aFp + NN * nv;
  double *slots = aFm + NN * nv;  // [3][ns][NT]
  const int lane = DIR == 0 ? 0 : (int)threadIdx.x;
  const int t = DIR == 0 ? (int)threadIdx.x : (int)threadIdx.y;
  const int tid = t * TXL + lane;
  const long long P = b.plane;
  const int nd = DIR == 0 ? b.mx : DIR == 1 ? b.my : b.mz;
  const int start = (DIR == 0 ? blockIdx.x : blockIdx.y) * (TD - 1);
  int i0, j0, k0;
  if (DIR == 0) {
    i0 = 0; j0 = blockIdx.y; k0 = blockIdx.z;
  } else if (DIR == 1) {
    i0 = blockIdx.x * TXL + lane; j0 = 0; k0 = blockIdx.z;
  } else {
    i0 = blockIdx.x * TXL + lane; j0 = blockIdx.z; k0 = 0;
  }
  const bool lane_ok = i0 < b.mx;
  auto pid = [&](int n) -> long long {
    return DIR == 0 ? b.id(n, j0, k0) : DIR == 1 ? b.id(i0, n, k0) : b.id(i0, j0, n);
  };
  auto qid = [&](int n) -> long long {
    return DIR == 0 ? b.iq(n, j0, k0) : DIR == 1 ? b.iq(i0, n, k0) : b.iq(i0, j0, n);
  };
  for (int e = tid; e < 2 * NN * nv; e += NT) aFp[e] = 0.0;
  if (lane_ok) {
    for (int st = t; st < NST; st += TD) {
      const int n = start - 4 + st;
      if (n > nd + 3) continue;
      const long long p = pid(n);
      double Q[Spec<NS>::A + 5];
      for (int l = 0; l < nv; ++l) Q[l] = s.cv[l * P + p];
      const double pk = s.bv[4 * P + p], c = s.acs[p];
      const double k0m = b.met[(DIR * 3 + 0) * P + p], k1m = b.met[(DIR * 3 + 1) * P + p],
                   k2m = b.met[(DIR * 3 + 2) * P + p];
      const double jac = b.jac[p];
      const double Uk = (Q[1] * k0m + Q[2] * k1m + Q[3] * k2m) / Q[0];
      const double l0 = fabs(Uk) + c * sqrt(k0m * k0m + k1m * k1m + k2m * k2m);
      double *fp = Fp + st * TXL + lane, *fm = Fm + st * TXL + lane;
      for (int l = 0; l < nv; ++l) {
        const double pt = l >= 1 && l <= 3 ? pk * (l == 1 ? k0m : l == 2 ? k1m : k2m) : 0.0;
        const double conv = l == 4 ? Uk * (Q[4] + pk) : Uk * Q[l] + pt;
        fp[l * NN] = 0.5 * jac * (conv + l0 * Q[l]);
        fm[l * NN] = 0.5 * jac * (conv - l0 * Q[l]);
      }
    }
  }
  __syncthreads();
  const int n = start - 1 + t;  // left node of this thread's face
  // a face carries an adjoint where this tile owns one of its nodes
  const bool own_l = lane_ok && n < nd && t >= 1, own_r = lane_ok && t <= TD - 2 && n + 1 < nd;
  auto afc = [&](int l) -> double {
    double a = 0.0;
    if (own_l) a -= dqb[l * b.n + qid(n)];
    if (own_r) a += dqb[l * b.n + qid(n + 1)];
    return a;
  };
  bool act = false;
  for (int l = 0; l < nv; ++l) act = act || afc(l) != 0.0;
  // Side sd (0: +, 1: -) of variable l at stencil place m, upwind first: + nodes t .. t + 6, - nodes t + 7
  // down to t + 1.
  auto at = [&](int sd, int m) -> int { return (t + (sd ? 7 - m : m)) * TXL + lane; };
  auto F = [&](int sd, int l, int m) -> double { return (sd ? Fm : Fp)[l * NN + at(sd, m)]; };
  // adds w[q] g[m] to the adjoints of variables l0 + q (q < N) of the 7 nodes of side sd
  auto scatter = [&](int sd, int l0, auto N, const double *w, const double *g) {
#pragma unroll
    for (int m = 0; m < 7; ++m) {
      if (act) {
        double *p = (sd ? aFm : aFp) + l0 * NN + at(sd, m);
#pragma unroll
        for (int q = 0; q < decltype(N)::value; ++q) p[q * NN] += w[q] * g[m];
      }
      __syncthreads();
    }
  };
  using One = std::integral_constant<int, 1>;
  using Five = std::integral_constant<int, 5>;
  const double one[1] = {1.0};
  if (scheme == 71) {
    double e0 = 0;
    if (act) {
      const long long pl = pid(n), pr = pid(n + 1);
      const double j1 = b.jac[pl], j2 = b.jac[pr];
      double a[3];
      for (int q = 0; q < 3; ++q) a[q] = b.met[(DIR * 3 + q) * P + pl] * j1 + b.met[(DIR * 3 + q) * P + pr] * j2;
      e0 = 1e-20 * c_mix.weno_eps_scale * 0.25 * (a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
    }
    const double e1 = e0 * c_mix.v_ref * c_mix.v_ref, e2 = e1 * c_mix.v_ref * c_mix.v_ref;
#pragma unroll 1
    for (int l = 0; l < nv; ++l)
#pragma unroll 1
      for (int sd = 0; sd < 2; ++sd) {
        double v[7], g[7];
        if (act) {
#pragma unroll
          for (int m = 0; m < 7; ++m) v[m] = F(sd, l, m);
          weno7_side_bwd(v, (l >= 1 && l <= 3) ? e1 : (l == 4 ? e2 : e0), afc(l), g);
        }
        scatter(sd, l, One(), one, g);
      }
  } else {
    auto AL_ = [&](int l) -> double & { return slots[l * NT + tid]; };             // alpha_l
    auto A_AL = [&](int l) -> double & { return slots[(ns + l) * NT + tid]; };     // its adjoint
    auto A_SV = [&](int l) -> double & { return slots[(2 * ns + l) * NT + tid]; };  // of the mass fraction
    double rli = 1, rri = 1, wl = 0, wr = 0, sl = 1, sr = 1;  // wl, wr: Roe weights over rho
    double um = 0, vm = 0, wm = 0, hm = 0, tm = 1, mw_inv = 1, gamma = 2, cm = 1, eps = 1, kx = 1, ky = 0, kz = 0;
    const long long pl = act ? pid(n) : 0, pr = act ? pid(n + 1) : 0;
    auto roe = [&](int l) -> double { return wl * s.cv[l * P + pl] + wr * s.cv[l * P + pr]; };
    if (act) {
      // forward: Roe-averaged mixture state at the face (as k_fvs)
      const double rl = s.cv[pl], rr = s.cv[pr];
      const double p_l = s.bv[4 * P + pl], p_r = s.bv[4 * P + pr];
      rli = 1.0 / rl;
      rri = 1.0 / rr;
      sl = sqrt(rl);
      sr = sqrt(rr);
      const double isum = 1.0 / (sl + sr);
      wl = sl * isum * rli;
      wr = sr * isum * rri;
      um = roe(1);
      vm = roe(2);
      wm = roe(3);
      hm = roe(4) + (wl * p_l + wr * p_r);
      mw_inv = 0;
#pragma unroll 1
      for (int l = 0; l < ns; ++l) {
        const double sv = roe(5 + l);
        mw_inv += sv * c_mix.imw[l];
        A_SV(l) = sv;
      }
      tm = (wl * p_l + wr * p_r) / (kRuD * mw_inv);
      double cp = 0, cvt = 0;
#pragma unroll 1
      for (int l = 0; l < ns; ++l) {
        double h, c;
        mix_h_cp_one<double>(l, tm, h, c);
        const double sv = A_SV(l);
        cp += sv * c;
        cvt += sv * (c - c_mix.ru_mw[l]);
        AL_(l) = h;
        A_SV(l) = A_AL(l) = 0.0;
      }
      gamma = cp / cvt;
      const double c2 = gamma * kRuD * mw_inv * tm;
      cm = sqrt(c2);
      const double jl = b.jac[pl], jr = b.jac[pr];
      kx = b.met[(DIR * 3 + 0) * P + pl] * jl + b.met[(DIR * 3 + 0) * P + pr] * jr;
      ky = b.met[(DIR * 3 + 1) * P + pl] * jl + b.met[(DIR * 3 + 1) * P + pr] * jr;
      kz = b.met[(DIR * 3 + 2) * P + pl] * jl + b.met[(DIR * 3 + 2) * P + pr] * jr;
      const double k2 = kx * kx + ky * ky + kz * kz, igk = 1.0 / sqrt(k2);
      eps = 1e-40 * c_mix.weno_eps_scale * 0.25 * k2;
      kx *= igk;
      ky *= igk;
      kz *= igk;
#pragma unroll 1
      for (int l = 0; l < ns; ++l) AL_(l) = (gamma * c_mix.ru_mw[l] * tm - (gamma - 1) * AL_(l)) / c2;
    }
    const double gm1 = gamma - 1, c2i = 1.0 / (cm * cm);
    const double ekm = 0.5 * (um * um + vm * vm + wm * wm);
    const double Ukb = kx * um + ky * vm + kz * wm, alpha = gm1 * ekm;
    const double cg = cm * cm / gm1;
    RoeBar r{};
    double a_hm = 0, a_cg = 0, ca = 0;
    // reverse of fc = R fch (WENO.cu:1069-1117): the adjoint of the flow field l and, once its face value f is
    // known, the adjoints of R
    const double f4 = act ? afc(4) : 0.0;
    double aca = 0;
    if (act) {
      aca = afc(0);
#pragma unroll 1
      for (int l = 0; l < ns; ++l) aca += roe(5 + l) * afc(5 + l);
    }
    auto flow_bar = [&](int l) -> double {
      const double hc = hm - cg;
      if (l == 0 || l == 4) {
        const double c = l == 0 ? -cm : cm;
        return aca + afc(1) * (um + kx * c) + afc(2) * (vm + ky * c) + afc(3) * (wm + kz * c) + f4 * (hm + Ukb * c);
      }
      if (l == 1)
        return aca * kx + afc(1) * kx * um + afc(2) * (kx * vm + kz * cm) + afc(3) * (kx * wm - ky * cm) +
               f4 * (kx * hc + (kz * vm - ky * wm) * cm);
      if (l == 2)
        return aca * ky + afc(1) * (ky * um - kz * cm) + afc(2) * ky * vm + afc(3) * (ky * wm + kx * cm) +
               f4 * (ky * hc + (kx * wm - kz * um) * cm);
      return aca * kz + afc(1) * (kz * um + ky * cm) + afc(2) * (kz * vm - kx * cm) + afc(3) * kz * wm +
             f4 * (kz * hc + (ky * um - kx * vm) * cm);
    };
    auto flow_face = [&](int l, double f) {
      if (l == 0 || l == 4) {
        const double sg = l == 0 ? -1.0 : 1.0;
        ca += f;
        r.um += afc(1) * f;
        r.vm += afc(2) * f;
        r.wm += afc(3) * f;
        r.cm += sg * f * (afc(1) * kx + afc(2) * ky + afc(3) * kz + f4 * Ukb);
        r.Ukb += sg * f * f4 * cm;
        a_hm += f4 * f;
      } else {
        const double k = l == 1 ? kx : l == 2 ? ky : kz;
        const double fk = k * f, c4 = f4 * cm * f;
        ca += fk;
        r.um += afc(1) * fk;
        r.vm += afc(2) * fk;
        r.wm += afc(3) * fk;
        if (l == 1) {
          r.vm += kz * c4;
          r.wm -= ky * c4;
          r.cm += f * (afc(2) * kz - afc(3) * ky + f4 * (kz * vm - ky * wm));
        } else if (l == 2) {
          r.um -= kz * c4;
          r.wm += kx * c4;
          r.cm += f * (afc(3) * kx - afc(1) * kz + f4 * (kx * wm - kz * um));
        } else {
          r.um += ky * c4;
          r.vm -= kx * c4;
          r.cm += f * (afc(1) * ky - afc(2) * kx + f4 * (ky * um - kx * vm));
        }
        a_hm += f4 * fk;
        a_cg -= f4 * fk;
      }
    };
#pragma unroll 1
    for (int sd = 0; sd < 2; ++sd) {
      double W[7];
#pragma unroll
      for (int m = 0; m < 7; ++m) W[m] = 0.0;
#pragma unroll 1
      for (int l = 0; l < 5; ++l) {
        double L[5], cs, g[7];
        if (act) {
          double v[7], AL[5];
          fvs_lrow(l, alpha, Ukb, cm, c2i, gm1, um, vm, wm, kx, ky, kz, L, cs);
#pragma unroll
          for (int m = 0; m < 7; ++m) v[m] = 0.0;
#pragma unroll 1
          for (int q = 0; q < ns; ++q) {
            const double al = cs * AL_(q);
#pragma unroll
            for (int m = 0; m < 7; ++m) v[m] += al * F(sd, 5 + q, m);
          }
#pragma unroll
          for (int m = 0; m < 7; ++m)
#pragma unroll
            for (int q = 0; q < 5; ++q) v[m] += L[q] * F(sd, q, m);
          flow_face(l, weno7_side_bwd(v, eps, flow_bar(l), g));
#pragma unroll
          for (int q = 0; q < 5; ++q) AL[q] = 0.0;
#pragma unroll
          for (int m = 0; m < 7; ++m) {
            W[m] += cs * g[m];
#pragma unroll
            for (int q = 0; q < 5; ++q) AL[q] += F(sd, q, m) * g[m];
          }
          fvs_lrow_bwd(l, AL, alpha, Ukb, cm, c2i, gm1, um, vm, wm, kx, ky, kz, r);
        }
        scatter(sd, 0, Five(), L, g);
      }
      double Z[7];
#pragma unroll
      for (int m = 0; m < 7; ++m) Z[m] = 0.0;
#pragma unroll 1
      for (int l = 0; l < ns; ++l) {
        double g[7];
        if (act) {
          const double sv = roe(5 + l), al = AL_(l), f5 = afc(5 + l);
          double v[7], s0 = 0, s1 = 0;
#pragma unroll
          for (int m = 0; m < 7; ++m) v[m] = F(sd, 5 + l, m) - sv * F(sd, 0, m);
          const double f = weno7_side_bwd(v, eps, f5 - f4 * al * cg, g);
#pragma unroll
          for (int m = 0; m < 7; ++m) {
            s0 += F(sd, 0, m) * g[m];
            s1 += F(sd, 5 + l, m) * W[m];
            Z[m] -= sv * g[m];
            g[m] += al * W[m];
          }
          A_SV(l) -= s0;
          A_AL(l) += s1 - f4 * f * cg;
          a_cg -= f4 * al * f;
        }
        scatter(sd, 5 + l, One(), one, g);
      }
      scatter(sd, 0, One(), one, Z);
    }
    if (act) {
      r.cm += a_cg * 2 * cm / gm1;
      r.gm1 -= a_cg * cg / gm1;
      // Roe symbols -> Roe averages
      r.gm1 += r.alpha * ekm;
      r.um += r.alpha * gm1 * um + r.Ukb * kx;
      r.vm += r.alpha * gm1 * vm + r.Ukb * ky;
      r.wm += r.alpha * gm1 * wm + r.Ukb * kz;
      double a_gamma = 0, a_tm = 0, a_mwinv = 0, a_al_sum = 0;
#pragma unroll 1
      for (int l = 0; l < ns; ++l) {
        double h, c;
        mix_h_cp_one<double>(l, tm, h, c);
        const double a = A_AL(l);
        a_gamma += a * c_mix.ru_mw[l] * tm * c2i;
        r.gm1 -= a * h * c2i;
        a_tm += a * gamma * c_mix.ru_mw[l] * c2i;
        a_al_sum += a * AL_(l);
      }
      r.c2i += a_al_sum / c2i;
      r.cm -= 2.0 * r.c2i * c2i / cm;
      a_gamma += r.gm1 + r.cm * cm / (2 * gamma);
      a_mwinv += r.cm * cm / (2 * mw_inv);
      a_tm += r.cm * cm / (2 * tm);
      // cvt = sum Y (cp - Ru / W) of the Roe average: cp - cvt = Ru mw_inv and gamma = cp / cvt
      const double cvt = kRuD * mw_inv / gm1;
      const double a_cp = a_gamma / cvt, a_cvt = -a_gamma * gamma / cvt;
#pragma unroll 1
      for (int l = 0; l < ns; ++l) {
        double h, c;
        mix_h_cp_one<double>(l, tm, h, c);
        const double sv = roe(5 + l);
        A_SV(l) += ca * afc(5 + l) + a_cp * c + a_cvt * (c - c_mix.ru_mw[l]);
        a_tm += -A_AL(l) * gm1 * c2i * c + (a_cp + a_cvt) * sv * mix_dcp_dt_one(l, tm);
      }
      const double a_prm = a_tm / (kRuD * mw_inv);
      a_mwinv -= a_tm * tm / mw_inv;
      // averages X = rlc X_l + rrc X_r of u, v, w, H, Y, p/rho; per side X = num / rho
      double a_rlc = 0, a_rrc = 0, g0l = 0, g0r = 0;
      auto avg = [&](double aX, double nl, double nr, double *plane) {
        // nl, nr: the numerators; their adjoints go to `plane` (of cv, or p)
        const double Xl = nl * rli, Xr = nr * rri, gl = aX * wl, gr = aX * wr;
        a_rlc += aX * Xl;
        a_rrc += aX * Xr;
        g0l -= gl * Xl;
        g0r -= gr * Xr;
        atomicAdd(plane + pl, gl);
        atomicAdd(plane + pr, gr);
      };
      const double p_l = s.bv[4 * P + pl], p_r = s.bv[4 * P + pr];
      avg(r.um, s.cv[P + pl], s.cv[P + pr], A.cv + P);
      avg(r.vm, s.cv[2 * P + pl], s.cv[2 * P + pr], A.cv + 2 * P);
      avg(r.wm, s.cv[3 * P + pl], s.cv[3 * P + pr], A.cv + 3 * P);
      avg(a_hm, s.cv[4 * P + pl] + p_l, s.cv[4 * P + pr] + p_r, A.cv + 4 * P);  // H = (rho E + p) / rho
      avg(a_prm, p_l, p_r, A.p);
      atomicAdd(A.p + pl, a_hm * wl);
      atomicAdd(A.p + pr, a_hm * wr);
#pragma unroll 1
      for (int l = 0; l < ns; ++l)
        avg(A_SV(l) + a_mwinv * c_mix.imw[l], s.cv[(5 + l) * P + pl], s.cv[(5 + l) * P + pr], A.cv + (5 + l) * P);
      const double den = sl + sr;
      g0l += (a_rlc - a_rrc) * sr / (den * den) / (2 * sl);
      g0r += (a_rrc - a_rlc) * sl / (den * den) / (2 * sr);
      atomicAdd(A.cv + pl, g0l);
      atomicAdd(A.cv + pr, g0r);
    }
  }
  __syncthreads();
  // staged nodes: split-flux adjoints -> node planes
  if (lane_ok) {
    for (int st = t; st < NST; st += TD) {
      const int nn = start - 4 + st;
      if (nn > nd + 3) continue;
      const long long p = pid(nn);
      double Q[Spec<NS>::A + 5], aQ[Spec<NS>::A + 5], ap, ac;
      for (int l = 0; l < nv; ++l) Q[l] = s.cv[l * P + p];
      fvs_node_bwd<NS>(Q, s.bv[4 * P + p], s.acs[p], b.met[(DIR * 3 + 0) * P + p], b.met[(DIR * 3 + 1) * P + p],
                       b.met[(DIR * 3 + 2) * P + p], b.jac[p], aFp + st * TXL + lane, aFm + st * TXL + lane, NN, aQ, ap, ac);
      for (int l = 0; l < nv; ++l)
        if (aQ[l] != 0.0) atomicAdd(A.cv + l * P + p, aQ[l]);
      if (ap != 0.0) atomicAdd(A.p + p, ap);
      if (ac != 0.0) atomicAdd(A.c + p, ac);
    }
  }
}

// Reverse of mix_visc_face (FP64) for the face between p0 and p0 + e[d] with face adjoint afv[nv]:
// adds to the adjoints of u, v, w, T, Y, mu, lambda and rho*D of the nodes its gradients read.
template <bool DIM3, int NS>
__device__ __forceinline__ void mix_visc_face_bwd(const DevBlock &b, const DevState &s, long long p0, int d,
                                                  const double *afv, const DevAdj &A) {
  const long long P = b.plane;
  const long long st[3] = {1, b.pitch, (long long)b.pitch * b.sy};
  const long long p1 = b.chk(p0 + st[d]);
  double m[9];
  for (int r = 0; r < 9; ++r) m[r] = 0.5 * (b.met[r * P + p0] + b.met[r * P + p1]);
  auto grad = [&](const double *B, double *out) {
    double g[3];
    for (int c = 0; c < 3; ++c) {
      if (c == d) {
        g[c] = B[p1] - B[p0];
      } else if (c == 2 && !DIM3) {
        g[c] = 0.0;
      } else {
        const long long a = st[c];
        g[c] = 0.25 * (B[p0 + a] - B[p0 - a] + B[p1 + a] - B[p1 - a]);
      }
    }
    out[0] = g[0] * m[0] + g[1] * m[3] + g[2] * m[6];
    out[1] = g[0] * m[1] + g[1] * m[4] + g[2] * m[7];
    out[2] = g[0] * m[2] + g[1] * m[5] + g[2] * m[8];
  };
  // reverse of grad: adjoint aout[3] of the metric-transformed gradient -> node adjoints of plane AB
  auto grad_bwd = [&](const double *aout, double *AB) {
    for (int c = 0; c < 3; ++c) {
      const double ag = aout[0] * m[c * 3 + 0] + aout[1] * m[c * 3 + 1] + aout[2] * m[c * 3 + 2];
      if (ag == 0.0) continue;
      if (c == d) {
        atomicAdd(AB + p1, ag);
        atomicAdd(AB + p0, -ag);
      } else if (c == 2 && !DIM3) {
      } else {
        const long long a = st[c];
        const double q = 0.25 * ag;
        atomicAdd(AB + p0 + a, q);
        atomicAdd(AB + p0 - a, -q);
        atomicAdd(AB + p1 + a, q);
        atomicAdd(AB + p1 - a, -q);
      }
    }
  };
  double gu[3], gv[3], gw[3], gt[3];
  grad(s.bv + P, gu);
  grad(s.bv + 2 * P, gv);
  grad(s.bv + 3 * P, gw);
  grad(s.bv + 5 * P, gt);
  const double mul = 0.5 * (s.mul[p0] + s.mul[p1]);
  const double txx = mul * (4 * gu[0] - 2 * gv[1] - 2 * gw[2]) / 3.0;
  const double tyy = mul * (4 * gv[1] - 2 * gu[0] - 2 * gw[2]) / 3.0;
  const double tzz = mul * (4 * gw[2] - 2 * gu[0] - 2 * gv[1]) / 3.0;
  const double txy = mul * (gu[1] + gv[0]);
  const double txz = mul * (gu[2] + gw[0]);
  const double tyz = mul * (gv[2] + gw[1]);
  const double j0 = b.jac[p0], j1 = b.jac[p1];
  const double nx = 0.5 * (b.met[(d * 3 + 0) * P + p0] * j0 + b.met[(d * 3 + 0) * P + p1] * j1);
  const double ny = 0.5 * (b.met[(d * 3 + 1) * P + p0] * j0 + b.met[(d * 3 + 1) * P + p1] * j1);
  const double nz = 0.5 * (b.met[(d * 3 + 2) * P + p0] * j0 + b.met[(d * 3 + 2) * P + p1] * j1);
  const double fv1 = nx * txx + ny * txy + nz * txz;
  const double fv2 = nx * txy + ny * tyy + nz * tyz;
  const double fv3 = nx * txz + ny * tyz + nz * tzz;
  const double um = 0.5 * (s.bv[P + p0] + s.bv[P + p1]);
  const double vm = 0.5 * (s.bv[2 * P + p0] + s.bv[2 * P + p1]);
  const double wm = 0.5 * (s.bv[3 * P + p0] + s.bv[3 * P + p1]);
  const double cond = 0.5 * (s.cond[p0] + s.cond[p1]);
  const int ns = OSTC_NS;
  double dif[Spec<NS>::A], yk[Spec<NS>::A], ddf[Spec<NS>::A];
  double sgw = 0, srdy = 0, corr = 0, mwt = 0;
  for (int l = 0; l < ns; ++l) {
    const double *Y = s.sv + (long long)l * P;
    yk[l] = 0.5 * (Y[p0] + Y[p1]);
    dif[l] = 0.5 * (s.rhod[l * P + p0] + s.rhod[l * P + p1]);
    double gy[3];
    grad(Y, gy);
    const double gdy = nx * gy[0] + ny * gy[1] + nz * gy[2];
    ddf[l] = gdy;
    corr += dif[l] * gdy;
    sgw += gdy / c_mix.mw[l];
    mwt += yk[l] / c_mix.mw[l];
    srdy += dif[l] * yk[l];
  }
  mwt = 1.0 / mwt;
  corr -= mwt * srdy * sgw;
  const double tf = 0.5 * (s.bv[5 * P + p0] + s.bv[5 * P + p1]);
  double h[Spec<NS>::A], cp[Spec<NS>::A];
  mix_h_cp<NS, double>(tf, h, cp);
  // ---- reverse
  const double a4 = afv[4];
  double a_tf = 0, a_corr = 0, a_sgw = 0, a_mwt = 0, a_srdy = 0;
  double a_yk[Spec<NS>::A], a_dif[Spec<NS>::A], a_gdy[Spec<NS>::A];
  for (int l = 0; l < ns; ++l) {
    const double flux = dif[l] * (ddf[l] - mwt * yk[l] * sgw) - yk[l] * corr;
    const double af = afv[5 + l] + a4 * h[l];
    a_tf += a4 * flux * cp[l];
    a_dif[l] = af * (ddf[l] - mwt * yk[l] * sgw);
    a_gdy[l] = af * dif[l];
    a_mwt -= af * dif[l] * yk[l] * sgw;
    a_yk[l] = -af * (dif[l] * mwt * sgw + corr);
    a_sgw -= af * dif[l] * mwt * yk[l];
    a_corr -= af * yk[l];
  }
  // corr = sum dif gdy - mwt srdy sgw
  for (int l = 0; l < ns; ++l) {
    a_dif[l] += a_corr * ddf[l];
    a_gdy[l] += a_corr * dif[l];
  }
  a_mwt -= a_corr * srdy * sgw;
  a_srdy -= a_corr * mwt * sgw;
  a_sgw -= a_corr * mwt * srdy;
  for (int l = 0; l < ns; ++l) {
    a_dif[l] += a_srdy * yk[l];
    a_yk[l] += a_srdy * dif[l] - a_mwt * mwt * mwt / c_mix.mw[l];
    a_gdy[l] += a_sgw / c_mix.mw[l];
    const double agy[3] = {a_gdy[l] * nx, a_gdy[l] * ny, a_gdy[l] * nz};
    grad_bwd(agy, A.Y + (long long)l * P);
    atomicAdd(A.Y + (long long)l * P + p0, 0.5 * a_yk[l]);
    atomicAdd(A.Y + (long long)l * P + p1, 0.5 * a_yk[l]);
    atomicAdd(A.rhod + (long long)l * P + p0, 0.5 * a_dif[l]);
    atomicAdd(A.rhod + (long long)l * P + p1, 0.5 * a_dif[l]);
  }
  atomicAdd(A.T + p0, 0.5 * a_tf);
  atomicAdd(A.T + p1, 0.5 * a_tf);
  // energy: fv4 = um fv1 + vm fv2 + wm fv3 + cond (n . gT) + sum h flux
  const double A1 = afv[1] + a4 * um, A2 = afv[2] + a4 * vm, A3 = afv[3] + a4 * wm;
  const double a_um = a4 * fv1, a_vm = a4 * fv2, a_wm = a4 * fv3;
  const double a_cond = a4 * (nx * gt[0] + ny * gt[1] + nz * gt[2]);
  const double agt[3] = {a4 * cond * nx, a4 * cond * ny, a4 * cond * nz};
  grad_bwd(agt, A.T);
  atomicAdd(A.lam + p0, 0.5 * a_cond);
  atomicAdd(A.lam + p1, 0.5 * a_cond);
  atomicAdd(A.vel + p0, 0.5 * a_um);
  atomicAdd(A.vel + p1, 0.5 * a_um);
  atomicAdd(A.vel + P + p0, 0.5 * a_vm);
  atomicAdd(A.vel + P + p1, 0.5 * a_vm);
  atomicAdd(A.vel + 2 * P + p0, 0.5 * a_wm);
  atomicAdd(A.vel + 2 * P + p1, 0.5 * a_wm);
  // stress
  const double a_txx = A1 * nx, a_tyy = A2 * ny, a_tzz = A3 * nz;
  const double a_txy = A1 * ny + A2 * nx, a_txz = A1 * nz + A3 * nx, a_tyz = A2 * nz + A3 * ny;
  const double a_mul = a_txx * (4 * gu[0] - 2 * gv[1] - 2 * gw[2]) / 3.0 +
                       a_tyy * (4 * gv[1] - 2 * gu[0] - 2 * gw[2]) / 3.0 +
                       a_tzz * (4 * gw[2] - 2 * gu[0] - 2 * gv[1]) / 3.0 + a_txy * (gu[1] + gv[0]) +
                       a_txz * (gu[2] + gw[0]) + a_tyz * (gv[2] + gw[1]);
  atomicAdd(A.mu + p0, 0.5 * a_mul);
  atomicAdd(A.mu + p1, 0.5 * a_mul);
  double agu[3], agv[3], agw[3];
  agu[0] = mul * (4 * a_txx - 2 * a_tyy - 2 * a_tzz) / 3.0;
  agv[1] = mul * (-2 * a_txx + 4 * a_tyy - 2 * a_tzz) / 3.0;
  agw[2] = mul * (-2 * a_txx - 2 * a_tyy + 4 * a_tzz) / 3.0;
  agu[1] = mul * a_txy;
  agv[0] = mul * a_txy;
  agu[2] = mul * a_txz;
  agw[0] = mul * a_txz;
  agv[2] = mul * a_tyz;
  agw[1] = mul * a_tyz;
  grad_bwd(agu, A.vel);
  grad_bwd(agv, A.vel + P);
  grad_bwd(agw, A.vel + 2 * P);
}

// Reverse of k_mix_visc: one thread per face; the face adjoint is dq_bar(n) - dq_bar(n + 1) over the
// nodes this tile owns (the forward adds fv(n + 1/2) to node n and subtracts it from node n + 1).
template <int DIR, bool DIM3, int NS>
__global__ void __launch_bounds__(FvsTile<DIR>::TD * FvsTile<DIR>::TXL, 3) k_adj_visc(DevBlock b, DevState s,
                                                                                    const double *__restrict__ dqb,
                                                                                    int nv, DevAdj A) {
  if (NS > 0) nv = 5 + NS;
  constexpr int TXL = FvsTile<DIR>::TXL, TD = FvsTile<DIR>::TD;
  const int lane = DIR == 0 ? 0 : (int)threadIdx.x;
  const int t = DIR == 0 ? (int)threadIdx.x : (int)threadIdx.y;
  const int nd = DIR == 0 ? b.mx : DIR == 1 ? b.my : b.mz;
  const int start = (DIR == 0 ? blockIdx.x : blockIdx.y) * (TD - 1);
  int i0, j0, k0;
  if (DIR == 0) {
    i0 = 0; j0 = blockIdx.y; k0 = blockIdx.z;
  } else if (DIR == 1) {
    i0 = blockIdx.x * TXL + lane; j0 = 0; k0 = blockIdx.z;
  } else {
    i0 = blockIdx.x * TXL + lane; j0 = blockIdx.z; k0 = 0;
  }
  const int n = start - 1 + t;
  if (!(i0 < b.mx && n < nd)) return;
  auto qid = [&](int m) -> long long {
    return DIR == 0 ? b.iq(m, j0, k0) : DIR == 1 ? b.iq(i0, m, k0) : b.iq(i0, j0, m);
  };
  double afv[Spec<NS>::A + 5];
  bool any = false;
  for (int l = 0; l < nv; ++l) {
    double a = 0.0;
    if (t >= 1) a += dqb[l * b.n + qid(n)];
    if (t <= TD - 2 && n + 1 < nd) a -= dqb[l * b.n + qid(n + 1)];
    afv[l] = a;
    any = any || a != 0.0;
  }
  if (!any) return;
  const long long p0 = DIR == 0 ? b.id(n, j0, k0) : DIR == 1 ? b.id(i0, n, k0) : b.id(i0, j0, n);
  mix_visc_face_bwd<DIM3, NS>(b, s, p0, DIR, afv, A);
}

// Reverse of the chemical source dq[5+l] += J omega_l(rho, T, Y) (compute_source<FR>,
// SourceTerm.cuh:11-35; finite_rate_chemistry, FiniteRateChem.cu:7-195), interior nodes.
// omega_l = 1e3 W_l sum_r (nu_b - nu_f)_rl (q1_r - q2_r), q1 = kf prod c^nu_f, q2 = kb prod c^nu_b,
// c_l = rho Y_l / W_l 1e-3: per reaction the adjoint of q1 - q2 goes to kf, kb and the
// concentrations; kf, kb are differentiated in T (and in the third-body sum) by Dual evaluations of
// the same rate-constant code.
template <int NS>
__global__ void __launch_bounds__(128, 4) k_adj_source(DevBlock b, DevState s, const double *__restrict__ dqb, DevAdj A) {
  const long long P = b.plane;
  const int ns = OSTC_NS, nr = c_mix.nr;
  constexpr int SA = Spec<NS>::A;
  for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < b.n; n += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(n % b.mx);
    const long long r0 = n / b.mx;
    const int j = (int)(r0 % b.my), k = (int)(r0 / b.my);
    const long long p = b.id(i, j, k);
    double aw[SA];
    bool any = false;
    for (int l = 0; l < ns; ++l) {
      aw[l] = b.jac[p] * dqb[(5 + l) * b.n + n] * c_mix.mw[l] * 1e+3;
      any = any || aw[l] != 0.0;
    }
    if (!any) continue;
    const double rho = s.bv[p], t = s.bv[5 * P + p];
    double y[SA], c[SA], ac[SA];
    for (int l = 0; l < ns; ++l) {
      y[l] = s.sv[l * P + p];
      c[l] = rho * y[l] * c_mix.imw[l] * 1e-3;
      ac[l] = 0.0;
    }
    const double lt = log(t), ti = 1.0 / t;
    const Dual tT(t, 1.0), ltT = log(tT), tiT = 1.0 / tT;
    Dual gT[SA], gC[SA];
    if (c_mix.use_gibbs) {
      mix_gibbs_rt<NS, Dual>(tT, gT);
      for (int l = 0; l < ns; ++l) gC[l] = Dual(gT[l].v, 0.0);
    }
    double aT = 0;
    for (int r = 0; r < nr; ++r) {
      double aq = 0;
      for (int l = 0; l < ns; ++l) aq += aw[l] * (c_mix.stoi_b[r][l] - c_mix.stoi_f[r][l]);
      if (aq == 0.0) continue;
      const int ty = c_mix.label[r];
      double cc = 0;
      if (ty >= 4)
        for (int l = 0; l < ns; ++l) cc += c[l] * c_mix.third_body[r][l];
      Dual kf, kb;
      reaction_rates<NS, Dual>(r, tT, ltT, tiT, Dual(cc), gT, kf, kb);
      double dkf_dcc = 0, dkb_dcc = 0;
      if (ty >= 4) {
        Dual kfc, kbc;
        reaction_rates<NS, Dual>(r, Dual(t), Dual(lt), Dual(ti), Dual(cc, 1.0), gC, kfc, kbc);
        dkf_dcc = kfc.d;
        dkb_dcc = kbc.d;
      }
      // concentration products as the forward forms them, and their partial derivatives
      auto fpow = [](double x, int nu) { return nu == 1 ? x : (nu == 2 ? x * x : pow(x, (double)nu)); };
      auto dpow = [](double x, int nu) { return nu == 1 ? 1.0 : (nu == 2 ? 2 * x : nu * pow(x, (double)(nu - 1))); };
      double p1 = 1.0, p2 = 1.0;
      for (int l = 0; l < ns; ++l) {
        if (c_mix.stoi_f[r][l]) p1 *= fpow(c[l], c_mix.stoi_f[r][l]);
        if (c_mix.stoi_b[r][l]) p2 *= fpow(c[l], c_mix.stoi_b[r][l]);
      }
      const double akf = aq * p1, akb = ty != 0 ? -aq * p2 : 0.0;
      aT += akf * kf.d + akb * kb.d;
      if (ty >= 4) {
        const double acc = akf * dkf_dcc + akb * dkb_dcc;
        for (int l = 0; l < ns; ++l) ac[l] += acc * c_mix.third_body[r][l];
      }
      for (int l = 0; l < ns; ++l) {
        const int nf = c_mix.stoi_f[r][l], nb = ty != 0 ? c_mix.stoi_b[r][l] : 0;
        if (nf) {
          double d = dpow(c[l], nf);
          for (int m = 0; m < ns; ++m)
            if (m != l && c_mix.stoi_f[r][m]) d *= fpow(c[m], c_mix.stoi_f[r][m]);
          ac[l] += aq * kf.v * d;
        }
        if (nb) {
          double d = dpow(c[l], nb);
          for (int m = 0; m < ns; ++m)
            if (m != l && c_mix.stoi_b[r][m]) d *= fpow(c[m], c_mix.stoi_b[r][m]);
          ac[l] -= aq * kb.v * d;
        }
      }
    }
    double arho = 0;
    for (int l = 0; l < ns; ++l) {
      arho += ac[l] * y[l] * c_mix.imw[l] * 1e-3;
      A.Y[(long long)l * P + p] += ac[l] * rho * c_mix.imw[l] * 1e-3;
    }
    A.rho[p] += arho;
    A.T[p] += aT;
  }
}

// The same over the reaction lists with the species arrays in shared memory (as mix_chemistry_listed):
// d ln kf / dT = b / T + Ea / T^2 for the Arrhenius types, d g / dT = -h / (Ru T^2) for the equilibrium constant;
// only fall-off reactions take Dual evaluations.  96 x 64 x 48, 19 reactions: 0.31 ms; dense 0.65.
template <int NS>
__global__ void __launch_bounds__(128, 4) k_adj_source_listed(DevBlock b, DevState s, const double *__restrict__ dqb,
                                                             DevAdj A) {
  extern __shared__ double adj_src_smem[];
  const long long P = b.plane;
  const int ns = OSTC_NS, nr = c_mix.nr;
  auto col = [&](int a) { return ChemColumn{adj_src_smem + a * ns * 128 + threadIdx.x, 128}; };
  const ChemColumn c = col(0), ac = col(1), aw = col(2), g = col(3), dg = col(4);
  for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < b.n; n += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(n % b.mx);
    const long long r0 = n / b.mx;
    const int j = (int)(r0 % b.my), k = (int)(r0 / b.my);
    const long long p = b.id(i, j, k);
    const double rho = s.bv[p], t = s.bv[5 * P + p], jac = b.jac[p];
    bool any = false;
    for (int l = 0; l < ns; ++l) {
      const double a = jac * dqb[(5 + l) * b.n + n] * c_mix.mw[l] * 1e+3;
      aw(l) = a;
      any = any || a != 0.0;
      c(l) = rho * s.sv[l * P + p] * c_mix.imw[l] * 1e-3;
      ac(l) = 0.0;
    }
    if (!any) continue;
    const double lt = log(t), ti = 1.0 / t;
    if (c_mix.use_gibbs) {
      double gr[Spec<NS>::A];
      mix_gibbs_rt<NS, double>(t, gr);
#pragma unroll
      for (int l = 0; l < ns; ++l) {
        double h, cp;
        mix_h_cp_one<double>(l, t, h, cp);
        g(l) = gr[l];
        // below t_low the Gibbs energy is evaluated at t_low, a constant
        dg(l) = t < c_mix.t_low[l] ? 0.0 : -h / c_mix.ru_mw[l] * (ti * ti);
      }
    }
    double aT = 0;
#pragma unroll 1
    for (int r = 0; r < nr; ++r) {
      const int ty = c_mix.label[r], nf = c_mix.n_f[r], nb = c_mix.n_b[r], nn = c_mix.n_net[r];
      double aq = 0, sg = 0, sdg = 0;
      for (int e = 0; e < nn; ++e) {
        const int m = c_mix.net[r][e];
        const double nu = c_mix.nu[r][e];
        aq += nu * aw(m);
        if (c_mix.use_gibbs) {
          sg += nu * g(m);
          sdg += nu * dg(m);
        }
      }
      if (aq == 0.0) continue;
      double cc = 0;
      if (ty >= 4)
        for (int l = 0; l < ns; ++l) cc += c(l) * c_mix.third_body[r][l];
      // kf with its derivatives in T and the third-body sum
      double kf, kf_t, kf_c = 0;
      if (ty > 4) {
        const Dual a = reaction_kf<Dual>(r, Dual(t, 1.0), Dual(lt, ti), Dual(ti, -ti * ti), Dual(cc));
        const Dual d = reaction_kf<Dual>(r, Dual(t), Dual(lt), Dual(ti), Dual(cc, 1.0));
        kf = a.v;
        kf_t = a.d;
        kf_c = d.d;
      } else {
        kf = arrhenius(lt, ti, c_mix.A[r], c_mix.b[r], c_mix.Ea[r]);
        kf_t = kf * (c_mix.b[r] + c_mix.Ea[r] * ti) * ti;
        if (ty == 3) {
          const double k2 = arrhenius(lt, ti, c_mix.A2[r], c_mix.b2[r], c_mix.Ea2[r]);
          kf += k2;
          kf_t += k2 * (c_mix.b2[r] + c_mix.Ea2[r] * ti) * ti;
        } else if (ty == 4) {
          kf_c = kf;
          kf *= cc;
          kf_t *= cc;
        }
      }
      // kb: kf over the equilibrium constant, whose ln changes with T by -sdg - order / T; else REV coefficients
      double kb = reaction_kb<double>(r, lt, ti, cc, kf, sg), kb_t = 0, kb_c = 0;
      if (ty != 0 && ty != 2 && c_mix.use_gibbs) {
        const double ratio = reaction_kb<double>(r, lt, ti, cc, 1.0, sg);
        kb_t = ratio * kf_t + kb * (sdg + c_mix.order[r] * ti);
        kb_c = ratio * kf_c;
      } else if (ty != 0 && c_mix.rev_type[r] == 1) {
        kb_t = kb * (c_mix.b2[r] + c_mix.Ea2[r] * ti) * ti;
        // times the third-body sum, which is zero where no collider is present (its derivative is not)
        if (ty == 4) kb_c = arrhenius(lt, ti, c_mix.A2[r], c_mix.b2[r], c_mix.Ea2[r]);
      }
      double p1 = 1.0, p2 = 1.0;
      for (int e = 0; e < nf; ++e) {
        double d = 1.0;  // product of the other molecules: d p1 / d c of this one
        for (int q = 0; q < nf; ++q)
          if (q != e) d *= c(c_mix.mol_f[r][q]);
        ac(c_mix.mol_f[r][e]) += aq * kf * d;
        p1 *= c(c_mix.mol_f[r][e]);
      }
      if (ty != 0) {
        for (int e = 0; e < nb; ++e) {
          double d = 1.0;
          for (int q = 0; q < nb; ++q)
            if (q != e) d *= c(c_mix.mol_b[r][q]);
          ac(c_mix.mol_b[r][e]) -= aq * kb * d;
          p2 *= c(c_mix.mol_b[r][e]);
        }
      }
      const double akf = aq * p1, akb = ty != 0 ? -aq * p2 : 0.0;
      aT += akf * kf_t + akb * kb_t;
      if (ty >= 4) {
        const double acc = akf * kf_c + akb * kb_c;
        for (int l = 0; l < ns; ++l) ac(l) += acc * c_mix.third_body[r][l];
      }
    }
    double arho = 0;
    for (int l = 0; l < ns; ++l) {
      const double a = ac(l) * c_mix.imw[l] * 1e-3;
      arho += a * s.sv[l * P + p];
      A.Y[(long long)l * P + p] += a * rho;
    }
    A.rho[p] += arho;
    A.T[p] += aT;
  }
}

// Reverse of the transport and acoustic properties (update_physical_properties<mixture>,
// FieldOperation.cuh:107-134, compute_transport_property, Transport.cu:43-136) at every padded node:
// adjoints of c, mu, lambda and rho*D_k -> adjoints of rho, p, T and Y.  Hand-written reverse of
// mix_properties (one forward sweep keeping its intermediates, then the reverse sweep).
// The powers, square roots and quotients are those of mix_properties (one log, one exp, one reciprocal
// square root a species, the powers of the collision integrals' constants in the tables): 0.27 ms at 96 x 64 x 48;
// with a pow per species and pair and a square root per ratio 1.7 ms.
template <int NS>
__global__ void __launch_bounds__(128, 2) k_adj_props(DevBlock b, DevState s, DevAdj A) {
  const long long P = b.plane;
  const int ns = OSTC_NS;
  constexpr int SA = Spec<NS>::A;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    const double rho = s.bv[p];
    if (!(rho > 0)) continue;
    const double ac = A.c[p], amu = A.mu[p], alam = A.lam[p];
    double ard[SA];
    bool any = ac != 0.0 || amu != 0.0 || alam != 0.0;
#pragma unroll
    for (int l = 0; l < ns; ++l) {
      ard[l] = A.rhod[(long long)l * P + p];
      any = any || ard[l] != 0.0;
    }
    if (!any) continue;
    const double pr = s.bv[4 * P + p], t = s.bv[5 * P + p], it = 1.0 / t;
    const double st = sqrt(t), tp = exp(-0.145 * log(t)), dtp = -0.145 * tp * it;  // T^-0.145
    double smw = 0, cpt = 0, cvt = 0;
#pragma unroll
    for (int l = 0; l < ns; ++l) {
      const double y = s.sv[l * P + p];
      double h, cp;
      mix_h_cp_one<double>(l, t, h, cp);
      smw += y * c_mix.imw[l];
      cpt += y * cp;
      cvt += y * (cp - c_mix.ru_mw[l]);
    }
    const double mw = 1 / smw, gamma = cpt / cvt;
    double X[SA], aX[SA];
#pragma unroll
    for (int l = 0; l < ns; ++l) {
      X[l] = s.sv[l * P + p] * mw * c_mix.imw[l];
      aX[l] = 0.0;
    }
    double arho = 0, aT = 0, ap = 0, amw = 0;
    {
      // rho D_l = rho t32p num_l / (den_l mw), den_l = sum (X_n + eps) w_ln, w = tp kbe_pow + q,
      // q = 1 / (D (T* + 0.5)^2)
      const double t32p = t * st / pr, eps = 1e-12;
      double num[SA], den[SA];
#pragma unroll
      for (int l = 0; l < ns; ++l) num[l] = den[l] = 0;
#pragma unroll
      for (int l = 0; l < ns; ++l)
#pragma unroll
        for (int n = l + 1; n < ns; ++n) {
          const double a = t * c_mix.kb_over_eps[l][n] + 0.5;
          const double w = tp * c_mix.kbe_pow[l][n] + c_mix.inv_diff[l][n] / (a * a);
          num[l] += (X[n] + eps) * c_mix.mw[n];
          den[l] += (X[n] + eps) * w;
          num[n] += (X[l] + eps) * c_mix.mw[l];
          den[n] += (X[l] + eps) * w;
        }
      double sum = 0, aden[SA], anum[SA];
#pragma unroll
      for (int l = 0; l < ns; ++l) {
        const double id = 1.0 / den[l], f = ard[l] * (rho * smw * t32p) * id;  // ard rho D / num
        sum += f * num[l];
        anum[l] = f;
        aden[l] = -f * num[l] * id;
      }
      arho += sum / rho;
      amw -= sum * smw;
      aT += 1.5 * sum * it;
      ap -= sum / pr;
#pragma unroll
      for (int l = 0; l < ns; ++l)
#pragma unroll
        for (int n = l + 1; n < ns; ++n) {
          const double kbe = c_mix.kb_over_eps[l][n], ia = 1.0 / (t * kbe + 0.5);
          const double q = c_mix.inv_diff[l][n] * ia * ia, w = tp * c_mix.kbe_pow[l][n] + q;
          aX[n] += aden[l] * w + anum[l] * c_mix.mw[n];
          aX[l] += aden[n] * w + anum[n] * c_mix.mw[l];
          aT += (aden[l] * (X[n] + eps) + aden[n] * (X[l] + eps)) * (c_mix.kbe_pow[l][n] * dtp - 2.0 * kbe * ia * q);
        }
    }
    double aTv = 0, acp[SA];
    {
      double vis[SA], isv[SA], avis[SA], dlv[SA];  // dlv = d ln(vis) / dT
#pragma unroll
      for (int l = 0; l < ns; ++l) {
        // vis = coeff sqrt(T) a^2 / d, d = lj_pow tp a^2 + 1
        const double lj = c_mix.lj_potent_inv[l], a = t * lj + 0.5, a2 = a * a, e = c_mix.lj_pow[l] * tp * a2, d = e + 1.0;
        const double q = 1.0 / (a * d);
        vis[l] = c_mix.vis_coeff[l] * st * a2 * (a * q);
        dlv[l] = 0.5 * it + (2.0 * lj + 0.145 * e * it * a) * q;
        isv[l] = rsqrt(vis[l]);
        avis[l] = 0.0;
      }
      // lambda = sum lam_m X_m / ct_m, lam_m = vis_m (cp_m + 1.25 Ru / W_m); mu = sum vis_m X_m / vt_m;
      // vt_m = sum_n pf_mn X_n, pf_mn = (1 + sqrt(vis_m / vis_n) w_mn)^2 s_mn
#pragma unroll
      for (int m = 0; m < ns; ++m) {
        const double svm = vis[m] * isv[m];
        double vt = X[m];
#pragma unroll
        for (int n = 0; n < ns; ++n) {
          if (m == n) continue;
          const double nm = 1 + svm * isv[n] * c_mix.wj_div_wi_1_4[m][n];
          vt += nm * nm * c_mix.sqrt_wiwj_8[m][n] * X[n];
        }
        const double ct = 1.065 * vt - 0.065 * X[m];
        const double q = 1.0 / (vt * ct), ivt = ct * q, ict = vt * q;
        double h, cp;
        mix_h_cp_one<double>(m, t, h, cp);
        const double lfac = cp + 1.25 * c_mix.ru_mw[m];
        const double al = alam * ict, au = amu * ivt;
        const double act = -al * vis[m] * lfac * X[m] * ict;
        const double avt = 1.065 * act - au * vis[m] * X[m] * ivt;
        acp[m] = al * X[m] * vis[m];
        aX[m] += al * vis[m] * lfac - 0.065 * act + au * vis[m] + avt;
        double av = (al * lfac + au) * X[m];
        const double ivm = isv[m] * isv[m];
#pragma unroll
        for (int n = 0; n < ns; ++n) {
          if (m == n) continue;
          const double w = c_mix.wj_div_wi_1_4[m][n], sw = c_mix.sqrt_wiwj_8[m][n];
          const double r = svm * isv[n], nm = 1 + r * w;
          aX[n] += avt * nm * nm * sw;
          const double ar = avt * X[n] * nm * sw * w * r;  // half the adjoint of ln(vis_m / vis_n) times 2
          av += ar * ivm;
          avis[n] -= ar * (isv[n] * isv[n]);
        }
        avis[m] += av;
      }
#pragma unroll
      for (int l = 0; l < ns; ++l) aTv += avis[l] * vis[l] * dlv[l];
    }
    aT += aTv;
    // c = sqrt(gamma Ru T / mw)
    const double acoustic = sqrt(gamma * kRuD * t * smw), hc = 0.5 * ac * acoustic;
    const double agamma = hc / gamma;
    aT += hc * it;
    amw -= hc * smw;
    // X_l = Y_l mw / W_l; gamma = cpt / cvt; mw = 1 / sum Y / W; cp_l(T)
#pragma unroll
    for (int l = 0; l < ns; ++l) amw += aX[l] * s.sv[l * P + p] * c_mix.imw[l];
    const double acpt = agamma / cvt, acvt = -agamma * gamma / cvt;
#pragma unroll
    for (int l = 0; l < ns; ++l) {
      double h, cp;
      mix_h_cp_one<double>(l, t, h, cp);
      A.Y[(long long)l * P + p] += aX[l] * mw * c_mix.imw[l] + acpt * cp + acvt * (cp - c_mix.ru_mw[l]) -
                                   amw * mw * mw * c_mix.imw[l];
      aT += (acp[l] + (acpt + acvt) * s.sv[l * P + p]) * mix_dcp_dt_one(l, t);
    }
    A.rho[p] += arho;
    A.p[p] += ap;
    A.T[p] += aT;
  }
}

// Ghost nodes hold copies of their source node's primitive state (bv, sv) and recompute their cv from
// it (compute_cv_from_bv_1_point<mixture>, FieldOperation.cuh:78-105): rho E = rho (sum h(T) Y +
// |V|^2 / 2) - p.  This moves a ghost's cv adjoint onto its primitive adjoints (rho, u, v, w, p, T, Y).
template <int NS>
__global__ void __launch_bounds__(128, 4) k_adj_ghost_cv(DevBlock b, DevState s, DevAdj A, int nv) {
  if (NS > 0) nv = 5 + NS;
  const long long P = b.plane;
  const int ns = OSTC_NS;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    if (!(s.bv[p] > 0)) continue;
    const int i = (int)(p % b.pitch) - b.g;
    const long long r = p / b.pitch;
    const int j = (int)(r % b.sy) - b.g, k = (int)(r / b.sy) - b.gz;
    if (i >= 0 && i < b.mx && j >= 0 && j < b.my && k >= 0 && k < b.mz) continue;
    const double rho = s.bv[p], u = s.bv[P + p], v = s.bv[2 * P + p], w = s.bv[3 * P + p], t = s.bv[5 * P + p];
    double a[Spec<NS>::A + 5];
    bool any = false;
    for (int l = 0; l < nv; ++l) {
      a[l] = A.cv[l * P + p];
      any = any || a[l] != 0.0;
      A.cv[l * P + p] = 0.0;
    }
    if (!any) continue;
    double h[Spec<NS>::A], cp[Spec<NS>::A];
    mix_h_cp<NS, double>(t, h, cp);
    double hy = 0, cpy = 0;
    for (int l = 0; l < ns; ++l) {
      const double y = s.sv[l * P + p];
      hy += h[l] * y;
      cpy += cp[l] * y;
    }
    const double ek = 0.5 * (u * u + v * v + w * w);
    double arho = a[0] + a[1] * u + a[2] * v + a[3] * w + a[4] * (hy + ek);
    for (int l = 0; l < ns; ++l) {
      arho += a[5 + l] * s.sv[l * P + p];
      A.Y[(long long)l * P + p] += a[4] * rho * h[l] + a[5 + l] * rho;
    }
    A.rho[p] += arho;
    A.vel[p] += (a[1] + a[4] * u) * rho;
    A.vel[P + p] += (a[2] + a[4] * v) * rho;
    A.vel[2 * P + p] += (a[3] + a[4] * w) * rho;
    A.T[p] += a[4] * rho * cpy;
    A.p[p] -= a[4];
  }
}

// Interior nodes: primitive adjoints -> cv (and T) adjoints.  rho = cv0, u = cv1 / rho (v, w
// alike), Y_l = cv_{5+l} / rho, p = rho Ru T sum Y / W.  With exact_t the node's T is the root of
// e = cv4 / rho - |V|^2 / 2 = sum Y h(T) - Ru T sum Y / W (compute_temperature_and_pressure,
// FieldOperation.cu:3-40) and its adjoint goes to cv by the implicit-function derivative; otherwise
// T is a state variable of its own and its adjoint is left in A.T.
template <int NS>
__global__ void __launch_bounds__(128, 4) k_adj_eos(DevBlock b, DevState s, DevAdj A, int exact_t) {
  const long long P = b.plane;
  const int ns = OSTC_NS;
  for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < b.n; n += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(n % b.mx);
    const long long r = n / b.mx;
    const int j = (int)(r % b.my), k = (int)(r / b.my);
    const long long p = b.id(i, j, k);
    const double rho = s.cv[p];
    const double t = s.bv[5 * P + p];
    const double irho = 1.0 / rho;
    const double u = s.cv[P + p] * irho, v = s.cv[2 * P + p] * irho, w = s.cv[3 * P + p] * irho;
    double y[Spec<NS>::A], ay[Spec<NS>::A];
    double gsum = 0;  // sum Y / W
    for (int l = 0; l < ns; ++l) {
      y[l] = s.cv[(5 + l) * P + p] * irho;
      ay[l] = A.Y[(long long)l * P + p];
      gsum += y[l] * c_mix.imw[l];
    }
    double arho = A.rho[p], aT = A.T[p];
    const double ap = A.p[p];
    double au = A.vel[p], av = A.vel[P + p], aw = A.vel[2 * P + p];
    // p = rho Ru T gsum
    arho += ap * kRuD * t * gsum;
    aT += ap * rho * kRuD * gsum;
    for (int l = 0; l < ns; ++l) ay[l] += ap * rho * kRuD * t * c_mix.imw[l];
    if (exact_t) {
      double h[Spec<NS>::A], cp[Spec<NS>::A];
      mix_h_cp<NS, double>(t, h, cp);
      double cvm = 0;
      for (int l = 0; l < ns; ++l) cvm += y[l] * (cp[l] - kRuD * c_mix.imw[l]);
      const double ae = aT / cvm;
      for (int l = 0; l < ns; ++l) ay[l] -= aT * (h[l] - kRuD * t * c_mix.imw[l]) / cvm;
      // e = cv4 / rho - (u^2 + v^2 + w^2) / 2
      A.cv[4 * P + p] += ae * irho;
      arho -= ae * s.cv[4 * P + p] * irho * irho;
      au -= ae * u;
      av -= ae * v;
      aw -= ae * w;
      aT = 0.0;
    }
    A.T[p] = aT;
    A.cv[P + p] += au * irho;
    A.cv[2 * P + p] += av * irho;
    A.cv[3 * P + p] += aw * irho;
    arho -= (au * u + av * v + aw * w) * irho;
    for (int l = 0; l < ns; ++l) {
      A.cv[(5 + l) * P + p] += ay[l] * irho;
      arho -= ay[l] * y[l] * irho;
    }
    A.cv[p] += arho;
  }
}

// Ghost fills in reverse (apply_outflow / apply_periodic, BoundCond.cuh:205-233, 1443-1486): each
// ghost node's primitive adjoints (rho, u, v, w, p, T, Y) move to the node it was copied from.  Faces
// run in the reverse of the forward order, so a ghost filled from another face's ghost passes its
// adjoint on in turn.
__global__ void __launch_bounds__(128) k_adj_bc_face(DevBlock b, DevAdj A, int ns, DevFace f) {
  const int t0 = f.face == 0 ? 1 : 0;
  const int t1 = f.face == 2 ? 1 : 2;
  const int n0 = f.re[t0] - f.rs[t0] + 1, n1 = f.re[t1] - f.rs[t1] + 1;
  const long long nn = (long long)n0 * n1;
  const long long P = b.plane;
  const long long st[3] = {1, b.pitch, (long long)b.pitch * b.sy};
  int dir[3] = {0, 0, 0};
  dir[f.face] = f.direction;
  const long long dstep = dir[0] * st[0] + dir[1] * st[1] + dir[2] * st[2];
  double *planes[6] = {A.rho, A.vel, A.vel + P, A.vel + 2 * P, A.p, A.T};
  for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < nn; n += (long long)gridDim.x * blockDim.x) {
    int idx[3];
    idx[f.face] = f.rs[f.face];
    idx[t0] = f.rs[t0] + (int)(n % n0);
    idx[t1] = f.rs[t1] + (int)(n / n0);
    const long long pb = b.id(idx[0], idx[1], idx[2]);
    long long po = pb;
    if (f.type == kPeriodic) {
      const int ext[3] = {b.mx, b.my, b.mz};
      int other[3] = {idx[0], idx[1], idx[2]};
      other[f.face] = f.direction < 0 ? ext[f.face] - 1 : 0;
      po = b.id(other[0], other[1], other[2]);
    }
    for (int g = b.g; g >= 1; --g) {
      const long long pg = b.chk(pb + g * dstep);
      const long long ps = b.chk(f.type == kPeriodic ? po + g * dstep : pb);
      for (int q = 0; q < 6; ++q) {
        planes[q][ps] += planes[q][pg];
        planes[q][pg] = 0.0;
      }
      for (int l = 0; l < ns; ++l) {
        A.Y[l * P + ps] += A.Y[l * P + pg];
        A.Y[l * P + pg] = 0.0;
      }
    }
  }
}

// Reverse of the stage's temperature Newton iteration (update_cv_and_bv_rk + compute_temperature_and_
// pressure, RK.cuh:230-284, FieldOperation.cu:3-40): T_out = N(T_start; e, Y) of the stage output's
// cv, started from the stage input's T, iterated to the reference's relative tolerance 1e-3.  The
// iterate (not the exact root) is differentiated, by Dual evaluations seeded on e, each Y and the
// start T: lam_cv += (dT_out / d cv_out)^T lam_t, lam_t_start += dT_out / dT_start * lam_t.
template <int NS>
__global__ void __launch_bounds__(128, 4) k_adj_newton(DevBlock b, DevState in, DevState out, const double *lam_t,
                                                    double *lam_cv, double *lam_t_start) {
  const long long P = b.plane;
  const int ns = OSTC_NS;
  for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < b.n; n += (long long)gridDim.x * blockDim.x) {
    const double lt = lam_t[n];
    if (lt == 0.0) continue;
    const int i = (int)(n % b.mx);
    const long long r = n / b.mx;
    const int j = (int)(r % b.my), k = (int)(r / b.my);
    const long long p = b.id(i, j, k);
    const double rho = out.cv[p], irho = 1.0 / rho;
    const double u = out.cv[P + p] * irho, v = out.cv[2 * P + p] * irho, w = out.cv[3 * P + p] * irho;
    const double e = out.cv[4 * P + p] / rho - 0.5 * (u * u + v * v + w * w);
    const double t0 = in.bv[5 * P + p];
    double yv[Spec<NS>::A];
    for (int l = 0; l < ns; ++l) yv[l] = out.cv[(5 + l) * P + p] * irho;
    double de = 0, dts = 0, dy[Spec<NS>::A];
    for (int in_ = 0; in_ < ns + 2; ++in_) {
      Dual y[Spec<NS>::A], pr;
      for (int l = 0; l < ns; ++l) y[l] = Dual(yv[l], in_ == 2 + l ? 1.0 : 0.0);
      const Dual t = mix_temperature<NS, Dual>(Dual(rho), Dual(e, in_ == 0 ? 1.0 : 0.0), Dual(t0, in_ == 1 ? 1.0 : 0.0),
                                               y, pr);
      if (in_ == 0) de = t.d;
      else if (in_ == 1) dts = t.d;
      else dy[in_ - 2] = t.d;
    }
    lam_t_start[n] += dts * lt;
    // e = cv4 / rho - |V|^2 / 2, Y = cv_{5+l} / rho
    const double ae = de * lt;
    double arho = -ae * out.cv[4 * P + p] * irho * irho + ae * (u * u + v * v + w * w) * irho;
    lam_cv[4 * b.n + n] += ae * irho;
    lam_cv[b.n + n] -= ae * u * irho;
    lam_cv[2 * b.n + n] -= ae * v * irho;
    lam_cv[3 * b.n + n] -= ae * w * irho;
    for (int l = 0; l < ns; ++l) {
      const double ay = dy[l] * lt;
      lam_cv[(5 + l) * b.n + n] += ay * irho;
      arho -= ay * yv[l] * irho;
    }
    lam_cv[n] += arho;
  }
}

// interior part of nv adjoint planes, in the layout of dq
__global__ void k_adj_gather(DevBlock b, const double *__restrict__ Acv, int nv, double *__restrict__ out) {
  for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < b.n; n += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(n % b.mx);
    const long long r = n / b.mx;
    const int j = (int)(r % b.my), k = (int)(r / b.my);
    const long long p = b.id(i, j, k);
    for (int l = 0; l < nv; ++l) out[l * b.n + n] = Acv[l * b.plane + p];
  }
}

// Seed of a stage's right-hand-side adjoint: dqb = c dt / J * lam (the stage adds c dt / J * dq to
// cv, update_cv_and_bv_rk, RK.cuh:230-284).  2-D blocks zero component 3 of lam in place first: the
// stage output's rho*w is set to 0, so its adjoint never reaches the stage's inputs.
__global__ void k_adj_stage_seed(DevBlock b, double *lam, double c, const double *dtp, double *dqb, int nv) {
  const double dt = *dtp;
  for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < b.n; n += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(n % b.mx);
    const long long r = n / b.mx;
    const int j = (int)(r % b.my), k = (int)(r / b.my);
    const double f = c * dt / b.jac[b.id(i, j, k)];
    if (b.mz == 1) lam[3 * b.n + n] = 0.0;
    for (int l = 0; l < nv; ++l) dqb[l * b.n + n] = f * lam[l * b.n + n];
  }
}

// y = a x + c y over n values
__global__ void k_axpby(long long n, double a, const double *__restrict__ x, double c, double *__restrict__ y) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = a * x[i] + c * y[i];
}

// lam_cv += (dT / dcv)^T lam_t for T the equation-of-state root of the node's cv (implicit-function
// derivative of sum Y h(T) - Ru T sum Y / W = cv4 / rho - |V|^2 / 2), interior nodes
template <int NS>
__global__ void __launch_bounds__(128) k_adj_t_to_cv(DevBlock b, DevState s, const double *lam_t, double *lam_cv) {
  const long long P = b.plane;
  const int ns = OSTC_NS;
  for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < b.n; n += (long long)gridDim.x * blockDim.x) {
    const double lt = lam_t[n];
    if (lt == 0.0) continue;
    const int i = (int)(n % b.mx);
    const long long r = n / b.mx;
    const int j = (int)(r % b.my), k = (int)(r / b.my);
    const long long p = b.id(i, j, k);
    const double rho = s.cv[p], irho = 1.0 / rho, t = s.bv[5 * P + p];
    const double u = s.cv[P + p] * irho, v = s.cv[2 * P + p] * irho, w = s.cv[3 * P + p] * irho;
    double y[Spec<NS>::A], h[Spec<NS>::A], cp[Spec<NS>::A];
    mix_h_cp<NS, double>(t, h, cp);
    double cvm = 0;
    for (int l = 0; l < ns; ++l) {
      y[l] = s.cv[(5 + l) * P + p] * irho;
      cvm += y[l] * (cp[l] - kRuD * c_mix.imw[l]);
    }
    const double ae = lt / cvm;
    double arho = -ae * s.cv[4 * P + p] * irho * irho + ae * (u * u + v * v + w * w) * irho;
    lam_cv[4 * b.n + n] += ae * irho;
    lam_cv[b.n + n] -= ae * u * irho;
    lam_cv[2 * b.n + n] -= ae * v * irho;
    lam_cv[3 * b.n + n] -= ae * w * irho;
    for (int l = 0; l < ns; ++l) {
      const double ay = -lt * (h[l] - kRuD * t * c_mix.imw[l]) / cvm;
      lam_cv[(5 + l) * b.n + n] += ay * irho;
      arho -= ay * y[l] * irho;
    }
    lam_cv[n] += arho;
  }
}

}  // namespace ostc
