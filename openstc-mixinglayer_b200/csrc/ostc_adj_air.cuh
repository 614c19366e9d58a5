// ostc_adj_air.cuh -- vector-Jacobian product of the calorically-perfect-air right-hand side
// (ostc_rhs_vjp on the AWENO path): cv_bar = (d dq / d cv)^T dq_bar at the current state.  The
// reference has no adjoint.  Every term of the forward sweep is a function of a few stencil nodes'
// cv, so its transposed Jacobian is assembled from local derivatives:
//   1. face fluxes (AWENO_interpolation + Riemann solver, AWENO.cu:15-154, RiemannSolver.cuh:9-461): the
//      reverse of aweno_face_flux by hand: Riemann solver, the two sides' primitive states, then field
//      by field the WENO-Z weights and interpolants, the eigenvector rows and the Roe averages;
//   2. the central correction (CDSPart1D, AWENO.cu:307-350): per node, the adjoint of its physical
//      flux collected from the nodes whose correction reads it, times d f_node / d cv (Dual);
//   3. viscous faces (viscous_flux_fv/gv/hv, ViscousScheme.cuh:24-911): the reverse of viscous_face onto
//      u, v, w, T of the up to ten nodes the face's gradients read (mu through Sutherland's law of T),
//      then per node through the equation of state onto cv;
//   4. ghost fills in reverse face order (apply_outflow / apply_periodic): a ghost's cv adjoint moves
//      to the node it was copied from (a ghost's cv is its source's cv).
// Evaluations are FP64 (the plain path's adjoint).  Accumulation into the node planes uses atomicAdd
// where several threads reach one node, so results are reproducible to rounding, not bitwise.
#pragma once

#include "dual.cuh"

namespace ostc {

// d p / d cv of one node (p = (gamma - 1)(rho E - |m|^2 / (2 rho))).
__device__ __forceinline__ void air_dp_dcv(const double *cv, double *dp) {
  const double ir = 1.0 / cv[0], u = cv[1] * ir, v = cv[2] * ir, w = cv[3] * ir;
  const double g1 = kGamma - 1;
  dp[0] = g1 * 0.5 * (u * u + v * v + w * w);
  dp[1] = -g1 * u;
  dp[2] = -g1 * v;
  dp[3] = -g1 * w;
  dp[4] = g1;
}

// Node index along a sweep: node c of direction DIR through the other two interior indices.
template <int DIR>
__device__ __forceinline__ long long sweep_id(const DevBlock &b, int c, int o1, int o2) {
  return DIR == 0 ? b.id(c, o1, o2) : DIR == 1 ? b.id(o1, c, o2) : b.id(o1, o2, c);
}
template <int DIR>
__device__ __forceinline__ long long sweep_iq(const DevBlock &b, int c, int o1, int o2) {
  return DIR == 0 ? b.iq(c, o1, o2) : DIR == 1 ? b.iq(o1, c, o2) : b.iq(o1, o2, c);
}
// Thread t of a sweep over `span` sweep positions starting at c0 and all interior (o1, o2).
template <int DIR>
__device__ __forceinline__ void sweep_pos(const DevBlock &b, long long t, int span, int c0, int &c, int &o1, int &o2) {
  if (DIR == 0) {
    c = c0 + (int)(t % span);
    const long long r = t / span;
    o1 = (int)(r % b.my);
    o2 = (int)(r / b.my);
  } else {
    o1 = (int)(t % b.mx);
    const long long r = t / b.mx;
    c = c0 + (int)(r % span);
    o2 = (int)(r / span);
  }
}

// ---- reverse of the Riemann solvers.  Sides are pl, pr = rho, u, v, w, p, rhoE; k the metric vector the
// solver projects on; fb the adjoint of the face flux; al, ar collect the adjoints of pl, pr (added).

// c (rho U, rho U v + p k, (rhoE + p) U), U = k . v
__device__ __forceinline__ void side_flux_bwd(const double *p, const double *k, double c, const double *fb, double *a) {
  const double U = k[0] * p[1] + k[1] * p[2] + k[2] * p[3], rU = p[0] * U;
  const double rUb = c * (fb[0] + fb[1] * p[1] + fb[2] * p[2] + fb[3] * p[3]);
  const double Ub = c * fb[4] * (p[5] + p[4]) + rUb * p[0];
  a[0] += rUb * U;
#pragma unroll
  for (int d = 0; d < 3; ++d) a[1 + d] += c * fb[1 + d] * rU + Ub * k[d];
  a[4] += c * (fb[1] * k[0] + fb[2] * k[1] + fb[3] * k[2] + fb[4] * U);
  a[5] += c * fb[4] * U;
}

// speed of sound c = sqrt(gamma p / rho) of one side
__device__ __forceinline__ void sound_bwd(const double *p, double c, double cb, double *a) {
  a[4] += cb * 0.5 * c / p[4];
  a[0] -= cb * 0.5 * c / p[0];
}

// Roe weights rl = sqrt(rho_l) / (sqrt(rho_l) + sqrt(rho_r)), rr: densities' adjoints
__device__ __forceinline__ void roe_weight_bwd(double sl, double sr, double isum, double rlb, double rrb, double &a0l,
                                               double &a0r) {
  const double t = (rlb - rrb) * isum * isum;
  a0l += t * sr * 0.5 / sl;
  a0r -= t * sl * 0.5 / sr;
}

__device__ __forceinline__ void hllc_bwd(const double *pl, const double *pr, const double *mt0, const double *mt1,
                                         double j0, double j1, const double *fb, double *al, double *ar) {
  const double k[3] = {0.5 * (mt0[0] + mt1[0]), 0.5 * (mt0[1] + mt1[1]), 0.5 * (mt0[2] + mt1[2])};
  const double gradK = sqrt(k[0] * k[0] + k[1] * k[1] + k[2] * k[2]), igk = 1.0 / gradK;
  const double jac = 0.5 * (j0 + j1), JG = jac * gradK;
  const double sql = sqrt(pl[0]), sqr = sqrt(pr[0]), isq = 1.0 / (sql + sqr);
  const double rlc = sql * isq, rrc = sqr * isq;
  double vt[3], ekt = 0, Ubar = 0, unl = 0, unr = 0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    vt[d] = pl[1 + d] * rlc + pr[1 + d] * rrc;
    ekt += 0.5 * vt[d] * vt[d];
    Ubar += k[d] * igk * vt[d];
    unl += k[d] * igk * pl[1 + d];
    unr += k[d] * igk * pr[1 + d];
  }
  const double hl = (pl[5] + pl[4]) / pl[0], hr = (pr[5] + pr[4]) / pr[0];
  const double ct = sqrt((kGamma - 1) * (hl * rlc + hr * rrc - ekt));
  const double cl = sqrt(kGamma * pl[4] / pl[0]);
  const bool l_roe = Ubar - ct < unl - cl;
  const double sl = l_roe ? Ubar - ct : unl - cl;
  if (sl >= 0) {
    side_flux_bwd(pl, k, jac, fb, al);
    return;
  }
  const double cr = sqrt(kGamma * pr[4] / pr[0]);
  const bool r_roe = Ubar + ct > unr + cr;
  const double sr = r_roe ? Ubar + ct : unr + cr;
  if (sr < 0) {
    side_flux_bwd(pr, k, jac, fb, ar);
    return;
  }
  const double dl = pl[0] * (sl - unl), dr = pr[0] * (sr - unr);
  const double iden = 1.0 / (dr - dl);
  const double sm = (dr * unr - dl * unl + pl[4] - pr[4]) * iden;
  const double pm = dl * (sm - unl) + pl[4];
  const bool left = sm >= 0;
  double q[6];
#pragma unroll
  for (int l = 0; l < 6; ++l) q[l] = left ? pl[l] : pr[l];
  const double sk = left ? sl : sr, un = left ? unl : unr;
  const double pc = 1.0 / (sk - sm), iq0 = 1.0 / q[0];
  const double Q = JG * pc * sm * (sk - un) * q[0];
  const double A = sk * pm - q[4] * un, B = sk * pm - sm * q[4];
  double slb = 0, srb = 0, unlb = 0, unrb = 0, skb = 0, unb = 0, smb, pmb, pcb;
  double qb[6] = {0, 0, 0, 0, 0, 0};
  // flux = Q (1, v, rhoE / rho) + dP k (momentum) + JG pc sm A (energy), dP = B pc jac
  const double Qb = fb[0] + fb[1] * q[1] + fb[2] * q[2] + fb[3] * q[3] + fb[4] * q[5] * iq0;
  const double dPb = fb[1] * k[0] + fb[2] * k[1] + fb[3] * k[2];
#pragma unroll
  for (int d = 0; d < 3; ++d) qb[1 + d] = fb[1 + d] * Q;
  qb[5] = fb[4] * Q * iq0;
  qb[0] = -fb[4] * Q * q[5] * iq0 * iq0;
  pcb = fb[4] * JG * sm * A;
  smb = fb[4] * JG * pc * A;
  const double Ab = fb[4] * JG * pc * sm, Bb = dPb * jac * pc;
  skb = (Ab + Bb) * pm;
  pmb = (Ab + Bb) * sk;
  qb[4] = -Ab * un - Bb * sm;
  unb = -Ab * q[4];
  pcb += dPb * jac * B;
  smb -= Bb * q[4];
  {
    const double c = JG * Qb;
    pcb += c * sm * (sk - un) * q[0];
    smb += c * pc * (sk - un) * q[0];
    skb += c * pc * sm * q[0];
    unb -= c * pc * sm * q[0];
    qb[0] += c * pc * sm * (sk - un);
  }
  {
    const double t = -pcb * pc * pc;
    skb += t;
    smb -= t;
  }
  double dlb = pmb * (sm - unl), drb;
  smb += pmb * dl;
  unlb -= pmb * dl;
  al[4] += pmb;
  {
    const double nb = smb * iden, db = -smb * sm * iden;
    drb = nb * unr + db;
    unrb += nb * dr;
    dlb -= nb * unl + db;
    unlb -= nb * dl;
    al[4] += nb;
    ar[4] -= nb;
  }
  if (left) {
    slb += skb;
    unlb += unb;
  } else {
    srb += skb;
    unrb += unb;
  }
#pragma unroll
  for (int l = 0; l < 6; ++l) {
    if (left) al[l] += qb[l];
    else ar[l] += qb[l];
  }
  al[0] += dlb * (sl - unl);
  slb += dlb * pl[0];
  unlb -= dlb * pl[0];
  ar[0] += drb * (sr - unr);
  srb += drb * pr[0];
  unrb -= drb * pr[0];
  double Ubb = 0, ctb = 0;
  if (l_roe) {
    Ubb += slb;
    ctb -= slb;
  } else {
    unlb += slb;
    sound_bwd(pl, cl, -slb, al);
  }
  if (r_roe) {
    Ubb += srb;
    ctb += srb;
  } else {
    unrb += srb;
    sound_bwd(pr, cr, srb, ar);
  }
  const double htb = ctb * 0.5 * (kGamma - 1) / ct;
  double rlb = htb * hl, rrb = htb * hr;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double vb = Ubb * k[d] * igk - htb * vt[d];
    al[1 + d] += vb * rlc + unlb * k[d] * igk;
    ar[1 + d] += vb * rrc + unrb * k[d] * igk;
    rlb += vb * pl[1 + d];
    rrb += vb * pr[1 + d];
  }
  {
    const double a = htb * rlc / pl[0], b = htb * rrc / pr[0];
    al[4] += a;
    al[5] += a;
    al[0] -= a * hl;
    ar[4] += b;
    ar[5] += b;
    ar[0] -= b * hr;
  }
  roe_weight_bwd(sql, sqr, isq, rlb, rrb, al[0], ar[0]);
}

// The AUSM+ splittings of one side (s = +1 left, -1 right): Mach and pressure parts and derivatives.
__device__ __forceinline__ void ausm_split(double m, double s, double &mp, double &dm, double &pp, double &dp) {
  if (fabs(m) > 1) {
    mp = 0.5 * (m + s * fabs(m));
    dm = s * m > 0 ? 1.0 : 0.0;
    pp = s * m > 0 ? 1.0 : 0.0;
    dp = 0;
  } else {
    const double a = 0.25 * (m + s) * (m + s), m2 = m * m - 1, b = m2 * m2;
    mp = s * (a + 0.125 * b);
    dm = s * (0.5 * (m + s) + 0.5 * m * m2);
    pp = a * (2 - s * m) + s * (3 / 16.0) * m * b;
    dp = 0.5 * (m + s) * (2 - s * m) - s * a + s * (3 / 16.0) * (b + 4 * m * m * m2);
  }
}

__device__ __forceinline__ void ausm_bwd(const double *pl, const double *pr, const double *mt0, const double *mt1,
                                         double j0, double j1, const double *fb, double *al, double *ar) {
  const double k[3] = {0.5 * (j0 * mt0[0] + j1 * mt1[0]), 0.5 * (j0 * mt0[1] + j1 * mt1[1]),
                       0.5 * (j0 * mt0[2] + j1 * mt1[2])};
  const double gkj = sqrt(k[0] * k[0] + k[1] * k[1] + k[2] * k[2]), ig = 1.0 / gkj;
  const double ul = (k[0] * pl[1] + k[1] * pl[2] + k[2] * pl[3]) * ig;
  const double ur = (k[0] * pr[1] + k[1] * pr[2] + k[2] * pr[3]) * ig;
  const double cl = sqrt(kGamma * pl[4] / pl[0]), cr = sqrt(kGamma * pr[4] / pr[0]);
  const double c = 0.5 * (cl + cr), ic = 1.0 / c, ml = ul * ic, mr = ur * ic;
  double mlp, dml, plp, dpl, mrn, dmr, prn, dpr;
  ausm_split(ml, 1.0, mlp, dml, plp, dpl);
  ausm_split(mr, -1.0, mrn, dmr, prn, dpr);
  const double mh = mlp + mrn, mpos = 0.5 * (mh + fabs(mh)), mneg = 0.5 * (mh - fabs(mh));
  const double rm = pl[0] * mpos + pr[0] * mneg, mass = c * rm, coeff = mass * gkj;
  const bool left = mass >= 0;
  double q[6], qb[6];
#pragma unroll
  for (int l = 0; l < 6; ++l) q[l] = left ? pl[l] : pr[l];
  const double iq0 = 1.0 / q[0], H = (q[5] + q[4]) * iq0;
  // flux = coeff (1, v, H) + p_coeff k (momentum)
  const double cfb = fb[0] + fb[1] * q[1] + fb[2] * q[2] + fb[3] * q[3] + fb[4] * H;
  const double pcb = fb[1] * k[0] + fb[2] * k[1] + fb[3] * k[2];
#pragma unroll
  for (int d = 0; d < 3; ++d) qb[1 + d] = fb[1 + d] * coeff;
  qb[4] = qb[5] = fb[4] * coeff * iq0;
  qb[0] = -fb[4] * coeff * iq0 * H;
#pragma unroll
  for (int l = 0; l < 6; ++l) {
    if (left) al[l] += qb[l];
    else ar[l] += qb[l];
  }
  al[4] += pcb * plp;
  ar[4] += pcb * prn;
  const double mb = cfb * gkj;
  al[0] += mb * c * mpos;
  ar[0] += mb * c * mneg;
  const double mhb = mb * c * (mh < 0 ? pr[0] : pl[0]);
  const double mlb = mhb * dml + pcb * pl[4] * dpl, mrb = mhb * dmr + pcb * pr[4] * dpr;
  const double cb = mb * rm - (mlb * ml + mrb * mr) * ic;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    al[1 + d] += mlb * ic * k[d] * ig;
    ar[1 + d] += mrb * ic * k[d] * ig;
  }
  sound_bwd(pl, cl, 0.5 * cb, al);
  sound_bwd(pr, cr, 0.5 * cb, ar);
}

__device__ __forceinline__ void lax_friedrichs_bwd(const double *pl, const double *pr, const double *mt0,
                                                   const double *mt1, double j0, double j1, const double *fb,
                                                   double *al, double *ar) {
  const double k[3] = {0.5 * (mt0[0] + mt1[0]), 0.5 * (mt0[1] + mt1[1]), 0.5 * (mt0[2] + mt1[2])};
  const double gradK = sqrt(k[0] * k[0] + k[1] * k[1] + k[2] * k[2]), hj = 0.25 * (j0 + j1);
  const double Ul = k[0] * pl[1] + k[1] * pl[2] + k[2] * pl[3], Ur = k[0] * pr[1] + k[1] * pr[2] + k[2] * pr[3];
  const double cl = sqrt(kGamma * pl[4] / pl[0]), cr = sqrt(kGamma * pr[4] / pr[0]);
  const double xl = fabs(Ul) + cl * gradK, xr = fabs(Ur) + cr * gradK;
  const bool right = xr > xl;
  const double sr = right ? xr : xl;
  side_flux_bwd(pl, k, hj, fb, al);
  side_flux_bwd(pr, k, hj, fb, ar);
  // - sr (U_r - U_l) hj over the conserved variables U = (rho, rho v, rhoE)
  const double c = hj * sr;
  double srb = fb[0] * (pr[0] - pl[0]) + fb[4] * (pr[5] - pl[5]);
  al[0] += c * fb[0];
  ar[0] -= c * fb[0];
  al[5] += c * fb[4];
  ar[5] -= c * fb[4];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    srb += fb[1 + d] * (pr[0] * pr[1 + d] - pl[0] * pl[1 + d]);
    al[0] += c * fb[1 + d] * pl[1 + d];
    al[1 + d] += c * fb[1 + d] * pl[0];
    ar[0] -= c * fb[1 + d] * pr[1 + d];
    ar[1 + d] -= c * fb[1 + d] * pr[0];
  }
  srb *= -hj;
  const double U = right ? Ur : Ul, sgn = U < 0 ? -srb : srb;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (right) ar[1 + d] += sgn * k[d];
    else al[1 + d] += sgn * k[d];
  }
  if (right) sound_bwd(pr, cr, srb * gradK, ar);
  else sound_bwd(pl, cl, srb * gradK, al);
}

// ---- reverse of the WENO-Z combinations

// Value f = sum w_k p_k / sum w_k, w_k = d_k (D_k + tau) prod_{i != k} D_i (WenoComb), D_k = (eps + beta_k)^2,
// and for its adjoint fb: pb[k] of the candidates, bb[k] of the indicators through D_k, tb of tau.  Products
// only, as the forward sweep, so that an eps + beta_k that passes through zero divides nothing.
template <int N>
__device__ __forceinline__ double weno_comb_bwd(const double *d, const double *beta, double tau, const double *p,
                                                double fb, double *pb, double *bb, double &tb) {
  const double eps = 1e-6;
  double g[N], D[N], w[N], S = 0, num = 0;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    g[k] = eps + beta[k];
    D[k] = g[k] * g[k];
  }
  double T[N];  // products of the other D
#pragma unroll
  for (int k = 0; k < N; ++k) {
    double t = 1.0;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (i != k) t = t * D[i];
    T[k] = t;
    w[k] = d[k] * (D[k] + tau) * t;
    S += w[k];
    num += w[k] * p[k];
  }
  const double is = 1.0 / S, f = num * is;
  double e[N];
  tb = 0;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    pb[k] = fb * w[k] * is;
    e[k] = fb * (p[k] - f) * is * d[k];
    tb += e[k] * T[k];
  }
#pragma unroll
  for (int j = 0; j < N; ++j) {
    double a = e[j] * T[j];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      if (k == j) continue;
      double t = 1.0;
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (i != k && i != j) t = t * D[i];
      a += e[k] * (D[k] + tau) * t;
    }
    bb[j] = 2 * g[j] * a;
  }
  return f;
}

// One side's WENO5-Z: points v[0..4] in the order of the forward sweep's indicators, candidates q0, q1, q2
// (linear in the face's six points, see below); adds to gv[0..4] the indicators' part.
__device__ __forceinline__ double weno5_side_bwd(const double *v, const double *d, const double *p, double fb, double *pb,
                                                 double *gv) {
  const double th = 13.0 / 12;
  const double a0 = v[0] + v[2] - 2 * v[1], c0 = v[0] + 3 * v[2] - 4 * v[1];
  const double a1 = v[1] + v[3] - 2 * v[2], c1 = v[3] - v[1];
  const double a2 = v[2] + v[4] - 2 * v[3], c2 = 3 * v[2] + v[4] - 4 * v[3];
  const double beta[3] = {th * a0 * a0 + 0.25 * c0 * c0, th * a1 * a1 + 0.25 * c1 * c1, th * a2 * a2 + 0.25 * c2 * c2};
  double bb[3], tb;
  const double dt = beta[0] - beta[2];
  const double f = weno_comb_bwd<3>(d, beta, dt * dt, p, fb, pb, bb, tb);
  bb[0] += 2 * tb * dt;
  bb[2] -= 2 * tb * dt;
  const double A0 = 2 * th * a0 * bb[0], C0 = 0.5 * c0 * bb[0], A1 = 2 * th * a1 * bb[1], C1 = 0.5 * c1 * bb[1],
               A2 = 2 * th * a2 * bb[2], C2 = 0.5 * c2 * bb[2];
  gv[0] += A0 + C0;
  gv[1] += -2 * A0 - 4 * C0 + A1 - C1;
  gv[2] += A0 + 3 * C0 - 2 * A1 + A2 + 3 * C2;
  gv[3] += A1 + C1 - 2 * A2 - 4 * C2;
  gv[4] += A2 + C2;
  return f;
}

// Gradient of weno_quad times s.
__device__ __forceinline__ void weno_quad_bwd(double a, double b, double c, double A, double B, double C, double D,
                                              double E, double F, double s, double &ga, double &gb, double &gc) {
  ga += s * (2 * A * a + B * b + C * c);
  gb += s * (B * a + 2 * D * b + E * c);
  gc += s * (C * a + E * b + 2 * F * c);
}

// One side's WENO7-Z (weno7_betas) from its differences d[0..5] and points v2, v3; candidates q as distances
// from the face's point i, whose adjoints go to qb; adds the indicators' part to gd[0..5], g2, g3.
__device__ __forceinline__ double weno7_side_bwd(const double *d, double v2, double v3, const double *w, const double *q,
                                                 double fb, double *qb, double *gd, double &g2, double &g3) {
  double b[4], bb[4], tb;
  weno7_betas<double>(d, v2, v3, b[0], b[1], b[2], b[3]);
  const double t = b[3] + 5 * (b[2] - b[1]) - b[0];
  const double f = weno_comb_bwd<4>(w, b, t * t, q, fb, qb, bb, tb);
  tb *= 2 * t;
  const double c = 1.0 / 2880;
  weno_quad_bwd(d[3], d[4], d[5], 25729, -63436, 22778, 45076, -33916, 6649, c * (bb[0] - tb), gd[3], gd[4], gd[5]);
  weno_quad_bwd(d[2], d[3], d[4], 6649, -17116, 5978, 17236, -13036, 3169, c * (bb[1] - 5 * tb), gd[2], gd[3], gd[4]);
  weno_quad_bwd(d[0], d[1], d[2], 6649, -33916, 22778, 45076, -63436, 25729, c * (bb[3] + tb), gd[0], gd[1], gd[2]);
  const double s = c * (bb[2] + 5 * tb);
  gd[1] += s * (2 * 3169 * d[1] - 13036 * d[2] + 5978 * d[3]);
  gd[2] += s * (-13036 * d[1] + 2 * 17236 * d[2] + 30414 * v3);
  gd[3] += s * (5978 * d[1] + 17116 * v2);
  g3 += s * 30414 * d[2];
  g2 += s * 17116 * d[3];
  return f;
}

// One characteristic field of a face: values v of the 2 NG points; returns the two sides' interpolated
// values and, for their adjoints fm, fp, adds the points' adjoints to gv.
template <int NG>
__device__ __forceinline__ void weno_char_bwd(const double *v, double fm, double fp, double &vm, double &vp, double *gv) {
  if constexpr (NG == 3) {
    const double dm[3] = {1.0 / 16, 5.0 / 8, 5.0 / 16}, dp[3] = {5.0 / 16, 5.0 / 8, 1.0 / 16};
    const double q0 = 0.125 * (3 * v[0] - 10 * v[1] + 15 * v[2]), q1 = 0.125 * (-v[1] + 6 * v[2] + 3 * v[3]);
    const double q2 = 0.125 * (3 * v[2] + 6 * v[3] - v[4]), q3 = 0.125 * (15 * v[3] - 10 * v[4] + 3 * v[5]);
    const double pm[3] = {q0, q1, q2}, pp[3] = {q1, q2, q3};
    double bm[3], bp[3];
    vm = weno5_side_bwd(v, dm, pm, fm, bm, gv);
    vp = weno5_side_bwd(v + 1, dp, pp, fp, bp, gv + 1);
    const double b0 = 0.125 * bm[0], b1 = 0.125 * (bm[1] + bp[0]), b2 = 0.125 * (bm[2] + bp[1]), b3 = 0.125 * bp[2];
    gv[0] += 3 * b0;
    gv[1] += -10 * b0 - b1;
    gv[2] += 15 * b0 + 6 * b1 + 3 * b2;
    gv[3] += 3 * b1 + 6 * b2 + 15 * b3;
    gv[4] += -b2 - 10 * b3;
    gv[5] += 3 * b3;
  } else {
    const double dm[4] = {7.0 / 64, 35.0 / 64, 21.0 / 64, 1.0 / 64}, dp[4] = {1.0 / 64, 21.0 / 64, 35.0 / 64, 7.0 / 64};
    double d[7], gd[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) {
      d[i] = v[i + 1] - v[i];
      gd[i] = 0;
    }
    // candidates as distances from v[3] (weno7)
    const double o16 = 0.0625;
    const double qa = o16 * (19 * d[2] - 16 * d[1] + 5 * d[0]), qb = o16 * (5 * d[3] + 4 * d[2] - d[1]);
    const double qc = o16 * (d[2] + 8 * d[3] - d[4]), qd = o16 * (11 * d[3] - 4 * d[4] + d[5]);
    const double qe = d[3] - o16 * (19 * d[4] - 16 * d[5] + 5 * d[6]);
    const double pm[4] = {qd, qc, qb, qa}, pp[4] = {qe, qd, qc, qb};
    double bm[4], bp[4];
    vm = v[3] + weno7_side_bwd(d, v[2], v[3], dm, pm, fm, bm, gd, gv[2], gv[3]);
    vp = v[3] + weno7_side_bwd(d + 1, v[3], v[4], dp, pp, fp, bp, gd + 1, gv[3], gv[4]);
    gv[3] += fm + fp;
    const double a = o16 * bm[3], b = o16 * (bm[2] + bp[3]), c = o16 * (bm[1] + bp[2]), e = o16 * (bm[0] + bp[1]),
                 h = o16 * bp[0];
    gd[0] += 5 * a;
    gd[1] += -16 * a - b;
    gd[2] += 19 * a + 4 * b + c;
    gd[3] += 5 * b + 8 * c + 11 * e + bp[0];
    gd[4] += -c - 4 * e - 19 * h;
    gd[5] += e + 16 * h;
    gd[6] -= 5 * h;
    gv[0] -= gd[0];
#pragma unroll
    for (int i = 1; i < 7; ++i) gv[i] += gd[i - 1] - gd[i];
    gv[7] += gd[6];
  }
}

// The Roe-averaged state of a face and the adjoints it collects (aweno_interp).
struct AirRoe {
  double k[3], u[3], h;
  double alpha, cm, icm, icm2, Uk;
  double ub[3], hb, alphab, cmb, icmb, icm2b, Ukb;
};

// Row l of L and column l of R of the face's eigenvectors (aweno_interp).
__device__ __forceinline__ void air_eigen(const AirRoe &f, int l, double *L, double *R) {
  const double g1 = kGamma - 1;
  if (l == 0 || l == 4) {
    const double s = l == 0 ? 1.0 : -1.0, c = s * f.cm, h2 = 0.5 * f.icm2;
    L[0] = (f.alpha + f.Uk * c) * h2;
    R[0] = 1.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      L[1 + d] = -(g1 * f.u[d] + f.k[d] * c) * h2;
      R[1 + d] = f.u[d] - f.k[d] * c;
    }
    L[4] = g1 * h2;
    R[4] = f.h - f.Uk * c;
  } else {
    const int e = l - 1, e1 = l % 3, e2 = (l + 1) % 3;
    const double ke = e == 0 ? f.k[0] : e == 1 ? f.k[1] : f.k[2];
    const double k1 = e1 == 0 ? f.k[0] : e1 == 1 ? f.k[1] : f.k[2], k2 = e2 == 0 ? f.k[0] : e2 == 1 ? f.k[1] : f.k[2];
    const double u1 = e1 == 0 ? f.u[0] : e1 == 1 ? f.u[1] : f.u[2], u2 = e2 == 0 ? f.u[0] : e2 == 1 ? f.u[1] : f.u[2];
    const double X = k2 * u1 - k1 * u2;
    L[0] = ke * (1 - f.alpha * f.icm2) - X * f.icm;
    R[0] = ke;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double rot = d == e1 ? k2 : d == e2 ? -k1 : 0.0;
      L[1 + d] = (ke * g1 * f.u[d] + rot * f.cm) * f.icm2;
      R[1 + d] = ke * f.u[d] + rot * f.cm;
    }
    L[4] = -ke * g1 * f.icm2;
    R[4] = ke * f.alpha / g1 + X * f.cm;
  }
}

// Adjoints a of row l of L and r of column l of R onto the Roe-averaged state.
__device__ __forceinline__ void air_eigen_bwd(AirRoe &f, int l, const double *a, const double *r) {
  const double g1 = kGamma - 1;
  if (l == 0 || l == 4) {
    const double s = l == 0 ? 1.0 : -1.0, c = s * f.cm, h2 = 0.5 * f.icm2;
    double h2b = a[0] * (f.alpha + f.Uk * c) + a[4] * g1, cb = a[0] * f.Uk * h2 - r[4] * f.Uk;
    f.alphab += a[0] * h2;
    f.Ukb += a[0] * c * h2 - r[4] * c;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      h2b -= a[1 + d] * (g1 * f.u[d] + f.k[d] * c);
      cb -= (a[1 + d] * h2 + r[1 + d]) * f.k[d];
      f.ub[d] += r[1 + d] - a[1 + d] * g1 * h2;
    }
    f.hb += r[4];
    f.cmb += s * cb;
    f.icm2b += 0.5 * h2b;
  } else {
    const int e = l - 1, e1 = l % 3, e2 = (l + 1) % 3;
    const double ke = e == 0 ? f.k[0] : e == 1 ? f.k[1] : f.k[2];
    const double k1 = e1 == 0 ? f.k[0] : e1 == 1 ? f.k[1] : f.k[2], k2 = e2 == 0 ? f.k[0] : e2 == 1 ? f.k[1] : f.k[2];
    const double u1 = e1 == 0 ? f.u[0] : e1 == 1 ? f.u[1] : f.u[2], u2 = e2 == 0 ? f.u[0] : e2 == 1 ? f.u[1] : f.u[2];
    const double X = k2 * u1 - k1 * u2;
    f.alphab += -a[0] * ke * f.icm2 + r[4] * ke / g1;
    f.icm2b -= a[0] * ke * f.alpha + a[4] * ke * g1;
    f.icmb -= a[0] * X;
    f.cmb += r[4] * X;
    const double Xb = r[4] * f.cm - a[0] * f.icm;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double rot = d == e1 ? k2 : d == e2 ? -k1 : 0.0;
      f.icm2b += a[1 + d] * (ke * g1 * f.u[d] + rot * f.cm);
      f.cmb += (a[1 + d] * f.icm2 + r[1 + d]) * rot;
      f.ub[d] += (a[1 + d] * g1 * f.icm2 + r[1 + d]) * ke + (d == e1 ? Xb * k2 : d == e2 ? -Xb * k1 : 0.0);
    }
  }
}

// 1. Face fluxes of direction DIR (faces c + 1/2, c = -1 .. n - 1): every face thread turns its face
// adjoint into cv adjoints of its 2 NG stencil nodes.  The forward sweep subtracts F(c + 1/2) from
// dq of node c and adds it to node c + 1.
// Two passes over the five characteristic fields: the first interpolates (the Riemann solver's sides),
// the second reverses each field and accumulates the stencil's adjoints in the thread's column of shared
// memory; the stencil is read again for each field (from L1: consecutive threads share its lines).  Both
// keep the registers for the field at hand.  One pass of 2 NG x 5 forward-mode evaluations of the whole face flux, which this replaces, took
// 9.2 ms a direction at 128 x 65 x 48 (WENO7 + HLLC); the whole VJP went from 30.4 to 1.33 ms.
template <int DIR, int NG, int RS>
__global__ void __launch_bounds__(128, 2) k_adj_air_face(DevBlock b, DevState s, const double *__restrict__ dqb,
                                                         double *__restrict__ acv) {
  __shared__ double sqb[2 * NG * 5][128];  // every thread's stencil adjoints
  const long long P = b.plane;
  const int nd = DIR == 0 ? b.mx : DIR == 1 ? b.my : b.mz;
  const long long other = DIR == 0 ? (long long)b.my * b.mz : DIR == 1 ? (long long)b.mx * b.mz : (long long)b.mx * b.my;
  const long long nf = (long long)(nd + 1) * other;
  const long long st = DIR == 0 ? 1 : DIR == 1 ? (long long)b.pitch : (long long)b.pitch * b.sy;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nf; t += (long long)gridDim.x * blockDim.x) {
    int c, o1, o2;
    sweep_pos<DIR>(b, t, nd + 1, -1, c, o1, o2);
    double fb[5];
    bool any = false;
#pragma unroll
    for (int l = 0; l < 5; ++l) {
      double a = 0.0;
      if (c >= 0) a -= dqb[l * b.n + sweep_iq<DIR>(b, c, o1, o2)];
      if (c + 1 < nd) a += dqb[l * b.n + sweep_iq<DIR>(b, c + 1, o1, o2)];
      fb[l] = a;
      any = any || a != 0.0;
    }
    if (!any) continue;
    const long long p0 = sweep_id<DIR>(b, c, o1, o2);  // left node of the face
    auto q = [&](int sn, int v) -> double { return s.cv[v * P + b.chk(p0 + (sn - NG + 1) * st)]; };
    const long long p1 = b.chk(p0 + st);
    AirRoe f;
    const double g1 = kGamma - 1;
    double ql[5] = {0, 0, 0, 0, 0}, qr[5] = {0, 0, 0, 0, 0};  // the sides' states, then their adjoints
    {
      const double rl0 = q(NG - 1, 0), rr0 = q(NG, 0), il = 1.0 / rl0, ir = 1.0 / rr0;
      const double sl = sqrt(rl0), sr = sqrt(rr0), isum = 1.0 / (sl + sr), rl = sl * isum, rr = sr * isum;
      double ek = 0, k2 = 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        f.u[d] = rl * q(NG - 1, 1 + d) * il + rr * q(NG, 1 + d) * ir;
        ek += 0.5 * f.u[d] * f.u[d];
        f.k[d] = 0.5 * (b.met[(DIR * 3 + d) * P + p0] + b.met[(DIR * 3 + d) * P + p1]);
        k2 += f.k[d] * f.k[d];
      }
      const double ik = 1.0 / sqrt(k2);
      f.h = rl * (q(NG - 1, 4) + s.bv[4 * P + p0]) * il + rr * (q(NG, 4) + s.bv[4 * P + p1]) * ir;
      f.alpha = g1 * ek;
      f.icm2 = 1.0 / (g1 * (f.h - ek));
      f.icm = sqrt(f.icm2);
      f.cm = 1.0 / f.icm;
      f.Uk = 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        f.k[d] *= ik;
        f.Uk += f.k[d] * f.u[d];
        f.ub[d] = 0;
      }
      f.hb = f.alphab = f.cmb = f.icmb = f.icm2b = f.Ukb = 0;
    }
#pragma unroll 1
    for (int l = 0; l < 5; ++l) {
      asm volatile("" ::: "memory");  // keeps the stencil out of the registers between the fields
      double L[5], R[5], vm, vp;
      air_eigen(f, l, L, R);
      auto qq = [&](int sn, int v) -> double { return q(sn, v); };
      weno_char<NG, double>(L, qq, vm, vp);
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        ql[m] += R[m] * vm;
        qr[m] += R[m] * vp;
      }
    }
    // Riemann solver and primitive states of the two sides
    {
      double pl[6], pr[6], al[6] = {0, 0, 0, 0, 0, 0}, ar[6] = {0, 0, 0, 0, 0, 0};
      const double iql = 1.0 / ql[0], iqr = 1.0 / qr[0];
      pl[0] = ql[0];
      pr[0] = qr[0];
      double el = 0, er = 0;
#pragma unroll
      for (int d = 1; d < 4; ++d) {
        pl[d] = ql[d] * iql;
        pr[d] = qr[d] * iqr;
        el += 0.5 * pl[d] * pl[d];
        er += 0.5 * pr[d] * pr[d];
      }
      pl[4] = g1 * (ql[4] - el * ql[0]);
      pr[4] = g1 * (qr[4] - er * qr[0]);
      pl[5] = ql[4];
      pr[5] = qr[4];
      const double j0 = b.jac[p0], j1 = b.jac[p1];
      double mt0[3], mt1[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        mt0[d] = b.met[(DIR * 3 + d) * P + p0];
        mt1[d] = b.met[(DIR * 3 + d) * P + p1];
      }
      if constexpr (RS == 4) hllc_bwd(pl, pr, mt0, mt1, j0, j1, fb, al, ar);
      else if constexpr (RS == 1) lax_friedrichs_bwd(pl, pr, mt0, mt1, j0, j1, fb, al, ar);
      else ausm_bwd(pl, pr, mt0, mt1, j0, j1, fb, al, ar);
      double bl = al[0] - g1 * el * al[4], br = ar[0] - g1 * er * ar[4];
#pragma unroll
      for (int d = 1; d < 4; ++d) {
        const double vl = al[d] - g1 * ql[0] * pl[d] * al[4], vr = ar[d] - g1 * qr[0] * pr[d] * ar[4];
        bl -= vl * pl[d] * iql;
        br -= vr * pr[d] * iqr;
        ql[d] = vl * iql;
        qr[d] = vr * iqr;
      }
      ql[0] = bl;
      qr[0] = br;
      ql[4] = al[5] + g1 * al[4];
      qr[4] = ar[5] + g1 * ar[4];
    }
    auto qb = [&](int sn, int v) -> double & { return sqb[sn * 5 + v][threadIdx.x]; };
#pragma unroll
    for (int sn = 0; sn < 2 * NG; ++sn)
#pragma unroll
      for (int v = 0; v < 5; ++v) qb(sn, v) = 0;
#pragma unroll 1
    for (int l = 0; l < 5; ++l) {
      asm volatile("" ::: "memory");
      double L[5], R[5], v[2 * NG], gv[2 * NG], vm, vp, fm = 0, fp = 0;
      air_eigen(f, l, L, R);
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        fm += R[m] * ql[m];
        fp += R[m] * qr[m];
      }
#pragma unroll
      for (int sn = 0; sn < 2 * NG; ++sn) {
        double a = 0;
#pragma unroll
        for (int m = 0; m < 5; ++m) a += L[m] * q(sn, m);
        v[sn] = a;
        gv[sn] = 0;
      }
      weno_char_bwd<NG>(v, fm, fp, vm, vp, gv);
      double Lb[5] = {0, 0, 0, 0, 0}, Rb[5];
#pragma unroll
      for (int sn = 0; sn < 2 * NG; ++sn)
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          qb(sn, m) += L[m] * gv[sn];
          Lb[m] += gv[sn] * q(sn, m);
        }
#pragma unroll
      for (int m = 0; m < 5; ++m) Rb[m] = vm * ql[m] + vp * qr[m];
      air_eigen_bwd(f, l, Lb, Rb);
    }
    // Roe averages: cm2 = (gamma - 1)(h - ek), alpha = (gamma - 1) ek, Uk = k . u
    {
      const double cm2b = -f.icm2b * f.icm2 * f.icm2 + 0.5 * f.icm * (f.cmb - f.icmb * f.icm2);
      const double hb = f.hb + g1 * cm2b, ekb = g1 * (f.alphab - cm2b);
      const double rl0 = q(NG - 1, 0), rr0 = q(NG, 0);
      const double sl = sqrt(rl0), sr = sqrt(rr0), isum = 1.0 / (sl + sr);
      double wb[2], a0[2];
#pragma unroll
      for (int sd = 0; sd < 2; ++sd) {
        const int sn = NG - 1 + sd;
        const double ir = 1.0 / (sd ? rr0 : rl0), w = (sd ? sr : sl) * isum * ir;
        const double h = (q(sn, 4) + s.bv[4 * P + (sd ? p1 : p0)]) * ir, a = hb * w;  // a: adjoint of rhoE + p
        double e2 = 0, b0 = -a * h;
        wb[sd] = hb * h;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const double u = q(sn, 1 + d) * ir, ub = f.ub[d] + f.Ukb * f.k[d] + ekb * f.u[d];
          wb[sd] += ub * u;
          b0 -= ub * w * u;
          e2 += 0.5 * u * u;
          // p = (gamma - 1)(rhoE - |m|^2 / (2 rho)) of the node
          qb(sn, 1 + d) += ub * w - a * g1 * u;
        }
        a0[sd] = b0 + a * g1 * e2;
        qb(sn, 4) += a * kGamma;
      }
      roe_weight_bwd(sl, sr, isum, wb[0], wb[1], a0[0], a0[1]);
      qb(NG - 1, 0) += a0[0];
      qb(NG, 0) += a0[1];
    }
#pragma unroll
    for (int sn = 0; sn < 2 * NG; ++sn) {
      const long long p = b.chk(p0 + (sn - NG + 1) * st);
#pragma unroll
      for (int v = 0; v < 5; ++v) atomicAdd(acv + v * P + p, qb(sn, v));
    }
  }
}

// 2. Central correction of direction DIR: node n (sweep positions -NG .. n + NG - 1) collects the
// adjoint of its physical flux from every node c = n -+ m whose correction reads it (c interior and
// c < n - 2 NG, as the forward sweep applies it), then maps it to its cv.  One thread per node.
template <int DIR, int NG>
__global__ void __launch_bounds__(128) k_adj_air_cds(DevBlock b, DevState s, const double *__restrict__ dqb,
                                                     double *__restrict__ acv) {
  const long long P = b.plane;
  const int nd = DIR == 0 ? b.mx : DIR == 1 ? b.my : b.mz;
  const long long other = DIR == 0 ? (long long)b.my * b.mz : DIR == 1 ? (long long)b.mx * b.mz : (long long)b.mx * b.my;
  const int span = nd + 2 * NG;
  const long long nn = (long long)span * other;
  // coefficients of f(c + m) - f(c - m), m = 1 .. NG (cds_correction)
  double cm[5];
  if (NG == 3) {
    cm[1] = -17.0 / 256; cm[2] = 13.0 / 320; cm[3] = -19.0 / 3840;
  } else {
    cm[1] = 421.0 / 5120; cm[2] = -289.0 / 5120; cm[3] = 1261.0 / 107520; cm[4] = -81.0 / 71680;
  }
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nn; t += (long long)gridDim.x * blockDim.x) {
    int n, o1, o2;
    sweep_pos<DIR>(b, t, span, -NG, n, o1, o2);
    double fb[5] = {0, 0, 0, 0, 0};
    bool any = false;
#pragma unroll
    for (int m = 1; m <= NG; ++m) {
      const int cu = n - m, cd = n + m;  // node n is f(cu + m) for cu, f(cd - m) for cd
      const bool use_u = cu >= 0 && cu < nd && cu < nd - 2 * NG;
      const bool use_d = cd >= 0 && cd < nd && cd < nd - 2 * NG;
#pragma unroll
      for (int l = 0; l < 5; ++l) {
        if (use_u) fb[l] += cm[m] * dqb[l * b.n + sweep_iq<DIR>(b, cu, o1, o2)];
        if (use_d) fb[l] -= cm[m] * dqb[l * b.n + sweep_iq<DIR>(b, cd, o1, o2)];
      }
      any = any || use_u || use_d;
    }
    if (!any) continue;
    const long long p = sweep_id<DIR>(b, n, o1, o2);
    double cv[5];
#pragma unroll
    for (int l = 0; l < 5; ++l) cv[l] = s.cv[l * P + p];
    double dp[5];
    air_dp_dcv(cv, dp);
    const double pn = s.bv[4 * P + p];
    const Dual k[3] = {Dual(b.met[(DIR * 3 + 0) * P + p]), Dual(b.met[(DIR * 3 + 1) * P + p]),
                       Dual(b.met[(DIR * 3 + 2) * P + p])};
    const Dual jac(b.jac[p]);
#pragma unroll 1
    for (int v = 0; v < 5; ++v) {
      Dual q[5];
#pragma unroll
      for (int l = 0; l < 5; ++l) q[l] = Dual(cv[l], l == v ? 1.0 : 0.0);
      const Dual ir = 1.0 / q[0];
      const Dual bb[5] = {q[0], q[1] * ir, q[2] * ir, q[3] * ir, Dual(pn, dp[v])};
      Dual f[5];
      node_flux<Dual>(bb, q[4], k, jac, f);
      double g = 0.0;
#pragma unroll
      for (int l = 0; l < 5; ++l) g += fb[l] * f[l].d;
      acv[v * P + p] += g;  // one thread per node in this launch
    }
  }
}

// 3. Viscous faces of direction DIR (faces c + 1/2, c = -1 .. n - 1; the forward adds F_v(c + 1/2) to
// dq of node c and subtracts it from node c + 1, components 1..4).  The reverse of viscous_face: stress,
// conduction and viscosity adjoints onto the face's gradients, means and viscosity, then onto the
// planes ap of u, v, w, T of the nodes {0, e_d} x {0, +-e_c} (c != d; c = 2 only in 3-D) they are formed
// from; mu's goes to T through Sutherland's law.  (Fifty forward-mode evaluations of the face, which this
// replaces, took 0.86 ms a direction at 128 x 65 x 48.)
template <int DIR, bool DIM3>
__global__ void __launch_bounds__(128) k_adj_air_visc(DevBlock b, DevState s, const double *__restrict__ dqb,
                                                      double prandtl, double *__restrict__ ap) {
  const long long P = b.plane;
  const int nd = DIR == 0 ? b.mx : DIR == 1 ? b.my : b.mz;
  const long long other = DIR == 0 ? (long long)b.my * b.mz : DIR == 1 ? (long long)b.mx * b.mz : (long long)b.mx * b.my;
  const long long nf = (long long)(nd + 1) * other;
  const long long st3[3] = {1, b.pitch, (long long)b.pitch * b.sy};
  const double *const pl[4] = {s.bv + P, s.bv + 2 * P, s.bv + 3 * P, s.bv + 5 * P};  // u, v, w, T
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nf; t += (long long)gridDim.x * blockDim.x) {
    int c, o1, o2;
    sweep_pos<DIR>(b, t, nd + 1, -1, c, o1, o2);
    double fb[4];
    bool any = false;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      double a = 0.0;
      if (c >= 0) a += dqb[(l + 1) * b.n + sweep_iq<DIR>(b, c, o1, o2)];
      if (c + 1 < nd) a -= dqb[(l + 1) * b.n + sweep_iq<DIR>(b, c + 1, o1, o2)];
      fb[l] = a;
      any = any || a != 0.0;
    }
    if (!any) continue;
    const long long p0 = sweep_id<DIR>(b, c, o1, o2), p1 = b.chk(p0 + st3[DIR]);
    // forward: mean metric, gradients, viscosity, face normal
    double m[9], g[4][3], um[3];
#pragma unroll
    for (int r = 0; r < 9; ++r) m[r] = 0.5 * (b.met[r * P + p0] + b.met[r * P + p1]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double *B = pl[q];
      double e[3];
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) {
        if (cc == DIR) {
          e[cc] = B[p1] - B[p0];
        } else if (cc == 2 && !DIM3) {
          e[cc] = 0;
        } else {
          const long long a = st3[cc];
          e[cc] = 0.25 * (B[b.chk(p0 + a)] - B[b.chk(p0 - a)] + B[b.chk(p1 + a)] - B[b.chk(p1 - a)]);
        }
      }
#pragma unroll
      for (int x = 0; x < 3; ++x) g[q][x] = e[0] * m[x] + e[1] * m[3 + x] + e[2] * m[6 + x];
      if (q < 3) um[q] = 0.5 * (B[p0] + B[p1]);
    }
    const double mu0 = s.mul[p0], mu1 = s.mul[p1], mu = 0.5 * (mu0 + mu1);
    const double j0 = b.jac[p0], j1 = b.jac[p1];
    double n[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) n[x] = 0.5 * (b.met[(DIR * 3 + x) * P + p0] * j0 + b.met[(DIR * 3 + x) * P + p1] * j1);
    // strain S (stress tau = mu S) and the flux F = tau n
    const double S[6] = {(4 * g[0][0] - 2 * g[1][1] - 2 * g[2][2]) / 3, (4 * g[1][1] - 2 * g[0][0] - 2 * g[2][2]) / 3,
                         (4 * g[2][2] - 2 * g[0][0] - 2 * g[1][1]) / 3, g[0][1] + g[1][0], g[0][2] + g[2][0],
                         g[1][2] + g[2][1]};
    const double Sn[3] = {n[0] * S[0] + n[1] * S[3] + n[2] * S[4], n[0] * S[3] + n[1] * S[1] + n[2] * S[5],
                          n[0] * S[4] + n[1] * S[5] + n[2] * S[2]};
    const double kc = kGamma * kRuD / kMwD / (kGamma - 1) / prandtl;  // conductivity over mu
    const double nT = n[0] * g[3][0] + n[1] * g[3][1] + n[2] * g[3][2];
    // reverse
    double Fb[3], umb[3], mub = fb[3] * kc * nT;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      Fb[x] = fb[x] + fb[3] * um[x];
      umb[x] = 0.5 * fb[3] * mu * Sn[x];
      mub += Fb[x] * Sn[x];
    }
    const double Sxx = mu * n[0] * Fb[0], Syy = mu * n[1] * Fb[1], Szz = mu * n[2] * Fb[2];
    const double Sxy = mu * (n[1] * Fb[0] + n[0] * Fb[1]), Sxz = mu * (n[2] * Fb[0] + n[0] * Fb[2]),
                 Syz = mu * (n[2] * Fb[1] + n[1] * Fb[2]);
    const double tr = (2.0 / 3.0) * (Sxx + Syy + Szz);
    const double gb[4][3] = {{2 * Sxx - tr, Sxy, Sxz}, {Sxy, 2 * Syy - tr, Syz}, {Sxz, Syz, 2 * Szz - tr},
                             {fb[3] * mu * kc * n[0], fb[3] * mu * kc * n[1], fb[3] * mu * kc * n[2]}};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      double *A = ap + q * P;
      double a0 = 0, a1 = 0;
      if (q < 3) {
        a0 = umb[q];
        a1 = umb[q];
      } else {
        const double t0 = s.bv[5 * P + p0], t1 = s.bv[5 * P + p1];
        a0 = 0.5 * mub * mu0 * (1.5 / t0 - 1.0 / (t0 + 110.0));
        a1 = 0.5 * mub * mu1 * (1.5 / t1 - 1.0 / (t1 + 110.0));
      }
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) {
        if (cc == 2 && !DIM3 && DIR != 2) continue;
        const double e = gb[q][0] * m[cc * 3] + gb[q][1] * m[cc * 3 + 1] + gb[q][2] * m[cc * 3 + 2];
        if (cc == DIR) {
          a0 -= e;
          a1 += e;
        } else {
          const long long a = st3[cc];
          const double h = 0.25 * e;
          atomicAdd(A + b.chk(p0 + a), h);
          atomicAdd(A + b.chk(p0 - a), -h);
          atomicAdd(A + b.chk(p1 + a), h);
          atomicAdd(A + b.chk(p1 - a), -h);
        }
      }
      atomicAdd(A + p0, a0);
      atomicAdd(A + p1, a1);
    }
  }
}

// The adjoints ap of u, v, w, T of every node that carries one (ghosts included) onto its cv:
// T = p W / (rho R_u), p = (gamma - 1)(rhoE - |m|^2 / (2 rho)).
__global__ void __launch_bounds__(128) k_adj_air_prim(DevBlock b, DevState s, const double *__restrict__ ap,
                                                      double *__restrict__ acv) {
  const long long P = b.plane;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    const double a[4] = {ap[p], ap[P + p], ap[2 * P + p], ap[3 * P + p]};
    if (a[0] == 0 && a[1] == 0 && a[2] == 0 && a[3] == 0) continue;
    double cv[5], dp[5];
#pragma unroll
    for (int l = 0; l < 5; ++l) cv[l] = s.cv[l * P + p];
    air_dp_dcv(cv, dp);
    const double ir = 1.0 / cv[0], tp = a[3] * ir * (kMwD / kRuD);
    acv[p] += tp * (dp[0] - s.bv[4 * P + p] * ir) - (a[0] * cv[1] + a[1] * cv[2] + a[2] * cv[3]) * ir * ir;
#pragma unroll
    for (int d = 0; d < 3; ++d) acv[(1 + d) * P + p] += a[d] * ir + tp * dp[1 + d];
    acv[4 * P + p] += tp * dp[4];
  }
}

// 4. Ghost fills in reverse (apply_outflow / apply_periodic, BoundCond.cuh:205-233, 1443-1486) on the
// cv adjoint planes: each ghost's adjoint moves to the node it was copied from.
__global__ void __launch_bounds__(128) k_adj_air_bc_face(DevBlock b, double *acv, DevFace f) {
  const int t0 = f.face == 0 ? 1 : 0;
  const int t1 = f.face == 2 ? 1 : 2;
  const int n0 = f.re[t0] - f.rs[t0] + 1, n1 = f.re[t1] - f.rs[t1] + 1;
  const long long nn = (long long)n0 * n1;
  const long long P = b.plane;
  const long long st[3] = {1, b.pitch, (long long)b.pitch * b.sy};
  int dir[3] = {0, 0, 0};
  dir[f.face] = f.direction;
  const long long dstep = dir[0] * st[0] + dir[1] * st[1] + dir[2] * st[2];
  for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < nn; n += (long long)gridDim.x * blockDim.x) {
    int idx[3];
    idx[f.face] = f.rs[f.face];
    idx[t0] = f.rs[t0] + (int)(n % n0);
    idx[t1] = f.rs[t1] + (int)(n / n0);
    const long long pb = b.id(idx[0], idx[1], idx[2]);
    long long po = pb;
    if (f.type == kPeriodic) {
      const int ext[3] = {b.mx, b.my, b.mz};
      int oth[3] = {idx[0], idx[1], idx[2]};
      oth[f.face] = f.direction < 0 ? ext[f.face] - 1 : 0;
      po = b.id(oth[0], oth[1], oth[2]);
    }
    for (int g = b.g; g >= 1; --g) {
      const long long pg = b.chk(pb + g * dstep);
      const long long ps = b.chk(f.type == kPeriodic ? po + g * dstep : pb);
#pragma unroll
      for (int l = 0; l < 5; ++l) {
        acv[l * P + ps] += acv[l * P + pg];
        acv[l * P + pg] = 0.0;
      }
    }
  }
}

}  // namespace ostc
