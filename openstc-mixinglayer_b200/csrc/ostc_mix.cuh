// ostc_mix.cuh -- kernels of the multi-component path (species = 1; included by ostc_b200.cu after
// DevBlock/DevState).  Per RK stage (RK.cuh:112-172): the chemical source initialises dq, the
// flux-split WENO7 sweeps and the viscous sweeps accumulate into it, the update kernel combines the
// stage and solves the temperature, the boundary faces fill the ghosts, and the properties kernel
// recomputes gamma, c, mu, lambda and rho*D over the padded block.
#pragma once

#include "mix_math.cuh"

namespace ostc {

// compute_cv_from_bv_1_point<mixture> (FieldOperation.cuh:78-105, total energy :17-32)
template <int NS>
__device__ __forceinline__ void mix_cv_from_bv_node(const DevBlock &b, const DevState &s, long long p) {
  const long long P = b.plane;
  const int ns = OSTC_NS;
  const double rho = s.bv[p], u = s.bv[P + p], v = s.bv[2 * P + p], w = s.bv[3 * P + p];
  s.cv[p] = rho;
  s.cv[P + p] = rho * u;
  s.cv[2 * P + p] = rho * v;
  s.cv[3 * P + p] = rho * w;
  double h[Spec<NS>::A];
  mix_h_cp<NS, double>(s.bv[5 * P + p], h, nullptr);
  double te = 0.5 * (u * u + v * v + w * w);
  for (int l = 0; l < ns; ++l) {
    const double y = s.sv[l * P + p];
    s.cv[(5 + l) * P + p] = rho * y;
    te += h[l] * y;
  }
  te *= rho;
  te -= s.bv[4 * P + p];
  s.cv[4 * P + p] = te;
}

// update_physical_properties<mixture> over every padded node (FieldOperation.cuh:107-134), with the
// node's state read in FP64 and the properties evaluated in T (FP32 in the mixed precision mode).
// Bound by latency: FP64 uncapped took 255 registers, two blocks an SM; five (spilling) 0.19 ms against 0.31 at
// 192 x 96 x 48 (four 0.19, three 0.25), 60 against 97 us at 97 x 65 x 33.  FP32 four blocks.
template <int NS, typename T>
__global__ void __launch_bounds__(128, sizeof(T) == 8 ? 5 : 4) k_mix_props(DevBlock b, DevState s) {
  const long long P = b.plane;
  const int ns = OSTC_NS;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    const double rho = s.bv[p];
    if (!(rho > 0)) continue;  // padding columns of the row pitch carry no state
    T y[Spec<NS>::A], rd[Spec<NS>::A];
    for (int l = 0; l < ns; ++l) y[l] = (T)s.sv[l * P + p];
    T g, a, mu, cd;
    mix_properties<NS, T>((T)rho, (T)s.bv[4 * P + p], (T)s.bv[5 * P + p], y, g, a, mu, cd, rd);
    s.gam[p] = g;
    s.acs[p] = a;
    s.mul[p] = mu;
    s.cond[p] = cd;
    for (int l = 0; l < ns; ++l) s.rhod[l * P + p] = rd[l];
  }
}

// conservative variables from bv and sv over the padded block (initialisation, RK.cuh:37-45)
template <int NS>
__global__ void k_mix_init_cv(DevBlock b, DevState s) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < b.plane; p += (long long)gridDim.x * blockDim.x)
    if (s.bv[p] > 0) mix_cv_from_bv_node<NS>(b, s, p);
}

// compute_source<FR> (SourceTerm.cuh:11-35) as the first contribution to dq: dq[5+l] = J omega_l
// (finite rate) or 0, dq[0..4] = 0.  LISTED: the reactions' species lists fit the tables and the species
// arrays sit in shared memory (mix_chemistry_listed); else the reactions run over every species from
// registers (mix_chemistry).  192 x 96 x 48, 19 reactions: 0.50 ms a sweep over every species, 0.34 ms listed.
template <int NS, bool LISTED>
__global__ void __launch_bounds__(128, 4) k_mix_source(DevBlock b, DevState s, double *__restrict__ dq, int nv,
                                                     int finite_rate) {
  extern __shared__ double chem_smem[];
  if (NS > 0) nv = 5 + NS;
  const long long P = b.plane;
  const int ns = OSTC_NS;
  const ChemColumn c{chem_smem + threadIdx.x, 128}, g{chem_smem + ns * 128 + threadIdx.x, 128},
      om{chem_smem + 2 * ns * 128 + threadIdx.x, 128};
  for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < b.n; n += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(n % b.mx);
    const long long r = n / b.mx;
    const int j = (int)(r % b.my), k = (int)(r / b.my);
    const long long p = b.id(i, j, k);
    for (int l = 0; l < 5; ++l) dq[l * b.n + n] = 0.0;
    if (finite_rate) {
      double y[Spec<NS>::A];
      for (int l = 0; l < ns; ++l) y[l] = s.sv[l * P + p];
      const double jac = b.jac[p];
      if constexpr (LISTED) {
        mix_chemistry_listed<NS, false>(s.bv[p], s.bv[5 * P + p], y, c, g, om, om);
        for (int l = 0; l < ns; ++l) dq[(5 + l) * b.n + n] = jac * om(l);
      } else {
        double w[Spec<NS>::A];
        mix_chemistry<NS>(s.bv[p], s.bv[5 * P + p], y, w);
        for (int l = 0; l < ns; ++l) dq[(5 + l) * b.n + n] = jac * w[l];
      }
    } else {
      for (int l = 5; l < nv; ++l) dq[l * b.n + n] = 0.0;
    }
  }
}

// Point-implicit chemistry (chem mode 1, an extension of the RK3 path): after the fluxes, add the
// chemical source J omega to dq and replace the species part by the solution of
// (I - dt J_chem) x = dq_species (EPI + solve_chem_system, FiniteRateChem.cu:233-254, 302-357, with the
// stage's global dt), one cell per thread, every cell of the block in one launch.  Block: 64 threads
// (LISTED, whose matrix sits in shared memory) or 128 (in local memory).  97 x 65 x 33: 0.50 ms -> 0.37 ms.
template <int NS, bool LISTED>
__global__ void __launch_bounds__(LISTED ? 64 : 128, 4) k_mix_chem_epi(DevBlock b, DevState s, double *__restrict__ dq,
                                                                      const double *dtp) {
  extern __shared__ double chem_smem[];
  const long long P = b.plane;
  const int ns = OSTC_NS;
  const double dt = *dtp;
  const ChemColumn c{chem_smem + threadIdx.x, 64}, g{chem_smem + ns * 64 + threadIdx.x, 64},
      x{chem_smem + 2 * ns * 64 + threadIdx.x, 64}, a{chem_smem + 3 * ns * 64 + threadIdx.x, 64};
  for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < b.n; n += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(n % b.mx);
    const long long r = n / b.mx;
    const int j = (int)(r % b.my), k = (int)(r / b.my);
    const long long p = b.id(i, j, k);
    double y[Spec<NS>::A];
    for (int l = 0; l < ns; ++l) y[l] = s.sv[l * P + p];
    const double jac = b.jac[p];
    if constexpr (LISTED) {
      mix_chemistry_listed<NS, true>(s.bv[p], s.bv[5 * P + p], y, c, g, x, a);
      for (int l = 0; l < ns; ++l) x(l) = dq[(5 + l) * b.n + n] + jac * x(l);
      for (int m = 0; m < ns; ++m)
        for (int q = 0; q < ns; ++q) a(m * ns + q) = (m == q ? 1.0 : 0.0) - dt * a(m * ns + q);
      mix_lu_solve_columns<NS>(a, x);
      for (int l = 0; l < ns; ++l) dq[(5 + l) * b.n + n] = x(l);
    } else {
      double om[Spec<NS>::A], jc[Spec<NS>::A * Spec<NS>::A], rhs[Spec<NS>::A];
      for (int l = 0; l < ns * ns; ++l) jc[l] = 0.0;
      mix_chemistry<NS>(s.bv[p], s.bv[5 * P + p], y, om, jc);
      for (int l = 0; l < ns; ++l) rhs[l] = dq[(5 + l) * b.n + n] + jac * om[l];
      for (int m = 0; m < ns; ++m)
        for (int q = 0; q < ns; ++q) jc[m * ns + q] = (m == q ? 1.0 : 0.0) - dt * jc[m * ns + q];
      mix_lu_solve<NS>(jc, rhs);
      for (int l = 0; l < ns; ++l) dq[(5 + l) * b.n + n] = rhs[l];
    }
  }
}

// ------------------------------------------------------------------ flux-split WENO7 sweeps

// Tile geometry of the sweeps: TD faces along the sweep direction (TD-1 nodes finalised per tile),
// and for the y / z sweeps TXL consecutive i per tile (coalesced rows).
template <int DIR> struct FvsTile {
  static constexpr int TXL = DIR == 0 ? 1 : 8;
  static constexpr int TD = DIR == 0 ? 128 : 16;
  static constexpr int NST = TD + 7;  // staged nodes: stencils of 8 nodes around TD faces
};

// split fluxes of the staged nodes [2][nv][NST][TXL], then per thread the species' slots [ns][TD][TXL] and
// the mass fractions', later the flow fluxes [max(ns, 5)][TD][TXL]
__host__ __device__ constexpr int fvs_slots(int ns) { return ns + (ns > 5 ? ns : 5); }
template <int DIR, typename T>
__host__ __device__ constexpr size_t fvs_smem_bytes(int nv) {
  return (size_t)(2 * FvsTile<DIR>::NST * nv + FvsTile<DIR>::TD * fvs_slots(nv - 5)) * FvsTile<DIR>::TXL * sizeof(T);
}

// compute_convective_term_weno_x/_y/_z (WENO.cu:8-461) for inviscid_scheme 72 (characteristic,
// compute_weno_flux_ch method 1, WENO.cu:722-758, 899-965, 1119-1142) or 71 (component-wise,
// compute_weno_flux_cp, :1455-1536).  Every node's split fluxes F+- (compute_flux, :697-720) are
// computed once into shared memory; each thread then forms one face flux from the 8-node stencil,
// and after a barrier the node threads difference neighbouring faces into dq.  T is the arithmetic
// type of the fluxes (FP32 in the mixed precision mode: state read in FP64, dq accumulated in FP64).
// Bound by FP64 arithmetic at the occupancy its shared memory and registers leave (40 % of the FP64 pipe;
// DRAM 8 %).  The staged values are laid out variable by variable, so that a warp's threads read
// consecutive words; with the variables of a node side by side (a stride of 14 doubles) every read is a
// two-way bank conflict.  Species arrays (the averaged mass fractions, then the fluxes) live in the thread's own
// slots and the staged values are read again per row, or 2.8 KB a thread would spill (0.3 KB now).  dq takes the
// differences by an atomicAdd whose result nobody reads (a reduction at L2; one thread adds to an entry), so that
// the block ends without waiting for a load of dq (10 % of the sweep).  Three sweeps: 192 x 96 x 48, FP64, 1.43 ms (2.50
// with node-wise staging, arrays in registers and a division per weight), 257 x 129 x 65, FP32, 2.17 ms (3.78).
// Resident blocks per SM: FP64 4 (3: 5 % slower), FP32 6 (8: 2 % slower); tiles of 4 lanes and 32 faces instead of 8
// and 16: 1.52 and 2.29 ms.
// EPS0: the epsilon of the weights is 0 (no reference state; fvs_weno7_core).  A kernel of its own, since a test per
// face value costs every case 1 % of the sweep.
template <int DIR, int NS, typename T, bool EPS0 = false>
__global__ void __launch_bounds__(FvsTile<DIR>::TD * FvsTile<DIR>::TXL, sizeof(T) == 8 ? 4 : 6) k_fvs(DevBlock b, DevState s,
                                                                               double *__restrict__ dq, int nv,
                                                                               int scheme) {
  constexpr int TXL = FvsTile<DIR>::TXL, TD = FvsTile<DIR>::TD, NST = FvsTile<DIR>::NST;
  extern __shared__ __align__(16) unsigned char mix_smem[];
  const int ns = OSTC_NS;
  if (NS > 0) nv = 5 + NS;
  T *Fp = reinterpret_cast<T *>(mix_smem);
  T *Fm = Fp + nv * NST * TXL;
  T *fcs = Fm + nv * NST * TXL;
  const int lane = DIR == 0 ? 0 : (int)threadIdx.x;
  const int t = DIR == 0 ? (int)threadIdx.x : (int)threadIdx.y;
  const long long P = b.plane;
  const int nd = DIR == 0 ? b.mx : DIR == 1 ? b.my : b.mz;
  const int start = (DIR == 0 ? blockIdx.x : blockIdx.y) * (TD - 1);
  int i0, j0, k0;  // coordinates of this lane's line
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
  const T half = T(0.5);
  // stage split fluxes of nodes start-4 .. start+TD+2
  if (lane_ok) {
    for (int st = t; st < NST; st += TD) {
      const int n = start - 4 + st;
      if (n > nd + 3) continue;
      const long long p = pid(n);
      T Q[Spec<NS>::A + 5];
#pragma unroll
      for (int l = 0; l < nv; ++l) Q[l] = (T)s.cv[l * P + p];
      const T pk = (T)s.bv[4 * P + p];
      const T c = (T)(s.acs ? s.acs[p] : sqrt(kGamma * (kRuD / kMwD) * s.bv[5 * P + p]));
      const T k0m = (T)b.met[(DIR * 3 + 0) * P + p], k1m = (T)b.met[(DIR * 3 + 1) * P + p],
              k2m = (T)b.met[(DIR * 3 + 2) * P + p];
      const T jac = (T)b.jac[p];
      const T Uk = (Q[1] * k0m + Q[2] * k1m + Q[3] * k2m) / Q[0];
      const T cg = c * tsqrt(k0m * k0m + k1m * k1m + k2m * k2m);
      const T l0 = tabs(Uk) + cg;
      const T hj = half * jac, up = hj * (Uk + l0), um = hj * (Uk - l0), pj = hj * pk;
      T *fp = Fp + st * TXL + lane, *fm = Fm + st * TXL + lane;
#pragma unroll
      for (int l = 0; l < nv; ++l) {
        const T pl = l == 1 ? pj * k0m : l == 2 ? pj * k1m : l == 3 ? pj * k2m : l == 4 ? pj * Uk : T(0);
        fp[l * NST * TXL] = up * Q[l] + pl;
        fm[l * NST * TXL] = um * Q[l] + pl;
      }
    }
  }
  __syncthreads();
  const int n = start - 1 + t;  // left node of this thread's face
  const bool face_ok = lane_ok && n < nd;
  auto FP = [&](int m, int l) -> T { return Fp[(l * NST + t + m) * TXL + lane]; };
  auto FM = [&](int m, int l) -> T { return Fm[(l * NST + t + m + 1) * TXL + lane]; };  // node m of the - side
  auto SP = [&](int tt, int l) -> T & { return fcs[(l * TD + tt) * TXL + lane]; };         // species l
  auto FL = [&](int tt, int l) -> T & { return fcs[((ns + l) * TD + tt) * TXL + lane]; };  // mass fractions, flow fluxes
  if (face_ok && scheme == 71) {
    const long long pl = pid(n), pr = pid(n + 1);
    const double j1 = b.jac[pl], j2 = b.jac[pr];
    double a[3];
    for (int q = 0; q < 3; ++q) a[q] = b.met[(DIR * 3 + q) * P + pl] * j1 + b.met[(DIR * 3 + q) * P + pr] * j2;
    const double eps_ref = 1e-20 * c_mix.weno_eps_scale * 0.25 * (a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
    const double e1 = eps_ref * c_mix.v_ref * c_mix.v_ref;
    const double e2 = e1 * c_mix.v_ref * c_mix.v_ref;
#pragma unroll 1
    for (int l = 0; l < nv; ++l) {
      const double e = (l >= 1 && l <= 3) ? e1 : (l == 4 ? e2 : eps_ref);
      T vp[7], vm[7];
#pragma unroll
      for (int m = 0; m < 7; ++m) {
        vp[m] = FP(m, l);
        vm[m] = FM(m, l);
      }
      (l < 5 ? FL(t, l) : SP(t, l - 5)) = fvs_weno7<EPS0>(vp, vm, e);
    }
  } else if (face_ok) {
    // Roe-averaged mixture eigensystem at the face (WENO.cu:747-821).  The averaged mass fractions and the
    // species' alpha_l of L wait in this thread's own slots until the fluxes replace them.
    const long long pl = pid(n), pr = pid(n + 1);
    const T rl = (T)s.cv[pl], rr = (T)s.cv[pr];
    const T p_l = (T)s.bv[4 * P + pl], p_r = (T)s.bv[4 * P + pr];
    const T rli = T(1) / rl, rri = T(1) / rr;
    const T sl = tsqrt(rl), sr = tsqrt(rr);
    const T isum = T(1) / (sl + sr);
    const T wl = sl * isum * rli, wr = sr * isum * rri;  // Roe weights over rho
    auto roe = [&](int l) -> T { return wl * (T)s.cv[l * P + pl] + wr * (T)s.cv[l * P + pr]; };
    const T um = roe(1), vm_ = roe(2), wm = roe(3);
    const T ekm = half * (um * um + vm_ * vm_ + wm * wm);
    const T hm = roe(4) + (wl * p_l + wr * p_r);
    T cm, gm1, c2i;
    T sp[7], sm[7];
    {
      T mw_inv = 0;
#pragma unroll 1
      for (int l = 0; l < ns; ++l) {
        const T sv = roe(5 + l);
        mw_inv += sv * (T)c_mix.imw[l];
        FL(t, l) = sv;
      }
      const T tm = (wl * p_l + wr * p_r) / (T(kRuD) * mw_inv);
      T cp = 0, cvt = 0;
#pragma unroll 1
      for (int l = 0; l < ns; ++l) {
        T h, c;
        mix_h_cp_one<T>(l, tm, h, c);
        const T sv = FL(t, l);
        cp += sv * c;
        cvt += sv * (c - (T)c_mix.ru_mw[l]);
        SP(t, l) = h;
      }
      const T gamma = cp / cvt;
      const T c2 = gamma * T(kRuD) * mw_inv * tm;
      cm = tsqrt(c2);
      gm1 = gamma - 1;
      c2i = T(1) / c2;
      // The species columns of the five flow rows of L are cs_l * al[q] (cs = 1/2, -kx, -ky, -kz, 1/2):
      // their products with the split fluxes share one sum per stencil node, formed once for all rows.
#pragma unroll
      for (int m = 0; m < 7; ++m) sp[m] = sm[m] = T(0);
#pragma unroll 1
      for (int l = 0; l < ns; ++l) {
        const T al = (gamma * (T)c_mix.ru_mw[l] * tm - gm1 * SP(t, l)) * c2i;
        SP(t, l) = al;
#pragma unroll
        for (int m = 0; m < 7; ++m) {
          sp[m] += al * FP(m, 5 + l);
          sm[m] += al * FM(m, 5 + l);
        }
      }
    }
    const double jld = b.jac[pl], jrd = b.jac[pr];
    const double kxJd = b.met[(DIR * 3 + 0) * P + pl] * jld + b.met[(DIR * 3 + 0) * P + pr] * jrd;
    const double kyJd = b.met[(DIR * 3 + 1) * P + pl] * jld + b.met[(DIR * 3 + 1) * P + pr] * jrd;
    const double kzJd = b.met[(DIR * 3 + 2) * P + pl] * jld + b.met[(DIR * 3 + 2) * P + pr] * jrd;
    const double k2 = kxJd * kxJd + kyJd * kyJd + kzJd * kzJd;
    const double eps = 1e-40 * c_mix.weno_eps_scale * 0.25 * k2;
    // the unit normal: the Jacobian-weighted mean metric, its length cancels.  In FP64 for either T: the square
    // of a face area leaves the FP32 range below 1e-19 (and above 1e19) square grid units
    const double igk = 1.0 / sqrt(k2);
    const T kx = (T)(kxJd * igk), ky = (T)(kyJd * igk), kz = (T)(kzJd * igk);
    const T Ukb = kx * um + ky * vm_ + kz * wm;
    const T alpha = gm1 * ekm, icm = cm * c2i, h2 = half * c2i;
    const T hc = hm - cm * cm / gm1;
    T fc[5] = {T(0), T(0), T(0), T(0), T(0)};
    // The staged values are read again for every row (the empty asm keeps the compiler from holding them
    // across the rows: their 70 values do not fit the registers).
#pragma unroll
    for (int l = 0; l < 5; ++l) {
      asm volatile("" ::: "memory");
      // row l of L over the flow variables, and column l of R
      T cs = half, L[5], R[5];
      if (l == 0) {
        L[0] = (alpha + Ukb * cm) * h2;
        L[1] = -(gm1 * um + kx * cm) * h2;
        L[2] = -(gm1 * vm_ + ky * cm) * h2;
        L[3] = -(gm1 * wm + kz * cm) * h2;
        L[4] = gm1 * h2;
        R[0] = T(1); R[1] = um - kx * cm; R[2] = vm_ - ky * cm; R[3] = wm - kz * cm; R[4] = hm - Ukb * cm;
      } else if (l == 1) {
        cs = -kx;
        L[0] = kx * (1 - alpha * c2i) - (kz * vm_ - ky * wm) * icm;
        L[1] = kx * gm1 * um * c2i;
        L[2] = (kx * gm1 * vm_ + kz * cm) * c2i;
        L[3] = (kx * gm1 * wm - ky * cm) * c2i;
        L[4] = -kx * gm1 * c2i;
        R[0] = kx; R[1] = kx * um; R[2] = kx * vm_ + kz * cm; R[3] = kx * wm - ky * cm;
        R[4] = kx * hc + (kz * vm_ - ky * wm) * cm;
      } else if (l == 2) {
        cs = -ky;
        L[0] = ky * (1 - alpha * c2i) - (kx * wm - kz * um) * icm;
        L[1] = (ky * gm1 * um - kz * cm) * c2i;
        L[2] = ky * gm1 * vm_ * c2i;
        L[3] = (ky * gm1 * wm + kx * cm) * c2i;
        L[4] = -ky * gm1 * c2i;
        R[0] = ky; R[1] = ky * um - kz * cm; R[2] = ky * vm_; R[3] = ky * wm + kx * cm;
        R[4] = ky * hc + (kx * wm - kz * um) * cm;
      } else if (l == 3) {
        cs = -kz;
        L[0] = kz * (1 - alpha * c2i) - (ky * um - kx * vm_) * icm;
        L[1] = (kz * gm1 * um + ky * cm) * c2i;
        L[2] = (kz * gm1 * vm_ - kx * cm) * c2i;
        L[3] = kz * gm1 * wm * c2i;
        L[4] = -kz * gm1 * c2i;
        R[0] = kz; R[1] = kz * um + ky * cm; R[2] = kz * vm_ - kx * cm; R[3] = kz * wm;
        R[4] = kz * hc + (ky * um - kx * vm_) * cm;
      } else {
        L[0] = (alpha - Ukb * cm) * h2;
        L[1] = -(gm1 * um - kx * cm) * h2;
        L[2] = -(gm1 * vm_ - ky * cm) * h2;
        L[3] = -(gm1 * wm - kz * cm) * h2;
        L[4] = gm1 * h2;
        R[0] = T(1); R[1] = um + kx * cm; R[2] = vm_ + ky * cm; R[3] = wm + kz * cm; R[4] = hm + Ukb * cm;
      }
      T vp[7], vmn[7];
#pragma unroll
      for (int m = 0; m < 7; ++m) {
        vp[m] = cs * sp[m];
        vmn[m] = cs * sm[m];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
          vp[m] += L[q] * FP(m, q);
          vmn[m] += L[q] * FM(m, q);
        }
      }
      const T fch = fvs_weno7<EPS0>(vp, vmn, eps);
#pragma unroll
      for (int q = 0; q < 5; ++q) fc[q] += R[q] * fch;
    }
    // species fields; fc[0] is also the factor of the mass fractions in their fluxes
    T p0[7], m0[7];
#pragma unroll
    for (int m = 0; m < 7; ++m) {
      p0[m] = FP(m, 0);
      m0[m] = FM(m, 0);
    }
    T add = 0;
#pragma unroll 1
    for (int l = 0; l < ns; ++l) {
      const T sv = FL(t, l);
      T vp[7], vmn[7];
#pragma unroll
      for (int m = 0; m < 7; ++m) {
        vp[m] = FP(m, 5 + l) - sv * p0[m];
        vmn[m] = FM(m, 5 + l) - sv * m0[m];
      }
      const T fch = fvs_weno7<EPS0>(vp, vmn, eps);
      add += SP(t, l) * fch;
      SP(t, l) = sv * fc[0] + fch;
    }
    fc[4] -= add * cm * cm / gm1;
#pragma unroll
    for (int l = 0; l < 5; ++l) FL(t, l) = fc[l];
  }
  __syncthreads();
  if (face_ok && t >= 1) {
    const long long q = DIR == 0 ? b.iq(n, j0, k0) : DIR == 1 ? b.iq(i0, n, k0) : b.iq(i0, j0, n);
#pragma unroll
    for (int l = 0; l < nv; ++l)
      atomicAdd(dq + l * b.n + q, (double)(l < 5 ? FL(t - 1, l) - FL(t, l) : SP(t - 1, l - 5) - SP(t, l - 5)));
  }
}

// ------------------------------------------------------------------ viscous sweeps (mixtures)

// compute_fv/gv/hv_2nd_order<mixture, Laminar> (ViscousScheme.cuh:24-318 and its y / z twins) at the
// face between node p0 and its neighbour p0 + e[d]: stress, Fourier conduction with the mixture
// conductivity, mixture-averaged species diffusion with the correction velocity and its enthalpy flux.
// The node differences of each gradient are taken in FP64 (they cancel the leading digits); the
// chain rule and the fluxes run in T.
template <bool DIM3, int NS, typename T>
__device__ __forceinline__ void mix_visc_face(const DevBlock &b, const DevState &s, long long p0, int d, int nv,
                                              T *fv) {
  const long long P = b.plane;
  const long long st[3] = {1, b.pitch, (long long)b.pitch * b.sy};
  const long long p1 = b.chk(p0 + st[d]);
  const T half = T(0.5);
  T m[9];
  for (int r = 0; r < 9; ++r) m[r] = (T)(0.5 * (b.met[r * P + p0] + b.met[r * P + p1]));
  // gradient of plane B at the face: 2-point normal difference, 4-point averages across
  auto diff = [&](const double *B, T *g) {
    for (int c = 0; c < 3; ++c) {
      if (c == d) {
        g[c] = (T)(B[p1] - B[p0]);
      } else if (c == 2 && !DIM3) {
        g[c] = T(0);
      } else {
        const long long a = st[c];
        g[c] = (T)(0.25 * (B[p0 + a] - B[p0 - a] + B[p1 + a] - B[p1 - a]));
      }
    }
  };
  auto grad = [&](const double *B, T *out) {
    T g[3];
    diff(B, g);
    out[0] = g[0] * m[0] + g[1] * m[3] + g[2] * m[6];
    out[1] = g[0] * m[1] + g[1] * m[4] + g[2] * m[7];
    out[2] = g[0] * m[2] + g[1] * m[5] + g[2] * m[8];
  };
  const double j0 = b.jac[p0], j1 = b.jac[p1];
  const T nx = (T)(0.5 * (b.met[(d * 3 + 0) * P + p0] * j0 + b.met[(d * 3 + 0) * P + p1] * j1));
  const T ny = (T)(0.5 * (b.met[(d * 3 + 1) * P + p0] * j0 + b.met[(d * 3 + 1) * P + p1] * j1));
  const T nz = (T)(0.5 * (b.met[(d * 3 + 2) * P + p0] * j0 + b.met[(d * 3 + 2) * P + p1] * j1));
  // T and the mass fractions enter by their derivative along the face normal alone: the weight of each
  // difference is the normal's product with that row of the mean metric.  Where the face normal is
  // orthogonal to the other two rows (every rectilinear grid) the cross differences have weight zero and
  // are not formed: 2 loads a field instead of 10.  192 x 96 x 48, three sweeps: 0.91 -> 0.69 ms (bound by
  // the latency of its loads; 24 % of HBM).
  T wn[3];
  for (int c = 0; c < 3; ++c) wn[c] = nx * m[c * 3] + ny * m[c * 3 + 1] + nz * m[c * 3 + 2];
  const bool cross = wn[(d + 1) % 3] != T(0) || wn[(d + 2) % 3] != T(0);
  auto along = [&](const double *B) -> T { return wn[d] * (T)(B[p1] - B[p0]); };
  auto mixed = [&](const double *B) -> T {
    T g[3];
    diff(B, g);
    return wn[0] * g[0] + wn[1] * g[1] + wn[2] * g[2];
  };
  T gu[3], gv[3], gw[3];
  grad(s.bv + P, gu);
  grad(s.bv + 2 * P, gv);
  grad(s.bv + 3 * P, gw);
  const T mul = (T)(0.5 * (s.mul[p0] + s.mul[p1]));
  const T m3 = mul * T(1.0 / 3.0);
  const T txx = m3 * (4 * gu[0] - 2 * gv[1] - 2 * gw[2]);
  const T tyy = m3 * (4 * gv[1] - 2 * gu[0] - 2 * gw[2]);
  const T tzz = m3 * (4 * gw[2] - 2 * gu[0] - 2 * gv[1]);
  const T txy = mul * (gu[1] + gv[0]);
  const T txz = mul * (gu[2] + gw[0]);
  const T tyz = mul * (gv[2] + gw[1]);
  fv[0] = 0;
  fv[1] = nx * txx + ny * txy + nz * txz;
  fv[2] = nx * txy + ny * tyy + nz * tyz;
  fv[3] = nx * txz + ny * tyz + nz * tzz;
  const T um = (T)(0.5 * (s.bv[P + p0] + s.bv[P + p1]));
  const T vm = (T)(0.5 * (s.bv[2 * P + p0] + s.bv[2 * P + p1]));
  const T wm = (T)(0.5 * (s.bv[3 * P + p0] + s.bv[3 * P + p1]));
  const T cond = (T)(0.5 * (s.cond[p0] + s.cond[p1]));
  fv[4] = um * fv[1] + vm * fv[2] + wm * fv[3] + cond * (cross ? mixed(s.bv + 5 * P) : along(s.bv + 5 * P));
  const int ns = OSTC_NS;
  T dif[Spec<NS>::A], yk[Spec<NS>::A], ddf[Spec<NS>::A];
  T sgw = 0, srdy = 0, corr = 0, mwt = 0;
  // one branch around the whole loop, so that the loads of all species can be in flight together
  auto species = [&](auto normal) {
#pragma unroll
    for (int l = 0; l < ns; ++l) {
      const double *Y = s.sv + (long long)l * P;
      yk[l] = (T)(0.5 * (Y[p0] + Y[p1]));
      dif[l] = (T)(0.5 * (s.rhod[l * P + p0] + s.rhod[l * P + p1]));
      const T gdy = normal(Y);
      ddf[l] = gdy;
      corr += dif[l] * gdy;
      sgw += gdy * (T)c_mix.imw[l];
      mwt += yk[l] * (T)c_mix.imw[l];
      srdy += dif[l] * yk[l];
    }
  };
  if (cross) species(mixed);
  else species(along);
  mwt = T(1) / mwt;
  corr -= mwt * srdy * sgw;
  T h[Spec<NS>::A];
  mix_h_cp<NS, T>((T)(0.5 * (s.bv[5 * P + p0] + s.bv[5 * P + p1])), h, nullptr);
  for (int l = 0; l < ns; ++l) {
    const T flux = dif[l] * (ddf[l] - mwt * yk[l] * sgw) - yk[l] * corr;
    fv[5 + l] = flux;
    fv[4] += h[l] * flux;
  }
}

// viscous_flux_fv/gv/hv (SchemeSelector.cuh:69-154) for mixtures: one thread per face of the tile,
// then dq += fv(i+1/2) - fv(i-1/2) through shared memory; tiles as the flux-split sweeps.
// Bound by the latency of its loads at the registers' occupancy, so the species' loads go out together
// (mix_visc_face) and dq takes the difference by an atomicAdd whose result nobody reads (a reduction at L2; one
// thread an entry), with no load of dq to wait for; the faces are laid out variable by variable, free of bank
// conflicts.  Three sweeps: 192 x 96 x 48, FP64, 0.33 ms (0.69 with a branch per species and a load of dq), 257 x 129 x
// 65, FP32, 0.79 ms (1.63).
template <int DIR, bool DIM3, int NS, typename T>
__global__ void __launch_bounds__(FvsTile<DIR>::TD * FvsTile<DIR>::TXL, sizeof(T) == 8 ? 4 : 5) k_mix_visc(DevBlock b, DevState s,
                                                                                    double *__restrict__ dq, int nv) {
  if (NS > 0) nv = 5 + NS;
  constexpr int TXL = FvsTile<DIR>::TXL, TD = FvsTile<DIR>::TD;
  extern __shared__ __align__(16) unsigned char mix_smem[];
  T *fsm = reinterpret_cast<T *>(mix_smem);
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
  const bool face_ok = i0 < b.mx && n < nd;
  T fv[Spec<NS>::A + 5] = {};
  if (face_ok) {
    const long long p0 = DIR == 0 ? b.id(n, j0, k0) : DIR == 1 ? b.id(i0, n, k0) : b.id(i0, j0, n);
    mix_visc_face<DIM3, NS, T>(b, s, p0, DIR, nv, fv);
  }
  for (int l = 0; l < nv; ++l) fsm[(l * TD + t) * TXL + lane] = fv[l];
  __syncthreads();
  if (face_ok && t >= 1) {
    const long long q = DIR == 0 ? b.iq(n, j0, k0) : DIR == 1 ? b.iq(i0, n, k0) : b.iq(i0, j0, n);
    for (int l = 0; l < nv; ++l)
      atomicAdd(dq + l * b.n + q, (double)(fv[l] - fsm[(l * TD + t - 1) * TXL + lane]));
  }
}

// update_cv_and_bv_rk<mixture> (RK.cuh:230-284) with compute_temperature_and_pressure
// (FieldOperation.cu:3-40): the Newton iteration starts from the stage-input temperature.  With dtl
// (per-node local time steps, interior-indexed) the step of each node is dtl[n] instead of *dtp: the
// steady driver's update_cv_and_bv (FieldOperation.cuh:189-232) with ca = 0, cb = cc = 1 and the state
// updated in place (in = qn = out).
template <int NS>
__global__ void __launch_bounds__(128, 4) k_mix_update(DevBlock b, DevState in, DevState qn, DevState out,
                                                     const double *__restrict__ dq, const double *dtp, double ca,
                                                     double cb, double cc, int nv, unsigned *flags,
                                                     const double *__restrict__ dtl = nullptr) {
  if (NS > 0) nv = 5 + NS;
  const long long P = b.plane;
  const int ns = OSTC_NS;
  const double dt = dtl ? 0.0 : *dtp;
  for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < b.n; n += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(n % b.mx);
    const long long r = n / b.mx;
    const int j = (int)(r % b.my), k = (int)(r / b.my);
    const long long p = b.id(i, j, k);
    const double dtj = (dtl ? dtl[n] : dt) / b.jac[p];
    double c[Spec<NS>::A + 5];
    for (int l = 0; l < nv; ++l) {
      c[l] = ca * qn.cv[l * P + p] + cb * in.cv[l * P + p] + cc * dtj * dq[l * b.n + n];
    }
    if (b.mz == 1) c[3] = 0;
    for (int l = 0; l < nv; ++l) out.cv[l * P + p] = c[l];
    const double rho = c[0];
    const double di = 1.0 / rho;
    const double u = c[1] * di, v = c[2] * di, w = c[3] * di;
    out.bv[p] = rho;
    out.bv[P + p] = u;
    out.bv[2 * P + p] = v;
    out.bv[3 * P + p] = w;
    double y[Spec<NS>::A];
    for (int l = 0; l < ns; ++l) {
      y[l] = c[5 + l] * di;
      out.sv[l * P + p] = y[l];
    }
    const double e = c[4] / rho - 0.5 * (u * u + v * v + w * w);
    double pr;
    const double t = mix_temperature<NS>(rho, e, in.bv[5 * P + p], y, pr);
    out.bv[4 * P + p] = pr;
    out.bv[5 * P + p] = t;
    if (!(rho > 0) || !(pr > 0) || !(t > 0)) atomicOr(flags, (rho != rho || pr != pr || t != t) ? 2u : 1u);
  }
}

}  // namespace ostc
