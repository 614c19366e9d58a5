// bc_faces.cuh -- the boundary faces whose ghosts are copies or characteristic states of the block's own
// nodes: apply_symmetry, apply_outflow, apply_periodic and apply_farfield (BoundCond.cuh:137-233,
// 755-1022, 1443-1486), for air and mixtures.  Walls, inflows and pressure faces are k_bc_face.
// Part of the ostc_b200.cu translation unit (included in order; not a standalone header).
#pragma once

namespace ostc {

// Face kinds k_bc_group runs.
__host__ __device__ inline bool bc_grouped(int type) {
  return type == kSymmetry || type == kOutflow || type == kPeriodic || type == kFarfield;
}

// One node's primitive state in registers (and, mixtures, its mass fractions).
template <bool MIX, int NS> struct BcNode {
  double v[6];
  double y[MIX ? Spec<NS>::A : 1];
};

template <bool MIX, int NS>
__device__ __forceinline__ BcNode<MIX, NS> bc_read(const DevBlock &b, const DevState &s, long long p) {
  BcNode<MIX, NS> q;
  const long long P = b.plane;
#pragma unroll
  for (int l = 0; l < 6; ++l) q.v[l] = s.bv[l * P + p];
  if constexpr (MIX) {
#pragma unroll
    for (int l = 0; l < OSTC_NS; ++l) q.y[l] = s.sv[l * P + p];
  }
  return q;
}

// Primitive state of node p (and its mass fractions), without the conservative variables.
template <bool MIX, int NS>
__device__ __forceinline__ void bc_write_bv(const DevBlock &b, const DevState &s, long long p, const BcNode<MIX, NS> &q) {
  const long long P = b.plane;
#pragma unroll
  for (int l = 0; l < 6; ++l) s.bv[l * P + p] = q.v[l];
  if constexpr (MIX) {
#pragma unroll
    for (int l = 0; l < OSTC_NS; ++l) s.sv[l * P + p] = q.y[l];
  }
}

// What finish_node computes at a node whose state is q, from the registers: the conservative
// variables (mu too for air; mixture ghosts get their properties from the properties sweep).
template <bool MIX, int NS> struct BcCv {
  double c[5], mu;
};
template <bool MIX, int NS>
__device__ __forceinline__ BcCv<MIX, NS> bc_cv(const BcNode<MIX, NS> &q) {
  BcCv<MIX, NS> r;
  const double rho = q.v[0], u = q.v[1], v = q.v[2], w = q.v[3];
  r.c[0] = rho;
  r.c[1] = rho * u;
  r.c[2] = rho * v;
  r.c[3] = rho * w;
  double te = 0.5 * (u * u + v * v + w * w);
  if constexpr (MIX) {
    double h[Spec<NS>::A];
    mix_h_cp<NS, double>(q.v[5], h, nullptr);
#pragma unroll
    for (int l = 0; l < OSTC_NS; ++l) te += h[l] * q.y[l];
    te *= rho;
    te -= q.v[4];
    r.mu = 0;
  } else {
    te *= rho;
    te += q.v[4] / (kGamma - 1);
    r.mu = sutherland(q.v[5]);
  }
  r.c[4] = te;
  return r;
}
template <bool MIX, int NS>
__device__ __forceinline__ void bc_write(const DevBlock &b, const DevState &s, long long p, const BcNode<MIX, NS> &q,
                                         const BcCv<MIX, NS> &r) {
  const long long P = b.plane;
  bc_write_bv<MIX, NS>(b, s, p, q);
#pragma unroll
  for (int l = 0; l < 5; ++l) s.cv[l * P + p] = r.c[l];
  if constexpr (MIX) {
#pragma unroll
    for (int l = 0; l < OSTC_NS; ++l) s.cv[(5 + l) * P + p] = r.c[0] * q.y[l];
  } else {
    s.mul[p] = r.mu;
  }
}
template <bool MIX, int NS>
__device__ __forceinline__ void bc_write(const DevBlock &b, const DevState &s, long long p, const BcNode<MIX, NS> &q) {
  bc_write<MIX, NS>(b, s, p, q, bc_cv<MIX, NS>(q));
}

// apply_farfield (BoundCond.cuh:755-1022) at a face node whose state is q, outward unit normal n: the
// state of the face node and of every ghost.  Supersonic outflow (returns false) leaves the face node
// as it is.  Mixtures: the molecular weight from the node's mass fractions, its gamma gb from the last
// properties sweep, and a face gamma iterated with cp of the face temperature until it changes by less
// than 1e-4; as in the reference, the entropy of the inflow branch is chosen for u_n <= 0 but its
// velocity and composition for u_n < 0.
template <bool MIX, int NS>
__device__ __forceinline__ bool bc_farfield(const DevFace &f, const double *n, double gb, BcNode<MIX, NS> &q) {
  const double ub = q.v[1], vb = q.v[2], wb = q.v[3], pbv = q.v[4], rb = q.v[0];
  const double uf = n[0] * ub + n[1] * vb + n[2] * wb;
  if (!MIX) gb = kGamma;
  const double ab = sqrt(gb * pbv / rb);
  const double mb = uf / ab;
  if (mb <= -1) {
    q.v[0] = f.density; q.v[1] = f.u; q.v[2] = f.v; q.v[3] = f.w; q.v[4] = f.pressure; q.v[5] = f.temperature;
    if constexpr (MIX)
      for (int l = 0; l < OSTC_NS; ++l) q.y[l] = f.y[l];
    return true;
  }
  if (mb >= 1) return false;
  const double rpos = uf + 2 * ab / (gb - 1);
  const double uinf = f.u * n[0] + f.v * n[1] + f.w * n[2];
  const double rneg = uinf - 2 * f.acoustic_speed / (f.gamma - 1);
  const double Un = 0.5 * (rpos + rneg);
  if constexpr (MIX) {
    double mw_inv = 0;
    for (int l = 0; l < OSTC_NS; ++l) mw_inv += q.y[l] / c_mix.mw[l];
    double mw = 1.0 / mw_inv;
    if (mb < 0) {
      q.v[1] = f.u + (Un - uinf) * n[0];
      q.v[2] = f.v + (Un - uinf) * n[1];
      q.v[3] = f.w + (Un - uinf) * n[2];
      for (int l = 0; l < OSTC_NS; ++l) q.y[l] = f.y[l];
      mw = f.mw;
    } else {
      q.v[1] = ub + (Un - uf) * n[0];
      q.v[2] = vb + (Un - uf) * n[1];
      q.v[3] = wb + (Un - uf) * n[2];
    }
    double gamma = kGamma, err = 1, rho = 0, pr = 0, t = 0;
    // the reference's loop has no bound; 100 iterations (far more than the few it takes) end it here
    for (int it = 0; err > 1e-4 && it < 100; ++it) {
      const double glast = gamma;
      const double cb = 0.25 * (gamma - 1) * (rpos - rneg);
      const double sb = mb <= 0 ? f.entropy : pbv / pow(rb, gamma);
      rho = pow(cb * cb / (gamma * sb), 1 / (gamma - 1));
      pr = rho * cb * cb / gamma;
      t = pr * mw / (rho * kRuD);
      double cp[Spec<NS>::A];
      mix_h_cp<NS>(t, (double *)nullptr, cp);
      double cpt = 0;
      for (int l = 0; l < OSTC_NS; ++l) cpt += cp[l] * q.y[l];
      gamma = cpt / (cpt - kRuD / mw);
      err = fabs(1 - gamma / glast);
    }
    q.v[0] = rho;
    q.v[4] = pr;
    q.v[5] = t;
  } else {
    const double cb = 0.25 * (kGamma - 1) * (rpos - rneg);
    double sb;
    if (mb <= 0) {
      sb = f.entropy;
      q.v[1] = f.u + (Un - uinf) * n[0];
      q.v[2] = f.v + (Un - uinf) * n[1];
      q.v[3] = f.w + (Un - uinf) * n[2];
    } else {
      sb = pbv / pow(rb, kGamma);
      q.v[1] = ub + (Un - uf) * n[0];
      q.v[2] = vb + (Un - uf) * n[1];
      q.v[3] = wb + (Un - uf) * n[2];
    }
    q.v[0] = pow(cb * cb / (kGamma * sb), 1 / (kGamma - 1));
    q.v[4] = q.v[0] * cb * cb / kGamma;
    q.v[5] = q.v[4] * kMwD / (q.v[0] * kRuD);
  }
  return true;
}

// A group of boundary faces in one launch: blockIdx.y is the face (consecutive in the block's face
// order and independent of one another, see launch_bcs), blockIdx.z the ghost layer, threads cover the
// two tangential index ranges, which include ngg ghost layers on each side (Mesh.cpp:14-32).
// Bound by latency (a face has 10^2 - 10^5 nodes): each thread makes one ghost, its loads before its
// stores and its conservative variables from registers.  One thread per face node that walked the ngg
// layers, re-reading each node it had stored, took 12-20 us a launch (257 x 129 to 192 x 96 x 48), a
// third to a half of a step on the small grids; the 257 x 129 step went from 0.237 to 0.123 ms, the
// 128 x 64 x 32 one from 1.08 to 0.84 ms.
// Far-field faces write the node they read, so there layer 0's threads do the whole column.
template <bool MIX, int NS>
__global__ void __launch_bounds__(128) k_bc_group(DevBlock b, DevState s, const DevFace *__restrict__ faces,
                                                  const double *gam_prev) {
  const DevFace &f = faces[blockIdx.y];
  const int face = f.face, type = f.type;
  const int layer = blockIdx.z;
  if (type == kFarfield && layer > 0) return;
  const int t0 = face == 0 ? 1 : 0, t1 = face == 2 ? 1 : 2;
  const int n0 = f.re[t0] - f.rs[t0] + 1, n1 = f.re[t1] - f.rs[t1] + 1;
  const int nn = n0 * n1;
  const long long P = b.plane;
  const long long st[3] = {1, b.pitch, (long long)b.pitch * b.sy};
  const long long dstep = f.direction * st[face];
  const int g = layer + 1;
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nn; n += gridDim.x * blockDim.x) {
    int idx[3];
    idx[face] = f.rs[face];
    idx[t0] = f.rs[t0] + n % n0;
    idx[t1] = f.rs[t1] + n / n0;
    const long long pb = b.id(idx[0], idx[1], idx[2]);
    if (type == kFarfield || type == kSymmetry) {
      double k[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) k[q] = b.met[(face * 3 + q) * P + pb];
      const double km = sqrt(k[0] * k[0] + k[1] * k[1] + k[2] * k[2]);
      if (type == kFarfield) {
        const double gni = f.direction / km;
#pragma unroll
        for (int q = 0; q < 3; ++q) k[q] *= gni;
        BcNode<MIX, NS> q = bc_read<MIX, NS>(b, s, pb);
        const bool face_too = bc_farfield<MIX, NS>(f, k, MIX ? gam_prev[pb] : kGamma, q);
        const BcCv<MIX, NS> r = bc_cv<MIX, NS>(q);
        for (int gg = face_too ? 0 : 1; gg <= b.g; ++gg) bc_write<MIX, NS>(b, s, b.chk(pb + gg * dstep), q, r);
        continue;
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) k[q] /= km;
      if (layer == 0) {
        // the face node: the first interior node's state with its tangential velocity (bv, not cv)
        BcNode<MIX, NS> q = bc_read<MIX, NS>(b, s, b.chk(pb - dstep));
        const double uk = k[0] * q.v[1] + k[1] * q.v[2] + k[2] * q.v[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) q.v[1 + d] -= k[d] * uk;
        bc_write_bv<MIX, NS>(b, s, pb, q);
        if constexpr (!MIX) s.mul[pb] = sutherland(q.v[5]);
      }
      BcNode<MIX, NS> q = bc_read<MIX, NS>(b, s, b.chk(pb - g * dstep));
      const double uk = k[0] * q.v[1] + k[1] * q.v[2] + k[2] * q.v[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) q.v[1 + d] -= 2 * uk * k[d];
      bc_write<MIX, NS>(b, s, b.chk(pb + g * dstep), q);
    } else {
      // outflow: every ghost takes the face node; periodic (node-coincident): the node as far inside
      // the opposite face
      long long src = pb, step = 0;
      if (type == kPeriodic) {
        const int ext[3] = {b.mx, b.my, b.mz};
        idx[face] = f.direction < 0 ? ext[face] - 1 : 0;
        src = b.id(idx[0], idx[1], idx[2]);
        step = dstep;
      }
      bc_write<MIX, NS>(b, s, b.chk(pb + g * dstep), bc_read<MIX, NS>(b, s, b.chk(src + g * step)));
    }
  }
}

}  // namespace ostc
