// D2Q13 lattice (src/dynamics.py:77-102): the staged step (boundary nodes,
// per-face fluxes, per-cell gather and update), the fused cell update for
// triangle meshes (boundary nodes, then one cell kernel) and the read-back
// helpers
// with 13 velocities, including the (+-2, 0), (0, +-2) ones, and the
// third-order equilibrium
//   feq_q = (W_q rho) * (((((1 + a/C^2) + a^2/(2C^4)) - u.u/(2C^2))
//                          + a^3/(2C^6)) - 3 a u.u/(2C^4)),   a = xi_q . u,
// evaluated in that order with a^3 = a*(a*a) (jax's integer_pow), so that
// results equal the reference's float32 step bit for bit.  The float32
// lattice constants come from the host (C = 1/sqrt(2) in float32).
//
// Layouts as the D2Q9 kernels: cell pdfs AoSoA [Np/32][13][32], face fluxes
// [13][Fp], node state [13][Mp] / [Mp] / [2][Mp].
#include "d2q13.cuh"

namespace fvdbm {

namespace {

// Boundary nodes (src/containers.py:339-404, utils/utils.py:34-60), one
// thread per computed node, its stencil entries folded in order.
__global__ void k13_nodes(DevPlan p, const float* __restrict__ f) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= p.Mc) return;
  const int type = p.nd_type[m];
  const int e0 = p.nd_ptr[m], e1 = p.nd_ptr[m + 1];
  float ar = 0.0f, ax = 0.0f, ay = 0.0f, an[Q13];
#pragma unroll
  for (int q = 0; q < Q13; ++q) an[q] = 0.0f;
  for (int e = e0; e < e1; ++e) {
    const unsigned code = p.nd_cell[e];
    const float w = p.nd_w[e];
    float fc[Q13], eq[Q13];
    load13(f, int(code & ~ND_NEQ_ZERO), fc);
    float rho, ux, uy;
    macros13(fc, rho, ux, uy);
    feq13(rho, ux, uy, p, eq);
    const bool zero = (code & ND_NEQ_ZERO) != 0;
    const bool first = e == e0;
    ar = first ? rho * w : ar + rho * w;
    ax = first ? ux * w : ax + ux * w;
    ay = first ? uy * w : ay + uy * w;
#pragma unroll
    for (int q = 0; q < Q13; ++q) {
      const float x = (zero ? 0.0f : fc[q] - eq[q]) * w;
      an[q] = first ? x : an[q] + x;
    }
  }
  if (p.nd_npad[m] > 0) {
    // padded (-1, weight 0) entries gather the last cell
    float fc[Q13];
    load13(f, p.last_cell, fc);
    float rho, ux, uy;
    macros13(fc, rho, ux, uy);
    const bool none = e1 == e0;
    ar = none ? rho * 0.0f : ar + rho * 0.0f;
    ax = none ? ux * 0.0f : ax + ux * 0.0f;
    ay = none ? uy * 0.0f : ay + uy * 0.0f;
  }
  const float sw = p.nd_sumw[m];
  float rho_p, ux_p, uy_p;
  if (type == 1) {
    rho_p = ar / sw;
    ux_p = p.node_vel[m];
    uy_p = p.node_vel[p.Mp + m];
    p.node_rho[m] = rho_p;
  } else {
    rho_p = p.node_rho[m];
    ux_p = ax / sw;
    uy_p = ay / sw;
    p.node_vel[m] = ux_p;
    p.node_vel[p.Mp + m] = uy_p;
  }
  float eqn[Q13];
  feq13(rho_p, ux_p, uy_p, p, eqn);
#pragma unroll
  for (int q = 0; q < Q13; ++q) p.node_pdf[size_t(q) * p.Mp + m] = eqn[q] + an[q] / sw;
}

// Face fluxes (src/containers.py:191-287), one thread per face.
__global__ void k13_face(DevPlan p, const float* __restrict__ f, float* __restrict__ flux) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= p.F) return;
  const int s0 = p.fs0[j], s1 = p.fs1[j];
  float lf[Q13], rf[Q13];
  if (s0 >= 0 && s1 >= 0) {
    load13(f, s0, lf);
    load13(f, s1, rf);
  } else {
    const int a = p.fna[j], b = p.fnb[j];
    float mq[Q13];
#pragma unroll
    for (int q = 0; q < Q13; ++q)
      mq[q] = (p.node_pdf[size_t(q) * p.Mp + a] + p.node_pdf[size_t(q) * p.Mp + b]) / 2.0f;
    if (s0 >= 0) {
      load13(f, s0, lf);
    } else {
      float kf[Q13];
      load13(f, p.fkl[j], kf);
#pragma unroll
      for (int q = 0; q < Q13; ++q) lf[q] = mq[q] + (mq[q] - kf[q]) * p.frl[j];
    }
    if (s1 >= 0) {
      load13(f, s1, rf);
    } else {
      float kf[Q13];
      load13(f, p.fkr[j], kf);
#pragma unroll
      for (int q = 0; q < Q13; ++q) rf[q] = mq[q] + (mq[q] - kf[q]) * p.frr[j];
    }
  }
  const float nx = p.fnx[j], ny = p.fny[j], L = p.fL[j];
#pragma unroll
  for (int q = 0; q < Q13; ++q) {
    const float v = c_kx13[q] * nx + c_ky13[q] * ny;
    float phi;
    if (p.scheme == 0) {
      phi = v >= 0.0f ? lf[q] : rf[q];
    } else {
      const float w = p.fr[j] - (v * p.dt) / p.fD2[j];
      phi = lf[q] + (rf[q] - lf[q]) * w;
    }
    flux[size_t(q) * p.Fp + j] = (phi * v) * L;
  }
}

// Cell update (src/containers.py:107-121), one thread per cell.
__global__ void k13_gather(DevPlan p, const float* __restrict__ fin, const float* __restrict__ flux,
                           float* __restrict__ fout) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.N) return;
  const size_t Np = p.Np;
  float f[Q13], eq[Q13], acc[Q13];
  load13(fin, i, f);
  float rho, ux, uy;
  macros13(f, rho, ux, uy);
  feq13(rho, ux, uy, p, eq);
#pragma unroll
  for (int q = 0; q < Q13; ++q) acc[q] = 0.0f;
  for (int k = 0; k < p.K; ++k) {
    const int fi = p.cf_face[k * Np + i];
    const float sg = p.cf_sign[k * Np + i];
#pragma unroll
    for (int q = 0; q < Q13; ++q) {
      const float x = flux[size_t(q) * p.Fp + fi] * sg;
      acc[q] = (k == 0) ? x : acc[q] + x;
    }
  }
  if (p.fv) {
    const float ia = p.inv_area[i];
#pragma unroll
    for (int q = 0; q < Q13; ++q) acc[q] = acc[q] * ia;
  }
  float* o = fout + base13(i);
#pragma unroll
  for (int q = 0; q < Q13; ++q) o[q * 32] = f[q] + p.dt * (p.inv_tau * (eq[q] - f[q]) - acc[q]);
}

// Fused cell update (k13_face + k13_gather in one pass), one thread per
// cell: macros, feq, the flux of each of the cell's three face slots from
// the canonical slot-0/slot-1 pair (both neighbours compute identical
// values), the signed sum and the update, with the per-cell face slots of
// the D2Q9 fused kernel ([Np/32][rows][32]: code, n, L*sigma, LW r and D2).
// ((phi*v)*L)*sigma == (phi*v)*(L*sigma) exactly for sigma = +-1.
template <int SCHEME>
__global__ void __launch_bounds__(256) k13_fused(DevPlan p, const float* __restrict__ fin,
                                                 float* __restrict__ fout) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.N) return;
  const HfRows HR{3, SCHEME, 0};
  const unsigned* hb = p.hf + size_t(i >> 5) * (HR.rows() * 32) + (i & 31);
  float f[Q13], acc[Q13];
  load13(fin, i, f);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int code = int(__ldg(hb + HR.code(k) * 32));
    const float nx = __uint_as_float(__ldg(hb + HR.nx(k) * 32));
    const float ny = __uint_as_float(__ldg(hb + HR.ny(k) * 32));
    const float Ls = __uint_as_float(__ldg(hb + HR.ls(k) * 32));
    const int other = code >> HF_SHIFT;
    const bool slot1 = (code & HF_SLOT1) != 0;
    float o[Q13];
    if (code & HF_GHOST) {
      // ghost = m + (m - f_known)*(d_ghost/d_known), the known cell this one
      const int a = __ldg(p.gh_a + other), b = __ldg(p.gh_b + other);
      const float rg = __ldg(p.gh_r + other);
#pragma unroll
      for (int q = 0; q < Q13; ++q) {
        const float mq = (p.node_pdf[size_t(q) * p.Mp + a] + p.node_pdf[size_t(q) * p.Mp + b]) / 2.0f;
        o[q] = mq + (mq - f[q]) * rg;
      }
    } else {
      load13(fin, other, o);
    }
    if (k == 0)
      face_flux13<SCHEME, true>(p, hb, k, slot1, nx, ny, Ls, f, o, acc);
    else
      face_flux13<SCHEME, false>(p, hb, k, slot1, nx, ny, Ls, f, o, acc);
  }
  float fn[Q13];
  cell_update13(p, p.fv ? p.inv_area[i] : 1.0f, p.fv != 0, f, acc, fn);
  float* o = fout + base13(i);
#pragma unroll
  for (int q = 0; q < Q13; ++q) o[q * 32] = fn[q];
}

// rho [Np], vel [2][Np], feq AoSoA of a pdf buffer (read-back)
__global__ void k13_macros(DevPlan p, const float* __restrict__ f, float* __restrict__ rho_o,
                           float* __restrict__ vel_o, float* __restrict__ feq_o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.N) return;
  float fc[Q13], eq[Q13];
  load13(f, i, fc);
  float rho, ux, uy;
  macros13(fc, rho, ux, uy);
  feq13(rho, ux, uy, p, eq);
  rho_o[i] = rho;
  vel_o[i] = ux;
  vel_o[size_t(p.Np) + i] = uy;
  float* o = feq_o + base13(i);
#pragma unroll
  for (int q = 0; q < Q13; ++q) o[q * 32] = eq[q];
}

inline int nblk(long long n, int t) { return int((n + t - 1) / t); }

}  // namespace

cudaError_t launch13_step(const DevPlan& p, const float* fin, float* flux, float* fout, cudaStream_t s) {
  if (p.Mc > 0) k13_nodes<<<nblk(p.Mc, 128), 128, 0, s>>>(p, fin);
  if (p.F > 0) k13_face<<<nblk(p.F, 256), 256, 0, s>>>(p, fin, flux);
  if (p.N > 0) k13_gather<<<nblk(p.N, 256), 256, 0, s>>>(p, fin, flux, fout);
  return cudaGetLastError();
}

cudaError_t launch13_fused(const DevPlan& p, const float* fin, float* fout, cudaStream_t s) {
  if (p.Mc > 0) k13_nodes<<<nblk(p.Mc, 128), 128, 0, s>>>(p, fin);
  if (p.N > 0) {
    if (p.scheme == 1)
      k13_fused<1><<<nblk(p.N, 256), 256, 0, s>>>(p, fin, fout);
    else
      k13_fused<0><<<nblk(p.N, 256), 256, 0, s>>>(p, fin, fout);
  }
  return cudaGetLastError();
}

cudaError_t launch13_nodes(const DevPlan& p, const float* fin, cudaStream_t s) {
  if (p.Mc > 0) k13_nodes<<<nblk(p.Mc, 128), 128, 0, s>>>(p, fin);
  return cudaGetLastError();
}

cudaError_t launch13_cells(const DevPlan& p, const float* fin, float* fout, cudaStream_t s) {
  if (p.N > 0) {
    if (p.scheme == 1)
      k13_fused<1><<<nblk(p.N, 256), 256, 0, s>>>(p, fin, fout);
    else
      k13_fused<0><<<nblk(p.N, 256), 256, 0, s>>>(p, fin, fout);
  }
  return cudaGetLastError();
}

cudaError_t launch13_face_flux(const DevPlan& p, const float* f, float* flux, cudaStream_t s) {
  if (p.F > 0) k13_face<<<nblk(p.F, 256), 256, 0, s>>>(p, f, flux);
  return cudaGetLastError();
}

cudaError_t launch13_macros(const DevPlan& p, const float* f, float* rho, float* vel, float* feq,
                            cudaStream_t s) {
  if (p.N > 0) k13_macros<<<nblk(p.N, 256), 256, 0, s>>>(p, f, rho, vel, feq);
  return cudaGetLastError();
}

}  // namespace fvdbm
