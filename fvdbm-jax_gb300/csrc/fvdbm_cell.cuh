// Device code of one cell's update shared by the step kernels (kernels.cu,
// resident.cu): the face flux, the update, the face-slot loads and the
// recording of node-stencil macros.
#pragma once
#include "fvdbm_math.cuh"

namespace fvdbm {

// Macros of a node-stencil cell for the next step's node kernel:
// rho, ux, uy, f_q - feq_q (src/containers.py:93-105,388-390).
__device__ __forceinline__ void record_stencil(const DevPlan& p, int i, const float fn[Q]) {
  float rho, ux, uy, eq[Q];
  macros(fn, rho, ux, uy);
  feq9(rho, ux, uy, p, eq);
  float* c = p.cprod + (i - p.stencil_start);
  c[0] = rho;
  c[size_t(p.Sp)] = ux;
  c[2 * size_t(p.Sp)] = uy;
#pragma unroll
  for (int q = 0; q < Q; ++q) c[(3 + q) * size_t(p.Sp)] = fn[q] - eq[q];
}

// Flux of face slot k from this cell's pdfs f and the pdfs o across it,
// signed for this cell, into acc (first slot: assigned).
template <int SCHEME, int VARIANT, bool FIRST>
__device__ __forceinline__ void face_flux(const DevPlan& p, const unsigned* __restrict__ hb, int k, int code,
                                          float nx, float ny, float Ls, float dt, const float f[Q],
                                          const float o[Q], float acc[Q]) {
  const HfRows HR{3, SCHEME, VARIANT};
  const bool slot1 = (code & HF_SLOT1) != 0;
  float v[Q];
  xi_dot_n(nx, ny, p.finite_n != 0, v);
  float w[Q];
  if (SCHEME == 1)
    lw_interp(v, __uint_as_float(__ldg(hb + HR.r(k) * 32)), __uint_as_float(__ldg(hb + HR.d2(k) * 32)),
              dt, p.finite_n != 0, w);
  const float scale = (VARIANT == 1) ? __uint_as_float(__ldg(hb + HR.sc(k) * 32)) : 1.0f;
#if FVDBM_PAIRED
  if constexpr (SCHEME == 0 && VARIANT == 0) {
    float phi[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) phi[q] = ((v[q] >= 0.0f) != slot1) ? f[q] : o[q];
    const float2 L2 = make_float2(Ls, Ls), one2 = make_float2(p.one, p.one);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x = mul2(mul2(make_float2(phi[2 * j], phi[2 * j + 1]), make_float2(v[2 * j], v[2 * j + 1])), L2);
      const float2 a = FIRST ? x : fold2(make_float2(acc[2 * j], acc[2 * j + 1]), one2, x);
      acc[2 * j] = a.x;
      acc[2 * j + 1] = a.y;
    }
    const float x8 = (phi[8] * v[8]) * Ls;
    acc[8] = FIRST ? x8 : acc[8] + x8;
  } else
#endif
  {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      float phi;
      if (SCHEME == 0) {
        // upwind: slot 0 when xi.n >= 0, else slot 1
        phi = ((v[q] >= 0.0f) != slot1) ? f[q] : o[q];
      } else {
        const float lq = slot1 ? o[q] : f[q], rq = slot1 ? f[q] : o[q];
        phi = lq + (rq - lq) * w[q];
      }
      float x = (phi * v[q]) * Ls;
      if (VARIANT == 1) x = x * scale;
      acc[q] = FIRST ? x : acc[q] + x;
    }
  }
}

// The relaxation and explicit-Euler update of one cell from its pdfs f and
// signed flux sum acc (times ia = 1/area in finite-volume mode).
template <bool FV>
__device__ __forceinline__ void cell_update(const DevPlan& p, float ia, const float f[Q], float acc[Q], float inv_tau,
                                            float dt, float fn[Q]) {
  float rho, ux, uy, eq[Q];
  macros(f, rho, ux, uy);
  feq9(rho, ux, uy, p, eq);
  if (FV) {
#pragma unroll
    for (int q = 0; q < Q; ++q) acc[q] = acc[q] * ia;
  }
#if FVDBM_PAIRED
  // f + dt*(inv_tau*(eq - f) - acc), pairwise
  const float2 it2 = make_float2(inv_tau, inv_tau), dt2 = make_float2(dt, dt);
  const float2 one2 = make_float2(p.one, p.one), m12 = make_float2(p.neg_one, p.neg_one);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f2 = make_float2(f[2 * j], f[2 * j + 1]);
    const float2 d = fold2(f2, m12, make_float2(eq[2 * j], eq[2 * j + 1]));    // eq - f
    const float2 u = fold2(make_float2(acc[2 * j], acc[2 * j + 1]), m12, mul2(it2, d));  // - acc
    const float2 r = fold2(f2, one2, mul2(dt2, u));                               // f + ...
    fn[2 * j] = r.x;
    fn[2 * j + 1] = r.y;
  }
  fn[8] = f[8] + dt * (inv_tau * (eq[8] - f[8]) - acc[8]);
#else
#pragma unroll
  for (int q = 0; q < Q; ++q) fn[q] = f[q] + dt * (inv_tau * (eq[q] - f[q]) - acc[q]);
#endif
}

template <int SCHEME, int VARIANT>
__device__ __forceinline__ void load_slots(const DevPlan& p, int i, const unsigned*& hb, int code[3],
                                           float nx[3], float ny[3], float Ls[3]) {
  constexpr int HROWS = (4 + (SCHEME == 1 ? 2 : 0) + (VARIANT == 1 ? 1 : 0)) * 3;
  const HfRows HR{3, SCHEME, VARIANT};
  hb = p.hf + cell_base(i < p.N ? i : 0, HROWS);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    code[k] = int(__ldg(hb + HR.code(k) * 32));
    nx[k] = __uint_as_float(__ldg(hb + HR.nx(k) * 32));
    ny[k] = __uint_as_float(__ldg(hb + HR.ny(k) * 32));
    Ls[k] = __uint_as_float(__ldg(hb + HR.ls(k) * 32));  // L * sigma
  }
}

// ---------------------------------------------------------------------------
// The fast family (FVDBM_KERNEL_FAST), on compact face slots (HfFastRows).
// Lax-Wendroff flux of one compact face slot:
// phi = l + (r - l) * (d0/(d0+d1) - (xi.n) dt/(2(d0+d1))), where
// (xi.n) dt/(2(d0+d1)) = (xi.a) * g.
__device__ __forceinline__ void face_lw_fast(int code, float ax, float ay, float r, float g, const float f[Q],
                                             const float o[Q], float acc[Q]) {
  const bool slot1 = (code & HF_SLOT1) != 0;
  const float a4[4] = {ax, ay, ax + ay, ay - ax};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int qp = j < 2 ? 1 + j : 5 + (j - 2), qm = qp + 2;  // xi.a = +a4[j], -a4[j]
    const float lp = slot1 ? o[qp] : f[qp], rp = slot1 ? f[qp] : o[qp];
    const float lm = slot1 ? o[qm] : f[qm], rm = slot1 ? f[qm] : o[qm];
    const float pp = __fmaf_rn(rp - lp, __fmaf_rn(-a4[j], g, r), lp);
    const float pm = __fmaf_rn(rm - lm, __fmaf_rn(a4[j], g, r), lm);
    acc[qp] = __fmaf_rn(pp, a4[j], acc[qp]);
    acc[qm] = __fmaf_rn(-pm, a4[j], acc[qm]);
  }
}

// Inflow rows of an upwind face: direction pair j is (qp, qp + 2) with xi.a =
// +a4[j], -a4[j]; up[j]: qp flows out (this cell's value) and qp + 2 flows in.
__device__ __forceinline__ void upwind_rows(int code, const float a4[4], bool up[4], int qn[4]) {
  const bool slot1 = (code & HF_SLOT1) != 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int qp = j < 2 ? 1 + j : 5 + (j - 2);
    up[j] = (a4[j] >= 0.0f) != slot1;
    qn[j] = up[j] ? qp + 2 : qp;
  }
}

// The face's flux sum from this cell's pdfs and the four inflow values.
__device__ __forceinline__ void upwind_sum(const float a4[4], const bool up[4], const float f[Q], const float o4[4],
                                           float acc[Q]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int qp = j < 2 ? 1 + j : 5 + (j - 2), qm = qp + 2;
    const float pp = up[j] ? f[qp] : o4[j];
    const float pm = up[j] ? o4[j] : f[qm];
    acc[qp] = __fmaf_rn(pp, a4[j], acc[qp]);
    acc[qm] = __fmaf_rn(-pm, a4[j], acc[qm]);
  }
}

// The fast family's update: f + dt*(inv_tau*(eq - f) - acc) (acc already
// carries 1/area in finite-volume mode).
__device__ __forceinline__ void cell_update_fast(const DevPlan& p, const float f[Q], const float acc[Q], float fn[Q]) {
  float rho, ux, uy, eq[Q];
  macros_fast(f, rho, ux, uy);
  feq9_fast(rho, ux, uy, p.d_c2.zr, p.d_c4x2.zr, p.d_c2x2.zr, eq);
  const float om = p.dt * p.inv_tau;
#pragma unroll
  for (int q = 0; q < Q; ++q) fn[q] = __fmaf_rn(-p.dt, acc[q], __fmaf_rn(om, eq[q] - f[q], f[q]));
}

template <int SCHEME>
__device__ __forceinline__ void load_slots_fast(const DevPlan& p, int i, const unsigned*& hb, int code[3],
                                                float ax[3], float ay[3]) {
  constexpr int HROWS = (3 + (SCHEME == 1 ? 2 : 0)) * 3;
  const HfFastRows HX{3, SCHEME};
  hb = p.hf + cell_base(i < p.N ? i : 0, HROWS);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    code[k] = int(__ldg(hb + HX.code(k) * 32));
    ax[k] = __uint_as_float(__ldg(hb + HX.ax(k) * 32));
    ay[k] = __uint_as_float(__ldg(hb + HX.ay(k) * 32));
  }
}

}  // namespace fvdbm
