// D2Q13 device arithmetic shared by d2q13.cu and resident.cu.
#pragma once
#include "fvdbm_math.cuh"

namespace fvdbm {

constexpr int Q13 = 13;
static __constant__ float c_kx13[Q13] = {0, 1, 0, -1, 0, 1, -1, -1, 1, 2, 0, -2, 0};
static __constant__ float c_ky13[Q13] = {0, 0, 1, 0, -1, 1, 1, -1, -1, 0, 2, 0, -2};
static __constant__ float c_w13[Q13] = {(float)(3.0 / 8.0),   (float)(1.0 / 12.0), (float)(1.0 / 12.0),
                                 (float)(1.0 / 12.0),  (float)(1.0 / 12.0), (float)(1.0 / 16.0),
                                 (float)(1.0 / 16.0),  (float)(1.0 / 16.0), (float)(1.0 / 16.0),
                                 (float)(1.0 / 96.0),  (float)(1.0 / 96.0), (float)(1.0 / 96.0),
                                 (float)(1.0 / 96.0)};

__device__ __forceinline__ size_t base13(int c) { return size_t(c >> 5) * (Q13 * 32) + size_t(c & 31); }

__device__ __forceinline__ void load13(const float* __restrict__ f, int c, float out[Q13]) {
  const float* b = f + base13(c);
#pragma unroll
  for (int q = 0; q < Q13; ++q) out[q] = __ldg(b + q * 32);
}

// rho = sum_q f_q; u = (xi^T f)/rho (src/dynamics.py:35-47).  For finite
// rho every f_q is finite: the 0*f_q terms of the literal fold are +-0 and
// leave the sum's value unchanged, +-1*f_q is +-f_q and 2*f_q is exact, so
// the fold runs over the nonzero directions only; otherwise every product is
// kept.
__device__ __forceinline__ void macros13(const float f[Q13], float& rho, float& ux, float& uy) {
  float r = f[0];
#pragma unroll
  for (int q = 1; q < Q13; ++q) r = r + f[q];
  float mx, my;
  if (fabsf(r) <= FLT_MAX) {
    mx = ((((((f[1] - f[3]) + f[5]) - f[6]) - f[7]) + f[8]) + 2.0f * f[9]) - 2.0f * f[11];
    my = ((((((f[2] - f[4]) + f[5]) + f[6]) - f[7]) - f[8]) + 2.0f * f[10]) - 2.0f * f[12];
  } else {
    mx = c_kx13[0] * f[0];
    my = c_ky13[0] * f[0];
#pragma unroll
    for (int q = 1; q < Q13; ++q) {
      mx = mx + c_kx13[q] * f[q];
      my = my + c_ky13[q] * f[q];
    }
  }
  rho = r;
  ux = mx / r;
  uy = my / r;
}

// v_q = xi_q . n (src/containers.py:235); for a finite normal the symmetric
// form (+-nx, +-ny, +-(nx+ny), +-(ny-nx), +-2nx, +-2ny), whose values equal
// the literal dot products'
__device__ __forceinline__ void xi13_dot_n(float nx, float ny, bool finite_n, float v[Q13]) {
  if (!finite_n) {
#pragma unroll
    for (int q = 0; q < Q13; ++q) v[q] = c_kx13[q] * nx + c_ky13[q] * ny;
    return;
  }
  const float s = nx + ny, d = ny - nx, x2 = 2.0f * nx, y2 = 2.0f * ny;
  v[0] = 0.0f;
  v[1] = nx;
  v[2] = ny;
  v[3] = -nx;
  v[4] = -ny;
  v[5] = s;
  v[6] = d;
  v[7] = -s;
  v[8] = -d;
  v[9] = x2;
  v[10] = y2;
  v[11] = -x2;
  v[12] = -y2;
}

// x == 0 or 2^-30 <= |x| <= 2^30: then x^2, x*x^2, 3x*u.u and their
// scalings by 2, 4, 8 stay in the normal range, where binary scaling commutes
// with rounding, and every dividend is one the known-divisor check covers.
__device__ __forceinline__ bool dom13(float x) {
  const float a = fabsf(x);
  return (a >= 0x1p-30f && a <= 0x1p30f) || x == 0.0f;
}

__device__ __forceinline__ float kdiv(float x, const CDiv& d, bool two) {
  return two ? cdiv_two(x, d.zr, d.zl) : cdiv_fast(x, d.y, d.zr);
}

__device__ __forceinline__ void feq13(float rho, float ux, float uy, const DevPlan& p, float out[Q13]) {
  const float uu = ux * ux + uy * uy;
  const float a5 = ux + uy, a6 = uy - ux;
  if (p.cdiv_mode != 0 && dom13(ux) && dom13(uy) && dom13(a5) && dom13(a6)) {
    // a_q = +-x or +-2x for x in (ux, uy, ux+uy, uy-ux) (a_0 = 0; the 0*u
    // terms of the literal dot product only change the sign of a zero a,
    // which leaves s unchanged).  Per x: t1 = x/C^2, t2 = x^2/(2C^4),
    // t4 = x*x^2/(2C^6), t5 = 3x*u.u/(2C^4); for -x the odd ones change sign
    // (RN(-y) = -RN(y)), for 2x they scale by 2, 4, 8, 2 exactly.  17
    // divisions instead of 65, each the known-divisor form.
    const bool two = p.cdiv_mode == 2;
    const float t3 = kdiv(uu, p.d_c2x2, two);
    const float b[4] = {ux, uy, a5, a6};
    float t1[4], t2[4], t4[4], t5[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float x = b[j], xx = x * x;
      t1[j] = kdiv(x, p.d_c2, two);
      t2[j] = kdiv(xx, p.d_c4x2, two);
      t4[j] = kdiv(x * xx, p.d_c6x2, two);
      t5[j] = kdiv((3.0f * x) * uu, p.d_c4x2, two);
    }
    auto S = [t3](float a1, float a2, float a4, float a5_) {
      float s = 1.0f + a1;
      s = s + a2;
      s = s - t3;
      s = s + a4;
      return s - a5_;
    };
    const float w0 = c_w13[0] * rho, w1 = c_w13[1] * rho, w5 = c_w13[5] * rho, w9 = c_w13[9] * rho;
    out[0] = w0 * S(0.0f, 0.0f, 0.0f, 0.0f);
    out[1] = w1 * S(t1[0], t2[0], t4[0], t5[0]);
    out[3] = w1 * S(-t1[0], t2[0], -t4[0], -t5[0]);
    out[2] = w1 * S(t1[1], t2[1], t4[1], t5[1]);
    out[4] = w1 * S(-t1[1], t2[1], -t4[1], -t5[1]);
    out[5] = w5 * S(t1[2], t2[2], t4[2], t5[2]);
    out[7] = w5 * S(-t1[2], t2[2], -t4[2], -t5[2]);
    out[6] = w5 * S(t1[3], t2[3], t4[3], t5[3]);
    out[8] = w5 * S(-t1[3], t2[3], -t4[3], -t5[3]);
    out[9] = w9 * S(2.0f * t1[0], 4.0f * t2[0], 8.0f * t4[0], 2.0f * t5[0]);
    out[11] = w9 * S(-2.0f * t1[0], 4.0f * t2[0], -8.0f * t4[0], -2.0f * t5[0]);
    out[10] = w9 * S(2.0f * t1[1], 4.0f * t2[1], 8.0f * t4[1], 2.0f * t5[1]);
    out[12] = w9 * S(-2.0f * t1[1], 4.0f * t2[1], -8.0f * t4[1], -2.0f * t5[1]);
    return;
  }
#pragma unroll
  for (int q = 0; q < Q13; ++q) {
    const float a = c_kx13[q] * ux + c_ky13[q] * uy;
    float s = 1.0f + a / p.c2;
    s = s + (a * a) / p.c4x2;
    s = s - uu / p.c2x2;
    s = s + (a * (a * a)) / p.c6x2;
    s = s - ((3.0f * a) * uu) / p.c4x2;
    out[q] = (c_w13[q] * rho) * s;
  }
}

// Flux of face slot k (paired with the neighbour's pdfs o) into acc; the
// first slot assigns.
template <int SCHEME, bool FIRST>
__device__ __forceinline__ void face_flux13(const DevPlan& p, const unsigned* __restrict__ hb, int k, bool slot1,
                                            float nx, float ny, float Ls, const float f[Q13], const float o[Q13],
                                            float acc[Q13]) {
  const HfRows HR{3, SCHEME, 0};
  float r = 0.0f, D2 = 1.0f;
  if (SCHEME == 1) {
    r = __uint_as_float(__ldg(hb + HR.r(k) * 32));
    D2 = __uint_as_float(__ldg(hb + HR.d2(k) * 32));
  }
  float vq[Q13];
  xi13_dot_n(nx, ny, p.finite_n != 0, vq);
  float w[Q13];
  if (SCHEME == 1) {
    // interp_q = d0/(d0+d1) - (v_q dt)/(2(d0+d1)) (src/containers.py:274);
    // for a finite normal v_{q'} = -v_q pairs share one quotient:
    // (-v dt)/D2 == -((v dt)/D2), and r - (-t) == r + t
    if (p.finite_n) {
      const float t1 = (vq[1] * p.dt) / D2, t2 = (vq[2] * p.dt) / D2, t5 = (vq[5] * p.dt) / D2;
      const float t6 = (vq[6] * p.dt) / D2, t9 = (vq[9] * p.dt) / D2, t10 = (vq[10] * p.dt) / D2;
      w[0] = r - (vq[0] * p.dt) / D2;
      w[1] = r - t1;
      w[3] = r + t1;
      w[2] = r - t2;
      w[4] = r + t2;
      w[5] = r - t5;
      w[7] = r + t5;
      w[6] = r - t6;
      w[8] = r + t6;
      w[9] = r - t9;
      w[11] = r + t9;
      w[10] = r - t10;
      w[12] = r + t10;
    } else {
#pragma unroll
      for (int q = 0; q < Q13; ++q) w[q] = r - (vq[q] * p.dt) / D2;
    }
  }
  float phi[Q13];
#pragma unroll
  for (int q = 0; q < Q13; ++q) {
    const float lq = slot1 ? o[q] : f[q], rq = slot1 ? f[q] : o[q];
    phi[q] = (SCHEME == 0) ? (vq[q] >= 0.0f ? lq : rq) : lq + (rq - lq) * w[q];
  }
#if FVDBM_PAIRED
  // paired products; a sum that takes one is the multiply-add acc*one + x
  const float2 L2 = make_float2(Ls, Ls), one2 = make_float2(p.one, p.one);
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    const float2 x = mul2(mul2(make_float2(phi[2 * j], phi[2 * j + 1]), make_float2(vq[2 * j], vq[2 * j + 1])), L2);
    const float2 a = FIRST ? x : fold2(make_float2(acc[2 * j], acc[2 * j + 1]), one2, x);
    acc[2 * j] = a.x;
    acc[2 * j + 1] = a.y;
  }
  {
    const float x = (phi[12] * vq[12]) * Ls;
    acc[12] = FIRST ? x : acc[12] + x;
  }
#else
#pragma unroll
  for (int q = 0; q < Q13; ++q) {
    const float x = (phi[q] * vq[q]) * Ls;
    acc[q] = FIRST ? x : acc[q] + x;
  }
#endif
}

// The relaxation and explicit-Euler update (times ia = 1/area when fv).
__device__ __forceinline__ void cell_update13(const DevPlan& p, float ia, bool fv, const float f[Q13],
                                              float acc[Q13], float fn[Q13]) {
  float rho, ux, uy, eq[Q13];
  macros13(f, rho, ux, uy);
  feq13(rho, ux, uy, p, eq);
  if (fv) {
#pragma unroll
    for (int q = 0; q < Q13; ++q) acc[q] = acc[q] * ia;
  }
#if FVDBM_PAIRED
  // f + dt*(inv_tau*(eq - f) - acc), pairwise
  const float2 it2 = make_float2(p.inv_tau, p.inv_tau), dt2 = make_float2(p.dt, p.dt);
  const float2 one2 = make_float2(p.one, p.one), m12 = make_float2(p.neg_one, p.neg_one);
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    const float2 f2 = make_float2(f[2 * j], f[2 * j + 1]);
    const float2 d = fold2(f2, m12, make_float2(eq[2 * j], eq[2 * j + 1]));
    const float2 u = fold2(make_float2(acc[2 * j], acc[2 * j + 1]), m12, mul2(it2, d));
    const float2 r = fold2(f2, one2, mul2(dt2, u));
    fn[2 * j] = r.x;
    fn[2 * j + 1] = r.y;
  }
  fn[12] = f[12] + p.dt * (p.inv_tau * (eq[12] - f[12]) - acc[12]);
#else
#pragma unroll
  for (int q = 0; q < Q13; ++q) fn[q] = f[q] + p.dt * (p.inv_tau * (eq[q] - f[q]) - acc[q]);
#endif
}

}  // namespace fvdbm
