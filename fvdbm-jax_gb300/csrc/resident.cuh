// Device code shared by the resident steps (resident.cu, resident_in_place.cu): the
// exchange words, the barriers and one cell's update.
#pragma once
#include "d2q13.cuh"
#include "fvdbm_cell.cuh"

namespace fvdbm {

// Limits of the waits.  A block's neighbour may not have started yet: other streams'
// kernels may hold the SM that it needs for as long as they run, so an import polls for
// about ten seconds.  Within a block the cell warps wait for the aux warps, which end an
// import that gives up: their limit (of tries of up to a microsecond) is the longer one.
// (Limits by the clock cost registers: 60k cells 3.65 us a step, 3.51 so.)
constexpr int RES_POLLS = 1 << 24, RES_TRIES = 1 << 28;

// One word of the exchange: three values and a tag, as a single 128-bit access
// (relaxed, gpu scope: atomic, through L2).
__device__ __forceinline__ uint4 ld_word(const uint4* ptr) {
  unsigned long long a, b;
  asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
               : "=l"(a), "=l"(b)
               : "l"(ptr)
               : "memory");
  return make_uint4(unsigned(a), unsigned(a >> 32), unsigned(b), unsigned(b >> 32));
}
__device__ __forceinline__ void st_word(uint4* ptr, float x, float y, float z, unsigned tag) {
  const unsigned long long a = __float_as_uint(x) | ((unsigned long long)__float_as_uint(y) << 32);
  const unsigned long long b = __float_as_uint(z) | ((unsigned long long)tag << 32);
  asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(ptr), "l"(a), "l"(b)
               : "memory");
}

// (the warp's lanes come together first: the barrier counts warps)
__device__ __forceinline__ void bar_sync(int id, int n) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int n) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Waits for phase `parity` of the barrier, a bounded number of polls.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
  for (int it = 0; it < RES_TRIES; ++it) {
    unsigned done;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000; selp.u32 %0, 1, 0, p; }"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Lattice-dependent pieces.  Directions beyond the rest one come in pairs
// (qp, qp + 2) with opposite velocities; pair j has xi_qp . n = pair_dot(j).
template <int LAT>
struct Lat;
template <>
struct Lat<9> {
  static constexpr int NQ = Q, NP = 4;
  static __device__ __forceinline__ void macros_(const float* f, float& r, float& x, float& y) { macros(f, r, x, y); }
  static __device__ __forceinline__ void feq_(float r, float x, float y, const DevPlan& p, float* o) {
    feq9(r, x, y, p, o);
  }
};
template <>
struct Lat<13> {
  static constexpr int NQ = Q13, NP = 6;
  static __device__ __forceinline__ void macros_(const float* f, float& r, float& x, float& y) { macros13(f, r, x, y); }
  static __device__ __forceinline__ void feq_(float r, float x, float y, const DevPlan& p, float* o) {
    feq13(r, x, y, p, o);
  }
};
__device__ __forceinline__ constexpr int pair_q(int j) { return j < 2 ? 1 + j : j < 4 ? 3 + j : 5 + j; }

// Rows of the resident face slots (non-fast families), field * 3 + face:
// code, nx, ny, L*sigma; Lax-Wendroff: d0/(d0+d1), then (xi.n dt)/(2(d0+d1)) of
// each direction pair; the face scale.
template <int LAT, int SCHEME, int VARIANT>
struct ResRows {
  static constexpr int NP = Lat<LAT>::NP;
  static constexpr int SC = SCHEME == 1 ? 5 + NP : 4;
  static constexpr int ROWS = 3 * (SC + (VARIANT == 1 ? 1 : 0));
};

template <int ROWS>
struct Slots {
  unsigned w[ROWS];
};
template <int ROWS>
__device__ __forceinline__ void load_rows(const unsigned* __restrict__ hf, int g, Slots<ROWS>& s) {
  const unsigned* b = hf + cell_base(g, ROWS);
#pragma unroll
  for (int i = 0; i < ROWS; ++i) s.w[i] = __ldg(b + i * 32);
}

// Neighbour pdfs from rows of NQ in shared memory (halo and ghost entries
// included).  inflow: of each direction pair the value that flows in; all: every
// direction's; read: no neighbour is read any more.
template <int NQ>
struct RowSource {
  const float* f0;
  template <int NP>
  __device__ __forceinline__ void inflow(int code, const bool (&up)[NP], const float*, float (&o)[NP]) const {
    const float* on = f0 + (code >> HF_SHIFT) * NQ;
#pragma unroll
    for (int j = 0; j < NP; ++j) o[j] = up[j] ? on[pair_q(j) + 2] : on[pair_q(j)];
  }
  __device__ __forceinline__ void all(int code, const float*, float (&o)[NQ]) const {
    const float* on = f0 + (code >> HF_SHIFT) * NQ;
#pragma unroll
    for (int q = 0; q < NQ; ++q) o[q] = on[q];
  }
  __device__ __forceinline__ void read() const {}
};

// One cell's new pdfs fn from its pdfs f and those of its neighbours.  LIT:
// the literal form, for inputs that are not all finite.
template <int LAT, int SCHEME, int VARIANT, bool FV, bool LIT, class Src>
__device__ __forceinline__ void cell_step(const DevPlan& p, const Src& nbr, const unsigned* w, float ia, float inv_tau,
                                          float dt, const float* f, float* fn) {
  using L = Lat<LAT>;
  constexpr int NQ = L::NQ, NP = L::NP;
  const float2 one2 = make_float2(p.one, p.one), m12 = make_float2(p.neg_one, p.neg_one);
  float2 acc[NP];  // pairs (qp, qp + 2)
  float acc0 = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int code = int(w[k]);
    const float nx = __uint_as_float(w[3 + k]), ny = __uint_as_float(w[6 + k]), Ls = __uint_as_float(w[9 + k]);
    const bool slot1 = (code & HF_SLOT1) != 0;
    const float2 L2 = make_float2(Ls, Ls);
    float a[NP], on[NQ], in[NP];
    bool up[NP];  // qp takes this cell's value
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      a[j] = j == 0 ? nx : j == 1 ? ny : j == 2 ? nx + ny : j == 3 ? ny - nx : j == 4 ? 2.0f * nx : 2.0f * ny;
      up[j] = (a[j] >= 0.0f) != slot1;
    }
    if (SCHEME == 0 && !LIT)
      nbr.inflow(code, up, f, in);
    else
      nbr.all(code, f, on);
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const int qp = pair_q(j), qm = qp + 2;
      float2 phi;
      if (SCHEME == 0) {
        if (LIT) {
          const bool um = (-a[j] >= 0.0f) != slot1;
          phi = make_float2(up[j] ? f[qp] : on[qp], um ? f[qm] : on[qm]);
        } else {
          phi = make_float2(up[j] ? f[qp] : in[j], up[j] ? in[j] : f[qm]);
        }
      } else {
        const float r = __uint_as_float(w[12 + k]), t = __uint_as_float(w[15 + 3 * j + k]);
        const float2 ff = make_float2(f[qp], f[qm]), oo = make_float2(on[qp], on[qm]);
        const float2 lq = make_float2(slot1 ? oo.x : ff.x, slot1 ? oo.y : ff.y);
        const float2 rq = make_float2(slot1 ? ff.x : oo.x, slot1 ? ff.y : oo.y);
        phi = fold2(lq, one2, mul2(sub2(rq, lq), add2(make_float2(r, r), make_float2(-t, t))));
      }
      float2 x = mul2(mul2(phi, make_float2(a[j], -a[j])), L2);
      if (VARIANT == 1) {
        const float sc = __uint_as_float(w[3 * ResRows<LAT, SCHEME, VARIANT>::SC + k]);
        x = mul2(x, make_float2(sc, sc));
      }
      acc[j] = k == 0 ? x : fold2(acc[j], one2, x);
    }
    if (LIT) {
      float phi = !slot1 ? f[0] : on[0];
      if (SCHEME == 1) {
        const float r = __uint_as_float(w[12 + k]);
        const float lq = slot1 ? on[0] : f[0], rq = slot1 ? f[0] : on[0];
        phi = __fadd_rn(lq, __fmul_rn(__fsub_rn(rq, lq), r));
      }
      float x = __fmul_rn(__fmul_rn(phi, 0.0f), Ls);
      if (VARIANT == 1) x = __fmul_rn(x, __uint_as_float(w[3 * ResRows<LAT, SCHEME, VARIANT>::SC + k]));
      acc0 = k == 0 ? x : __fadd_rn(acc0, x);
    }
  }
  nbr.read();
  float rho, ux, uy, eq[NQ];
  L::macros_(f, rho, ux, uy);
  L::feq_(rho, ux, uy, p, eq);
  if (FV) {
    acc0 = acc0 * ia;
#pragma unroll
    for (int j = 0; j < NP; ++j) acc[j] = mul2(acc[j], make_float2(ia, ia));
  }
  const float2 it2 = make_float2(inv_tau, inv_tau), dt2 = make_float2(dt, dt);
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const int qp = pair_q(j), qm = qp + 2;
    const float2 f2 = make_float2(f[qp], f[qm]);
    const float2 d = fold2(f2, m12, make_float2(eq[qp], eq[qm]));     // eq - f
    const float2 u = fold2(acc[j], m12, mul2(it2, d));                // - acc
    const float2 r = fold2(f2, one2, mul2(dt2, u));                   // f + ...
    fn[qp] = r.x;
    fn[qm] = r.y;
  }
  fn[0] = f[0] + dt * (inv_tau * (eq[0] - f[0]) - acc0);
}

// The fast family's cell (contracted arithmetic on compact slots).
template <int SCHEME, class Src>
__device__ __forceinline__ void cell_step_fast(const DevPlan& p, const Src& nbr, const unsigned* w, const float* f,
                                               float* fn) {
  const HfFastRows HX{3, SCHEME};
  float acc[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) acc[q] = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int code = int(w[HX.code(k)]);
    const float ax = __uint_as_float(w[HX.ax(k)]), ay = __uint_as_float(w[HX.ay(k)]);
    if (SCHEME == 0) {
      const float a4[4] = {ax, ay, ax + ay, ay - ax};
      bool up[4];
      int qn[4];
      float o4[4];
      upwind_rows(code, a4, up, qn);
      nbr.inflow(code, up, f, o4);
      upwind_sum(a4, up, f, o4, acc);
    } else {
      float o[Q];
      nbr.all(code, f, o);
      face_lw_fast(code, ax, ay, __uint_as_float(w[HX.r(k)]), __uint_as_float(w[HX.g(k)]), f, o, acc);
    }
  }
  nbr.read();
  cell_update_fast(p, f, acc, fn);
}

}  // namespace fvdbm
