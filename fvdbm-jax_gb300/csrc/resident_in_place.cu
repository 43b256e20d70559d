// The resident step for meshes of many cells per block, whose state need not fit on
// the chip twice (resident.cu): a block's interior pdfs move through a ring in
// shared memory.
//
// A step in each block, one per SM, its two halves side by side:
//   cell warps   sweep the interior cells (whose neighbours are all the block's
//                own) in chunks along the longer side of its part, so that a
//                cell's neighbours lie in its own chunk, the ones beside it or
//                among the boundary cells.  The new state lies a chunk before the old
//                one in the ring: a chunk's new pdfs take the place of the chunk
//                before it, once every warp has read its neighbours.
//   aux warps    macros of the node stencils, the halo import, nodes, ghosts, then
//                the boundary cells (with halo or ghost faces, or exported): two copies in shared
//                memory.  These read every neighbour as a row: imported,
//                ghost, interior or boundary cell, the latter two by the step's parity.
//
// Rows are the block's own scratch in global memory (L1 and L2).
//
// Bound by latency, at 425k cells: the sweep takes about 3,200 clocks per chunk of 512
// cells (525 instructions per cell on 16 warps), the aux warps' chain of rounds
// through the halo import about 18,000; both run at once.  us per step in runs of 512,
// one or two launches of a step / here: porous, 249k cells 12.1 / 6.6, 420k 13.7 / 9.9, contracted
// family 10.6 / 6.0 and 11.6 / 8.7; cavity, 425k 10.8 / 9.1, contracted 9.2 / 7.2; 24 cases of
// 423k cells in all 17.1 / 11.2.  Boundary cells after the sweep, by the cell warps: porous,
// 420k 11.1 and 8.8.
#include "resident.cuh"

namespace fvdbm {

namespace {

constexpr int IP_THREADS = 1024;
constexpr int IP_ROW = 12;  // floats of a row: q = 1..8, 0, and padding
constexpr int IP_SR = 12;   // floats of a stencil cell: macros, f - feq

// A face's code: HF_SLOT1, the neighbour (16 bits from HF_SHIFT); in the first
// one, from bit IP_LINK on, 1 + the row of an interior cell that boundary cells
// read, or 1 + a boundary cell's export slot (of the block's); 0: none.
__device__ __forceinline__ int ip_neighbour(int code) { return (code >> HF_SHIFT) & 0xffff; }

// The block's own pdfs in shared memory, in groups of 32 cells (pdf q is 32 q
// on): the ring, whose state begins at rot, then two copies of the boundary cells.
constexpr int IP_GROUP = Q * 32;
__device__ __forceinline__ int ip_index(int l) { return (l >> 5) * IP_GROUP + (l & 31); }
struct State {
  float* pd;
  int size, rot;  // of the ring
  int bnd0, bnd;  // first boundary cell; offset of this state's copy
  __device__ __forceinline__ float* at(int i) const {
    const int j = i + rot;
    return pd + (i >= size ? i + bnd : j >= size ? j - size : j);
  }
  __device__ __forceinline__ float* cell(int l) const { return at(l < bnd0 ? ip_index(l) : size + ip_index(l - bnd0)); }
  __device__ __forceinline__ void load(int l, float* f) const {
    const float* c = cell(l);
#pragma unroll
    for (int q = 0; q < Q; ++q) f[q] = c[q * 32];
  }
  __device__ __forceinline__ void store(int l, const float* f) const {
    float* c = cell(l);
#pragma unroll
    for (int q = 0; q < Q; ++q) c[q * 32] = f[q];
  }
  // of the next step; copy: floats of the boundary cells' one
  __device__ __forceinline__ State next(int chunk, int copy) const {
    const int n = rot - chunk / 32 * IP_GROUP;
    return State{pd, size, n < 0 ? n + size : n, bnd0, bnd ? 0 : copy};
  }
};

// Neighbours of an interior cell.  read() tells the other warps that
// this one has read what it needs of the old state.
struct StateSource {
  State state;
  unsigned guard;
  template <int NP>
  __device__ __forceinline__ void inflow(int code, const bool (&up)[NP], const float*, float (&o)[NP]) const {
    const float* on = state.at(ip_neighbour(code));
#pragma unroll
    for (int j = 0; j < NP; ++j) o[j] = on[(up[j] ? pair_q(j) + 2 : pair_q(j)) * 32];
  }
  __device__ __forceinline__ void all(int code, const float*, float (&o)[Q]) const {
    const float* on = state.at(ip_neighbour(code));
#pragma unroll
    for (int q = 0; q < Q; ++q) o[q] = on[q * 32];
  }
  __device__ __forceinline__ void read() const {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(guard);
  }
};

// Neighbours of a boundary cell: rows; those from row `own` on are the block's
// cells, two rows each, by the parity of the step.
struct ScratchSource {
  const float* rows;
  int own, shift;
  __device__ __forceinline__ const float4* row(int code) const {
    const int i = ip_neighbour(code);
    return reinterpret_cast<const float4*>(rows + size_t(i >= own ? i + shift : i) * IP_ROW);
  }
  template <int NP>
  __device__ __forceinline__ void inflow(int code, const bool (&up)[NP], const float*, float (&o)[NP]) const {
    const float4 *r = row(code), a = r[0], b = r[1];
    o[0] = up[0] ? a.z : a.x;
    o[1] = up[1] ? a.w : a.y;
    o[2] = up[2] ? b.z : b.x;
    o[3] = up[3] ? b.w : b.y;
  }
  __device__ __forceinline__ void all(int code, const float*, float (&o)[Q]) const {
    const float4 *r = row(code), a = r[0], b = r[1];
    o[0] = r[2].x;
    o[1] = a.x, o[2] = a.y, o[3] = a.z, o[4] = a.w;
    o[5] = b.x, o[6] = b.y, o[7] = b.z, o[8] = b.w;
  }
  __device__ __forceinline__ void read() const {}
};

__device__ __forceinline__ void put_row(float* row, const float* f) {
  float4* r = reinterpret_cast<float4*>(row);
  r[0] = make_float4(f[1], f[2], f[3], f[4]);
  r[1] = make_float4(f[5], f[6], f[7], f[8]);
  row[8] = f[0];
}

// A cell whose inputs are not all finite, out of line (rarely taken).
struct Pdfs {
  float f[Q];
};
template <int SCHEME, bool FV, class Src>
__device__ __noinline__ Pdfs in_place_literal(const DevPlan& p, const Src nbr, const unsigned* __restrict__ hf, int g,
                                              float ia, float inv_tau, float dt, const Pdfs f) {
  Slots<ResRows<9, SCHEME, 0>::ROWS> s;
  load_rows(hf, g, s);
  Pdfs o;
  cell_step<9, SCHEME, 0, FV, true>(p, nbr, s.w, ia, inv_tau, dt, f.f, o.f);
  return o;
}

// One cell's new pdfs.
template <int SCHEME, bool FV, bool FAST, int ROWS, class Src>
__device__ __forceinline__ void in_place_cell(const DevPlan& p, const Src& nbr, const Slots<ROWS>& slots,
                                              const unsigned* __restrict__ hf, int g, bool literal, float ia,
                                              float inv_tau, float dt, const float* f, float* fn) {
  if constexpr (FAST) {
    cell_step_fast<SCHEME>(p, nbr, slots.w, f, fn);
  } else if (literal) {
    Pdfs x;
#pragma unroll
    for (int q = 0; q < Q; ++q) x.f[q] = f[q];
    const Pdfs o = in_place_literal<SCHEME, FV>(p, nbr, hf, g, ia, inv_tau, dt, x);
#pragma unroll
    for (int q = 0; q < Q; ++q) fn[q] = o.f[q];
  } else {
    cell_step<9, SCHEME, 0, FV, false>(p, nbr, slots.w, ia, inv_tau, dt, f, fn);
  }
}

template <int SCHEME, bool FV, bool FAST>
__global__ void __launch_bounds__(IP_THREADS, 1)
    k_resident_in_place(DevPlan p, DevResident r, const float* fin, float* f_prev, float* f_last, int n_steps,
                        unsigned tag) {
  constexpr int ROWS = FAST ? HfFastRows{3, SCHEME}.rows() : ResRows<9, SCHEME, 0>::ROWS;
  extern __shared__ __align__(16) float sm[];
  __shared__ unsigned long long s_bar[2];  // stencils taken; chunk read (a phase per chunk)
  __shared__ int s_bad;                    // 1 + step of a failed wait
  __shared__ int s_nf[3], s_nfx[3];        // a pdf of state s % 3 is not finite: own cells; halo or ghosts
  const int tid = threadIdx.x, T = IP_THREADS, TA = T - r.cell_threads;
  const ResidentBlock b = r.block[blockIdx.x];
  // a batch's case: see k_resident
  const bool retired = p.case_active && !__ldg(p.case_active + b.cs);
  if (retired) n_steps = 1;
  const float inv_tau = p.case_active ? __ldg(p.case_inv_tau + b.cs) : p.inv_tau;
  const float dt = p.case_active ? __ldg(p.case_dt + b.cs) : p.dt;
  const int bnd0 = (b.nin + 31) / 32 * 32, nb = b.nown - b.nin, slots = bnd0 + (nb + 31) / 32 * 32;
  const int sp = (9 * r.stride + 12 * r.max_st), tab = sp + (r.max_table + 3) / 4 * 4;
  float* sprod = sm + 9 * r.stride;  // [max_st][IP_SR]
  float* npdf = sm + tab;            // [max_nodes][Q]
  // the block's node, ghost and import tables, read every step
  int4* t_nd = reinterpret_cast<int4*>(sm + sp);
  float4* t_set = reinterpret_cast<float4*>(t_nd + b.nn);  // {sum of weights, set values, -}
  int4* t_gh = reinterpret_cast<int4*>(t_set + b.nn);
  int2* t_en = reinterpret_cast<int2*>(t_gh + b.ng);  // {stencil index | ND_NEQ_ZERO, weight}
  int* t_st = reinterpret_cast<int*>(t_en + b.ne);
  int* t_ex = t_st + b.nst_own;
  int* t_hs = t_ex + b.nhalo;  // stencil index of a halo cell, -1: none
  float* rows = r.rows + size_t(b.row_off) * IP_ROW;
  const int copy = (slots - bnd0) / 32 * IP_GROUP;
  State state{sm, (bnd0 + b.chunk) / 32 * IP_GROUP, 0, bnd0, 0};
  // rows: halo, ghosts, then twice the interior cells that are read so and the boundary cells
  const int grow = b.nhalo, orow = b.nhalo + b.ng, own_rows = b.nsave + nb;
  const unsigned bar_st = unsigned(__cvta_generic_to_shared(&s_bar[0])), guard = bar_st + 8;

  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_st) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(guard), "r"(r.cell_threads / 32) : "memory");
    s_bad = 0;
    for (int k = 0; k < 3; ++k) s_nf[k] = s_nfx[k] = k == 0 ? 1 : 0;  // the first state is not checked: literal
  }
  // state 0: own and halo cells, frozen nodes
  for (int l = tid; l < slots + b.nhalo; l += T) {
    const bool own = l < slots;
    const int c = own ? __ldg(r.dev + b.own_off + l) : __ldg(r.halo_dev + b.halo_off + l - slots);
    if (c < 0) continue;
    const float* src = fin + cell_base(c, Q);
    float f[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) f[q] = __ldcg(src + q * 32);
    if (own) state.store(l, f);
    if (!own)
      put_row(rows + size_t(l - slots) * IP_ROW, f);
    else if (l >= bnd0)
      put_row(rows + size_t(orow + b.nsave + l - bnd0) * IP_ROW, f);
    else if (const int link = int(__ldg(r.hf + cell_base(b.own_off + l, ROWS)) >> IP_LINK))
      put_row(rows + size_t(orow + link - 1) * IP_ROW, f);
  }
  for (int j = tid; j < b.nn; j += T) {
    int4 nd = r.nd[b.nd_off + j];
    nd.z -= b.en_off;
    t_nd[j] = nd;
    const bool vel = (nd.y & 3) == 1;  // the set values: they do not change
    t_set[j] = make_float4(r.nd_sw[b.nd_off + j], vel ? __ldcg(p.node_vel + nd.x) : __ldcg(p.node_rho + nd.x),
                           vel ? __ldcg(p.node_vel + p.Mp + nd.x) : 0.0f, 0.0f);
  }
  for (int j = tid; j < b.ng; j += T) t_gh[j] = r.gh[b.gh_off + j];
  for (int j = tid; j < b.ne; j += T) t_en[j] = make_int2(int(r.en_st[b.en_off + j]), __float_as_int(r.en_w[b.en_off + j]));
  for (int j = tid; j < b.nst_own; j += T) t_st[j] = __ldg(r.st_loc + b.st_off + j);
  for (int j = tid; j < b.nhalo; j += T) {
    t_ex[j] = __ldg(r.halo_exp + b.halo_off + j);
    t_hs[j] = __ldg(r.halo_st + b.halo_off + j);
  }
  for (int j = tid; j < b.nf; j += T) {
    const int d = __ldg(r.fz_dev + b.fz_off + j);
#pragma unroll
    for (int q = 0; q < Q; ++q) npdf[(b.nn + j) * Q + q] = __ldcg(p.node_pdf + size_t(q) * p.Mp + d);
  }
  __syncthreads();

  // the last two states, and the stencil macros of the last one
  auto finish = [&](int l, const float* f, const float* fn) {
    const int c = __ldg(r.dev + b.own_off + l);
    const size_t o = cell_base(c, Q);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      f_last[o + q * 32] = fn[q];
      if (n_steps > 1) f_prev[o + q * 32] = f[q];
    }
    if (c >= p.stencil_start && c < p.stencil_end) record_stencil(p, c, fn);
  };

  if (tid < TA) {
    const int at = tid;
    for (int s = 0; s < n_steps; ++s, state = state.next(b.chunk, copy)) {
      // macros and f - feq of a stencil cell
      auto stencil = [&](int j, const float* f) {
        float eq[Q], rho, ux, uy;
        macros(f, rho, ux, uy);
        feq9(rho, ux, uy, p, eq);
        float4* o = reinterpret_cast<float4*>(sprod + j * IP_SR);
        o[0] = make_float4(rho, ux, uy, f[0] - eq[0]);
        o[1] = make_float4(f[1] - eq[1], f[2] - eq[2], f[3] - eq[3], f[4] - eq[4]);
        o[2] = make_float4(f[5] - eq[5], f[6] - eq[6], f[7] - eq[7], f[8] - eq[8]);
      };
      for (int j = at; j < b.nst_own; j += TA) {
        float f[Q];
        state.load(t_st[j], f);
        stencil(j, f);
      }
      bar_sync(1, TA);
      if (at == 0) {
        s_nfx[(s + 1) % 3] = 0;
        mbar_arrive(bar_st);
      }
      int nf = 0;
      if (s > 0) {
        const uint4* ex = r.ex + size_t(s & 1) * 3 * r.n_export;
        const unsigned want = tag + unsigned(s);
        for (int j = at; j < b.nhalo; j += TA) {
          const uint4* src = ex + t_ex[j];
          uint4 w[3];
          bool ok = false;
          for (int it = 0; it < RES_POLLS && !ok; ++it) {
#pragma unroll
            for (int k = 0; k < 3; ++k) w[k] = ld_word(src + size_t(k) * r.n_export);
            ok = w[0].w == want && w[1].w == want && w[2].w == want;
            if (!ok && (it & 1023) == 1023 && *reinterpret_cast<volatile int*>(p.status) != 0) break;
          }
          if (!ok) {
            atomicExch(p.status, STATUS_WAIT_TIMEOUT);
            atomicCAS(&s_bad, 0, s + 1);
            break;
          }
          float f[Q], sum = 0.0f;
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            f[q] = __uint_as_float(q % 3 == 0 ? w[q / 3].x : q % 3 == 1 ? w[q / 3].y : w[q / 3].z);
            sum += f[q];
          }
          put_row(rows + size_t(j) * IP_ROW, f);
          if (t_hs[j] >= 0) stencil(t_hs[j], f);
          nf |= !finite(sum);
        }
      } else {
        for (int j = at; j < b.nhalo; j += TA)
          if (t_hs[j] >= 0) {
            const float* row = rows + size_t(j) * IP_ROW;
            float f[Q];
            f[0] = row[8];
#pragma unroll
            for (int q = 1; q < Q; ++q) f[q] = row[q - 1];
            stencil(t_hs[j], f);
          }
      }
      if (b.nn > 0) {
        // nodes: each folds rho, ux, uy, then f - feq by direction over its entries in order
        bar_sync(1, TA);
        for (int m = at; m < b.nn; m += TA) {
          const int4 nd = t_nd[m];
          const float4 set = t_set[m];
          float acc[IP_SR];
#pragma unroll
          for (int i = 0; i < IP_SR; ++i) acc[i] = 0.0f;
          for (int e = 0; e < nd.w; ++e) {
            const int2 en = t_en[nd.z + e];
            const unsigned st = unsigned(en.x);
            const float wt = __int_as_float(en.y);
            const float4* v = reinterpret_cast<const float4*>(sprod + int(st & ~ND_NEQ_ZERO) * IP_SR);
            const float4 v0 = v[0], v1 = v[1], v2 = v[2];
            const float x[IP_SR] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w, v2.x, v2.y, v2.z, v2.w};
#pragma unroll
            for (int i = 0; i < IP_SR; ++i) {
              const float y = ((st & ND_NEQ_ZERO) && i >= 3 ? 0.0f : x[i]) * wt;
              acc[i] = e ? acc[i] + y : y;
            }
          }
          if (nd.y & 4)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              const float z = sprod[b.last_st * IP_SR + i] * 0.0f;
              acc[i] = nd.w ? acc[i] + z : z;
            }
#pragma unroll
          for (int i = 0; i < IP_SR; ++i) acc[i] = acc[i] / set.x;
          const bool vel = (nd.y & 3) == 1;
          const float rho = vel ? acc[0] : set.y, ux = vel ? set.y : acc[1], uy = vel ? set.z : acc[2];
          float eq[Q];
          feq9(rho, ux, uy, p, eq);
          const bool out = s == n_steps - 1 && (nd.y & 8);
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            const float v = eq[q] + acc[3 + q];
            npdf[m * Q + q] = v;
            if (out) p.node_pdf[size_t(q) * p.Mp + nd.x] = v;
          }
          if (out) {
            if (vel) {
              p.node_rho[nd.x] = rho;
            } else {
              p.node_vel[nd.x] = ux;
              p.node_vel[p.Mp + nd.x] = uy;
            }
          }
        }
        bar_sync(1, TA);
      }
      for (int j = at; j < b.ng; j += TA) {
        const int4 g = t_gh[j];
        const float rg = __int_as_float(g.w);
        const float *na = npdf + g.y * Q, *nc = npdf + g.z * Q;
        float f[Q], v[Q], sum = 0.0f;
        state.load(g.x, f);
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          if (FAST) {
            const float mq = (na[q] + nc[q]) * 0.5f;
            v[q] = __fmaf_rn(mq - f[q], rg, mq);
          } else {
            const float mq = (na[q] + nc[q]) / 2.0f;
            v[q] = __fadd_rn(mq, __fmul_rn(__fsub_rn(mq, f[q]), rg));
          }
          sum += v[q];
        }
        put_row(rows + size_t(grow + j) * IP_ROW, v);
        nf |= !finite(sum);
      }
      if (nf) s_nfx[s % 3] = 1;
      bar_sync(1, TA);
      // boundary cells
      const int lit = s_nf[s % 3] | s_nfx[s % 3];
      const bool last = s == n_steps - 1;
      const State out = state.next(b.chunk, copy);
      int nf_new = 0;
      const ScratchSource bs{rows, orow, (s & 1) * own_rows};
      float* brows = rows + size_t(orow + ((s & 1) ^ 1) * own_rows + b.nsave) * IP_ROW;
      uint4* ex = r.ex + size_t((s & 1) ^ 1) * 3 * r.n_export;
      for (int j = at; j < (retired ? 0 : nb); j += TA) {
        const int l = bnd0 + j, g = b.own_off + l;
        Slots<ROWS> cur;
        load_rows(r.hf, g, cur);
        float f[Q], fn[Q], ia = 1.0f;
        state.load(l, f);
        const int exp = int(cur.w[0] >> IP_LINK) - 1;
        if (FV) ia = __ldg(r.inv_area + g);
        in_place_cell<SCHEME, FV, FAST>(p, bs, cur, r.hf, g, lit != 0, ia, inv_tau, dt, f, fn);
        if (exp >= 0 && !last) {
          const unsigned t = tag + unsigned(s + 1);
#pragma unroll
          for (int k = 0; k < 3; ++k)
            st_word(ex + size_t(k) * r.n_export + b.exp_off + exp, fn[3 * k], fn[3 * k + 1], fn[3 * k + 2], t);
        }
        if (!FAST) {
          float sum = 0.0f;
#pragma unroll
          for (int q = 0; q < Q; ++q) sum += fn[q];
          nf_new |= !finite(sum);
        }
        out.store(l, fn);
        put_row(brows + size_t(j) * IP_ROW, fn);
        if (last) finish(l, f, fn);
      }
      if (nf_new) s_nf[(s + 1) % 3] = 1;
      bar_sync(2, T);
      const int bad = *reinterpret_cast<volatile int*>(&s_bad);
      if (bad && bad <= s + 1) return;
    }
  } else {
    const int ct = tid - TA, w0 = ct & ~31;
    const int chunk = b.chunk, K = (b.nin + chunk - 1) / chunk;
    unsigned ph = 0;  // chunks done: phases of the guard
    auto fail = [&](int s) {
      atomicExch(p.status, STATUS_WAIT_TIMEOUT);
      atomicCAS(&s_bad, 0, s + 1);
    };
    for (int s = 0; s < n_steps && !retired; ++s) {
      const int nf_own = *reinterpret_cast<volatile int*>(&s_nf[s % 3]);
      int nf_new = 0;
      const bool last = s == n_steps - 1;
      const StateSource src{state, guard};
      const State out = state.next(b.chunk, copy);
      float* own = rows + size_t(orow + ((s & 1) ^ 1) * own_rows) * IP_ROW;
      for (int k = 0; k < K; ++k) {
        const int l = k * chunk + ct;
        const bool mine = ct < chunk && l < b.nin;
        float fn[Q];
        if (w0 < chunk && k * chunk + w0 < b.nin) {
          float f[Q], ia = 1.0f;
          const int lc = min(l, b.nin - 1), g = b.own_off + lc;
          Slots<ROWS> cur;
          load_rows(r.hf, g, cur);
          if (FV) ia = __ldg(r.inv_area + g);
          state.load(lc, f);
          in_place_cell<SCHEME, FV, FAST>(p, src, cur, r.hf, g, nf_own != 0, ia, inv_tau, dt, f, fn);
          if (!FAST) {
            float sum = 0.0f;
#pragma unroll
            for (int q = 0; q < Q; ++q) sum += fn[q];
            nf_new |= mine && !finite(sum);
          }
          const int row = int(cur.w[0] >> IP_LINK) - 1;
          if (row >= 0 && mine) put_row(own + size_t(row) * IP_ROW, fn);
          if (last && mine) finish(l, f, fn);
        } else {
          src.read();
        }
        // chunk k - 1's old pdfs are read by chunk k at the latest (the first
        // chunk goes to the free part of the ring)
        if (!mbar_wait(guard, ph & 1)) fail(s);
        ++ph;
        if (k == 1 && !mbar_wait(bar_st, unsigned(s & 1))) fail(s);
        if (mine) out.store(l, fn);
      }

      if (nf_new) s_nf[(s + 1) % 3] = 1;
      if (ct == 0) s_nf[(s + 2) % 3] = 0;
      state = out;
      bar_sync(2, T);
      const int bad = *reinterpret_cast<volatile int*>(&s_bad);
      if (bad && bad <= s + 1) return;
    }
    if (retired) bar_sync(2, T);
  }
}

using InPlaceKern = void (*)(DevPlan, DevResident, const float*, float*, float*, int, unsigned);

InPlaceKern pick_in_place(const DevPlan& p) {
  if (p.fast) return k_resident_in_place<0, false, true>;
  return p.fv ? k_resident_in_place<0, true, false> : k_resident_in_place<0, false, false>;
}

}  // namespace

// Threads of a block: the cell warps, then the aux warps.  A chunk takes about as
// long with fewer cell threads (latency) and a round of the aux warps 2-4
// thousand clocks, so half of the threads each; 576 to the cells where that saves
// the largest block a chunk.  us per step (exact, fast; porous, 420k cells): 12.3,
// 11.8 with 768 cell threads, 11.4, 11.1 with 640, 9.9, 8.7 with 576, 10.0, 8.7 with 512, 11.3,
// 8.7 with 384.
void in_place_threads(int max_in, int* cell_threads, int* threads) {
  *cell_threads = (max_in + 575) / 576 < (max_in + 511) / 512 ? 576 : 512;
  *threads = IP_THREADS;
}

cudaError_t prepare_in_place(const DevPlan& p, const ResidentPlan& rp, DevResident& r, bool* fits) {
  *fits = false;
  r.n_blocks = int(rp.block.size());
  r.n_export = rp.n_export;
  r.stride = rp.stride;
  r.max_nodes = rp.max_nodes;
  r.max_st = rp.max_st;
  r.cell_threads = rp.cell_threads;
  r.threads = rp.threads;
  int dev = 0, lim = 0, sms = 0, coop = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  lim -= 1024;  // the static shared memory
  r.max_table = rp.max_table;
  r.smem = sizeof(float) * (size_t(Q) * rp.stride + size_t(IP_SR) * rp.max_st + (rp.max_table + 3) / 4 * 4 + size_t(Q) * rp.max_nodes);
  if (!coop || r.smem > size_t(lim)) return cudaSuccess;
  InPlaceKern k = pick_in_place(p);
  r.kern = reinterpret_cast<const void*>(k);
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, r.threads, r.smem);
  if (e != cudaSuccess) return e;
  *fits = per_sm * sms >= r.n_blocks;
  return cudaSuccess;
}

}  // namespace fvdbm
