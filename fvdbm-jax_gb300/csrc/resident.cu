// Resident step: n steps in one cooperative launch with the state on the
// chip.  Each block owns a compact part of the cells (resident_plan.cpp) whose
// pdfs stay in its shared memory, double-buffered; the face slots, which do
// not change, come through L1/L2.  Per step
//   * the aux warps import the halo cells from the other blocks, then evaluate
//     the boundary nodes that the block's ghost faces read and the ghost
//     values (Nodes.calc_pdfs, src/containers.py:339-404; :280-287);
//   * the cell warps update the cells (src/containers.py:107-121, :191-291),
//     interior ones first: only a group of cells with halo faces, ghost faces
//     or exports waits for the aux warps.  Cells that other blocks import are
//     exported as soon as they are updated.
// An exported cell travels as 16-byte words {three pdfs, tag} written and read
// with one 128-bit access each, so a reader that finds the step's tag has the
// values too: no fence, no flag and no grid barrier, and a block waits only
// for the blocks it borders.  Two exchange buffers alternate: a block writes
// state s + 1 over state s - 1 only after its aux warps have imported state s
// from every block that reads it, which those blocks export after their import of
// s - 1 (every link goes both ways).  The cooperative launch makes all blocks
// resident; a wait that runs out sets the status word and ends the launch.
//
// What bounds it: on small meshes (up to ~400 cells per block) the chain
// import, stencil macros, nodes, ghosts, boundary cells, export of the blocks at the
// boundary, about 6,500 clocks; beyond, the cell warps' issue and shared-memory
// slots.  us per step in runs of 512, per-step launches / here: cavity 3.2k cells 7.3 / 3.3;
// channel with cylinder, 60k, upwind 8.2 / 3.2, Lax-Wendroff 9.9 / 3.4, D2Q13 12.9 / 4.9; porous
// 129k 10.7 / 5.0, 179k 10.5 / 5.6, Lax-Wendroff 204k 14.0 / 6.6, 328k 14.5 / 10.1, D2Q13 179k
// 17.0 / 8.4 (D2Q9 upwind takes resident_in_place.cu from 206k on; two copies there: porous 249k
// 7.9, cavity 251k 5.6).  Tried on meshes of 3.2k to 400k cells: one
// barrier for all warps and the nodes in line with the cells took 1.1 to 1.7 times as
// long, row-wise tables read through L1 each step 1.0 to 1.1 times.
//
// The states are bit for bit those of the same number of single steps: every
// sum and product is that of fvdbm_cell.cuh and d2q13.cuh, element by element.
// Two things are left out while every pdf a block reads is finite, where they
// only add +-0: the rest direction's flux (xi.n = 0) and, upwind, the value on
// the far side of the outflow directions.  A step whose inputs are not all finite
// takes the literal form.
#include <algorithm>

#include "resident.cuh"

namespace fvdbm {

namespace {

// The same in the literal form, out of line (rarely taken).
template <int LAT, int SCHEME, int VARIANT, bool FV>
__device__ __noinline__ void cell_step_literal(const DevPlan& p, const unsigned* __restrict__ hf, int g,
                                               const float* f0, const float* own, float ia, float inv_tau, float dt,
                                               float* out) {
  constexpr int NQ = Lat<LAT>::NQ;
  Slots<ResRows<LAT, SCHEME, VARIANT>::ROWS> s;
  load_rows(hf, g, s);
  float f[NQ], fn[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) f[q] = own[q];
  cell_step<LAT, SCHEME, VARIANT, FV, true>(p, RowSource<NQ>{f0}, s.w, ia, inv_tau, dt, f, fn);
#pragma unroll
  for (int q = 0; q < NQ; ++q) out[q] = fn[q];
}

// ONE: every block has at most one cell per cell thread; its slots and pdfs
// then stay in registers over the steps.
template <int LAT, int SCHEME, int VARIANT, bool FV, bool FAST, bool ONE>
__global__ void __launch_bounds__(ONE ? 640 : 1024, 1)
    k_resident(DevPlan p, DevResident r, const float* fin, float* f_prev, float* f_last, int n_steps, unsigned tag) {
  using L = Lat<LAT>;
  constexpr int NQ = L::NQ, NW = (NQ + 2) / 3, SR = NQ + 4;  // SR: row of sprod (odd)
  constexpr int ROWS = FAST ? HfFastRows{3, SCHEME}.rows() : ResRows<LAT, SCHEME, VARIANT>::ROWS;
  extern __shared__ __align__(16) float sm[];
  __shared__ unsigned long long s_bar[2];  // halo imported, ghosts evaluated
  __shared__ int s_bad;                    // 1 + step of a failed wait
  __shared__ int s_nf[3], s_nfx[3];        // a pdf of state s % 3 is not finite: own cells; halo or ghosts
  const int S = r.stride, tid = threadIdx.x, T = blockDim.x, TC = r.cell_threads, TA = T - TC;
  float* npdf = sm + size_t(2) * NQ * S;           // [max_nodes][NQ]
  float* sprod = npdf + size_t(NQ) * r.max_nodes;  // [max_st][SR]: macros and f - feq of the stencil cells
  const ResidentBlock b = r.block[blockIdx.x];
  // a batch's case: its own constants; the blocks of a retired one only evaluate
  // its nodes, once (no block imports from another case, and both buffers hold
  // its final state)
  const bool retired = p.case_active && !__ldg(p.case_active + b.cs);
  if (retired) n_steps = 1;
  const float inv_tau = p.case_active ? __ldg(p.case_inv_tau + b.cs) : p.inv_tau;
  const float dt = p.case_active ? __ldg(p.case_dt + b.cs) : p.dt;
  // the block's node, ghost and import tables, read every step
  int4* t_nd = reinterpret_cast<int4*>(sm + (size_t(2) * NQ * S + size_t(NQ) * r.max_nodes + size_t(SR) * r.max_st + 3) / 4 * 4);
  float4* t_set = reinterpret_cast<float4*>(t_nd + b.nn);   // {sum of weights, set values, -}
  int4* t_gh = reinterpret_cast<int4*>(t_set + b.nn);
  int2* t_en = reinterpret_cast<int2*>(t_gh + b.ng);        // {stencil index | ND_NEQ_ZERO, weight}
  int* t_st = reinterpret_cast<int*>(t_en + b.ne);
  int* t_ex = t_st + b.nst;
  const int halo0 = (b.nown + 31) / 32 * 32, ghost0 = halo0 + b.nhalo;
  const unsigned bar_halo = unsigned(__cvta_generic_to_shared(&s_bar[0])), bar_ghost = bar_halo + 8;

  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_halo) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_ghost) : "memory");
    s_bad = 0;
    for (int k = 0; k < 3; ++k) s_nf[k] = s_nfx[k] = k == 0 ? 1 : 0;  // the first state is not checked: literal
  }
  // state 0: own and halo cells, frozen nodes
  for (int l = tid; l < b.nown + b.nhalo; l += T) {
    const bool own = l < b.nown;
    const float* s = fin + cell_base(own ? __ldg(r.dev + b.own_off + l) : __ldg(r.halo_dev + b.halo_off + l - b.nown), NQ);
    float* d = sm + (own ? l : halo0 + l - b.nown) * NQ;
#pragma unroll
    for (int q = 0; q < NQ; ++q) d[q] = __ldcg(s + q * 32);
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
  for (int j = tid; j < b.nst; j += T) t_st[j] = r.st_loc[b.st_off + j] * NQ;
  for (int j = tid; j < b.nhalo; j += T) t_ex[j] = r.halo_exp[b.halo_off + j];
  for (int j = tid; j < b.nf; j += T) {
    const int d = __ldg(r.fz_dev + b.fz_off + j);
#pragma unroll
    for (int q = 0; q < NQ; ++q) npdf[(b.nn + j) * NQ + q] = __ldcg(p.node_pdf + size_t(q) * p.Mp + d);
  }
  __syncthreads();

  if (tid < TA) {
    // ---- aux warps (the first ones of the block: they were seen to be served
    // last otherwise, behind every busy cell warp)
    const int at = tid;
    for (int s = 0; s < n_steps; ++s) {
      float* f0 = sm + size_t(s & 1) * NQ * S;
      int nf = 0;
      if (s > 0) {
        const uint4* ex = r.ex + size_t(s & 1) * NW * r.n_export;
        const unsigned want = tag + unsigned(s);
        for (int j = at; j < b.nhalo; j += TA) {
          const uint4* src = ex + t_ex[j];
          uint4 w[NW];
          bool ok = false;
          for (int it = 0; it < RES_POLLS && !ok; ++it) {
            ok = true;
#pragma unroll
            for (int k = 0; k < NW; ++k) w[k] = ld_word(src + size_t(k) * r.n_export);
#pragma unroll
            for (int k = 0; k < NW; ++k) ok = ok && w[k].w == want;
            // (D2Q13: the last word holds one pdf; its spare components carry
            // the tag too, so that every component of the access is used and
            // the compiler cannot narrow it into parts that may tear)
            if (NQ % 3 == 1) ok = ok && w[NW - 1].y == want && w[NW - 1].z == want;
            if (!ok && (it & 1023) == 1023 && *reinterpret_cast<volatile int*>(p.status) != 0) break;
          }
          if (!ok) {
            atomicExch(p.status, STATUS_WAIT_TIMEOUT);
            atomicCAS(&s_bad, 0, s + 1);
            break;
          }
          float sum = 0.0f;
#pragma unroll
          for (int q = 0; q < NQ; ++q) {
            const float v = __uint_as_float(q % 3 == 0 ? w[q / 3].x : q % 3 == 1 ? w[q / 3].y : w[q / 3].z);
            f0[(halo0 + j) * NQ + q] = v;
            sum += v;
          }
          nf |= !finite(sum);
        }
        if (nf) s_nfx[s % 3] = 1;
      }
      // the own cells of this state are complete, and no cell warp still
      // waits for the previous step's phase.  The flag of state s + 1 is cleared
      // before the barrier (state 1's starts clear): a warp sets it while it imports
      // that state, which in a block without nodes and ghosts it may do right after the
      // barrier.  The cell warps read it last for state s - 2, two barriers ago.
      if (s > 0) {
        if (at == 0) s_nfx[(s + 1) % 3] = 0;
        bar_sync(2, T);
      }
      if (at == 0) mbar_arrive(bar_halo);
      if (b.nn > 0) {
        // macros and f - feq of the stencil cells
        for (int j = at; j < b.nst; j += TA) {
          const float* c = f0 + t_st[j];
          float fc[NQ], eq[NQ], rho, ux, uy;
#pragma unroll
          for (int q = 0; q < NQ; ++q) fc[q] = c[q];
          L::macros_(fc, rho, ux, uy);
          L::feq_(rho, ux, uy, p, eq);
          float* o = sprod + j * SR;
          o[0] = rho;
          o[1] = ux;
          o[2] = uy;
#pragma unroll
          for (int q = 0; q < NQ; ++q) o[3 + q] = fc[q] - eq[q];
        }
        bar_sync(1, TA);
        // nodes, 4 lanes each: lane k folds the quantities k, k + 4, ... (rho,
        // ux, uy, then f - feq by direction) over the entries in order
        constexpr int NI = (3 + NQ) / 4;
        const int k = at & 3;
        for (int m0 = (at >> 5) * 8; m0 < b.nn; m0 += TA / 4) {
          const int mi = m0 + ((at >> 2) & 7), m = min(mi, b.nn - 1);
          const int4 nd = t_nd[m];
          const float4 set = t_set[m];
          const int type = nd.y & 3;
          const float sw = set.x;
          float acc[NI];
#pragma unroll
          for (int i = 0; i < NI; ++i) acc[i] = 0.0f;
          for (int e = 0; e < nd.w; ++e) {
            const int2 en = t_en[nd.z + e];
            const unsigned st = unsigned(en.x);
            const float wt = __int_as_float(en.y);
            const float* v = sprod + int(st & ~ND_NEQ_ZERO) * SR + k;
#pragma unroll
            for (int i = 0; i < NI; ++i) {
              const bool zero = (st & ND_NEQ_ZERO) && k + 4 * i >= 3;
              const float x = (zero ? 0.0f : v[4 * i]) * wt;
              acc[i] = e ? acc[i] + x : x;
            }
          }
          if ((nd.y & 4) && k < 3) {
            const float z = sprod[b.last_st * SR + k] * 0.0f;
            acc[0] = nd.w ? acc[0] + z : z;
          }
          float avg[NI];
#pragma unroll
          for (int i = 0; i < NI; ++i) avg[i] = acc[i] / sw;
          const float a0 = __shfl_sync(0xffffffffu, avg[0], 0, 4), a1 = __shfl_sync(0xffffffffu, avg[0], 1, 4);
          const float a2 = __shfl_sync(0xffffffffu, avg[0], 2, 4);
          const float rho = type == 1 ? a0 : set.y, ux = type == 1 ? set.y : a1, uy = type == 1 ? set.z : a2;
          float eq[NQ];
          L::feq_(rho, ux, uy, p, eq);
          if (mi < b.nn) {
            const bool out = s == n_steps - 1 && (nd.y & 8);
#pragma unroll
            for (int i = 0; i < NI; ++i) {
              const int q = k + 4 * i - 3;
              if (q < 0) continue;
              const float e0 = i == 0 ? eq[0] : k == 0 ? eq[4 * i - 3] : k == 1 ? eq[4 * i - 2] : k == 2 ? eq[4 * i - 1] : eq[4 * i];
              const float v = e0 + avg[i];
              npdf[m * NQ + q] = v;
              if (out) p.node_pdf[size_t(q) * p.Mp + nd.x] = v;
            }
            if (out) {
              if (type == 1 && k == 0) p.node_rho[nd.x] = rho;
              if (type != 1 && (k == 1 || k == 2)) p.node_vel[size_t(k - 1) * p.Mp + nd.x] = avg[0];
            }
          }
        }
        bar_sync(1, TA);
      }
      if (b.ng > 0) {
        nf = 0;
        for (int j = at; j < b.ng; j += TA) {
          const int4 g = t_gh[j];
          const float rg = __int_as_float(g.w);
          const float *na = npdf + g.y * NQ, *nb = npdf + g.z * NQ, *fk = f0 + g.x * NQ;
          float* o = f0 + (ghost0 + j) * NQ;
          float sum = 0.0f;
#pragma unroll
          for (int q = 0; q < NQ; ++q) {
            float v;
            if (FAST) {
              const float mq = (na[q] + nb[q]) * 0.5f;
              v = __fmaf_rn(mq - fk[q], rg, mq);
            } else {
              const float mq = (na[q] + nb[q]) / 2.0f;
              v = __fadd_rn(mq, __fmul_rn(__fsub_rn(mq, fk[q]), rg));
            }
            o[q] = v;
            sum += v;
          }
          nf |= !finite(sum);
        }
        if (nf) s_nfx[s % 3] = 1;
        bar_sync(1, TA);
      }
      if (at == 0) mbar_arrive(bar_ghost);
      bar_arrive(3, T);
      const int bad = *reinterpret_cast<volatile int*>(&s_bad);
      if (bad && bad <= s + 1) return;
    }
  } else {
    // ---- cell warps
    const int ct = tid - TA;
    Slots<ROWS> hold;
    float keep[NQ], ia = 1.0f;
    int exp = -1, cls = 0;
    if (ONE) {
      const int g = b.own_off + min(ct, b.nown - 1);
      load_rows(r.hf, g, hold);
      exp = __ldg(r.exp + g);
      cls = __ldg(r.cls + (g >> 5));
      if (FV) ia = __ldg(r.inv_area + g);
#pragma unroll
      for (int q = 0; q < NQ; ++q) keep[q] = sm[(g - b.own_off) * NQ + q];
    }
    for (int s = 0; s < n_steps; ++s) {
      const float* f0 = sm + size_t(s & 1) * NQ * S;
      float* f1 = sm + size_t((s & 1) ^ 1) * NQ * S;
      uint4* ex = r.ex + size_t((s & 1) ^ 1) * NW * r.n_export;
      const int nf_own = *reinterpret_cast<volatile int*>(&s_nf[s % 3]);
      int nf_new = 0;
      for (int l0 = ct & ~31; l0 < (retired ? 0 : b.nown); l0 += TC) {
        const int l = l0 + (tid & 31), g = b.own_off + l;
        if (!ONE) cls = __ldg(r.cls + (g >> 5));
        int nf = nf_own;
        if (cls) {
          if (!mbar_wait(cls == 2 ? bar_ghost : bar_halo, unsigned(s & 1))) {
            atomicExch(p.status, STATUS_WAIT_TIMEOUT);
            atomicCAS(&s_bad, 0, s + 1);
          }
          nf |= *reinterpret_cast<volatile int*>(&s_nfx[s % 3]);
        }
        if (l < b.nown) {
          float f[NQ], fn[NQ];
          if (!ONE) {
            load_rows(r.hf, g, hold);
            exp = __ldg(r.exp + g);
            if (FV) ia = __ldg(r.inv_area + g);
          }
#pragma unroll
          for (int q = 0; q < NQ; ++q) f[q] = ONE ? keep[q] : f0[l * NQ + q];
          if constexpr (FAST) {
            cell_step_fast<SCHEME>(p, RowSource<NQ>{f0}, hold.w, f, fn);
          } else {
            if (nf) {
              cell_step_literal<LAT, SCHEME, VARIANT, FV>(p, r.hf, g, f0, f0 + l * NQ, ia, inv_tau, dt, f1 + l * NQ);
#pragma unroll
              for (int q = 0; q < NQ; ++q) fn[q] = f1[l * NQ + q];
            } else {
              cell_step<LAT, SCHEME, VARIANT, FV, false>(p, RowSource<NQ>{f0}, hold.w, ia, inv_tau, dt, f, fn);
            }
          }
          if (exp >= 0 && s + 1 < n_steps) {
            const float t = __uint_as_float(tag + unsigned(s + 1));
#pragma unroll
            for (int k = 0; k < NW; ++k)
              st_word(ex + size_t(k) * r.n_export + exp, fn[3 * k], 3 * k + 1 < NQ ? fn[(3 * k + 1) % NQ] : t,
                      3 * k + 2 < NQ ? fn[(3 * k + 2) % NQ] : t, tag + unsigned(s + 1));
          }
          float sum = 0.0f;
#pragma unroll
          for (int q = 0; q < NQ; ++q) {
            f1[l * NQ + q] = fn[q];
            if (ONE) keep[q] = fn[q];
            sum += fn[q];
          }
          if (!FAST) nf_new |= !finite(sum);
        }
      }
      if (nf_new) s_nf[(s + 1) % 3] = 1;
      if (ct == 0) s_nf[(s + 2) % 3] = 0;
      bar_sync(3, T);
      const int bad = *reinterpret_cast<volatile int*>(&s_bad);
      if (bad && bad <= s + 1) return;
      if (s + 1 < n_steps) bar_arrive(2, T);
    }
  }
  if (retired) return;
  __syncthreads();

  // the last two states, and the stencil macros of the last one
  const float* fl = sm + size_t(n_steps & 1) * NQ * S;
  const float* fp = sm + size_t((n_steps & 1) ^ 1) * NQ * S;
  for (int l = tid; l < b.nown; l += T) {
    const int c = __ldg(r.dev + b.own_off + l);
    const size_t o = cell_base(c, NQ);
    float fn[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      fn[q] = fl[l * NQ + q];
      f_last[o + q * 32] = fn[q];
    }
    if (n_steps > 1)
#pragma unroll
      for (int q = 0; q < NQ; ++q) f_prev[o + q * 32] = fp[l * NQ + q];
    if constexpr (LAT == 9)
      if (c >= p.stencil_start && c < p.stencil_end) record_stencil(p, c, fn);
  }
}

using ResKern = void (*)(DevPlan, DevResident, const float*, float*, float*, int, unsigned);

template <bool ONE>
ResKern pick(const DevPlan& p) {
  if (p.q == 13) {
    if (p.scheme == 0) return p.fv ? k_resident<13, 0, 0, true, false, ONE> : k_resident<13, 0, 0, false, false, ONE>;
    return p.fv ? k_resident<13, 1, 0, true, false, ONE> : k_resident<13, 1, 0, false, false, ONE>;
  }
  if (p.fast) return p.scheme == 0 ? k_resident<9, 0, 0, false, true, ONE> : k_resident<9, 1, 0, false, true, ONE>;
  if (p.variant == 0) {
    if (p.scheme == 0) return p.fv ? k_resident<9, 0, 0, true, false, ONE> : k_resident<9, 0, 0, false, false, ONE>;
    return p.fv ? k_resident<9, 1, 0, true, false, ONE> : k_resident<9, 1, 0, false, false, ONE>;
  }
  if (p.scheme == 0) return p.fv ? k_resident<9, 0, 1, true, false, ONE> : k_resident<9, 0, 1, false, false, ONE>;
  return p.fv ? k_resident<9, 1, 1, true, false, ONE> : k_resident<9, 1, 1, false, false, ONE>;
}

}  // namespace

// Threads of a block: the cell warps, then the aux warps.
void resident_threads(int max_own, int* cell_threads, int* threads) {
  const int own = (max_own + 31) / 32 * 32;
  const int aux = own <= 512 ? 128 : 256;
  *cell_threads = own <= 512 ? own : std::min(own, 1024 - aux);
  *threads = *cell_threads + aux;
}

cudaError_t prepare_resident(const DevPlan& p, const ResidentPlan& rp, DevResident& r, bool* fits) {
  *fits = false;
  r.n_blocks = int(rp.block.size());
  r.n_export = rp.n_export;
  r.stride = rp.stride;
  r.max_nodes = rp.max_nodes;
  r.max_st = rp.max_st;
  r.cell_threads = rp.cell_threads;
  r.threads = rp.threads;
  r.smem = sizeof(float) * ((size_t(2) * p.q * rp.stride + size_t(p.q) * rp.max_nodes + size_t(4 + p.q) * rp.max_st + 3) / 4 * 4 +
                            rp.max_table);
  int dev = 0, lim = 0, sms = 0, coop = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  lim -= 1024;  // the static shared memory
  if (!coop || r.smem > size_t(lim)) return cudaSuccess;
  ResKern k = rp.max_own <= r.cell_threads && r.threads <= 640 ? pick<true>(p) : pick<false>(p);
  r.kern = reinterpret_cast<const void*>(k);
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, r.threads, r.smem);
  if (e != cudaSuccess) return e;
  *fits = per_sm * sms >= r.n_blocks;
  return cudaSuccess;
}

cudaError_t launch_resident(const DevPlan& p, const DevResident& r, const float* fin, float* f_prev, float* f_last,
                            int n_steps, unsigned tag, cudaStream_t s) {
  DevPlan pp = p;
  DevResident rr = r;
  void* args[] = {&pp, &rr, &fin, &f_prev, &f_last, &n_steps, &tag};
  return cudaLaunchCooperativeKernel(r.kern, dim3(r.n_blocks), dim3(r.threads), args, r.smem, s);
}

}  // namespace fvdbm
