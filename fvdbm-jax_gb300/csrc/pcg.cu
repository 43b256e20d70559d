// Jacobi-preconditioned conjugate gradients on the GPU: the potential-flow
// estimate of the warm start's features solves a cell Laplacian per case
// (all held-out cases together as one block-diagonal system).  No
// counterpart in the reference.
//
// Vectors are float32.  Every dot product is summed by each thread in
// float32 (multiply-adds; the rows of a thread are few) and then in double
// over the block and over the blocks in block order by one block, so an
// iteration is bitwise reproducible (float64 arithmetic is slow on this GPU,
// so it is kept to the reductions).  The scalars of the recurrence (alpha,
// beta, r.z) stay on the device; the host reads ||r||^2 every check_every
// iterations to stop.
//
// Recurrence (Saad, Iterative Methods for Sparse Linear Systems, 2nd ed.,
// Algorithm 9.1, with M = diag(A)):
//   r = b - A x, z = M^-1 r, p = z
//   repeat: q = A p; alpha = (r.z)/(p.q); x += alpha p; r -= alpha q;
//           z = M^-1 r; beta = (r.z)_new/(r.z); p = z + beta p
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "fvdbm.h"
#include "fvdbm_mpnn.h"

namespace {

constexpr int PT = 256;       // threads per block
constexpr int PB_MAX = 1216;  // blocks of the vector kernels (8 per SM of a 152-SM GB300, at most)

// scalar slots (double) at the start of the work buffer
enum { S_RZ = 0, S_RR, S_BB, S_PQ, S_ALPHA, S_BETA, S_COUNT = 8 };

// Row i of A times x, in entry order (column indices outside [0, n) are
// skipped, so a malformed matrix cannot read out of bounds).
__device__ __forceinline__ float row_dot(int n, const int* __restrict__ ip, const int* __restrict__ ix,
                                         const float* __restrict__ v, const float* __restrict__ x, int i) {
  float s = 0.0f;
  for (int e = ip[i]; e < ip[i + 1]; ++e) {
    const int c = ix[e];
    if (unsigned(c) < unsigned(n)) s += v[e] * x[c];
  }
  return s;
}

// Sum of up to 3 doubles over the block in a fixed order; thread 0 writes them.
template <int K>
__device__ __forceinline__ void block_sum_store(double v[K], double* __restrict__ out) {
  __shared__ double sh[PT / 32][K];
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) sh[w][k] = v[k];
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double s = sh[0][k];
      for (int j = 1; j < PT / 32; ++j) s += sh[j][k];
      out[k] = s;
    }
}

// diag^-1 (1 where the row has no positive diagonal), r = b - A x, z = r/diag,
// p = z; partials (r.z, r.r, b.b)
__global__ void __launch_bounds__(PT) k_init(int n, const int* __restrict__ ip, const int* __restrict__ ix,
                                            const float* __restrict__ v, const float* __restrict__ b,
                                            const float* __restrict__ x, float* __restrict__ dinv,
                                            float* __restrict__ r, float* __restrict__ z, float* __restrict__ p,
                                            double* __restrict__ part) {
  float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f;
  for (int i = blockIdx.x * PT + threadIdx.x; i < n; i += gridDim.x * PT) {
    float d = 0.0f;
    for (int e = ip[i]; e < ip[i + 1]; ++e)
      if (ix[e] == i) d += v[e];
    const float di = d > 0.0f ? 1.0f / d : 1.0f;
    const float ri = b[i] - row_dot(n, ip, ix, v, x, i);
    const float zi = ri * di;
    dinv[i] = di;
    r[i] = ri;
    z[i] = zi;
    p[i] = zi;
    a0 = __fmaf_rn(ri, zi, a0);
    a1 = __fmaf_rn(ri, ri, a1);
    a2 = __fmaf_rn(b[i], b[i], a2);
  }
  double acc[3] = {a0, a1, a2};
  block_sum_store<3>(acc, part + size_t(blockIdx.x) * 3);
}

// q = A p; partial p.q
__global__ void __launch_bounds__(PT) k_spmv(int n, const int* __restrict__ ip, const int* __restrict__ ix,
                                            const float* __restrict__ v, const float* __restrict__ p,
                                            float* __restrict__ q, double* __restrict__ part) {
  float a0 = 0.0f;
  for (int i = blockIdx.x * PT + threadIdx.x; i < n; i += gridDim.x * PT) {
    const float qi = row_dot(n, ip, ix, v, p, i);
    q[i] = qi;
    a0 = __fmaf_rn(p[i], qi, a0);
  }
  double acc[1] = {a0};
  block_sum_store<1>(acc, part + size_t(blockIdx.x) * 3);
}

// One block: sums the k-th partial of every block in block order.
// mode 0 (after init): rz, rr, bb.  mode 1: pq and alpha = rz / pq.
// mode 2: beta = rz_new / rz, rz = rz_new, rr.
__global__ void __launch_bounds__(PT) k_scalars(int nblk, const double* __restrict__ part, double* __restrict__ s,
                                               int mode) {
  double acc[3] = {0.0, 0.0, 0.0};
  for (int j = threadIdx.x; j < nblk; j += PT)
#pragma unroll
    for (int k = 0; k < 3; ++k) acc[k] += part[size_t(j) * 3 + k];
  __shared__ double tot[3];
  block_sum_store<3>(acc, tot);
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (mode == 0) {
    s[S_RZ] = tot[0];
    s[S_RR] = tot[1];
    s[S_BB] = tot[2];
  } else if (mode == 1) {
    s[S_PQ] = tot[0];
    s[S_ALPHA] = tot[0] != 0.0 ? s[S_RZ] / tot[0] : 0.0;
  } else {
    s[S_BETA] = s[S_RZ] != 0.0 ? tot[0] / s[S_RZ] : 0.0;
    s[S_RZ] = tot[0];
    s[S_RR] = tot[1];
  }
}

// x += alpha p; r -= alpha q; z = r/diag; partials (r.z, r.r)
__global__ void __launch_bounds__(PT) k_update(int n, const double* __restrict__ s, const float* __restrict__ p,
                                              const float* __restrict__ q, const float* __restrict__ dinv,
                                              float* __restrict__ x, float* __restrict__ r, float* __restrict__ z,
                                              double* __restrict__ part) {
  const float a = float(s[S_ALPHA]);
  float a0 = 0.0f, a1 = 0.0f;
  for (int i = blockIdx.x * PT + threadIdx.x; i < n; i += gridDim.x * PT) {
    x[i] = __fmaf_rn(a, p[i], x[i]);
    const float ri = __fmaf_rn(-a, q[i], r[i]);
    const float zi = ri * dinv[i];
    r[i] = ri;
    z[i] = zi;
    a0 = __fmaf_rn(ri, zi, a0);
    a1 = __fmaf_rn(ri, ri, a1);
  }
  double acc[3] = {a0, a1, 0.0};
  block_sum_store<3>(acc, part + size_t(blockIdx.x) * 3);
}

// p = z + beta p
__global__ void __launch_bounds__(PT) k_direction(int n, const double* __restrict__ s, const float* __restrict__ z,
                                                 float* __restrict__ p) {
  const float bt = float(s[S_BETA]);
  for (int i = blockIdx.x * PT + threadIdx.x; i < n; i += gridDim.x * PT) p[i] = __fmaf_rn(bt, p[i], z[i]);
}

// ---------------------------------------------------------------------------
// The whole solve in one cooperative launch, for systems of at most PB_MAX
// blocks of PT rows (every thread of the launch-per-kernel form then has one
// row).  Each block owns the rows of a few of those PT-row groups and keeps
// their x, r, q, dinv, z and p in registers; the other blocks' directions are read
// through L2: p_new = z + beta p_old is formed again by every reader, so an
// iteration has two exchanges, p.q and (r.z, r.r), instead of five launches.
// An exchange doubles as the grid barrier: a block publishes the partial sums of
// its groups as 16-byte words {double, tag}, each one 128-bit access, and
// every block collects all of them.  Sums run in the order of the kernels above
// (group partials by the same tree, then k_scalars' order), so the iterates
// are the same bits.  Waits are bounded (other work on the GPU may keep a block
// from starting): one that runs out sets *fail and ends the launch, whose solution
// is then not taken (it waits in the rows' words) and the kernels above solve the system.
constexpr int PV = 4;                  // row groups a block works on side by side (PV * PT threads)
constexpr int PCG_POLLS = 1 << 20;     // of one wait (about a second)

__device__ __forceinline__ bool get_word(const uint4* ptr, unsigned tag, double* v) {
  unsigned long long a, b;
  asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
               : "=l"(a), "=l"(b)
               : "l"(ptr)
               : "memory");
  *v = __longlong_as_double((long long)a);
  // (both halves of the second word carry the tag: every part of the access is used)
  return unsigned(b) == tag && unsigned(b >> 32) == tag;
}
// Waits for the row's word of iteration `tag` (bounded).
__device__ __forceinline__ bool get_row(const uint4* ptr, unsigned tag, int polls, float* z, float* p) {
  for (int it = 0; it < polls; ++it) {
    double v;
    if (get_word(ptr, tag, &v)) {
      const unsigned long long a = (unsigned long long)__double_as_longlong(v);
      *z = __uint_as_float(unsigned(a));
      *p = __uint_as_float(unsigned(a >> 32));
      return true;
    }
  }
  return false;
}
__device__ __forceinline__ void put_word(uint4* ptr, unsigned tag, double v) {
  const unsigned long long a = (unsigned long long)__double_as_longlong(v), b = tag | ((unsigned long long)tag << 32);
  asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(ptr), "l"(a), "l"(b)
               : "memory");
}

__device__ __forceinline__ void put_row(uint4* ptr, unsigned tag, float z, float p) {
  put_word(ptr, tag, __longlong_as_double((long long)(__float_as_uint(z) | ((unsigned long long)__float_as_uint(p) << 32))));
}

struct SolveArgs {
  int n, groups, per_block, max_iter, check_every, polls;
  double rtol;
  const int *ip, *ix;
  const float *v, *b, *x;
  uint4* zp;    // [n]: {z, p of the iteration before, tag, tag}; out: {x, -, -, -}
  uint4* ex;    // [2][3][groups]: the exchange words of even and odd exchanges
  double* s;    // out: S_RZ, S_RR, S_BB
  int* fail;    // out: {a wait ran out, iterations}
};

__device__ __forceinline__ void pcg_bar(int n) { asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory"); }

// The five levels of a warp's shuffle tree over `chunks` runs of 32 values at
// stride 32 of d (in place; the sums end at each run's first entry), with the
// adds of all runs packed into full warps: double adds run at about 2 per clock
// and SM here, whether or not a warp's lanes are needed (per lane, as the kernels
// above form them, they took 3/4 of an iteration).  Two levels per barrier.
template <bool ALL>
__device__ __forceinline__ void packed_tree(double* d, int chunks, int nt) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 2) {  // lanes l + {0, o, 2o, 3o}, l < o: levels 2o and o
    const int sh = o == 8 ? 3 : 1;
    for (int t = threadIdx.x; t < (chunks << sh); t += nt) {
      double* c = d + (t >> sh) * 32 + (t & (o - 1));
      c[0] = (c[0] + c[2 * o]) + (c[o] + c[3 * o]);
    }
    if (ALL)
      __syncthreads();
    else
      pcg_bar(nt);
  }
}

// The tree's last level of a group's runs, and their sum in order.
__device__ __forceinline__ double run_sum(const double* c) {
  double v[PT / 32];
#pragma unroll
  for (int j = 0; j < PT / 32; ++j) v[j] = c[32 * j] + c[32 * j + 1];
  double s = v[0];
#pragma unroll
  for (int j = 1; j < PT / 32; ++j) s += v[j];
  return s;
}

// One exchange of K sums: part[g][k] are this block's group partials in shared
// memory; tot receives the totals over all groups, summed as k_scalars does, and
// tot[K] the recurrence's quotient: alpha = rz / tot[0] (K = 1) or beta =
// tot[0] / rz (K = 2).
template <int K>
__device__ __forceinline__ bool exchange(const SolveArgs& a, double (*part)[3], int g0, int ng, unsigned tag,
                                         double* d, double rz, double* tot, int* s_ok) {
  constexpr int NWD = 4;  // words per thread, at most: 3 * 1216 groups over 1024 threads
  __shared__ double s_tot[4];
  __shared__ int s_go;
  __syncthreads();
  uint4* ex = a.ex + size_t(tag & 1) * 3 * a.groups;
  const int tid = threadIdx.x, nt = blockDim.x, words = K * a.groups;
  if (tid < ng * K) put_word(ex + size_t(tid % K) * a.groups + g0 + tid / K, tag, part[tid / K][tid % K]);
  double v[NWD];
  bool all = false;
  for (int it = 0; it < a.polls && !all; ++it) {
    all = true;
#pragma unroll
    for (int i = 0; i < NWD; ++i)
      if (tid + i * nt < words) all &= get_word(ex + tid + i * nt, tag, &v[i]);
  }
  if (!all) *s_ok = 0;
#pragma unroll
  for (int i = 0; i < NWD; ++i)
    if (tid + i * nt < words) d[tid + i * nt] = v[i];
  __syncthreads();
  if (tid < PT) {
    double acc[K];
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k] = 0.0;
    for (int j = tid; j < a.groups; j += PT)
#pragma unroll
      for (int k = 0; k < K; ++k) acc[k] += d[k * a.groups + j];
    pcg_bar(PT);
#pragma unroll
    for (int k = 0; k < K; ++k) d[k * PT + tid] = acc[k];
    pcg_bar(PT);
    packed_tree<false>(d, K * (PT / 32), PT);
    if (tid < K) {
      const double s = run_sum(d + tid * PT);
      s_tot[tid] = s;
      // (one thread divides: 1024 would take 7,000 clocks)
      if (tid == 0 && K == 1) s_tot[1] = s != 0.0 ? rz / s : 0.0;
      if (tid == 0 && K == 2) s_tot[2] = rz != 0.0 ? s / rz : 0.0;
      if (tid == 0) s_go = *s_ok;  // (one answer for the block: a thread that is ahead may clear *s_ok again)
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k <= (K < 3 ? K : 2); ++k) tot[k] = s_tot[k];
  if (!s_go && tid == 0) atomicExch(a.fail, 1);
  return s_go != 0;
}

template <int R>
__global__ void __launch_bounds__(PV* PT, 1) k_solve(SolveArgs a) {
  constexpr int NG = PV * R;
  extern __shared__ double d[];  // [3][NG * PT] tree values
  __shared__ double part[NG][3];
  __shared__ int s_ok;
  const int tid = threadIdx.x, lg = tid / PT, nlg = blockDim.x / PT;
  const int g0 = blockIdx.x * a.per_block, ng = min(a.per_block, a.groups - g0);
  if (tid == 0) s_ok = 1;
  int row[R];
  float x[R], r[R], z[R], p[R], q[R], dinv[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int lgi = lg + i * nlg, rr = (g0 + lgi) * PT + (tid & (PT - 1));
    row[i] = lgi < ng && rr < a.n ? rr : -1;
  }
  // the group partials of K quantities from the rows' float products, summed
  // by block_sum_store's tree
  auto reduce = [&](float (*f)[3], int K) {
#pragma unroll
    for (int i = 0; i < R; ++i)
      for (int k = 0; k < K; ++k)
        if (lg + i * nlg < ng) d[(k * ng + lg + i * nlg) * PT + (tid & (PT - 1))] = f[i][k];
    __syncthreads();
    packed_tree<true>(d, K * ng * (PT / 32), blockDim.x);
    if (tid < ng * K) part[tid / K][tid % K] = run_sum(d + (tid % K * ng + tid / K) * PT);
  };
  float f[R][3];
  // the first four entries of each row stay in registers
  int col[R][4], rest[R], end[R];
  float w[R][4];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    rest[i] = end[i] = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      col[i][k] = -1;
      w[i][k] = 0.0f;
    }
    if (row[i] < 0) continue;
    end[i] = a.ip[row[i] + 1];
    rest[i] = a.ip[row[i]] + 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int e = rest[i] - 4 + k;
      if (e < end[i] && unsigned(a.ix[e]) < unsigned(a.n)) {
        col[i][k] = a.ix[e];
        w[i][k] = a.v[e];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    f[i][0] = f[i][1] = f[i][2] = 0.0f;
    x[i] = r[i] = z[i] = p[i] = q[i] = 0.0f;
    dinv[i] = 1.0f;
    if (row[i] < 0) continue;
    const int c = row[i];
    float d = 0.0f;
    for (int e = a.ip[c]; e < a.ip[c + 1]; ++e)
      if (a.ix[e] == c) d += a.v[e];
    dinv[i] = d > 0.0f ? 1.0f / d : 1.0f;
    x[i] = a.x[c];
    r[i] = a.b[c] - row_dot(a.n, a.ip, a.ix, a.v, a.x, c);
    z[i] = r[i] * dinv[i];
    p[i] = z[i];
    put_row(a.zp + c, 1, z[i], 0.0f);
    f[i][0] = __fmaf_rn(r[i], z[i], 0.0f);
    f[i][1] = __fmaf_rn(r[i], r[i], 0.0f);
    f[i][2] = __fmaf_rn(a.b[c], a.b[c], 0.0f);
  }
  reduce(f, 3);
  unsigned tag = 1;
  double tot[3];
  bool ok = exchange<3>(a, part, g0, ng, tag, d, 0.0, tot, &s_ok);
  double rz = tot[0], rr = tot[1];
  const double bb = tot[2], bn = bb > 0.0 ? bb : 1.0;
  double rel = rr > 0.0 ? sqrt(rr / bn) : 0.0;
  int it = 0;
  float bt = 0.0f;  // float(beta) of the direction that is formed next
  while (ok && it < a.max_iter && rel > a.rtol) {
    const int steps = min(a.max_iter - it, a.check_every);
    for (int j = 0; j < steps && ok; ++j) {
      // p of this iteration: stored already at the start, else z + beta p
      const bool first = it == 0 && j == 0;
      const unsigned ztag = unsigned(it + j) + 1;
      // direction of row c
      auto dir = [&](int c) {
        float zc = 0.0f, pc = 0.0f;
        if (!get_row(a.zp + c, ztag, a.polls, &zc, &pc)) s_ok = 0;
        return first ? zc : __fmaf_rn(bt, pc, zc);
      };
      float t[R][4];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (!first) p[i] = __fmaf_rn(bt, p[i], z[i]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int c = col[i][k];
          t[i][k] = c < 0 ? 0.0f : c == row[i] ? p[i] : dir(c);
        }
      }
#pragma unroll
      for (int i = 0; i < R; ++i) {
        float s = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (col[i][k] >= 0) s = __fadd_rn(s, __fmul_rn(w[i][k], t[i][k]));
        for (int e = rest[i]; e < end[i]; ++e) {  // rows of more than four entries
          const int c = __ldg(a.ix + e);
          if (unsigned(c) < unsigned(a.n)) s = __fadd_rn(s, __fmul_rn(__ldg(a.v + e), c == row[i] ? p[i] : dir(c)));
        }
        q[i] = s;
        f[i][0] = row[i] < 0 ? 0.0f : __fmaf_rn(p[i], s, 0.0f);
        f[i][1] = f[i][2] = 0.0f;
      }
      reduce(f, 1);
      ok = exchange<1>(a, part, g0, ng, ++tag, d, rz, tot, &s_ok);
      const float al = float(tot[1]);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        f[i][0] = f[i][1] = f[i][2] = 0.0f;
        if (row[i] < 0) continue;
        x[i] = __fmaf_rn(al, p[i], x[i]);
        r[i] = __fmaf_rn(-al, q[i], r[i]);
        z[i] = r[i] * dinv[i];
        put_row(a.zp + row[i], ztag + 1, z[i], p[i]);
        f[i][0] = __fmaf_rn(r[i], z[i], 0.0f);
        f[i][1] = __fmaf_rn(r[i], r[i], 0.0f);
      }
      reduce(f, 2);
      ok = ok && exchange<2>(a, part, g0, ng, ++tag, d, rz, tot, &s_ok);
      bt = float(tot[2]);
      rz = tot[0];
      rr = tot[1];
    }
    it += steps;
    rel = rr > 0.0 ? sqrt(rr / bn) : 0.0;
    if (!(rel == rel)) break;
  }
#pragma unroll
  for (int i = 0; i < R; ++i)
    if (row[i] >= 0) reinterpret_cast<float*>(a.zp + row[i])[0] = x[i];  // (no block reads it after the last exchange)
  if (blockIdx.x == 0 && tid == 0) {
    a.s[S_RZ] = rz;
    a.s[S_RR] = rr;
    a.s[S_BB] = bb;
    a.fail[1] = it;
  }
}

// x from the rows' words when every wait of the solve was met
__global__ void __launch_bounds__(PT) k_take(int n, const int* __restrict__ fail, const uint4* __restrict__ zp,
                                            float* __restrict__ x) {
  const int i = blockIdx.x * PT + threadIdx.x;
  if (i < n && !*fail) x[i] = __uint_as_float(zp[i].x);
}

int grid_blocks(int n) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int g = (n + PT - 1) / PT;
  const int cap = sms > 0 ? sms * 8 : PB_MAX;
  if (g > cap) g = cap;
  if (g > PB_MAX) g = PB_MAX;
  return g < 1 ? 1 : g;
}

size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

}  // namespace

extern "C" size_t fvdbm_pcg_work_bytes(int32_t n) {
  if (n < 0) return 0;
  return align256(S_COUNT * sizeof(double)) + align256(size_t(PB_MAX) * 3 * sizeof(double)) +
         5 * align256(size_t(n) * sizeof(float));
}

extern "C" int fvdbm_pcg(int32_t n, const int32_t* indptr, const int32_t* indices, const float* values,
                         const float* b, float* x, int32_t max_iter, double rtol, int32_t check_every, void* work,
                         size_t work_bytes, void* stream, int32_t* iters, double* rel_res) {
  return fvdbm_pcg_bounded(n, indptr, indices, values, b, x, max_iter, rtol, check_every, PCG_POLLS, work, work_bytes,
                           stream, iters, rel_res);
}

extern "C" int fvdbm_pcg_bounded(int32_t n, const int32_t* indptr, const int32_t* indices, const float* values,
                                 const float* b, float* x, int32_t max_iter, double rtol, int32_t check_every,
                                 int32_t polls, void* work, size_t work_bytes, void* stream, int32_t* iters,
                                 double* rel_res) {
  if (iters) *iters = 0;
  if (rel_res) *rel_res = 0.0;
  if (n < 0 || max_iter < 0 || check_every <= 0 || polls < 0 || polls > PCG_POLLS || !(rtol >= 0.0)) return FVDBM_EINVAL;
  if (n == 0) return FVDBM_OK;
  if (!indptr || !indices || !values || !b || !x || !work || work_bytes < fvdbm_pcg_work_bytes(n))
    return FVDBM_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  char* w = static_cast<char*>(work);
  double* s = reinterpret_cast<double*>(w);
  w += align256(S_COUNT * sizeof(double));
  double* part = reinterpret_cast<double*>(w);
  w += align256(size_t(PB_MAX) * 3 * sizeof(double));
  float* vec[5];
  for (int k = 0; k < 5; ++k) {
    vec[k] = reinterpret_cast<float*>(w);
    w += align256(size_t(n) * sizeof(float));
  }
  float *dinv = vec[0], *r = vec[1], *z = vec[2], *p = vec[3], *q = vec[4];
  const int g = grid_blocks(n);
  // one launch for the whole solve while every thread has one row and the
  // row groups fit the blocks (227k rows: 37 us per iteration as five
  // launches, 14.7 in one, of which the double sums' latency is about half);
  // larger systems stream their vectors
  {
    int dev = 0, sms = 0, coop = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    const int groups = (n + PT - 1) / PT, per_block = sms > 0 ? (groups + sms - 1) / sms : 0;
    if (coop && groups <= g && per_block >= 1 && per_block <= 2 * PV && (reinterpret_cast<uintptr_t>(work) & 15) == 0) {
      const int blocks = (groups + per_block - 1) / per_block, threads = PT * (per_block < PV ? per_block : PV);
      void (*kern)(SolveArgs) = per_block <= PV ? k_solve<1> : k_solve<2>;
      const size_t smem = sizeof(double) * 3 * size_t(per_block) * PT;
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(double) * 6 * PV * PT)) !=
              cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) != cudaSuccess)
        return FVDBM_ECUDA;
      if (per_sm * sms >= blocks) {
        // (the exchange words, 96 bytes per 256 rows, fit in one of the five
        // vectors, the rows' words in the four after it)
        SolveArgs a{n, groups, per_block, max_iter, check_every, polls, rtol, indptr, indices, values, b, x,
                    reinterpret_cast<uint4*>(r), reinterpret_cast<uint4*>(dinv), s, reinterpret_cast<int*>(s + S_COUNT)};
        void* args[] = {&a};
        struct {
          double s[S_COUNT];
          int fail[2];
        } out;
        if (cudaMemsetAsync(s, 0, sizeof(out), st) != cudaSuccess ||
            cudaMemsetAsync(a.ex, 0, size_t(6) * groups * sizeof(uint4), st) != cudaSuccess ||
            cudaMemsetAsync(a.zp, 0, size_t(n) * sizeof(uint4), st) != cudaSuccess ||
            cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern), dim3(blocks), dim3(threads), args,
                                        smem, st) != cudaSuccess)
          return FVDBM_ECUDA;
        k_take<<<groups, PT, 0, st>>>(n, a.fail, a.zp, x);
        if (cudaGetLastError() != cudaSuccess ||
            cudaMemcpyAsync(&out, s, sizeof(out), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
          return FVDBM_ECUDA;
        if (!out.fail[0]) {
          const double bn = out.s[S_BB] > 0.0 ? out.s[S_BB] : 1.0;
          if (iters) *iters = out.fail[1];
          if (rel_res) *rel_res = out.s[S_RR] > 0.0 ? std::sqrt(out.s[S_RR] / bn) : 0.0;
          return FVDBM_OK;
        }
      }
    }
  }
  double* hs = nullptr;
  if (cudaMallocHost(reinterpret_cast<void**>(&hs), 3 * sizeof(double)) != cudaSuccess) return FVDBM_ECUDA;
  int rc = FVDBM_OK;
  int it = 0;
  double rel = 0.0;
  auto read_rr = [&]() -> bool {
    if (cudaMemcpyAsync(hs, s, 3 * sizeof(double), cudaMemcpyDeviceToHost, st) != cudaSuccess) return false;
    return cudaStreamSynchronize(st) == cudaSuccess;
  };
  k_init<<<g, PT, 0, st>>>(n, indptr, indices, values, b, x, dinv, r, z, p, part);
  k_scalars<<<1, PT, 0, st>>>(g, part, s, 0);
  if (cudaGetLastError() != cudaSuccess || !read_rr()) {
    rc = FVDBM_ECUDA;
  } else {
    const double bn = hs[S_BB] > 0.0 ? hs[S_BB] : 1.0;
    rel = hs[S_RR] > 0.0 ? std::sqrt(hs[S_RR] / bn) : 0.0;
    while (it < max_iter && rel > rtol) {
      const int k = (max_iter - it) < check_every ? (max_iter - it) : check_every;
      for (int j = 0; j < k; ++j) {
        k_spmv<<<g, PT, 0, st>>>(n, indptr, indices, values, p, q, part);
        k_scalars<<<1, PT, 0, st>>>(g, part, s, 1);
        k_update<<<g, PT, 0, st>>>(n, s, p, q, dinv, x, r, z, part);
        k_scalars<<<1, PT, 0, st>>>(g, part, s, 2);
        k_direction<<<g, PT, 0, st>>>(n, s, z, p);
      }
      it += k;
      if (cudaGetLastError() != cudaSuccess || !read_rr()) {
        rc = FVDBM_ECUDA;
        break;
      }
      rel = hs[S_RR] > 0.0 ? std::sqrt(hs[S_RR] / bn) : 0.0;
      if (!(rel == rel)) break;  // NaN: not SPD or bad input; reported through rel_res
    }
  }
  cudaFreeHost(hs);
  if (iters) *iters = it;
  if (rel_res) *rel_res = rel;
  return rc;
}
