// Fused kernels of the warm-start network's hidden width (64): one pass over
// the cells per layer and direction.  mpnn.cu holds the same quantities as
// separate dense, aggregation and ReLU kernels for any width up to its limits.
//
// A hidden layer is h' = h + relu([h | m] W^T + b) with m = A h, where A's last
// sparse stage (at most a few entries per cell: mesh neighbours, or a cell's bin)
// is gathered while the rows are loaded, so m never goes through memory; the
// backward pass gathers it again, and folds the pending A^T rows of the layer
// above into its load of dh in the same way.  The sign of the pre-activation is
// kept as one bit.
//
// The backward products run on the 5th-generation tensor cores (tcgen05,
// accumulators in tensor memory).  Weights are bfloat16; an FP32 operand x is written as three
// bfloat16 pieces x = p1 + p2 + p3 (p1 = bf16(x), p2 = bf16(x - p1), p3 =
// bf16(x - p1 - p2); the differences are exact), which hold all 24 of its bits,
// so a product with a weight is three exact bf16 products.  Where both operands are FP32
// (the weight gradient) the six products down to 2^-16 relative are kept; the
// rest is below an ulp.  Products are issued from the smallest piece up.  The weight
// gradient's accumulator is drained every tile and summed in FP32 registers:
// the tensor core truncates where it adds, and a chain over a block's thousands of
// cells would drift (each tile's is 24 long: six pairs of pieces by four steps of 16 cells).
//
// Operand tiles are [rows][64] bfloat16 in the 128-byte swizzle (row r's 16-byte
// chunk c at chunk c ^ (r & 7)).  Read along the rows' 64 entries they are the
// K-major operand of dz W; read along the rows (cells) they are the MN-major
// operands of dz^T [h | m], so each tile is written once.
#include <cuda_bf16.h>

#include <algorithm>

#include "../../include/fvdbm_mpnn.h"

namespace fvdbm {
namespace {

constexpr int H = 64;         // hidden width
constexpr int TM = 128;       // cells per tile of the forward pass
constexpr int WT_B = H * 128;     // bytes of one [64][64] bf16 weight tile

__device__ __forceinline__ unsigned smem_addr(const void* p) { return unsigned(__cvta_generic_to_shared(p)); }

// Shared-memory matrix descriptor, 128-byte swizzle.  lbo: between 64-wide
// column groups (MN-major operands; not read for the others); rows in groups of 8 are 1024 bytes.
__device__ __forceinline__ unsigned long long mma_desc(unsigned addr, unsigned lbo) {
  return ((unsigned long long)((addr >> 4) & 0x3fff)) | ((unsigned long long)((lbo >> 4) & 0x3fff) << 16) |
         ((unsigned long long)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor: bf16 x bf16 -> f32; ta/tb: operand is MN-major.
__host__ __device__ constexpr unsigned mma_idesc(int m, int n, int ta, int tb) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (unsigned(ta) << 15) | (unsigned(tb) << 16) | (unsigned(n >> 3) << 17) |
         (unsigned(m >> 4) << 24);
}
__device__ __forceinline__ void mma(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, bool acc) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(unsigned(acc))
      : "memory");
}
__device__ __forceinline__ void mma_commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
template <int N>
__device__ __forceinline__ void tmem_ld(unsigned addr, float (&v)[N]);
template <>
__device__ __forceinline__ void tmem_ld<16>(unsigned addr, float (&v)[16]) {
  unsigned u[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
        "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
      : "r"(addr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(u[i]);
}
__device__ __forceinline__ void tmem_alloc(unsigned* slot, int cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(unsigned base, int cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void bar_init(unsigned bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
// Waits for the barrier's phase, a bounded number of polls.
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity) {
  for (int it = 0; it < (1 << 22); ++it) {
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

// Four values as three bf16 pieces at column 4*c4 of row r of a tile set
// (pieces `step` bytes apart).
__device__ __forceinline__ unsigned pack2(float a, float b) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const unsigned*>(&t);
}
__device__ __forceinline__ void put_pieces(unsigned char* tile, int step, int r, int c4, float4 v) {
  unsigned char* o = tile + r * 128 + (((c4 >> 1) ^ (r & 7)) << 4) + ((c4 & 1) << 3);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const unsigned lo = pack2(v.x, v.y), hi = pack2(v.z, v.w);
    *reinterpret_cast<uint2*>(o + k * step) = make_uint2(lo, hi);
    v.x -= __uint_as_float(lo << 16);
    v.y -= __uint_as_float(lo & 0xffff0000u);
    v.z -= __uint_as_float(hi << 16);
    v.w -= __uint_as_float(hi & 0xffff0000u);
  }
}

// The weights [64][128] as two swizzled tiles (columns of h, columns of m).
__device__ __forceinline__ void put_weights(unsigned char* tile, const uint16_t* __restrict__ w) {
  for (int e = threadIdx.x; e < H * 16; e += blockDim.x) {
    const int o = e >> 4, c = e & 15;  // 16-byte chunk c of row o
    uint4 v;
    uint16_t* p = reinterpret_cast<uint16_t*>(&v);
#pragma unroll
    for (int i = 0; i < 8; ++i) p[i] = w[o * 128 + c * 8 + i];
    *reinterpret_cast<uint4*>(tile + (c >> 3) * WT_B + o * 128 + (((c & 7) ^ (o & 7)) << 4)) = v;
  }
}

// FP32 staging tile [rows][64]: 16-byte chunks swizzled by the row, so that both
// a thread per row and 16 threads per row access it without bank conflicts.
__device__ __forceinline__ float4* stage_at(unsigned char* base, int r, int c4) {
  return reinterpret_cast<float4*>(base + r * 256 + ((c4 ^ (r & 7)) << 4));
}

__device__ __forceinline__ float4 load4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 fma4(float w, float4 x, float4 s) {
  return make_float4(fmaf(w, x.x, s.x), fmaf(w, x.y, s.y), fmaf(w, x.z, s.z), fmaf(w, x.w, s.w));
}
// Columns 4*c4.. of sum_e wt[e] src[col[e]] over row i's entries, in order.
template <int NR>
__device__ __forceinline__ void gather_rows(const int* __restrict__ ptr, const int* __restrict__ col,
                                            const float* __restrict__ wt, const float* __restrict__ src, int row0,
                                            int stride, int n, int c4, float4 (&s)[NR]) {
  int e[NR], end[NR], longest = 0;
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int r = row0 + i * stride;
    s[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    e[i] = r < n ? __ldg(ptr + r) : 0;
    end[i] = r < n ? __ldg(ptr + r + 1) : 0;
    longest = max(longest, end[i] - e[i]);
  }
  for (int k = 0; k < longest; ++k) {
    int c[NR];
    float w[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const bool in = e[i] + k < end[i];
      c[i] = in ? __ldg(col + e[i] + k) : -1;
      w[i] = in ? __ldg(wt + e[i] + k) : 0.0f;
    }
    float4 v[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i)
      if (c[i] >= 0) v[i] = load4(src + size_t(c[i]) * H + 4 * c4);
#pragma unroll
    for (int i = 0; i < NR; ++i)
      if (c[i] >= 0) s[i] = fma4(w[i], v[i], s[i]);
  }
}

// ---------------------------------------------------------------------------
// Forward: z = [h | m] W^T + b for the layers, the encoder (h = x) and the
// decoder.  The products are mpnn.cu's dense kernel's, bit for bit: mma.sync m16n8k8
// TF32 with the FP32 operand split into hi + lo, the same order over k (a
// prediction or a loss does not change with the route that computes it; three
// bf16 pieces on tcgen05 round differently).
// Around them everything is one pass: the rows of h arrive by cp.async, m is gathered
// beside them, the weights wait in shared memory in fragment order (one 16-byte
// load per two column blocks instead of four 2-byte ones and their conversions), and
// a row's fragment is one ldmatrix.  256 threads, 16 rows per warp, two blocks per SM.
// A layer of 500k cells: 119 us (144 with mesh neighbours; tensor pipe 49 % busy
// with the legacy products), as aggregation and dense kernel 517-606.
__device__ __forceinline__ unsigned to_tf32(float x) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

enum { LAYER, ENC, DEC };
constexpr int FT = 256;
// KS: steps of 8 inputs; NB: blocks of 8 outputs
template <int KS>
__host__ __device__ constexpr int row_stride() { return 8 * KS + 4; }  // floats; rows 4 banks apart
template <int KS, int NB>
constexpr int fwd_smem() { return 4 * (TM * row_stride<KS>() + KS * ((NB + 1) / 2) * 32 * 4); }

template <int MODE, int KS, int NB>
__global__ void __launch_bounds__(FT, 2) k_fwd(const float* __restrict__ x, int n, int din,
                                               const int* __restrict__ ptr, const int* __restrict__ col,
                                               const float* __restrict__ wt, const float* __restrict__ src,
                                               const uint16_t* __restrict__ w, const float* __restrict__ bias, int dout,
                                               float* __restrict__ out, unsigned* __restrict__ mask) {
  extern __shared__ __align__(1024) unsigned char sm[];
  constexpr int RS = row_stride<KS>(), NP = (NB + 1) / 2;
  float* xs = reinterpret_cast<float*>(sm);                       // [TM][RS]
  uint4* ws = reinterpret_cast<uint4*>(sm + 4 * TM * RS);         // [KS][NP][32] fragments
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int K = MODE == ENC ? din : 8 * KS;
  // fragment (k step, pair of column blocks, lane): {b0, b1} of both blocks, b0 =
  // W[8j + g][8k + t], b1 = W[8j + g][8k + t + 4]
  for (int e = tid; e < KS * NP * 32; e += FT) {
    const int l = e & 31, jp = (e >> 5) % NP, ks = e / (32 * NP), lg = l >> 2, lt = l & 3;
    unsigned v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int o = 8 * (2 * jp + (i >> 1)) + lg, k = 8 * ks + lt + 4 * (i & 1);
      v[i] = o < dout && k < K ? unsigned(w[size_t(o) * K + k]) << 16 : 0u;
    }
    ws[e] = make_uint4(v[0], v[1], v[2], v[3]);
  }
  if (MODE == ENC)
    for (int e = tid; e < TM * RS; e += FT) xs[e] = 0.0f;  // (the columns past din stay zero)
  __syncthreads();
  const int ntile = (n + TM - 1) / TM;
  for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int row0 = tile * TM;
    if (MODE == ENC) {
      const int lim = min(TM, n - row0) * din;
      for (int e = tid; e < lim; e += FT) xs[e / din * RS + e % din] = x[size_t(row0) * din + e];
    } else {
      const int c4 = tid & 15, r0 = tid >> 4;
#pragma unroll
      for (int i = 0; i < TM / 16; ++i) {
        const int rl = r0 + 16 * i;
        if (row0 + rl < n)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(xs + rl * RS + 4 * c4)),
                       "l"(x + size_t(row0 + rl) * H + 4 * c4)
                       : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (MODE == LAYER) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float4 m[4];
          gather_rows<4>(ptr, col, wt, src, row0 + r0 + 64 * half, 16, n, c4, m);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<float4*>(xs + (r0 + 64 * half + 16 * i) * RS + H + 4 * c4) = m[i];
        }
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    float acc[NB][4];
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[j][r] = 0.0f;
    // ldmatrix: lane l gives the address of row (l & 15), columns 4 * (l >> 4)
    const unsigned abase = smem_addr(xs + (16 * warp + (lane & 15)) * RS + 4 * (lane >> 4));
#pragma unroll 4
    for (int ks = 0; ks < KS; ++ks) {
      unsigned a[4], hi[4], lo[4];
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                   : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
                   : "r"(abase + 32 * ks)
                   : "memory");
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        hi[i] = to_tf32(__uint_as_float(a[i]));
        lo[i] = to_tf32(__uint_as_float(a[i]) - __uint_as_float(hi[i]));
      }
#pragma unroll
      for (int jp = 0; jp < NP; ++jp) {
        const uint4 b = ws[(ks * NP + jp) * 32 + lane];
        mma_tf32(acc[2 * jp], lo, b.x, b.y);
        if (2 * jp + 1 < NB) mma_tf32(acc[(2 * jp + 1) % NB], lo, b.z, b.w);
        mma_tf32(acc[2 * jp], hi, b.x, b.y);
        if (2 * jp + 1 < NB) mma_tf32(acc[(2 * jp + 1) % NB], hi, b.z, b.w);
      }
    }
    // lane (g, t): rows g and g + 8 of the warp's 16, columns 2t, 2t + 1 of a block
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int rl = 16 * warp + g + 8 * half, r = row0 + rl;
      unsigned bits[2] = {0u, 0u};
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const int o = 8 * j + 2 * t;
        if (MODE == DEC) {
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (r < n && o + i < dout) out[size_t(r) * dout + o + i] = acc[j][2 * half + i] + (bias ? bias[o + i] : 0.0f);
          continue;
        }
        const float2 b = bias ? __ldg(reinterpret_cast<const float2*>(bias + o)) : make_float2(0.0f, 0.0f);
        const float z0 = acc[j][2 * half] + b.x, z1 = acc[j][2 * half + 1] + b.y;
        bits[j >> 2] |= ((z0 > 0.0f ? 1u : 0u) | (z1 > 0.0f ? 2u : 0u)) << (8 * (j & 3) + 2 * t);
        float2 y = make_float2(fmaxf(z0, 0.0f), fmaxf(z1, 0.0f));
        if (MODE == LAYER) {
          const float2 res = *reinterpret_cast<const float2*>(xs + rl * RS + o);
          y = make_float2(y.x + res.x, y.y + res.y);
        }
        if (r < n) *reinterpret_cast<float2*>(out + size_t(r) * H + o) = y;
      }
      if (MODE != DEC) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          bits[k] |= __shfl_xor_sync(0xffffffffu, bits[k], 1);
          bits[k] |= __shfl_xor_sync(0xffffffffu, bits[k], 2);
        }
        if (r < n && t < 2) mask[2 * size_t(r) + t] = t ? bits[1] : bits[0];
      }
    }
    __syncthreads();  // the tile is consumed before it is refilled
  }
}

// ---------------------------------------------------------------------------
// Backward.  Tiles of 64 cells, 256 threads, two blocks per SM: a tile is a chain
// (indices, gathered rows, pieces, products, results) beside which the other
// block runs.  Bound by that chain's load latency at 16 warps per SM (2 of 6.8
// TB/s): 183-266 us per layer at 500k cells, where ReLU, weight gradient, data
// gradient and aggregation as separate kernels took 980.  dh and the pending rows
// are loaded before h and m (226-327 us the other way round); one block of 512
// threads and 128 cells took 208-276; an L2 prefetch of the next tile's rows
// changed nothing.  Shared memory: three piece tiles of dz, of h and m (72
// KB), the weights (16 KB); dx is staged over the h and m tiles.  Tensor memory:
// dx = dz W [cell][128] in columns 0-127 (the product has 128 rows; those past
// the 64 cells read whatever follows the tile and are not used), dW^T [128
// inputs][64 outputs] in 128-191.
constexpr int BT = 256, BM = 64, BRW = BM / (BT / 16);
constexpr int BTILE = BM * 128;                       // bytes of one [64][64] bf16 tile
constexpr int X_PIECE = 2 * BTILE;                    // h tile, m tile of one piece
constexpr int B_X = 3 * BTILE;                        // x tiles after the dz pieces
constexpr int B_W = B_X + 3 * X_PIECE;
constexpr int B_SMEM = B_W + 2 * WT_B + 32;

__global__ void __launch_bounds__(BT, 2) k_layer_bwd(float* dh, int n, const int* __restrict__ pptr,
                                                     const int* __restrict__ pcol, const float* __restrict__ pwt,
                                                     const float* __restrict__ psrc, const unsigned* __restrict__ mask,
                                                     const float* __restrict__ h, const int* __restrict__ ptr,
                                                     const int* __restrict__ col, const float* __restrict__ wt,
                                                     const float* __restrict__ src, const uint16_t* __restrict__ w,
                                                     float* __restrict__ dm, float* __restrict__ part) {
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned long long& s_bar = *reinterpret_cast<unsigned long long*>(sm + B_W + 2 * WT_B);
  unsigned& s_tmem = *reinterpret_cast<unsigned*>(sm + B_W + 2 * WT_B + 16);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, c4 = tid & 15;
  if (warp == 0) tmem_alloc(&s_tmem, 256);
  if (tid == 0) bar_init(smem_addr(&s_bar));
  put_weights(sm + B_W, w);
  __syncthreads();
  const unsigned tmem = s_tmem, bar = smem_addr(&s_bar);
  const unsigned a_dz = smem_addr(sm), a_x = a_dz + B_X, a_w = a_dz + B_W;
  const unsigned quarter = (unsigned(warp & 3) * 32) << 16;
  float dw[32];  // dW^T[32 (warp & 3) + lane][32 (warp >> 2) + j]
#pragma unroll
  for (int j = 0; j < 32; ++j) dw[j] = 0.0f;
  float4 db = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const int ntile = (n + BM - 1) / BM;
  unsigned phase = 0;
  bool ok = true;
  for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x, phase ^= 1) {
    const int r0 = tid >> 4, row0 = tile * BM + r0;
    float4 g[BRW];
    unsigned mk[BRW];
#pragma unroll
    for (int i = 0; i < BRW; ++i) {
      const int r = row0 + i * (BT / 16);
      g[i] = r < n ? *reinterpret_cast<const float4*>(dh + size_t(r) * H + 4 * c4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      mk[i] = r < n ? __ldg(mask + 2 * size_t(r) + (c4 >> 3)) >> (4 * (c4 & 7)) : 0u;
    }
    if (psrc) {
      float4 s[BRW];
      gather_rows<BRW>(pptr, pcol, pwt, psrc, row0, BT / 16, n, c4, s);
#pragma unroll
      for (int i = 0; i < BRW; ++i) g[i] = make_float4(g[i].x + s[i].x, g[i].y + s[i].y, g[i].z + s[i].z, g[i].w + s[i].w);
    }
    {
      float4 hv[BRW], m[BRW];
#pragma unroll
      for (int i = 0; i < BRW; ++i) {
        const int r = row0 + i * (BT / 16);
        hv[i] = r < n ? load4(h + size_t(r) * H + 4 * c4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
      gather_rows<BRW>(ptr, col, wt, src, row0, BT / 16, n, c4, m);
#pragma unroll
      for (int i = 0; i < BRW; ++i) {
        put_pieces(sm + B_X, X_PIECE, r0 + i * (BT / 16), c4, hv[i]);
        put_pieces(sm + B_X + BTILE, X_PIECE, r0 + i * (BT / 16), c4, m[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < BRW; ++i) {
      const float4 dz = make_float4(mk[i] & 1u ? g[i].x : 0.0f, mk[i] & 2u ? g[i].y : 0.0f, mk[i] & 4u ? g[i].z : 0.0f,
                                    mk[i] & 8u ? g[i].w : 0.0f);
      put_pieces(sm, BTILE, r0 + i * (BT / 16), c4, dz);
      db = make_float4(db.x + dz.x, db.y + dz.y, db.z + dz.z, db.w + dz.w);
    }
    fence_proxy();
    __syncthreads();
    if (tid == 0) {
      fence_after();
      constexpr unsigned id_dx = mma_idesc(128, 128, 0, 1), id_dw = mma_idesc(128, H, 1, 1);
      for (int piece = 2; piece >= 0; --piece)
#pragma unroll
        for (int k = 0; k < 4; ++k)  // 16 outputs a step: columns of dz, rows of W
          mma(tmem, mma_desc(a_dz + piece * BTILE + k * 32, 16), mma_desc(a_w + k * 2048, WT_B), id_dx,
              !(piece == 2 && k == 0));
      // piece pairs (x, dz) from the smallest product up
      const int px[6] = {2, 1, 0, 1, 0, 0}, pz[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
      for (int t = 0; t < 6; ++t)
#pragma unroll
        for (int k = 0; k < BM / 16; ++k)  // 16 cells a step: rows of both tiles
          mma(tmem + 128, mma_desc(a_x + px[t] * X_PIECE + k * 2048, BTILE), mma_desc(a_dz + pz[t] * BTILE + k * 2048, BTILE),
              id_dw, !(t == 0 && k == 0));
      mma_commit(bar);
    }
    ok = bar_wait(bar, phase) && ok;
    fence_after();
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float v[16];
      tmem_ld<16>(tmem + quarter + 128 + (warp >> 2) * 32 + half * 16, v);
#pragma unroll
      for (int j = 0; j < 16; ++j) dw[half * 16 + j] += v[j];
    }
    if ((warp & 3) < 2) {  // the lanes of the 64 cells; 64 columns each
      unsigned char* st = sm + B_X + (warp >> 2) * BM * 256;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float v[16];
        tmem_ld<16>(tmem + quarter + (warp >> 2) * 64 + q * 16, v);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *stage_at(st, (warp & 3) * 32 + lane, 4 * q + i) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
      }
    }
    fence_before();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < BRW; ++i) {
      const int rl = r0 + i * (BT / 16), r = tile * BM + rl;
      if (r >= n) continue;
      const float4 a = *stage_at(sm + B_X, rl, c4);
      *reinterpret_cast<float4*>(dh + size_t(r) * H + 4 * c4) =
          make_float4(g[i].x + a.x, g[i].y + a.y, g[i].z + a.z, g[i].w + a.w);
      *reinterpret_cast<float4*>(dm + size_t(r) * H + 4 * c4) = *stage_at(sm + B_X + BM * 256, rl, c4);
    }
    __syncthreads();  // the staged rows are consumed before the tiles are refilled
  }
  // this block's partials: dW [64][128] and the column sums of dz
  float* o = part + size_t(blockIdx.x) * (H * 128 + H);
#pragma unroll
  for (int j = 0; j < 32; ++j)
    o[((warp >> 2) * 32 + j) * 128 + (warp & 3) * 32 + lane] = ok ? dw[j] : __int_as_float(0x7fc00000);
  float4* sd = reinterpret_cast<float4*>(sm);
  sd[tid] = db;
  __syncthreads();
  if (tid < 16) {
    float4 s = sd[tid];
    for (int k = 1; k < BT / 16; ++k) {
      const float4 v = sd[tid + 16 * k];
      s = make_float4(s.x + v.x, s.y + v.y, s.z + v.z, s.w + v.w);
    }
    *reinterpret_cast<float4*>(o + H * 128 + 4 * tid) = s;
  }
  if (warp == 0) tmem_free(tmem, 256);
}

// Sums of the block partials in a fixed order: 8 threads per entry take every
// eighth block, then a shuffle tree.
__global__ void __launch_bounds__(256) k_sum_blocks(const float* __restrict__ part, int parts, int E,
                                                    float* __restrict__ dw, float* __restrict__ dbias, int wentries) {
  const int e = blockIdx.x * 32 + (threadIdx.x & 31), s = threadIdx.x >> 5;
  __shared__ float sh[8][32];
  float a = 0.0f;
  if (e < E)
    for (int b = s; b < parts; b += 8) a += part[size_t(b) * E + e];
  sh[s][threadIdx.x & 31] = a;
  __syncthreads();
  if (s == 0 && e < E) {
    for (int k = 1; k < 8; ++k) a += sh[k][threadIdx.x];
    if (e < wentries)
      dw[e] = a;
    else if (dbias)
      dbias[e - wentries] = a;
  }
}

// ---------------------------------------------------------------------------
// Backward of the encoder (DIN features -> 64) and the decoder (64 -> DOUT), a few
// products per value: bound by the 256 bytes per cell of h and dh, so plain FP32
// multiply-adds.  16 threads per cell, 4 columns each.
__device__ __forceinline__ float bf(const uint16_t v) { return __uint_as_float(unsigned(v) << 16); }
constexpr int EMAX = 16, DMAX = 4;

// dW [64][din] and the bias gradient of the encoder: dz = (dh + pending) where
// the mask is set; a thread keeps its 4 columns' sums over its cells.
template <int DIN>  // at least din
__global__ void __launch_bounds__(256, DIN <= 10 ? 2 : 1) k_enc_bwd(const float* __restrict__ dh, int n, const int* __restrict__ pptr,
                                                 const int* __restrict__ pcol, const float* __restrict__ pwt,
                                                 const float* __restrict__ psrc, const unsigned* __restrict__ mask,
                                                 const float* __restrict__ x, int din, float* __restrict__ part) {
  constexpr int NR = 4;
  __shared__ float red[16][H];
  __shared__ float sx[16 * NR][DIN + 1];
  const int tid = threadIdx.x, c4 = tid & 15, rl = tid >> 4;
  float4 s[DIN + 1];  // the last one: the bias
#pragma unroll
  for (int k = 0; k <= DIN; ++k) s[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int r0 = blockIdx.x * 16 * NR; r0 < n; r0 += gridDim.x * 16 * NR) {
    float4 g[NR], p[NR];
    unsigned mk[NR];
    __syncthreads();
    {
      const int lim = min(16 * NR, n - r0) * din;
      for (int q = tid; q < lim; q += 256) sx[q / din][q % din] = x[size_t(r0) * din + q];
    }
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int r = r0 + rl + 16 * i;
      g[i] = r < n ? load4(dh + size_t(r) * H + 4 * c4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      mk[i] = r < n ? __ldg(mask + 2 * size_t(r) + (c4 >> 3)) >> (4 * (c4 & 7)) : 0u;
    }
    if (psrc) {
      gather_rows<NR>(pptr, pcol, pwt, psrc, r0 + rl, 16, n, c4, p);
#pragma unroll
      for (int i = 0; i < NR; ++i) g[i] = make_float4(g[i].x + p[i].x, g[i].y + p[i].y, g[i].z + p[i].z, g[i].w + p[i].w);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NR; ++i) {  // (rows past n: dz = 0)
      const float4 dz = make_float4(mk[i] & 1u ? g[i].x : 0.0f, mk[i] & 2u ? g[i].y : 0.0f, mk[i] & 4u ? g[i].z : 0.0f,
                                    mk[i] & 8u ? g[i].w : 0.0f);
#pragma unroll
      for (int k = 0; k < DIN; ++k)
        if (k < din && r0 + rl + 16 * i < n) s[k] = fma4(sx[rl + 16 * i][k], dz, s[k]);
      s[DIN] = make_float4(s[DIN].x + dz.x, s[DIN].y + dz.y, s[DIN].z + dz.z, s[DIN].w + dz.w);
    }
  }
  float* o = part + size_t(blockIdx.x) * (H * din + H);
#pragma unroll
  for (int k = 0; k <= DIN; ++k) {
    if (k >= din && k < DIN) continue;
    __syncthreads();
    *reinterpret_cast<float4*>(&red[rl][4 * c4]) = s[k];
    __syncthreads();
    if (tid < H) {
      float a = red[0][tid];
      for (int j = 1; j < 16; ++j) a += red[j][tid];
      o[k < DIN ? tid * din + k : H * din + tid] = a;
    }
  }
}

// Decoder backward in one pass: dh = dy W, and dW [dout][64], db.
__global__ void __launch_bounds__(256) k_dec_bwd(const float* __restrict__ dy, const float* __restrict__ h, int n,
                                                 const uint16_t* __restrict__ w, int dout, float* __restrict__ dh,
                                                 float* __restrict__ part) {
  __shared__ float red[16][H];
  const int tid = threadIdx.x, c4 = tid & 15, rl = tid >> 4;
  float4 wv[DMAX], s[DMAX];
  float db[DMAX];
#pragma unroll
  for (int o = 0; o < DMAX; ++o) {
    const uint16_t* p = w + o * H + 4 * c4;
    wv[o] = o < dout ? make_float4(bf(p[0]), bf(p[1]), bf(p[2]), bf(p[3])) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    s[o] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    db[o] = 0.0f;
  }
  constexpr int NR = 4;
  for (int r0 = blockIdx.x * 16 * NR; r0 < n; r0 += gridDim.x * 16 * NR) {
    float4 v[NR];
    float g[NR][DMAX];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int r = r0 + rl + 16 * i;
      v[i] = r < n ? load4(h + size_t(r) * H + 4 * c4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
      for (int o = 0; o < DMAX; ++o) g[i][o] = r < n && o < dout ? __ldg(dy + size_t(r) * dout + o) : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int r = r0 + rl + 16 * i;
      float4 d = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
      for (int o = 0; o < DMAX; ++o) {
        d = fma4(g[i][o], wv[o], d);
        s[o] = fma4(g[i][o], v[i], s[o]);
        db[o] += g[i][o];
      }
      if (r < n) *reinterpret_cast<float4*>(dh + size_t(r) * H + 4 * c4) = d;
    }
  }
  float* out = part + size_t(blockIdx.x) * (dout * H + dout);
#pragma unroll
  for (int o = 0; o < DMAX; ++o) {
    if (o >= dout) break;
    __syncthreads();
    *reinterpret_cast<float4*>(&red[rl][4 * c4]) = s[o];
    __syncthreads();
    if (tid < H) {
      float a = red[0][tid];
      for (int j = 1; j < 16; ++j) a += red[j][tid];
      out[o * H + tid] = a;
    }
    __syncthreads();
    if (c4 == 0) red[0][rl] = db[o];
    __syncthreads();
    if (tid == 0) {
      float a = red[0][0];
      for (int j = 1; j < 16; ++j) a += red[0][j];
      out[dout * H + o] = a;
    }
  }
}

int sms() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}
int grid_of(int n, int rows, int cap) { return std::max(1, std::min((n + rows - 1) / rows, cap)); }
bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
template <int MODE, int KS, int NB>
int launch_fwd(const float* x, int n, int din, const int* ptr, const int* col, const float* wt, const float* src,
               const uint16_t* w, const float* bias, int dout, float* out, unsigned* mask, void* stream) {
  if (n == 0) return 0;
  auto kern = k_fwd<MODE, KS, NB>;
  constexpr int smem = fwd_smem<KS, NB>();
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -2;
  kern<<<grid_of(n, TM, 2 * sms()), FT, smem, static_cast<cudaStream_t>(stream)>>>(x, n, din, ptr, col, wt, src, w, bias,
                                                                                 dout, out, mask);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
int layer_grid(int n) { return grid_of(n, BM, 2 * sms()); }
int enc_grid(int n) { return grid_of(n, 64, 4 * sms()); }

}  // namespace
}  // namespace fvdbm

using namespace fvdbm;

extern "C" {

int fvdbm_mp_layer_fwd(const float* h, int32_t n, const int32_t* row_ptr, const int32_t* col, const float* wt,
                       const float* src, const uint16_t* w, const float* bias, float* hout, uint32_t* mask,
                       void* stream) {
  if (n < 0 || !h || !row_ptr || !col || !wt || !src || !w || !hout || !mask || !al16(h) || !al16(src) || !al16(bias) ||
      !al16(hout))
    return -1;
  return launch_fwd<LAYER, 16, 8>(h, n, H, row_ptr, col, wt, src, w, bias, H, hout, mask, stream);
}

size_t fvdbm_mp_fused_scratch(int32_t n) {
  return sizeof(float) * std::max(size_t(layer_grid(n)) * (H * 128 + H), size_t(enc_grid(n)) * (H * EMAX + H));
}

int fvdbm_mp_layer_bwd(float* dh, int32_t n, const int32_t* pend_ptr, const int32_t* pend_col, const float* pend_wt,
                       const float* pend_src, const uint32_t* mask, const float* h, const int32_t* row_ptr,
                       const int32_t* col, const float* wt, const float* src, const uint16_t* w, float* dm, float* dw,
                       float* dbias, float* scratch, size_t scratch_bytes, void* stream) {
  if (n <= 0 || !dh || !mask || !h || !row_ptr || !col || !wt || !src || !w || !dm || !dw || !scratch ||
      (pend_src && (!pend_ptr || !pend_col || !pend_wt)) || !al16(dh) || !al16(h) || !al16(src) || !al16(dm) ||
      !al16(pend_src) || dm == pend_src || !al16(scratch) || scratch_bytes < fvdbm_mp_fused_scratch(n))
    return -1;
  if (cudaFuncSetAttribute(k_layer_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, B_SMEM) != cudaSuccess) return -2;
  const int g = layer_grid(n), E = H * 128 + H;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  k_layer_bwd<<<g, BT, B_SMEM, s>>>(dh, n, pend_ptr, pend_col, pend_wt, pend_src, mask, h, row_ptr, col, wt, src, w, dm,
                                    scratch);
  k_sum_blocks<<<(E + 31) / 32, 256, 0, s>>>(scratch, g, E, dw, dbias, H * 128);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int fvdbm_mp_enc_fwd(const float* x, int32_t n, int32_t din, const uint16_t* w, const float* bias, float* h,
                     uint32_t* mask, void* stream) {
  if (n < 0 || din <= 0 || din > EMAX || !x || !w || !h || !mask || !al16(bias) || !al16(h)) return -1;
  return launch_fwd<ENC, 2, 8>(x, n, din, nullptr, nullptr, nullptr, nullptr, w, bias, H, h, mask, stream);
}

int fvdbm_mp_enc_bwd(const float* dh, int32_t n, const int32_t* pend_ptr, const int32_t* pend_col,
                     const float* pend_wt, const float* pend_src, const uint32_t* mask, const float* x, int32_t din,
                     float* dw, float* dbias, float* scratch, size_t scratch_bytes, void* stream) {
  if (n <= 0 || din <= 0 || din > EMAX || !dh || !mask || !x || !dw || !scratch ||
      (pend_src && (!pend_ptr || !pend_col || !pend_wt)) || !al16(dh) || !al16(pend_src) ||
      scratch_bytes < fvdbm_mp_fused_scratch(n))
    return -1;
  const int g = enc_grid(n), E = H * din + H;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  auto kern = din <= 10 ? k_enc_bwd<10> : k_enc_bwd<EMAX>;
  kern<<<g, 256, 0, s>>>(dh, n, pend_ptr, pend_col, pend_wt, pend_src, mask, x, din, scratch);
  k_sum_blocks<<<(E + 31) / 32, 256, 0, s>>>(scratch, g, E, dw, dbias, H * din);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int fvdbm_mp_dec_fwd(const float* h, int32_t n, const uint16_t* w, const float* bias, int32_t dout, float* y,
                     void* stream) {
  if (n < 0 || dout <= 0 || dout > DMAX || !h || !w || !y || !al16(h)) return -1;
  return launch_fwd<DEC, 8, 1>(h, n, H, nullptr, nullptr, nullptr, nullptr, w, bias, dout, y, nullptr, stream);
}

int fvdbm_mp_dec_bwd(const float* dy, const float* h, int32_t n, const uint16_t* w, int32_t dout, float* dh, float* dw,
                     float* dbias, float* scratch, size_t scratch_bytes, void* stream) {
  if (n <= 0 || dout <= 0 || dout > DMAX || !dy || !h || !w || !dh || !dw || !scratch || !al16(h) || !al16(dh) ||
      scratch_bytes < fvdbm_mp_fused_scratch(n))
    return -1;
  const int g = enc_grid(n), E = dout * H + dout;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  k_dec_bwd<<<g, 256, 0, s>>>(dy, h, n, w, dout, dh, scratch);
  k_sum_blocks<<<(E + 31) / 32, 256, 0, s>>>(scratch, g, E, dw, dbias, dout * H);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // extern "C"
