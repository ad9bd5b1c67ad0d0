// Chunked gated delta rule without gradients (scoring, prefill, the first pass of a rematerialised layer).
//
// Reference: crates/ferrl/src/gdn.rs - gated_delta_rule_chunked :451-556, which composes it from ~40 tensor ops per chunk.
//
// Per head and chunk of 64 tokens, with raw 16-bit rows k, q, v, their L2 factors kn, qn (qn with 1/sqrt(128)), the
// cumulative log decay G and gamma = exp(G):
//   A_ij = beta_i kn_i kn_j exp(G_i - G_j) <k_i, k_j>  (i > j),   T = (I + A)^-1
//   P_ij = qn_i kn_j exp(G_i - G_j) <q_i, k_j>         (i >= j)
//   R  = beta (v - gamma kn (k S)),   Vn = T R,   O = gamma qn (q S) + P Vn
//   S' = gamma_C S + k^T (kn exp(G_C - G) Vn)
// The L2 factors multiply rows of products instead of the rows themselves, so k and q enter every product as the exact
// 16-bit values that they are.  The other operands (T, P, S, R, Vn) are 32-bit: each is the exact sum of three 16-bit
// pieces (8 + 8 + 8 bits of the fraction), and the products of pieces down to 2^-24 of the whole are kept - three with k
// or q, six between two of them - so the tensor cores give what 32-bit multiply-adds give.  The leading products and
// the small ones have accumulators of their own, which keeps the chain that rounds at the leading size short.
//
//   gdn_chunk_prep_kernel   one CTA per (chunk, head): T and P as pieces, the row factors
//   gdn_chunk_scan_kernel   one CTA per head: chunks in order, the state in registers and, as pieces, in tensor memory
//
// The scan on warp-level products, two CTAs a head (four where they all ran at once), took 9 us a chunk, bound by issuing the
// products and their fragments: 5119 tokens x 48 heads 549 us, 4 x 2047 x 48 677 (a round of 26 chunks), 1024 x 16 73.  On
// tcgen05 with the state as an operand in tensor memory: 321, 295 and 69 us, 4 us a chunk.  A chunk is a chain of four
// products, 3300 cycles of the tensor cores' time, with the threads' work between them: 5500 cycles, of which splitting an
// entry into pieces takes 10 a pair of warps (28 with shifts and conversions of its own, 13 with cut-off pieces).  The state's
// distance from float64 is 1.2e-7 to 1.7e-7 (2-norm), as it was.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../api.h"
#include "../common.cuh"
#include "../gemm/tc_common.cuh"
#include "mma_sync.cuh"

namespace ferrl {
namespace {

using namespace mmah;
constexpr int GC = 64;                       // chunk length
constexpr int GD = 128;                      // key and value head dim
constexpr int NTH = 256;
constexpr int PIECE = GC * GC;               // entries of one piece of T or P
constexpr int VEC = 5;                       // row factors: beta, beta gamma kn, gamma qn, kn exp(G_C - G), [gamma_C]
constexpr uint32_t TILE = GC * GC * 2;       // bytes of a [64, 64] 16-bit tile

// x - the upper or lower half of a pair of 16-bit values, in one instruction
template <bool UPPER>
__device__ __forceinline__ float less(uint32_t pair, float x) {
  float d;
  if constexpr (UPPER)
    asm("{.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %1;\n\tfma.rn.f32.bf16 %0, hi, %2, %3;}" : "=f"(d) : "r"(pair), "h"(static_cast<unsigned short>(0xBF80)), "f"(x));
  else
    asm("{.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %1;\n\tfma.rn.f32.bf16 %0, lo, %2, %3;}" : "=f"(d) : "r"(pair), "h"(static_cast<unsigned short>(0xBF80)), "f"(x));
  return d;
}
// pieces of two neighbouring entries: x = h + m + l
__device__ __forceinline__ void split3(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16(x, y);
  x = less<false>(h, x);
  y = less<true>(h, y);
  m = pack_bf16(x, y);
  l = pack_bf16(less<false>(m, x), less<true>(m, y));
}

struct ChunkArgs {
  const __nv_bfloat16 *q, *k, *v;
  long long q_bs, q_ts, k_bs, k_ts, v_bs, v_ts;
  const float *g, *beta;
  int T, Hk, Hv, c0, n;                      // chunks c0 .. c0 + n of every row
  __nv_bfloat16* pieces;                     // [B * Hv, n, 6, 64, 64]: T then P, rows swizzled as the products read them
  float* vec;                                // [B * Hv, n, VEC, 64]
  int* status;
};

// entry (i, c) of a piece: rows of 128 bytes, 16-byte chunks exchanged within groups of eight rows
__device__ __forceinline__ int piece_at(int i, int c) { return i * GC + (((c >> 3) ^ (i & 7)) << 3) + (c & 7); }

// Shared: k, q [64, 256 bytes] swizzled, later the pieces of P, then of T; A, T [64, 68]; G (two floats), kn, qn, beta [64].
//
// T comes from its 16 x 16 diagonal blocks, each by substitution, a thread a column, and from products: with
// [[T0, 0], [-T1 A10 T0, T1]] pairs of blocks become one, twice.  By substitution over all 64 rows, on 64 threads, it was 13 of
// the block's 31 thousand cycles, the L2 factors (a warp a row) 7 thousand and stores of single words 6 thousand.
// 5119 tokens x 48 heads: 167 -> 120 us, a chunk of one head 13 -> 8.
constexpr int LA = GC + 4;
constexpr size_t kPrepSmem = 2 * GC * GD * 2 + (2 * GC * LA + 5 * GC) * sizeof(float);

__global__ void __launch_bounds__(NTH, 3)
gdn_chunk_prep_kernel(ChunkArgs a, int l2norm, float eps) {
  extern __shared__ __align__(128) unsigned char sm8[];
  const uint32_t ks = smem_addr(sm8), qs = ks + GC * GD * 2;
  float* A = reinterpret_cast<float*>(sm8 + 2 * GC * GD * 2);
  float* Ts = A + GC * LA;
  float *Gs = Ts + GC * LA, *Gl = Gs + GC, *kn = Gl + GC, *qn = kn + GC, *bs = qn + GC;
  const int ci = blockIdx.x % a.n, bh = blockIdx.x / a.n, b = bh / a.Hv, hv = bh % a.Hv;
  pdl_trigger();                             // the scan sets up while the last of these run
  const int hk = hv / (a.Hv / a.Hk), t0 = (a.c0 + ci) * GC, n = min(GC, a.T - t0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < 2 * GC * 16; e += NTH) {
    const int which = e >> 10, r = (e >> 4) & 63, c = e & 15;
    const __nv_bfloat16* src = which ? a.q + b * a.q_bs + (t0 + min(r, n - 1)) * a.q_ts : a.k + b * a.k_bs + (t0 + min(r, n - 1)) * a.k_ts;
    cp_async16((which ? qs : ks) + sw_off<256>(r, c), src + hk * GD + c * 8, r < n);
  }
  cp_commit();
  const long long go = (static_cast<long long>(b) * a.T + t0) * a.Hv + hv;
  if (tid < GC) bs[tid] = tid < n ? a.beta[go + static_cast<long long>(tid) * a.Hv] : 0.f;
  if (warp == 2) {                           // inclusive scan of 64 log decays, kept as two floats: differences of large sums matter
    const double a0 = 2 * lane < n ? a.g[go + static_cast<long long>(2 * lane) * a.Hv] : 0.f;
    const double a1 = 2 * lane + 1 < n ? a.g[go + static_cast<long long>(2 * lane + 1) * a.Hv] : 0.f;
    double sum = a0 + a1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double t = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += t;
    }
    const double even = sum - a1;
    Gs[2 * lane + 1] = static_cast<float>(sum);
    Gl[2 * lane + 1] = static_cast<float>(sum - Gs[2 * lane + 1]);
    Gs[2 * lane] = static_cast<float>(even);
    Gl[2 * lane] = static_cast<float>(even - Gs[2 * lane]);
  }
  cp_wait<0>();
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {              // L2 factors: eight threads a row of k, then of q
    const int r = i * 32 + (tid >> 3);
    float sum = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 w = *reinterpret_cast<const uint4*>(sm8 + (r >> 6) * GC * GD * 2 + sw_off<256>(r & 63, h * 8 + (tid & 7)));
      const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x = __uint_as_float(u[e] << 16), y = __uint_as_float(u[e] & 0xFFFF0000u);
        sum += x * x + y * y;
      }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float f = l2norm ? rsqrtf(sum + eps) : 1.f;
    if ((tid & 7) == 0) (r < GC ? kn : qn)[r & 63] = r < GC ? f : f * rsqrtf(static_cast<float>(GD));
  }
  // <k_i, k_j> and <q_i, k_j>: a warp has 16 rows and 32 columns of both
  const int mt = warp >> 1, nh = warp & 1;
  float kk[4][4] = {}, qk[4][4] = {};
#pragma unroll
  for (int s = 0; s < GD / 16; ++s) {
    uint32_t fa[4], fq[4], fb[4][2];
    const int ar = mt * 16 + (lane & 15), ac = 2 * s + (lane >> 4);
    ldsm4(ks + sw_off<256>(ar, ac), fa[0], fa[1], fa[2], fa[3]);
    ldsm4(qs + sw_off<256>(ar, ac), fq[0], fq[1], fq[2], fq[3]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {            // 16 columns: rows of k, k16 of the head dim
      const int br = nh * 32 + j * 16 + (lane & 7) + ((lane >> 4) << 3), bc = 2 * s + ((lane >> 3) & 1);
      ldsm4(ks + sw_off<256>(br, bc), fb[2 * j][0], fb[2 * j][1], fb[2 * j + 1][0], fb[2 * j + 1][1]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      mma16816(kk[j], fa, fb[j][0], fb[j][1]);
      mma16816(qk[j], fq, fb[j][0], fb[j][1]);
    }
  }
  __syncthreads();                           // kn, qn; k and q are read
  const long long co = static_cast<long long>(bh) * a.n + ci;
  __nv_bfloat16 *pc = a.pieces + co * 6 * PIECE, *stage = reinterpret_cast<__nv_bfloat16*>(sm8);
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = mt * 16 + (lane >> 2) + 8 * h, c = nh * 32 + j * 8 + (lane & 3) * 2;
      float p[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float d = i >= c + e ? __expf((Gs[i] - Gs[c + e]) + (Gl[i] - Gl[c + e])) * kn[c + e] : 0.f;
        p[e] = qk[j][2 * h + e] * (qn[i] * d);
        A[i * LA + c + e] = i > c + e ? kk[j][2 * h + e] * (bs[i] * kn[i] * d) : 0.f;
      }
      uint32_t w[3];
      split3(p[0], p[1], w[0], w[1], w[2]);
#pragma unroll
      for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(stage + s * PIECE + piece_at(i, c)) = w[s];
    }
  const float glast = Gs[GC - 1], llast = Gl[GC - 1];
  if (tid < GC) {
    const float gamma = __expf(Gs[tid] + Gl[tid]);
    float* vp = a.vec + co * VEC * GC + tid;
    vp[0] = bs[tid];
    vp[GC] = bs[tid] * gamma * kn[tid];
    vp[2 * GC] = gamma * qn[tid];
    vp[3 * GC] = kn[tid] * __expf((glast - Gs[tid]) + (llast - Gl[tid]));
    vp[4 * GC] = __expf(glast + llast);
  }
  tc::fence_async_smem();
  __syncthreads();
  if (tid == 0) {
    tc::bulk_store(pc + 3 * PIECE, stage, 3 * PIECE * 2);
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
  if (warp >= 4 && lane < 16) {              // column `lane` of a diagonal block: t[i] = [i == lane] - sum_{j<i} A[i][j] t[j]
    const float* D = A + (warp - 4) * 16 * (LA + 1);
    float t[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float a0 = (i == lane) ? 1.f : 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
      for (int j = 0; j + 3 < i; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(D + i * LA + j);
        a0 -= x.x * t[j];
        a1 -= x.y * t[j + 1];
        a2 -= x.z * t[j + 2];
        a3 -= x.w * t[j + 3];
      }
#pragma unroll
      for (int j = i & ~3; j < i; ++j) a0 -= D[i * LA + j] * t[j];
      t[i] = (a0 + a1) + (a2 + a3);
      Ts[(warp - 4) * 16 * (LA + 1) + i * LA + lane] = t[i];
    }
  }
  __syncthreads();
  // a row of one operand with N columns of the other, k0 .. k1; the products on their way lie where T has its zeros
  {                                          // blocks 0 and 1, 2 and 3: a thread has two columns
    const int o = (tid >> 7) * 32 * (LA + 1), r = (tid >> 3) & 15, c = (tid & 7) * 2;
    auto product = [&](const float* x, const float* y) {
      float2 acc = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        const float4 u = *reinterpret_cast<const float4*>(x + j);
        const float w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 z = *reinterpret_cast<const float2*>(y + (j + e) * LA);
          acc.x += w[e] * z.x;
          acc.y += w[e] * z.y;
        }
      }
      return acc;
    };
    *reinterpret_cast<float2*>(Ts + o + r * LA + 16 + c) = product(A + o + (16 + r) * LA, Ts + o + c);
    __syncthreads();
    const float2 x = product(Ts + o + (16 + r) * LA + 16, Ts + o + 16 + c);
    *reinterpret_cast<float2*>(Ts + o + (16 + r) * LA + c) = make_float2(-x.x, -x.y);
  }
  __syncthreads();
  {                                          // rows 32 on, columns up to 32: a thread has four columns
    const int r = tid >> 3, c = (tid & 7) * 4;
    auto product = [&](const float* x, const float* y, int j0, int j1) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int j = j0; j < j1; j += 4) {
        const float4 u = *reinterpret_cast<const float4*>(x + j);
        const float w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float4 z = *reinterpret_cast<const float4*>(y + (j + e) * LA);
          acc.x += w[e] * z.x;
          acc.y += w[e] * z.y;
          acc.z += w[e] * z.z;
          acc.w += w[e] * z.w;
        }
      }
      return acc;
    };
    // the columns from 16 on meet zeros above (products of the step before, not to be read), the rows below 16 likewise
    *reinterpret_cast<float4*>(Ts + r * LA + 32 + c) = product(A + (32 + r) * LA, Ts + c, c & 16, 32);
    __syncthreads();
    const float4 x = product(Ts + (32 + r) * LA + 32, Ts + 32 + c, 0, (r & 16) + 16);
    *reinterpret_cast<float4*>(Ts + (32 + r) * LA + c) = make_float4(-x.x, -x.y, -x.z, -x.w);
  }
  if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  __syncthreads();                           // T is whole, the pieces of P are on their way to memory
  for (int e = tid; e < PIECE / 2; e += NTH) {
    const int i = e >> 5, c = (e & 31) * 2;
    const float2 x = c >> 4 <= i >> 4 ? *reinterpret_cast<const float2*>(Ts + i * LA + c) : make_float2(0.f, 0.f);
    uint32_t w[3];
    split3(x.x, x.y, w[0], w[1], w[2]);
#pragma unroll
    for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(stage + s * PIECE + piece_at(i, c)) = w[s];
  }
  tc::fence_async_smem();
  __syncthreads();
  if (tid == 0) {
    tc::bulk_store(pc, stage, 3 * PIECE * 2);
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
}

// The scan.  Everything is transposed: a lane of tensor memory is a value column, so the state, R and Vn are operands that
// the products read from tensor memory, written there by the threads that own the column, and k, q, T and P are the
// operands in shared memory.  All 512 columns (32 bits each) are taken, X = 192 and Y = 320 changing places from chunk to
// chunk; leading and small parts of a sum are 64 columns apart where nothing else is said:
//   [0, 192) [448, 512)   pieces of the state; then Vn; then the state's increment, leading [0, 128), small [128, 192) [448, 512)
//   X, 128 columns        k S; then pieces of R; then of the scaled Vn; then P Vn
//   Y, 128 columns        q S; then pieces of Vn
// A warp has 32 value columns and one half of the tokens (of the key dim, in the state): it alone reads and writes its
// parts of these, so pieces may lie over the sums that they were made of.
constexpr int CW = 8;                        // computing warps; one issues the products, three copy
constexpr uint32_t KQ = 4 * TILE;            // k then q of a chunk, each as two tiles of 64 of the key dim
constexpr uint32_t VT = GC * GD * 2;         // v of a chunk, rows as they are; then O
constexpr uint32_t kScanTiles = 2 * KQ + 2 * 6 * TILE + 3 * VT;
constexpr uint32_t kScanSmem = kScanTiles + 2 * VEC * GC * sizeof(float) + 20 * sizeof(uint64_t);
constexpr uint32_t kMnMajorB = 1u << 16;     // operand B of a product lies with its columns, not its contraction, in rows
constexpr uint32_t TM = 0;                   // tensor memory that is all of one block's starts at its first column

__device__ __forceinline__ void tmem_st8(uint32_t at, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(at), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// pieces of 32 entries of a lane: 16 columns each
__device__ __forceinline__ void put_pieces(const float* x, uint32_t at_h, uint32_t at_m, uint32_t at_l) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    uint32_t h[8], m[8], l[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) split3(x[16 * i + 2 * e], x[16 * i + 2 * e + 1], h[e], m[e], l[e]);
    tmem_st8(at_h + 8 * i, h);
    tmem_st8(at_m + 8 * i, m);
    tmem_st8(at_l + 8 * i, l);
  }
}
// leading + small part of 32 columns
__device__ __forceinline__ void read_sums(uint32_t hi, uint32_t lo, float* x) {
  uint32_t c[32];
  tc::tmem_ld32(hi, reinterpret_cast<uint32_t*>(x));
  tc::tmem_ld32(lo, c);
  tc::tmem_ld_wait();
#pragma unroll
  for (int e = 0; e < 32; ++e) x[e] += __uint_as_float(c[e]);
}

__global__ void __launch_bounds__((CW + 4) * 32, 1)
gdn_chunk_scan_kernel(ChunkArgs a, const float* S0, float* S_out, __nv_bfloat16* __restrict__ out) {
  using namespace tc;
  extern __shared__ __align__(1024) unsigned char scan_sm[];
  unsigned char *kq = scan_sm, *tp = scan_sm + 2 * KQ, *vs = tp + 2 * 6 * TILE;
  float* vec = reinterpret_cast<float*>(scan_sm + kScanTiles);
  uint64_t* bars = reinterpret_cast<uint64_t*>(vec + 2 * VEC * GC);
  // T and P, and the rows and factors of a chunk, are here
  uint64_t *tp_full = bars, *row_full = bars + 2;
  // halves of the state's pieces, R's, the scaled Vn's, Vn's, O in v's place, O's sums read
  uint64_t *s_full = bars + 4, *r_full = bars + 6, *w_full = bars + 7, *v_full = bars + 8, *o_full = bars + 9, *o_read = bars + 11;
  uint64_t *ks_done = bars + 12, *qs_done = bars + 13, *vn_done = bars + 14, *inc_done = bars + 15, *o_done = bars + 16;
  uint64_t* o_taken = bars + 18;             // the copying warps have read O out of v's place
  uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 19);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(slot + 1);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bh = blockIdx.x, b = bh / a.Hv, hv = bh % a.Hv, hk = hv / (a.Hv / a.Hk);
  if (smem_u32(scan_sm) & 1023) {            // the swizzled tiles start on a 1024-byte boundary, the same in every thread
    if (tid == 0) atomicCAS(a.status, kStatusOk, kStatusBadShape);
    return;
  }
  if (tid == 0) {
    for (int i = 0; i < 19; ++i) mbar_init(&bars[i], i == 2 || i == 3 || i == 18 ? 3 : i >= 4 && i < 12 ? CW : 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == CW) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();                                // the pieces and factors are written

  // 168 registers a thread at launch: 56 for the last four warps and 224 for the others are the same sum
  if (warp >= CW) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == CW) {
      const uint32_t base = smem_u32(scan_sm);
      auto load_tp = [&](int ci) {
        if (elect_one()) {
          mbar_expect_tx(&tp_full[ci & 1], 6 * TILE);
          bulk_load(tp + (ci & 1) * 6 * TILE, a.pieces + (static_cast<long long>(bh) * a.n + ci) * 6 * PIECE, 6 * TILE, &tp_full[ci & 1]);
        }
        __syncwarp();
      };
      constexpr uint32_t n64 = make_idesc_bf16(128, 64), inc64 = n64 | kMnMajorB, inc128 = make_idesc_bf16(128, 128) | kMnMajorB;
      // 128 value columns x 64 tokens: the pieces of one half of each warp's part of the state with the rows of k or q
      auto rows = [&](uint32_t to, uint64_t d, int half) {
#pragma unroll
        for (int p = 2; p >= 0; --p)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t at = (i >> 1) ? (p == 2 ? 448u : 64u + 32u * p) : (p == 2 ? 128u : 32u * p);
            umma_ts(TM + to + (p ? 64 : 0), TM + at + 16 * half + 8 * (i & 1), desc_adv(d, (i >> 1) * TILE + half * 64 + (i & 1) * 32), n64,
                    p != 1 && half == 0 && i == 0 ? 0u : 1u);
          }
      };
      // pieces of R or Vn with those of T or P, lower triangular: 16 tokens j reach the rows from j on
      auto product6 = [&](uint32_t to, uint32_t from, uint64_t d, uint64_t* done) {
        if (elect_one()) {
          constexpr int pa[6] = {0, 1, 2, 0, 1, 0}, pb[6] = {2, 1, 0, 1, 0, 0};
#pragma unroll
          for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int s = 0; s < GC / 16; ++s)
              umma_ts(TM + to + (i == 5 ? 0 : 64) + 16 * s, TM + from + (pa[i] == 2 ? 64u : 16u * pa[i]) + 32 * (s >> 1) + 8 * (s & 1),
                      desc_adv(d, pb[i] * TILE + s * (16 * 128 + 32)), make_idesc_bf16(128, 64 - 16 * s), (i == 0 || i == 5) && s == 0 ? 0u : 1u);
          umma_commit(done);
        }
        __syncwarp();
      };
      auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp(bar, parity, abort_flag, a.status, kStatusWaitTimeoutMma); };
      auto chunk = [&](int ci) {
        const uint32_t ph = ci & 1, X = 192 + 128 * ph, Y = 320 - 128 * ph;
        const uint32_t twice = (ci >> 1) & 1;
        const uint32_t at_k = base + (ci & 1) * KQ;
        const uint64_t kd = make_smem_desc(at_k), td = make_smem_desc(base + 2 * KQ + (ci & 1) * 6 * TILE);
        if ((ci > 0 && !wait(&o_done[ph ^ 1], ((ci - 1) >> 1) & 1)) || !wait(&s_full[0], ph)) return false;      // X held Vn
        tc_fence_after();
        if (elect_one()) rows(X, kd, 0);
        __syncwarp();
        if (!wait(&s_full[1], ph)) return false;
        tc_fence_after();
        if (elect_one()) {
          rows(X, kd, 1);
          umma_commit(ks_done);
        }
        __syncwarp();
        if (ci + 1 < a.n) load_tp(ci + 1);   // the last chunk's products have all retired: its buffer is free
        if (ci > 0 && !wait(o_read, ph ^ 1)) return false;     // Y held O
        tc_fence_after();
        if (elect_one()) {
          rows(Y, desc_adv(kd, 2 * TILE), 0);
          rows(Y, desc_adv(kd, 2 * TILE), 1);
          umma_commit(qs_done);
        }
        __syncwarp();
        if (!wait(&tp_full[ph], twice) || !wait(qs_done, ph) || !wait(r_full, ph)) return false;
        tc_fence_after();
        product6(0, X, td, vn_done);
        if (ci + 1 < a.n && !wait(&row_full[ph ^ 1], ((ci + 1) >> 1) & 1)) return false;       // here, where there is time
        if (!wait(w_full, ph)) return false;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t kn = make_smem_desc_mn(at_k, TILE);
#pragma unroll
          for (int p = 2; p >= 0; --p)
#pragma unroll
            for (int s = 0; s < GC / 16; ++s) {
              const uint32_t at = TM + X + (p == 2 ? 64u : 16u * p) + 32 * (s >> 1) + 8 * (s & 1);
              if (p == 0) {
                umma_ts(TM, at, desc_adv(kn, s * 16 * 128), inc128, s ? 1u : 0u);
              } else {
                umma_ts(TM + 128, at, desc_adv(kn, s * 16 * 128), inc64, p == 2 && s == 0 ? 0u : 1u);
                umma_ts(TM + 448, at, desc_adv(kn, TILE + s * 16 * 128), inc64, p == 2 && s == 0 ? 0u : 1u);
              }
            }
          umma_commit(inc_done);
        }
        __syncwarp();
        if (!wait(v_full, ph) || !wait(inc_done, ph)) return false;      // P Vn goes where the scaled Vn was
        tc_fence_after();
        product6(X, Y, desc_adv(td, 3 * TILE), &o_done[ph]);
        return true;
      };
      load_tp(0);
      bool ok = wait(&row_full[0], 0);
      for (int ci = 0; ci < a.n && ok; ++ci) ok = chunk(ci);
    } else {
      const int id = tid - (CW + 1) * 32;    // three warps: O to memory, the rows and factors of the chunk after the next from there
      auto load = [&](int ci) {
        const int t0 = (a.c0 + ci) * GC, n = min(GC, a.T - t0), buf = ci & 1;
        const uint32_t dk = smem_u32(kq) + buf * KQ, dv = smem_u32(vs) + ci % 3 * VT;
        const __nv_bfloat16 *kp = a.k + b * a.k_bs + t0 * a.k_ts + hk * GD, *qp = a.q + b * a.q_bs + t0 * a.q_ts + hk * GD;
        const __nv_bfloat16* vp = a.v + b * a.v_bs + t0 * a.v_ts + hv * GD;
#pragma unroll 2
        for (int e = id; e < GC * 16; e += 96) {
          const int r = e >> 4, c = e & 15, t = min(r, n - 1);
          const uint32_t at = dk + (c >> 3) * TILE + sw_off<128>(r, c & 7);
          cp_async16(at, kp + t * a.k_ts + c * 8, r < n);
          cp_async16(at + 2 * TILE, qp + t * a.q_ts + c * 8, r < n);
          cp_async16(dv + e * 16, vp + t * a.v_ts + c * 8, r < n);
        }
        const float* fp = a.vec + (static_cast<long long>(bh) * a.n + ci) * VEC * GC;
        if (id < VEC * GC / 4) cp_async16(smem_u32(vec + buf * VEC * GC) + id * 16, fp + id * 4, true);
        cp_commit();
        cp_wait<0>();
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&row_full[buf]);
      };
      load(0);
      if (a.n > 1) load(1);
      auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp(bar, parity, abort_flag, a.status, kStatusWaitTimeoutProducer); };
      for (int ci = 0; ci <= a.n; ++ci) {
        if (ci > 0) {
          if (!wait(&o_full[(ci - 1) & 1], ((ci - 1) >> 1) & 1)) break;
          const int t0 = (a.c0 + ci - 1) * GC;
#pragma unroll 2
          for (int e = id; e < GC * 16; e += 96) {
            const int t = t0 + (e >> 4);
            if (t < a.T)
              *reinterpret_cast<uint4*>(out + ((static_cast<long long>(b) * a.T + t) * a.Hv + hv) * GD + (e & 15) * 8) =
                  *reinterpret_cast<const uint4*>(vs + (ci - 1) % 3 * VT + e * 16);
          }
        }
        if (ci + 2 < a.n) {
          if (!wait(&o_done[ci & 1], (ci >> 1) & 1)) break;
          __syncwarp();                      // all of O is read before v takes its place
          if (lane == 0) mbar_arrive(o_taken);
          if (!wait(o_taken, ci & 1)) break;
          load(ci + 2);
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    const int w = warp >> 2;                 // half of the tokens; of the key dim in the state
    const int col = (warp & 3) * 32 + lane;  // value column
    const uint32_t tl = TM + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const uint32_t lo_s = tl + (w ? 448u : 128u);
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      const bool ok = mbar_wait_warp(bar, parity, abort_flag, a.status, kStatusWaitTimeoutEpilogue);
      tc_fence_after();
      return ok;
    };
    auto arrive = [&](uint64_t* bar) {       // what this warp stored in tensor memory is there
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    float S[64];                             // the state: row 64 w + e, this thread's column
#pragma unroll
    for (int e = 0; e < 64; ++e) S[e] = S0 ? S0[(static_cast<long long>(bh) * GD + 64 * w + e) * GD + col] : 0.f;
    auto put_state = [&](int h) {
      put_pieces(S + 32 * h, tl + 64 * w + 16 * h, tl + 64 * w + 32 + 16 * h, lo_s + 16 * h);
      arrive(&s_full[h]);
    };
    put_state(0);
    put_state(1);
    float vv[32];                            // v of the chunk at hand, read while the state's increment of the last one is formed
    uint32_t ob[16];                         // O of the last chunk, stored while Vn of the one at hand is formed
    auto rows_of = [&](int ci) { return reinterpret_cast<unsigned short*>(vs + ci % 3 * VT) + 32 * w * GD + col; };
    auto load_v = [&](int ci) {
      if (!wait(&row_full[ci & 1], (ci >> 1) & 1)) return false;
      const unsigned short* vr = rows_of(ci);
#pragma unroll
      for (int e = 0; e < 32; ++e) vv[e] = __uint_as_float(static_cast<uint32_t>(vr[e * GD]) << 16);
      return true;
    };
    auto store_o = [&](int ci) {             // each where its thread read v
      unsigned short* vr = rows_of(ci);
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        vr[2 * e * GD] = static_cast<unsigned short>(ob[e]);
        vr[(2 * e + 1) * GD] = static_cast<unsigned short>(ob[e] >> 16);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&o_full[ci & 1]);
    };
    bool ok = load_v(0);
    for (int ci = 0; ci < a.n && ok; ++ci) {
      const uint32_t ph = ci & 1, X = tl + (ph ? 320u : 192u) + 32 * w, Y = tl + (ph ? 192u : 320u) + 32 * w;
      const float* vf = vec + ph * VEC * GC + 32 * w;
      float x[32], q[32], f[32];
      if (!(ok = wait(ks_done, ph))) break;
      read_sums(X, X + 64, x);
#pragma unroll
      for (int e = 0; e < 32; e += 4) {
        const float4 bt = *reinterpret_cast<const float4*>(vf + e), f1 = *reinterpret_cast<const float4*>(vf + GC + e);
        x[e] = fmaf(bt.x, vv[e], -(f1.x * x[e]));              // the product with v is the large one: it does not round
        x[e + 1] = fmaf(bt.y, vv[e + 1], -(f1.y * x[e + 1]));
        x[e + 2] = fmaf(bt.z, vv[e + 2], -(f1.z * x[e + 2]));
        x[e + 3] = fmaf(bt.w, vv[e + 3], -(f1.w * x[e + 3]));
      }
      put_pieces(x, X, X + 16, X + 64);
      arrive(r_full);
      if (ci > 0) store_o(ci - 1);
      if (!(ok = wait(qs_done, ph))) break;
      read_sums(Y, Y + 64, q);
#pragma unroll
      for (int e = 0; e < 32; e += 4) {
        const float4 f2 = *reinterpret_cast<const float4*>(vf + 2 * GC + e);
        q[e] *= f2.x;
        q[e + 1] *= f2.y;
        q[e + 2] *= f2.z;
        q[e + 3] *= f2.w;
        *reinterpret_cast<float4*>(f + e) = *reinterpret_cast<const float4*>(vf + 3 * GC + e);
      }
      const float gC = vec[ph * VEC * GC + 4 * GC];
      if (!(ok = wait(vn_done, ph))) break;
      read_sums(tl + 32 * w, tl + 64 + 32 * w, x);
#pragma unroll
      for (int e = 0; e < 32; ++e) f[e] *= x[e];
      put_pieces(f, X, X + 16, X + 64);
      arrive(w_full);
      put_pieces(x, Y, Y + 16, Y + 64);
      arrive(v_full);
      if (ci + 1 < a.n && !(ok = load_v(ci + 1))) break;
      if (!(ok = wait(inc_done, ph))) break;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        read_sums(tl + 64 * w + 32 * h, lo_s + 32 * h, x);
#pragma unroll
        for (int e = 0; e < 32; ++e) S[32 * h + e] = S[32 * h + e] * gC + x[e];
      }
      if (ci + 1 < a.n) {
        put_state(0);
        put_state(1);
      }
      if (!(ok = wait(&o_done[ph], (ci >> 1) & 1))) break;
      read_sums(X, X + 64, x);
      arrive(o_read);
#pragma unroll
      for (int e = 0; e < 16; ++e) ob[e] = pack_bf16(q[2 * e] + x[2 * e], q[2 * e + 1] + x[2 * e + 1]);
    }
    if (ok) store_o(a.n - 1);
#pragma unroll
    for (int e = 0; e < 64; ++e) S_out[(static_cast<long long>(bh) * GD + 64 * w + e) * GD + col] = S[e];
  }
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(10000);         // let a copy in flight land before shared memory goes away
  }
  if (warp == CW) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(TM), "r"(512));
}

constexpr size_t kChunkBytes = 6 * PIECE * 2 + VEC * GC * sizeof(float);      // workspace of one chunk of one head

}  // namespace

// Chunks of every row that go through the two kernels together: 256 MB of pieces, or one chunk of every row and head (50 KB each)
// where that is more; a longer sequence takes several rounds, the state carried between them.
static int chunk_round(int B, int T, int Hv) {
  const long long chunks = (T + GC - 1) / GC, heads = std::max(1LL, static_cast<long long>(B) * Hv);
  return static_cast<int>(std::max(1LL, std::min(chunks, (256LL << 20) / (heads * static_cast<long long>(kChunkBytes)))));
}

size_t gdn_chunk_workspace(int B, int T, int Hv) {
  return static_cast<size_t>(chunk_round(B, T, Hv)) * B * Hv * kChunkBytes;
}

const char* gdn_chunk_fwd(const void* q, const void* k, const void* v, long long q_bs, long long q_ts, long long k_bs,
                          long long k_ts, long long v_bs, long long v_ts, const float* g, const float* beta,
                          const float* S0, float* S_out, void* out, int B, int T, int Hk, int Hv, int KD, int VD,
                          bool l2norm, float eps, void* workspace, int* status, cudaStream_t stream) {
  if (KD != GD || VD != GD) return "gdn_chunk_fwd: key and value head dim must be 128";
  if (Hk <= 0 || Hv % Hk) return "gdn_chunk_fwd: value heads must be a multiple of key heads";
  if (B == 0 || T == 0) return nullptr;
  if (!FERRL_ONCE_PER_DEVICE(
          cudaFuncSetAttribute(gdn_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kPrepSmem)) == cudaSuccess &&
          cudaFuncSetAttribute(gdn_chunk_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kScanSmem)) == cudaSuccess))
    return "gdn_chunk_fwd: cannot reserve shared memory";
  const int round = chunk_round(B, T, Hv), chunks = (T + GC - 1) / GC;
  ChunkArgs a{static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v),
              q_bs, q_ts, k_bs, k_ts, v_bs, v_ts, g, beta, T, Hk, Hv, 0, 0, static_cast<__nv_bfloat16*>(workspace), nullptr, status};
  for (int c0 = 0; c0 < chunks; c0 += round) {
    a.c0 = c0;
    a.n = std::min(round, chunks - c0);
    a.vec = reinterpret_cast<float*>(a.pieces + static_cast<long long>(B) * Hv * a.n * 6 * PIECE);
    const float* from = c0 == 0 ? S0 : S_out;
    gdn_chunk_prep_kernel<<<a.n * B * Hv, NTH, kPrepSmem, stream>>>(a, l2norm ? 1 : 0, eps);
    launch_pdl(gdn_chunk_scan_kernel, dim3(B * Hv), dim3((CW + 4) * 32), kScanSmem, stream, a, from, S_out, static_cast<__nv_bfloat16*>(out));
    count_launch(2);
  }
  return cudaGetLastError() == cudaSuccess ? nullptr : "gdn_chunk_fwd launch failed";
}

}  // namespace ferrl
