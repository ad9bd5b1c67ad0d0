// Chunked gated delta rule on tensor cores, forward and backward (GatedDeltaNet training and scoring).
//
// Reference: crates/ferrl/src/gdn.rs - gated_delta_rule_chunked (WY form, chunk 64) :451-556 and its
// block forward substitution ut_solve :400-431; the reference composes them from tensor ops with a
// Python-style loop over chunks and differentiates through that loop with the autograd tape.
//
// Per head, with chunk length C = 64, head dims 128 and for one chunk (rows = tokens of the chunk):
//   G   cumulative log decay inside the chunk, gamma = exp(G), D_ij = exp(G_i - G_j) (i >= j)
//   A   = tril(diag(beta) K K^T o D, -1),  T = (I + A)^-1
//   U   = T diag(beta) V,   W = T diag(gamma beta) K
//   Vn  = U - W S                              (S: state entering the chunk, [dk, dv] fp32)
//   O   = diag(gamma) Q S + tril(Q K^T o D) Vn
//   S'  = gamma_C S + (diag(gamma_C / gamma) K)^T Vn
// q and k arrive L2-normalised (q also scaled by 1/sqrt(dk)); those elementwise steps and their
// derivatives stay with the caller.
//
// All matrix products run on the tensor cores (mma m16n8k8, tf32 operands, fp32 accumulation).  Only the two products per
// chunk that carry the state are sequential; everything else is one CTA per (chunk, head):
//   gdn_prep_kernel       G, T (forward substitution), U, Wn = -W, Kd = diag(gamma_C / gamma) K
//   gdn_scan_kernel<fwd>  one CTA per (head, slice of the value columns), chunks in order, state in registers:
//                         Vn = U + Wn S and S' = gamma_C S + Kd^T Vn; saves the entering state of each chunk
//   gdn_out_kernel        O of a chunk from its saved entering state
//   gdn_bwd_prep_kernel   X0 = P^T dO and Y0 = (gamma Q)^T dO
//   gdn_scan_kernel<bwd>  chunks in reverse: dVn = X0 + Kd dS', dS = gamma_C dS' + Y0 + Wn^T dVn
//   gdn_bwd_chunk_kernel  everything else of a chunk: dq, dk, dv, dbeta and dG (the caller turns dG into dg with a reverse
//                         cumulative sum inside each chunk)
//
// What bounds them is reading operands from shared memory: a fragment of 32-bit operands costs as many of its cycles as a
// product of the tensor cores takes, so a warp has the largest tile that its registers hold and tiles lie so that no read
// conflicts, whichever way round a product wants them.  5119 tokens, 48 heads (us, before with 16 x 16 tiles of wmma and a kernel
// of its own for the products with the states): prep 413 -> 201, scan 836 -> 309, out 509 -> 198, bwd_prep 477 -> 174, reverse
// scan 892 -> 432, chunk gradients 2433 -> 780; 4 x 1535 tokens, 16 heads: forward 576 -> 268, backward 1315 -> 522.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../api.h"
#include "../common.cuh"

namespace ferrl {

namespace {

constexpr int GC = 64;      // chunk length
constexpr int GD = 128;     // key and value head dim
constexpr int TILE = GC * GD;      // floats of a [64, 128] tile
constexpr int SQ = GC * GC;        // floats of a [64, 64] tile

// ---------------------------------------------------------------------------------------------
// Shared-memory tiles are rows of 32, 64 or 128 floats whose column is XORed with a function of the row.  A fragment is read
// either as 8 rows x 4 columns or as 4 rows x 8 columns (the stored tile transposed); with these eight values both touch
// all 32 banks once.  16-byte groups stay whole, so tiles are filled by 16-byte copies.
__device__ __forceinline__ int swz(int row) { return ((row & 3) << 3) | (row & 4); }
template <int LD>
__device__ __forceinline__ int at(int row, int col) { return row * LD + (col ^ swz(row)); }

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))),
               "l"(gsrc)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// ROWS x LD floats from global (row stride lds) into a tile, whole CTA of THREADS
template <int ROWS, int LD, int THREADS>
__device__ __forceinline__ void tile_async(float* dst, const float* src, long long lds) {
#pragma unroll 4
  for (int e = threadIdx.x; e < ROWS * LD / 4; e += THREADS) {
    const int r = e / (LD / 4), x = (e % (LD / 4)) * 4;
    cp_async16(dst + at<LD>(r, x), src + r * lds + x);
  }
}

// acc += op(A) op(B) for a warp's tile of 16 MT x 8 NT at (m0, n0), contraction over k0 .. k0 + K; m0 and k0 are multiples of 8,
// n0 of 8.  A is stored [M, K] (AT: [K, M]), B [K, N] (BT: [N, K]).  m16n8k8, tf32 operands, fp32 accumulation; the fp32
// operands go to the tensor cores as they are, which read the top 19 bits.
template <int MT, int NT, int K, bool AT, bool BT, int LDA, int LDB>
__device__ __forceinline__ void warp_mma(float (&acc)[MT][NT][4], const float* A, int m0, const float* B, int n0, int k0 = 0) {
  const int g = (threadIdx.x >> 2) & 7, t = threadIdx.x & 3;
  const int sg = swz(g), st = swz(t);
  constexpr int KI = K < 32 ? K : 32;            // unrolled: more would only hold more fragments in registers
#pragma unroll 1
  for (int kb = k0; kb < k0 + K; kb += KI)
#pragma unroll
  for (int kk = 0; kk < KI; kk += 8) {
    const int k = kb + kk;
    uint32_t a[MT][4], b[NT][2];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int dm = 16 * i + 8 * (e & 1), dk = 4 * (e >> 1);
        if (!AT) a[i][e] = __float_as_uint(A[(m0 + dm + g) * LDA + (KI == 32 ? kb + ((kk + dk + t) ^ sg) : ((k + dk + t) ^ sg))]);
        else a[i][e] = __float_as_uint(A[(k + dk + t) * LDA + ((m0 + dm + g) ^ (st ^ dk))]);
      }
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int dk = 4 * e;
        if (BT) b[j][e] = __float_as_uint(B[(n0 + 8 * j + g) * LDB + (KI == 32 ? kb + ((kk + dk + t) ^ sg) : ((k + dk + t) ^ sg))]);
        else b[j][e] = __float_as_uint(B[(k + dk + t) * LDB + ((n0 + 8 * j + g) ^ (st ^ dk))]);
      }
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
        asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(acc[i][j][0]), "+f"(acc[i][j][1]), "+f"(acc[i][j][2]), "+f"(acc[i][j][3])
                     : "r"(a[i][0]), "r"(a[i][1]), "r"(a[i][2]), "r"(a[i][3]), "r"(b[j][0]), "r"(b[j][1]));
  }
}
// f(row, column, first of two neighbouring accumulators) over a warp's tile
template <int MT, int NT, typename F>
__device__ __forceinline__ void each_pair(float (&acc)[MT][NT][4], int m0, int n0, F f) {
  const int g = (threadIdx.x >> 2) & 7, t = threadIdx.x & 3;
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < NT; ++j) f(m0 + 16 * i + 8 * h + g, n0 + 8 * j + 2 * t, acc[i][j] + 2 * h);
}
template <int MT, int NT>
__device__ __forceinline__ void clear(float (&acc)[MT][NT][4]) {
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
}
template <int LD, int MT, int NT>
__device__ __forceinline__ void put_tile(float* dst, float (&acc)[MT][NT][4], int m0, int n0) {
  each_pair(acc, m0, n0, [&](int r, int c, float* v) { *reinterpret_cast<float2*>(dst + at<LD>(r, c)) = make_float2(v[0], v[1]); });
}
template <int MT, int NT>
__device__ __forceinline__ void put_rows(float* dst, long long ld, float (&acc)[MT][NT][4], int m0, int n0) {
  each_pair(acc, m0, n0, [&](int r, int c, float* v) { *reinterpret_cast<float2*>(dst + r * ld + c) = make_float2(v[0], v[1]); });
}

struct GdnDims {
  int B, T, Hk, Hv, n;        // T is a multiple of GC, n = T / GC chunks
};
// row pointer helpers: q,k are [B, T, Hk, GD], v/out/dO [B, T, Hv, GD], g/beta [B, T, Hv]
__device__ __forceinline__ long long qk_off(const GdnDims& d, int b, int t, int hk) {
  return ((static_cast<long long>(b) * d.T + t) * d.Hk + hk) * GD;
}
__device__ __forceinline__ long long v_off(const GdnDims& d, int b, int t, int hv) {
  return ((static_cast<long long>(b) * d.T + t) * d.Hv + hv) * GD;
}
__device__ __forceinline__ long long ch_off(const GdnDims& d, int b, int hv, int c) {      // chunk-indexed saves
  return (static_cast<long long>(b) * d.Hv + hv) * d.n + c;
}

// P = tril(Q K^T o D) of a chunk into Ps (which may be where K lies), eight warps; the caller has synchronised after the loads
__device__ __forceinline__ void chunk_p(float* Ps, const float* Qs, const float* Ks, const float* Gs) {
  const int warp = threadIdx.x >> 5, m0 = (warp >> 2) * 32, n0 = (warp & 3) * 16;
  float acc[2][2][4];
  clear(acc);
  if (n0 < m0 + 32) warp_mma<2, 2, GD, false, true, GD, GD>(acc, Qs, m0, Ks, n0);
  __syncthreads();
  each_pair(acc, m0, n0, [&](int i, int j, float* v) {
    const float gi = Gs[i];
    *reinterpret_cast<float2*>(Ps + at<GC>(i, j)) =
        make_float2(i >= j ? v[0] * __expf(gi - Gs[j]) : 0.f, i >= j + 1 ? v[1] * __expf(gi - Gs[j + 1]) : 0.f);
  });
  __syncthreads();
}

// ---------------------------------------------------------------------------------------------
// prep: per chunk G, T, U, Wn = -W, Kd = diag(exp(G_C - G)) K and gl = G_C.
// T = (I + A)^-1 with A strictly lower triangular: column c of T depends on A and on that column's own
// earlier rows only, so thread c solves its column in registers (fully unrolled, four partial sums per row
// to shorten the dependent chain) with no synchronisation at all.
// Shared: K, V [64, 128]; A, then -T diag(gamma beta) [64, 64]; T diag(beta) [64, 64]; two vectors.
constexpr size_t kPrepSmem = (2 * TILE + 2 * SQ + 2 * GC) * sizeof(float);

__global__ void __launch_bounds__(256, 2)
gdn_prep_kernel(const float* __restrict__ k, const float* __restrict__ v, const float* __restrict__ g,
                const float* __restrict__ beta, GdnDims d, float* __restrict__ Gc, float* __restrict__ gl,
                float* __restrict__ Tm, float* __restrict__ U, float* __restrict__ Wn, float* __restrict__ Kd) {
  extern __shared__ __align__(128) float sm[];
  float* Ks = sm;
  float* Vs = Ks + TILE;
  float* Y1 = Vs + TILE;
  float* Y2 = Y1 + SQ;
  float* Gs = Y2 + SQ;
  float* bs = Gs + GC;
  const int c = blockIdx.x, hv = blockIdx.y, b = blockIdx.z;
  const int hk = hv / (d.Hv / d.Hk);
  const int tid = threadIdx.x, warp = tid >> 5;
  const long long ldk = static_cast<long long>(d.Hk) * GD, ldv = static_cast<long long>(d.Hv) * GD;
  const long long co = ch_off(d, b, hv, c);
  tile_async<GC, GD, 256>(Ks, k + qk_off(d, b, c * GC, hk), ldk);
  cp_async_commit();
  tile_async<GC, GD, 256>(Vs, v + v_off(d, b, c * GC, hv), ldv);
  cp_async_commit();
  if (tid < GC) bs[tid] = beta[(static_cast<long long>(b) * d.T + c * GC + tid) * d.Hv + hv];
  if (tid < 32) {                  // inclusive scan of 64 log decays by one warp
    const long long o = (static_cast<long long>(b) * d.T + c * GC) * d.Hv + hv;
    float a0 = g[o + static_cast<long long>(2 * tid) * d.Hv], a1 = g[o + static_cast<long long>(2 * tid + 1) * d.Hv];
    float sum = a0 + a1;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, sum, off);
      if (tid >= off) sum += t;
    }
    Gs[2 * tid + 1] = sum;
    Gs[2 * tid] = sum - a1;
  }
  cp_async_wait<1>();
  __syncthreads();
  {                                                    // A = tril(diag(beta) K K^T o D, -1)
    const int m0 = (warp >> 2) * 32, n0 = (warp & 3) * 16;
    float acc[2][2][4];
    clear(acc);
    if (n0 < m0 + 32) warp_mma<2, 2, GD, false, true, GD, GD>(acc, Ks, m0, Ks, n0);
    each_pair(acc, m0, n0, [&](int i, int j, float* x) {
      const float gi = Gs[i], bi = bs[i];
      *reinterpret_cast<float2*>(Y1 + at<GC>(i, j)) =
          make_float2(i > j ? bi * x[0] * __expf(gi - Gs[j]) : 0.f, i > j + 1 ? bi * x[1] * __expf(gi - Gs[j + 1]) : 0.f);
    });
  }
  const float glast = Gs[GC - 1];
  __syncthreads();
  float t[GC];
  if (tid < GC) {
    // column tid of T: t[i] = [i == tid] - sum_{j<i} A[i][j] t[j]; rows above the diagonal stay zero
#pragma unroll
    for (int i = 0; i < GC; ++i) {
      float a0 = (i == tid) ? 1.f : 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
      for (int j = 0; j < i; j += 4) {                 // entries on and above the diagonal are zeros of A
        const float4 a = *reinterpret_cast<const float4*>(Y1 + at<GC>(i, j));
        a0 -= a.x * t[j];
        if (j + 1 < i) a1 -= a.y * t[j + 1];
        if (j + 2 < i) a2 -= a.z * t[j + 2];
        if (j + 3 < i) a3 -= a.w * t[j + 3];
      }
      t[i] = (a0 + a1) + (a2 + a3);
    }
  } else {
    // meanwhile the others write Kd = diag(exp(G_C - G)) K
    for (int e = tid - GC; e < TILE / 4; e += 256 - GC) {
      const int i = e / (GD / 4), x = (e % (GD / 4)) * 4;
      const float4 w = *reinterpret_cast<const float4*>(Ks + at<GD>(i, x));
      const float f = __expf(glast - Gs[i]);
      reinterpret_cast<float4*>(Kd + co * TILE)[e] = make_float4(w.x * f, w.y * f, w.z * f, w.w * f);
    }
  }
  cp_async_wait<0>();
  __syncthreads();                                     // A has been read, V is here
  if (tid < GC) {
    const float fb = bs[tid], fg = -fb * __expf(Gs[tid]);
    float* tm = Tm + co * SQ + tid;
#pragma unroll
    for (int i = 0; i < GC; ++i) {
      tm[i * GC] = t[i];
      Y2[at<GC>(i, tid)] = t[i] * fb;
      Y1[at<GC>(i, tid)] = t[i] * fg;
    }
    Gc[co * GC + tid] = Gs[tid];
    if (tid == 0) gl[co] = glast;
  }
  __syncthreads();
  const int m0 = (warp >> 2) * 32, n0 = (warp & 3) * 32;
  float acc[2][4][4];
  clear(acc);                                          // U = T diag(beta) V; T is lower triangular
  warp_mma<2, 4, 32, false, false, GC, GD>(acc, Y2, m0, Vs, n0);
  if (m0) warp_mma<2, 4, 32, false, false, GC, GD>(acc, Y2, m0, Vs, n0, 32);
  put_rows(U + co * TILE, GD, acc, m0, n0);
  clear(acc);                                          // Wn = -T diag(gamma beta) K
  warp_mma<2, 4, 32, false, false, GC, GD>(acc, Y1, m0, Ks, n0);
  if (m0) warp_mma<2, 4, 32, false, false, GC, GD>(acc, Y1, m0, Ks, n0, 32);
  put_rows(Wn + co * TILE, GD, acc, m0, n0);
}

// ---------------------------------------------------------------------------------------------
// The two scans.  The state's value columns never mix (Vn[:, j] and S'[:, j] depend on S[:, j] only), so a CTA
// owns DV of the 128 value columns of one head and walks the chunks with two products per chunk:
//   forward   Vn  = U  + Wn S              S' = gamma_C S   + Kd^T Vn
//   backward  dVn = X0 + Kd dS'            dS = gamma_C dS' + Y0 + Wn^T dVn      (chunks in reverse)
// Both have the form  V = V0 + A1 R;  R = g R + R0 + A2^T V  with per-chunk [64,128] matrices A1, A2, a
// [64, DV] start V0 and (backward only) a [128, DV] addend R0.  R stays in registers as accumulators, with a copy in shared
// memory as the next chunk's operand.  A1, A2 and V0 of the next chunk are fetched with cp.async while the current chunk
// computes; everything elementwise was folded into the per-chunk kernels.
template <int DV>
struct ScanSmem {
  static constexpr int R = GD * DV, V = GC * DV;
  static constexpr size_t BYTES = static_cast<size_t>(R + 2 * (2 * TILE + V)) * sizeof(float);
};

constexpr int kScanThreads = 512;
constexpr int kMaxChunks = 1024;

template <int DV, bool BWD>
__global__ void __launch_bounds__(kScanThreads, 1)
gdn_scan_kernel(const float* __restrict__ A1g,    // [.., n, 64, 128]: Wn (forward) / Kd (backward)
                const float* __restrict__ A2g,    // [.., n, 64, 128]: Kd (forward) / Wn (backward)
                const float* __restrict__ V0g,    // [.., n, 64, 128]: U (forward) / X0 (backward)
                const float* __restrict__ R0g,    // backward: Y0 [.., n, 128, 128]; forward: null
                const float* __restrict__ gl,     // [.., n] last cumulative log decay of every chunk
                const float* __restrict__ Rinit,  // [.., 128, 128] initial state (S0 / dS_final) or null
                int n, int n_slices,
                float* __restrict__ Vout,         // [.., n, 64, 128]: Vn / dVn
                float* __restrict__ Rchunks,      // [.., n, 128, 128]: forward Sin[c] = state entering chunk c;
                                                  //                    backward dSout[c] = gradient of the state leaving c
                float* __restrict__ Rfinal) {     // [.., 128, 128]: S after the last chunk / dS0 (may be null)
  using SM = ScanSmem<DV>;
  extern __shared__ __align__(128) float sm[];
  float* Rs = sm;
  float* buf0 = Rs + SM::R;                       // two of A1, A2, V0
  constexpr int BUF = 2 * TILE + SM::V;
  __shared__ float gls[kMaxChunks];
  const int slice = blockIdx.x % n_slices;
  const long long bh = blockIdx.x / n_slices + static_cast<long long>(blockIdx.y) * (gridDim.x / n_slices);
  const int col0 = slice * DV;
  const int tid = threadIdx.x, warp = tid >> 5;
  const long long cbase = bh * n;
  // tiles of the 16 warps: 16 rows of V x DV / 4 columns, 32 rows of R x DV / 4 columns
  constexpr int NT = DV / 32;
  const int mv = (warp >> 2) * 16, mr = (warp >> 2) * 32, nc = (warp & 3) * (DV / 4);
  auto fetch = [&](int c, int buf) {
    float* at0 = buf0 + buf * BUF;
    const long long co = (cbase + c) * TILE;
    tile_async<GC, GD, kScanThreads>(at0, A1g + co, GD);
    tile_async<GC, DV, kScanThreads>(at0 + 2 * TILE, V0g + co + col0, GD);
    tile_async<GC, GD, kScanThreads>(at0 + TILE, A2g + co, GD);
    cp_async_commit();
  };
  const int first = BWD ? n - 1 : 0, step = BWD ? -1 : 1;
  fetch(first, 0);
  for (int e = tid; e < n; e += kScanThreads) gls[e] = gl[cbase + e];
  float r[2][NT][4];                              // the state
  clear(r);
  if (Rinit)
    each_pair(r, mr, nc, [&](int i, int j, float* x) {
      const float2 w = *reinterpret_cast<const float2*>(Rinit + bh * GD * GD + i * GD + col0 + j);
      x[0] = w.x;
      x[1] = w.y;
    });
  put_tile<DV>(Rs, r, mr, nc);
  put_rows(Rchunks + (cbase + first) * GD * GD + col0, GD, r, mr, nc);      // the state as the first chunk sees it
  for (int i = 0; i < n; ++i) {
    const int c = first + i * step, buf = i & 1;
    cp_async_wait<0>();
    __syncthreads();                        // this chunk's tiles have landed, the state is written; the other buffer is free
    if (i + 1 < n) fetch(c + step, buf ^ 1);
    const float* a1 = buf0 + buf * BUF;
    const float* a2 = a1 + TILE;
    float* vs = buf0 + buf * BUF + 2 * TILE;
    float add[2][NT][4];
    if (BWD)
      each_pair(add, mr, nc, [&](int row, int j, float* x) {
        const float2 w = *reinterpret_cast<const float2*>(R0g + (cbase + c) * GD * GD + row * GD + col0 + j);
        x[0] = w.x;
        x[1] = w.y;
      });
    // V = V0 + A1 R    [64, DV], K = 128
    float v[1][NT][4];
    each_pair(v, mv, nc, [&](int row, int j, float* x) {
      const float2 w = *reinterpret_cast<const float2*>(vs + at<DV>(row, j));
      x[0] = w.x;
      x[1] = w.y;
    });
    warp_mma<1, NT, GD, false, false, GD, DV>(v, a1, mv, Rs, nc);
    put_tile<DV>(vs, v, mv, nc);
    put_rows(Vout + (cbase + c) * TILE + col0, GD, v, mv, nc);
    __syncthreads();
    // R = g R (+ R0) + A2^T V    [128, DV], K = 64
    const float eg = __expf(gls[c]);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) r[a][j][e] = BWD ? r[a][j][e] * eg + add[a][j][e] : r[a][j][e] * eg;
    warp_mma<2, NT, GC, true, false, GD, DV>(r, a2, mr, vs, nc);
    const bool last = i + 1 == n;
    if (!last) put_tile<DV>(Rs, r, mr, nc);
    float* rdst = last ? (Rfinal ? Rfinal + bh * GD * GD : nullptr) : Rchunks + (cbase + c + step) * GD * GD;
    if (rdst) put_rows(rdst + col0, GD, r, mr, nc);
  }
}

// ---------------------------------------------------------------------------------------------
// output of one chunk from the saved entering state:  O = diag(gamma) (Q Sin) + tril(Q K^T o D) Vn.  A CTA has half of the
// value columns, so two fit a multiprocessor and one loads while the other multiplies.
// Shared: Q [64, 128]; K [64, 128], then P [64, 64]; Sin [128, 64]; Vn [64, 64]; G [64].
constexpr size_t kOutSmem = (2 * TILE + GD * 64 + SQ + GC) * sizeof(float);

__global__ void __launch_bounds__(256, 2)
gdn_out_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ Gc,
               const float* __restrict__ Sin, const float* __restrict__ Vn, GdnDims d, float* __restrict__ out) {
  extern __shared__ __align__(128) float sm[];
  float* Qs = sm;
  float* Ks = Qs + TILE;
  float* Ss = Ks + TILE;
  float* Vs = Ss + GD * 64;
  float* Gs = Vs + SQ;
  const int c = blockIdx.x >> 1, col0 = (blockIdx.x & 1) * 64, hv = blockIdx.y, b = blockIdx.z;
  const int hk = hv / (d.Hv / d.Hk);
  const int tid = threadIdx.x, warp = tid >> 5;
  const long long ldk = static_cast<long long>(d.Hk) * GD, ldv = static_cast<long long>(d.Hv) * GD;
  const long long co = ch_off(d, b, hv, c);
  tile_async<GC, GD, 256>(Qs, q + qk_off(d, b, c * GC, hk), ldk);
  tile_async<GC, GD, 256>(Ks, k + qk_off(d, b, c * GC, hk), ldk);
  cp_async_commit();
  tile_async<GD, 64, 256>(Ss, Sin + co * GD * GD + col0, GD);
  tile_async<GC, 64, 256>(Vs, Vn + co * TILE + col0, GD);
  cp_async_commit();
  if (tid < GC) Gs[tid] = Gc[co * GC + tid];
  cp_async_wait<1>();
  __syncthreads();
  float* Ps = Ks;
  chunk_p(Ps, Qs, Ks, Gs);
  cp_async_wait<0>();
  __syncthreads();
  const int m0 = (warp >> 2) * 32, n0 = (warp & 3) * 16;
  float acc[2][2][4];
  clear(acc);
  warp_mma<2, 2, GD, false, false, GD, 64>(acc, Qs, m0, Ss, n0);
  each_pair(acc, m0, n0, [&](int i, int, float* x) {
    const float f = __expf(Gs[i]);
    x[0] *= f;
    x[1] *= f;
  });
  warp_mma<2, 2, 32, false, false, GC, 64>(acc, Ps, m0, Vs, n0);
  if (m0) warp_mma<2, 2, 32, false, false, GC, 64>(acc, Ps, m0, Vs, n0, 32);
  put_rows(out + v_off(d, b, c * GC, hv) + col0, ldv, acc, m0, n0);
}

// ---------------------------------------------------------------------------------------------
// backward, chunk-local inputs of the reverse scan:  X0 = P^T dO  [64,128],  Y0 = (gamma Q)^T dO  [128,128]
// Shared: Q [64, 128]; K [64, 128], then P [64, 64]; dO [64, 128]; G [64].
constexpr size_t kBwdPrepSmem = (3 * TILE + GC) * sizeof(float);

__global__ void __launch_bounds__(256, 2)
gdn_bwd_prep_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ Gc,
                    const float* __restrict__ dO, GdnDims d, float* __restrict__ X0, float* __restrict__ Y0) {
  extern __shared__ __align__(128) float sm[];
  float* Qs = sm;
  float* Ks = Qs + TILE;
  float* Os = Ks + TILE;
  float* Gs = Os + TILE;
  const int c = blockIdx.x, hv = blockIdx.y, b = blockIdx.z;
  const int hk = hv / (d.Hv / d.Hk);
  const int tid = threadIdx.x, warp = tid >> 5;
  const long long ldk = static_cast<long long>(d.Hk) * GD, ldv = static_cast<long long>(d.Hv) * GD;
  const long long co = ch_off(d, b, hv, c);
  tile_async<GC, GD, 256>(Qs, q + qk_off(d, b, c * GC, hk), ldk);
  tile_async<GC, GD, 256>(Ks, k + qk_off(d, b, c * GC, hk), ldk);
  cp_async_commit();
  tile_async<GC, GD, 256>(Os, dO + v_off(d, b, c * GC, hv), ldv);
  cp_async_commit();
  if (tid < GC) Gs[tid] = Gc[co * GC + tid];
  cp_async_wait<1>();
  __syncthreads();
  float* Ps = Ks;
  chunk_p(Ps, Qs, Ks, Gs);
  for (int e = tid; e < TILE / 4; e += 256) {           // Q diag(gamma): a row's factor, wherever its columns lie
    float4* w = reinterpret_cast<float4*>(Qs) + e;
    const float f = __expf(Gs[e / (GD / 4)]);
    *w = make_float4(w->x * f, w->y * f, w->z * f, w->w * f);
  }
  cp_async_wait<0>();
  __syncthreads();
  {                                                      // X0 = P^T dO: P_ij = 0 for i < j
    const int m0 = (warp >> 2) * 32, n0 = (warp & 3) * 32;
    float acc[2][4][4];
    clear(acc);
    if (m0 == 0) warp_mma<2, 4, 32, true, false, GC, GD>(acc, Ps, m0, Os, n0);
    warp_mma<2, 4, 32, true, false, GC, GD>(acc, Ps, m0, Os, n0, 32);
    put_rows(X0 + co * TILE, GD, acc, m0, n0);
  }
#pragma unroll 1
  for (int t = warp; t < 16; t += 8) {                   // Y0 = (gamma Q)^T dO
    const int m0 = (t >> 2) * 32, n0 = (t & 3) * 32;
    float acc[2][4][4];
    clear(acc);
    warp_mma<2, 4, GC, true, false, GD, GD>(acc, Qs, m0, Os, n0);
    put_rows(Y0 + co * GD * GD, GD, acc, m0, n0);
  }
}

// ---------------------------------------------------------------------------------------------
// Backward of a chunk, given dVn and dS' from the reverse scan.  One CTA per (chunk, head):
//   E1 = dO Sin^T,  dW = -dVn Sin^T,  E2 = Vn dS'^T
//   dq = gamma o E1 + (dP o D) K                          dP o D = tril(dO Vn^T) o D
//   dk = (gamma_C / gamma) o E2 + (dP o D)^T Q + (Ab + Ab^T) K + diag(gamma beta) T^T dW
//   dv = diag(beta) T^T dVn
//   Z1 = dVn V^T,  Z2 = dW K^T,  dT = tril(Z1 + Z2 diag(gamma)) diag(beta)      (T is lower triangular: the rest moves nothing)
//   dA o D = -tril(T^T dT T^T, -1) o D,  Ab = diag(beta) (dA o D)
//   dbeta_i = sum_k T_ki (Z1_ki + gamma_i Z2_ki) + sum_j (dA o D)_ij (K K^T)_ij
//   dG_i  = gamma <Q, E1> - R_i + rowsum - colsum of (dP o D) o (Q K^T) and of Ab o (K K^T), + gamma_i beta_i sum_k T_ki Z2_ki
//   dG_last += gamma_C <Sin, dS'> + sum R,  R_i = (gamma_C / gamma_i) <K_i, E2_i>
// Warps 0..7 hold dq as accumulators and warps 8..15 dk, a tile of 32 x 32 each, from the first product to the last; the [64, 64]
// products are tiles of 32 x 16 whose elementwise steps and sums happen in registers.  What a later step needs is fetched into
// tiles as they fall free, so only the first loads are waited for.
// Shared: seven [64, 128] tiles, G and beta, block sums.
//   0,1: Sin, then dS' (through registers), then 0: dW, 1: dP o D and dT [64, 64]
//   2: dO, then V      3: dVn      4: Vn, then T [64, 64] and partial sums      5: K      6: Q, then T^T dT and Ab + Ab^T [64, 64]
constexpr int kChunkThreads = 512;
constexpr size_t kBwdChunkSmem = (7 * TILE + 2 * GC + 16) * sizeof(float);
static_assert(kBwdChunkSmem <= 227 * 1024, "shared memory");

__global__ void __launch_bounds__(kChunkThreads, 1)
gdn_bwd_chunk_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                     const float* __restrict__ beta, const float* __restrict__ Gc, const float* __restrict__ Tm,
                     const float* __restrict__ Vn, const float* __restrict__ dVn, const float* __restrict__ Sin,
                     const float* __restrict__ dSout, const float* __restrict__ dO, GdnDims d, float* __restrict__ dq,
                     float* __restrict__ dk, float* __restrict__ dv, float* __restrict__ dbeta, float* __restrict__ dG) {
  extern __shared__ __align__(128) float sm[];
  float *sS = sm, *sW = sm, *sP = sm + TILE, *sdT = sP + SQ;
  float *sO = sm + 2 * TILE, *sV = sO, *sdV = sm + 3 * TILE, *sVn = sm + 4 * TILE, *sT = sVn;
  float *sK = sm + 5 * TILE, *sQ = sm + 6 * TILE, *sY = sQ, *sSym = sQ + SQ;
  float* Gs = sm + 7 * TILE;
  float* bs = Gs + GC;
  float* red = bs + GC;                          // [16]
  // partial sums of the warps that share a row or a column
  float* pQ = sVn + SQ;                          // [4][64] <dq, Q>
  float* pK = pQ + 4 * GC;                       // [4][64] R
  float* pMr = pK + 4 * GC;                      // [4][64] rows of (dP o D) o (Q K^T)
  float* pMc = pMr + 4 * GC;                     // [2][64] columns
  float* pZ1 = pMc + 2 * GC;                     // [2][64] columns of T o Z1
  float* pZ2 = pZ1 + 2 * GC;                     // [2][64] of T o Z2
  float* pAr = pZ2 + 2 * GC;                     // [4][64] rows of (dA o D) o (K K^T)
  float* pAc = pAr + 4 * GC;                     // [2][64] columns of Ab o (K K^T)
  const int c = blockIdx.x, hv = blockIdx.y, b = blockIdx.z;
  const int hk = hv / (d.Hv / d.Hk);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const bool hi = warp >= 8;                     // warps of dk
  const int w8 = warp & 7, m0 = (w8 >> 2) * 32, n0 = (w8 & 3) * 32, s0 = (w8 & 3) * 16;      // tiles [m0, n0] of 32 x 32, [m0, s0] of 32 x 16
  const long long ldk = static_cast<long long>(d.Hk) * GD, ldv = static_cast<long long>(d.Hv) * GD;
  const long long co = ch_off(d, b, hv, c);
  const long long vo = v_off(d, b, c * GC, hv), qo = qk_off(d, b, c * GC, hk);
  tile_async<GD, GD, kChunkThreads>(sS, Sin + co * GD * GD, GD);
  tile_async<GC, GD, kChunkThreads>(sO, dO + vo, ldv);
  tile_async<GC, GD, kChunkThreads>(sdV, dVn + co * TILE, GD);
  cp_async_commit();
  tile_async<GC, GD, kChunkThreads>(sVn, Vn + co * TILE, GD);
  tile_async<GC, GD, kChunkThreads>(sQ, q + qo, ldk);
  tile_async<GC, GD, kChunkThreads>(sK, k + qo, ldk);
  cp_async_commit();
  float4 ds[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) ds[e] = __ldg(reinterpret_cast<const float4*>(dSout + co * GD * GD) + tid + e * kChunkThreads);
  if (tid < GC) {
    Gs[tid] = Gc[co * GC + tid];
    bs[tid] = beta[(static_cast<long long>(b) * d.T + c * GC + tid) * d.Hv + hv];
  }
  cp_async_wait<1>();
  __syncthreads();
  // ---- E1 = dO Sin^T (warps 0..7), dVn Sin^T (8..15)
  float acc[2][4][4];
  clear(acc);
  warp_mma<2, 4, GD, false, true, GD, GD>(acc, hi ? sdV : sO, m0, sS, n0);
  cp_async_wait<0>();
  __syncthreads();
  {                                              // <Sin, dS'>, and dS' in its place
    float part = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int at4 = tid + e * kChunkThreads;
      float4* w = reinterpret_cast<float4*>(sS + at<GD>(at4 / (GD / 4), (at4 % (GD / 4)) * 4));
      part += w->x * ds[e].x + w->y * ds[e].y + w->z * ds[e].z + w->w * ds[e].w;
      *w = ds[e];
    }
    part = warp_sum(part);
    if (lane == 0) red[warp] = part;
  }
  __syncthreads();
  // ---- E2 = Vn dS'^T (8..15); dP = dO Vn^T and Q K^T where rows reach columns (0..7)
  float ek[2][4][4], p[2][2][4], qk[2][2][4];
  const bool low = s0 < m0 + 32;                 // tile [m0, s0] is not all above the diagonal
  clear(p);
  clear(qk);
  if (hi) {
    clear(ek);
    warp_mma<2, 4, GD, false, true, GD, GD>(ek, sVn, m0, sS, n0);
  } else if (low) {
    warp_mma<2, 2, GD, false, true, GD, GD>(p, sO, m0, sVn, s0);
    warp_mma<2, 2, GD, false, true, GD, GD>(qk, sQ, m0, sK, s0);
  }
  __syncthreads();
  tile_async<GC, GD, kChunkThreads>(sV, v + vo, ldv);
  tile_async<GC, GC, kChunkThreads>(sT, Tm + co * SQ, GC);
  cp_async_commit();
  const float glast = Gs[GC - 1];
  // a row's sum over the lanes that share it, a column's over its rows of the tile
  auto row_sum = [&](float* dst, float x, int row) {
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    if (t4 == 0) dst[row] = x;
  };
  auto col_sum = [&](float* dst, float x, int col) {
    x += __shfl_xor_sync(0xffffffffu, x, 4);
    x += __shfl_xor_sync(0xffffffffu, x, 8);
    x += __shfl_xor_sync(0xffffffffu, x, 16);
    if (g == 0) dst[col] = x;
  };
  auto tile_sums = [&](float (&x)[2][2][4], float* rows, float* cols) {      // of a [32, 16] tile; either may be null
    if (rows)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          row_sum(rows, (x[i][0][2 * h] + x[i][0][2 * h + 1]) + (x[i][1][2 * h] + x[i][1][2 * h + 1]), m0 + 16 * i + 8 * h + g);
    if (cols)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          col_sum(cols, (x[0][j][e] + x[0][j][2 + e]) + (x[1][j][e] + x[1][j][2 + e]), s0 + 8 * j + 2 * t4 + e);
  };
  // rows scaled by f, and their dots with the same rows of X
  auto scale_dot = [&](float (&x)[2][4][4], const float* X, float* dots, auto f) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = m0 + 16 * i + 8 * h + g;
        const float s = f(row);
        float dot = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 w = *reinterpret_cast<const float2*>(X + at<GD>(row, n0 + 8 * j + 2 * t4));
          x[i][j][2 * h] *= s;
          x[i][j][2 * h + 1] *= s;
          dot += x[i][j][2 * h] * w.x + x[i][j][2 * h + 1] * w.y;
        }
        row_sum(dots, dot, row);
      }
  };
  if (!hi) {
    scale_dot(acc, sQ, pQ + (w8 & 3) * GC, [&](int i) { return __expf(Gs[i]); });
    each_pair(p, m0, s0, [&](int i, int j, float* x) {                 // dP o D
      const float gi = Gs[i];
      x[0] = i >= j ? x[0] * __expf(gi - Gs[j]) : 0.f;
      x[1] = i >= j + 1 ? x[1] * __expf(gi - Gs[j + 1]) : 0.f;
    });
    put_tile<GC>(sP, p, m0, s0);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) qk[i][j][e] *= p[i][j][e];
    tile_sums(qk, pMr + (w8 & 3) * GC, pMc + (w8 >> 2) * GC);
  } else {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][j][e] = -acc[i][j][e];
    put_tile<GD>(sW, acc, m0, n0);
    scale_dot(ek, sK, pK + (w8 & 3) * GC, [&](int i) { return __expf(glast - Gs[i]); });
  }
  __syncthreads();
  // ---- dq += (dP o D) K;  dk += (dP o D)^T Q
  if (!hi) {
    warp_mma<2, 4, 32, false, false, GC, GD>(acc, sP, m0, sK, n0);
    if (m0) warp_mma<2, 4, 32, false, false, GC, GD>(acc, sP, m0, sK, n0, 32);
    put_rows(dq + vo, ldv, acc, m0, n0);
  } else {
    if (m0 == 0) warp_mma<2, 4, 32, true, false, GC, GD>(ek, sP, m0, sQ, n0);
    warp_mma<2, 4, 32, true, false, GC, GD>(ek, sP, m0, sQ, n0, 32);
  }
  cp_async_wait<0>();
  __syncthreads();
  // ---- Z1, Z2 and dT (0..7);  dk += diag(gamma beta) T^T dW, K K^T (8..15)
  float kk[2][2][4];
  clear(kk);
  if (!hi) {
    float z1[2][2][4], z2[2][2][4];
    clear(z1);
    clear(z2);
    if (low) {
      warp_mma<2, 2, GD, false, true, GD, GD>(z1, sdV, m0, sV, s0);
      warp_mma<2, 2, GD, false, true, GD, GD>(z2, sW, m0, sK, s0);
    }
    float dt[2][2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int row = m0 + 16 * i + 8 * (e >> 1) + g, col = s0 + 8 * j + 2 * t4 + (e & 1);
          const float tv = sT[at<GC>(row, col)];
          dt[i][j][e] = row >= col ? bs[col] * (z1[i][j][e] + __expf(Gs[col]) * z2[i][j][e]) : 0.f;
          z1[i][j][e] *= tv;
          z2[i][j][e] *= tv;
        }
    put_tile<GC>(sdT, dt, m0, s0);
    tile_sums(z1, nullptr, pZ1 + (w8 >> 2) * GC);
    tile_sums(z2, nullptr, pZ2 + (w8 >> 2) * GC);
  } else {
    clear(acc);
    if (m0 == 0) warp_mma<2, 4, 32, true, false, GC, GD>(acc, sT, m0, sW, n0);
    warp_mma<2, 4, 32, true, false, GC, GD>(acc, sT, m0, sW, n0, 32);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = m0 + 16 * i + 8 * h + g;
        const float f = bs[row] * __expf(Gs[row]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          ek[i][j][2 * h] += f * acc[i][j][2 * h];
          ek[i][j][2 * h + 1] += f * acc[i][j][2 * h + 1];
        }
      }
    if (low) warp_mma<2, 2, GD, false, true, GD, GD>(kk, sK, m0, sK, s0);
  }
  __syncthreads();
  {                                              // T^T dT: both lower triangular, so k starts at the later of row and column
    const int ma = (warp >> 2) * 16, na = (warp & 3) * 16;
    float y[1][2][4];
    clear(y);
    for (int k0 = max(ma, na); k0 < GC; k0 += 16) warp_mma<1, 2, 16, true, false, GC, GC>(y, sT, ma, sdT, na, k0);
    put_tile<GC>(sY, y, ma, na);
  }
  __syncthreads();
  // ---- dA = -tril(Y T^T, -1) o D, Ab + Ab^T and its sums (8..15);  dv = diag(beta) T^T dVn (0..7)
  if (!hi) {
    clear(acc);
    if (m0 == 0) warp_mma<2, 4, 32, true, false, GC, GD>(acc, sT, m0, sdV, n0);
    warp_mma<2, 4, 32, true, false, GC, GD>(acc, sT, m0, sdV, n0, 32);
    each_pair(acc, m0, n0, [&](int i, int, float* x) {
      const float f = bs[i];
      x[0] *= f;
      x[1] *= f;
    });
    put_rows(dv + vo, ldv, acc, m0, n0);
  } else {
    float a[2][2][4], ab[2][2][4];
    clear(a);
    if (low) {
      warp_mma<2, 2, 32, false, true, GC, GC>(a, sY, m0, sT, s0);
      if (m0) warp_mma<2, 2, 32, false, true, GC, GC>(a, sY, m0, sT, s0, 32);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int row = m0 + 16 * i + 8 * (e >> 1) + g, col = s0 + 8 * j + 2 * t4 + (e & 1);
          const float x = row > col ? -a[i][j][e] * __expf(Gs[row] - Gs[col]) : 0.f, y = x * bs[row];
          if (row >= col) {
            sSym[at<GC>(row, col)] = y;
            if (row > col) sSym[at<GC>(col, row)] = y;
          }
          ab[i][j][e] = y * kk[i][j][e];
          a[i][j][e] = x * kk[i][j][e];
        }
    tile_sums(a, pAr + (w8 & 3) * GC, nullptr);
    tile_sums(ab, nullptr, pAc + (w8 >> 2) * GC);
  }
  __syncthreads();
  if (hi) {
    warp_mma<2, 4, GC, false, false, GC, GD>(ek, sSym, m0, sK, n0);
    put_rows(dk + vo, ldv, ek, m0, n0);
  } else if (warp < 2) {
    const int i = tid;
    auto sum4 = [&](const float* x) { return (x[i] + x[GC + i]) + (x[2 * GC + i] + x[3 * GC + i]); };
    auto sum2 = [&](const float* x) { return x[i] + x[GC + i]; };
    const float eg = __expf(Gs[i]), z2 = sum2(pZ2), ar = sum4(pAr), rk = sum4(pK);
    dbeta[(static_cast<long long>(b) * d.T + c * GC + i) * d.Hv + hv] = sum2(pZ1) + eg * z2 + ar;
    float out = sum4(pQ) - rk + sum4(pMr) - sum2(pMc) + bs[i] * (eg * z2 + ar) - sum2(pAc);
    if (warp == 1) {                             // the last row takes the state's decay and every R
      float all = rk + (pK[lane] + pK[GC + lane]) + (pK[2 * GC + lane] + pK[3 * GC + lane]);
      all = warp_sum(all);
      if (lane == 31) {
        float ss = 0.f;
        for (int x = 0; x < 16; ++x) ss += red[x];
        out += __expf(glast) * ss + all;
      }
    }
    dG[(static_cast<long long>(b) * d.T + c * GC + i) * d.Hv + hv] = out;
  }
}

template <bool BWD>
const char* launch_scan(const float* A1, const float* A2, const float* V0, const float* R0, const float* gl, const float* Rinit,
                        int B, int Hv, int n, float* Vout, float* Rchunks, float* Rfinal, cudaStream_t stream) {
  if (n > kMaxChunks) return "gdn_tc: at most 1024 chunks (65536 tokens) per sequence";
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // narrower column slices when all of them still run at once
  const bool narrow = static_cast<long long>(B) * Hv * 4 <= sms;
  if (!FERRL_ONCE_PER_DEVICE(
          cudaFuncSetAttribute(gdn_scan_kernel<64, BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(ScanSmem<64>::BYTES)) == cudaSuccess &&
          cudaFuncSetAttribute(gdn_scan_kernel<32, BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(ScanSmem<32>::BYTES)) == cudaSuccess))
    return "gdn_tc: cannot reserve shared memory";
  if (narrow)
    gdn_scan_kernel<32, BWD><<<dim3(Hv * 4, B), kScanThreads, ScanSmem<32>::BYTES, stream>>>(A1, A2, V0, R0, gl, Rinit, n, 4, Vout, Rchunks,
                                                                                    Rfinal);
  else
    gdn_scan_kernel<64, BWD><<<dim3(Hv * 2, B), kScanThreads, ScanSmem<64>::BYTES, stream>>>(A1, A2, V0, R0, gl, Rinit, n, 2, Vout, Rchunks,
                                                                                    Rfinal);
  count_launch();
  return nullptr;
}

}  // namespace

const char* gdn_tc_forward(const float* q, const float* k, const float* v, const float* g, const float* beta, const float* S0,
                           int B, int T, int Hk, int Hv, float* Gc, float* gl, float* Tm, float* U, float* Wn, float* Kd,
                           float* out, float* S_out, float* Sin, float* Vn, cudaStream_t stream) {
  if (T % GC) return "gdn_tc: the sequence length must be a multiple of 64 (pad with beta = 0, g = 0)";
  if (Hk <= 0 || Hv % Hk) return "gdn_tc: value heads must be a multiple of key heads";
  if (B == 0 || T == 0) return nullptr;
  GdnDims d{B, T, Hk, Hv, T / GC};
  if (!FERRL_ONCE_PER_DEVICE(
          cudaFuncSetAttribute(gdn_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kPrepSmem)) == cudaSuccess &&
          cudaFuncSetAttribute(gdn_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kOutSmem)) == cudaSuccess))
    return "gdn_tc: cannot reserve shared memory";
  gdn_prep_kernel<<<dim3(d.n, Hv, B), 256, kPrepSmem, stream>>>(k, v, g, beta, d, Gc, gl, Tm, U, Wn, Kd);
  count_launch();
  if (const char* e = launch_scan<false>(Wn, Kd, U, nullptr, gl, S0, B, Hv, d.n, Vn, Sin, S_out, stream)) return e;
  gdn_out_kernel<<<dim3(d.n * 2, Hv, B), 256, kOutSmem, stream>>>(q, k, Gc, Sin, Vn, d, out);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "gdn_tc forward launch failed";
}

const char* gdn_tc_backward(const float* q, const float* k, const float* v, const float* beta, const float* Gc, const float* gl,
                            const float* Tm, const float* Wn, const float* Kd, const float* Vn, const float* Sin,
                            const float* dO, const float* dS_final, int B, int T, int Hk, int Hv, float* X0, float* Y0,
                            float* dVn, float* dSout, float* dq, float* dk, float* dv, float* dbeta,
                            float* dG, float* dS0, cudaStream_t stream) {
  if (T % GC) return "gdn_tc: the sequence length must be a multiple of 64";
  if (Hk <= 0 || Hv % Hk) return "gdn_tc: value heads must be a multiple of key heads";
  if (B == 0 || T == 0) return nullptr;
  GdnDims d{B, T, Hk, Hv, T / GC};
  if (!FERRL_ONCE_PER_DEVICE(
          cudaFuncSetAttribute(gdn_bwd_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kBwdPrepSmem)) == cudaSuccess &&
          cudaFuncSetAttribute(gdn_bwd_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kBwdChunkSmem)) == cudaSuccess))
    return "gdn_tc: cannot reserve shared memory";
  gdn_bwd_prep_kernel<<<dim3(d.n, Hv, B), 256, kBwdPrepSmem, stream>>>(q, k, Gc, dO, d, X0, Y0);
  count_launch();
  if (const char* e = launch_scan<true>(Kd, Wn, X0, Y0, gl, dS_final, B, Hv, d.n, dVn, dSout, dS0, stream)) return e;
  gdn_bwd_chunk_kernel<<<dim3(d.n, Hv, B), kChunkThreads, kBwdChunkSmem, stream>>>(q, k, v, beta, Gc, Tm, Vn, dVn, Sin, dSout, dO, d, dq, dk,
                                                                                 dv, dbeta, dG);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "gdn_tc backward launch failed";
}

}  // namespace ferrl
