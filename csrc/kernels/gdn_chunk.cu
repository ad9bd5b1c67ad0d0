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
//   gdn_chunk_scan_kernel   one CTA per (head, DV value columns): chunks in order, the state in registers
//
// One CTA per head with everything in 32-bit multiply-adds was bound by them and by its serial chain, on 48 SMs for 48
// heads: 5119 tokens x 48 heads 5057 -> 722 us, 4 x 2047 x 48 4053 -> 958 us, 1024 x 16 966 -> 95 us.  The state is now
// 1.1e-7 to 1.8e-7 off float64 (2-norm), 1.7e-7 to 6.9e-7 before.  What bounds the scan is issuing the warp-level products
// and their fragments (four barriers a chunk, 9 us a chunk for 64 columns); 16-bit pieces of a third the size would halve it and
// lose the last eight bits of every sum.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../api.h"
#include "../common.cuh"
#include "mma_sync.cuh"

namespace ferrl {
namespace {

using namespace mmah;
constexpr int GC = 64;                       // chunk length
constexpr int GD = 128;                      // key and value head dim
constexpr int NTH = 256;
constexpr int PIECE = GC * GC;               // entries of one piece of T or P
constexpr int VEC = 5;                       // row factors: beta, beta gamma kn, gamma qn, kn exp(G_C - G), [gamma_C]
constexpr int TILE = GC * GC * 2;            // bytes of a [64, 64] 16-bit tile

// pieces of two neighbouring entries: x = h + m + l
__device__ __forceinline__ void split3(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16(x, y);
  x -= __uint_as_float(h << 16);
  y -= __uint_as_float(h & 0xFFFF0000u);
  m = pack_bf16(x, y);
  x -= __uint_as_float(m << 16);
  y -= __uint_as_float(m & 0xFFFF0000u);
  l = pack_bf16(x, y);
}

struct ChunkArgs {
  const __nv_bfloat16 *q, *k, *v;
  long long q_bs, q_ts, k_bs, k_ts, v_bs, v_ts;
  const float *g, *beta;
  int T, Hk, Hv, c0, n;                      // chunks c0 .. c0 + n of every row
  __nv_bfloat16* pieces;                     // [B * Hv, n, 6, 64, 64]: T then P
  float* vec;                                // [B * Hv, n, VEC, 64]
};

// Shared: k, q [64, 256 bytes] swizzled; A [64, 68]; T [64, 65]; G (two floats), kn, qn, beta [64].
constexpr int LA = GC + 4, LT = GC + 1;
constexpr size_t kPrepSmem = 2 * GC * GD * 2 + (GC * LA + GC * LT + 5 * GC) * sizeof(float);

__global__ void __launch_bounds__(NTH, 3)
gdn_chunk_prep_kernel(ChunkArgs a, int l2norm, float eps) {
  extern __shared__ __align__(128) unsigned char sm8[];
  const uint32_t ks = smem_addr(sm8), qs = ks + GC * GD * 2;
  float* A = reinterpret_cast<float*>(sm8 + 2 * GC * GD * 2);
  float* Ts = A + GC * LA;
  float *Gs = Ts + GC * LT, *Gl = Gs + GC, *kn = Gl + GC, *qn = kn + GC, *bs = qn + GC;
  const int ci = blockIdx.x % a.n, bh = blockIdx.x / a.n, b = bh / a.Hv, hv = bh % a.Hv;
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
  for (int r = warp; r < 2 * GC; r += 8) {   // L2 factors: a warp per row of k, then of q
    const uint2 w = *reinterpret_cast<const uint2*>(sm8 + (r >> 6) * GC * GD * 2 + sw_off<256>(r & 63, lane >> 1) + (lane & 1) * 8);
    const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w.x));
    const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w.y));
    const float s = warp_sum(x.x * x.x + x.y * x.y + y.x * y.x + y.y * y.y);
    const float f = l2norm ? rsqrtf(s + eps) : 1.f;
    if (lane == 0) (r < GC ? kn : qn)[r & 63] = r < GC ? f : f * rsqrtf(static_cast<float>(GD));
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
  __syncthreads();                           // kn, qn
  const long long co = static_cast<long long>(bh) * a.n + ci;
  __nv_bfloat16* pc = a.pieces + co * 6 * PIECE;
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
      for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(pc + (3 + s) * PIECE + i * GC + c) = w[s];
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
  __syncthreads();
  if (tid < GC) {
    // column tid of T: t[i] = [i == tid] - sum_{j<i} A[i][j] t[j]; a column depends on its own earlier rows only
    float t[GC];
#pragma unroll
    for (int i = 0; i < GC; ++i) {
      float a0 = (i == tid) ? 1.f : 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
      for (int j = 0; j + 3 < i; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(A + i * LA + j);
        a0 -= x.x * t[j];
        a1 -= x.y * t[j + 1];
        a2 -= x.z * t[j + 2];
        a3 -= x.w * t[j + 3];
      }
#pragma unroll
      for (int j = i & ~3; j < i; ++j) a0 -= A[i * LA + j] * t[j];
      t[i] = (a0 + a1) + (a2 + a3);
      Ts[i * LT + tid] = t[i];
    }
  }
  __syncthreads();
  for (int e = tid; e < PIECE / 2; e += NTH) {
    const int i = e >> 5, c = (e & 31) * 2;
    uint32_t w[3];
    split3(Ts[i * LT + c], Ts[i * LT + c + 1], w[0], w[1], w[2]);
#pragma unroll
    for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(pc + s * PIECE + i * GC + c) = w[s];
  }
}

// Shared: k and q of a chunk [128, 256 bytes], two buffers; three pieces each of T, P [64, 64], S [128, DV], R (later the
// scaled Vn) and Vn [64, DV]; row factors, two buffers.  A warp has rows 16 mt of k and q, of R, Vn and O, rows 32 mt of the
// state, and the columns of one half of DV.
template <int DV>
constexpr size_t scan_smem() {
  return 2 * 2 * GC * GD * 2 + 6 * TILE + 3 * (GD + 2 * GC) * DV * 2 + 2 * VEC * GC * sizeof(float);
}

template <int DV>
__global__ void __launch_bounds__(NTH, 1)
gdn_chunk_scan_kernel(ChunkArgs a, const float* S0, float* S_out, __nv_bfloat16* __restrict__ out) {
  constexpr int NT = DV / 16;                // columns of a warp in eights
  constexpr int RB = DV * 2;                 // bytes of a row of S, R, Vn
  constexpr int KQ = 2 * GC * GD * 2;
  extern __shared__ __align__(128) unsigned char sm8[];
  const uint32_t kq = smem_addr(sm8), Ts = kq + 2 * KQ, Ps = Ts + 3 * TILE, Ss = Ps + 3 * TILE, Rs = Ss + 3 * GD * RB, Vs = Rs + 3 * GC * RB;
  float* vec = reinterpret_cast<float*>(sm8 + 2 * KQ + 6 * TILE + 3 * (GD + 2 * GC) * RB);
  constexpr int SL = GD / DV;
  const int slice = blockIdx.x % SL, bh = blockIdx.x / SL, b = bh / a.Hv, hv = bh % a.Hv, hk = hv / (a.Hv / a.Hk);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, mt = warp >> 1, nh = warp & 1;
  const int col0 = slice * DV + nh * (DV / 2);         // the warp's columns in the head
  const int g4 = lane >> 2, c2 = (lane & 3) * 2;
  // 16-byte chunk of a [*, DV] tile, rows of RB bytes
  auto at = [&](uint32_t base, int row, int chunk) {
    if constexpr (RB == 128) return base + sw_off<128>(row, chunk);
    else return base + static_cast<uint32_t>(row * RB + ((chunk ^ ((row >> 1) & 3)) << 4));
  };
  auto put = [&](uint32_t base, int rows, int row, int col, float x, float y) {      // pieces of two entries
    uint32_t w[3];
    split3(x, y, w[0], w[1], w[2]);
#pragma unroll
    for (int s = 0; s < 3; ++s)
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(at(base + s * rows * RB, row, col >> 3) + (col & 7) * 2), "r"(w[s]) : "memory");
  };
  auto load_kq = [&](int ci, int buf) {
    const int t0 = (a.c0 + ci) * GC, n = min(GC, a.T - t0);
    for (int e = tid; e < 2 * GC * 16; e += NTH) {
      const int which = e >> 10, r = (e >> 4) & 63, c = e & 15, t = t0 + min(r, n - 1);
      const __nv_bfloat16* src = which ? a.q + b * a.q_bs + t * a.q_ts : a.k + b * a.k_bs + t * a.k_ts;
      cp_async16(kq + buf * KQ + sw_off<256>(which * GC + r, c), src + hk * GD + c * 8, r < n);
    }
    const float* vp = a.vec + (static_cast<long long>(bh) * a.n + ci) * VEC * GC;
    if (tid < VEC * GC / 4) cp_async16(smem_addr(vec + buf * VEC * GC) + tid * 16, vp + tid * 4, true);
  };
  auto load_tp = [&](int ci, int which) {    // 0: T, 1: P
    const __nv_bfloat16* pc = a.pieces + (static_cast<long long>(bh) * a.n + ci) * 6 * PIECE + which * 3 * PIECE;
    for (int e = tid; e < 3 * GC * 8; e += NTH) {
      const int s = e >> 9, r = (e >> 3) & 63, c = e & 7;
      cp_async16((which ? Ps : Ts) + s * TILE + sw_off<128>(r, c), pc + s * PIECE + r * GC + c * 8, true);
    }
  };
  // three pieces of B fragments: rows k0 .. k0 + 16 of a [*, DV] tile, the warp's columns
  auto load_b = [&](uint32_t base, int rows, int k0, uint32_t (*f)[NT][2]) {
#pragma unroll
    for (int s = 0; s < 3; ++s)
#pragma unroll
      for (int j = 0; j < NT; j += 2)
        ldsm4t(at(base + s * rows * RB, k0 + (lane & 15), nh * (DV / 16) + j + (lane >> 4)), f[s][j][0], f[s][j][1], f[s][j + 1][0], f[s][j + 1][1]);
  };
  // leading and small products of 32-bit [64, 64] pieces with a 32-bit [64, DV] tile; both lower triangular in blocks
  auto product6 = [&](uint32_t base, uint32_t tile, float (*hi)[4], float (*lo)[4]) {
    for (int s = 0; s <= mt; ++s) {
      uint32_t fa[3][4], fb[3][NT][2];
#pragma unroll
      for (int p = 0; p < 3; ++p)
        ldsm4(base + p * TILE + sw_off<128>(mt * 16 + (lane & 15), 2 * s + (lane >> 4)), fa[p][0], fa[p][1], fa[p][2], fa[p][3]);
      load_b(tile, GC, s * 16, fb);
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        mma16816(lo[j], fa[2], fb[0][j][0], fb[0][j][1]);
        mma16816(lo[j], fa[1], fb[1][j][0], fb[1][j][1]);
        mma16816(lo[j], fa[0], fb[2][j][0], fb[2][j][1]);
        mma16816(lo[j], fa[1], fb[0][j][0], fb[0][j][1]);
        mma16816(lo[j], fa[0], fb[1][j][0], fb[1][j][1]);
        mma16816(hi[j], fa[0], fb[0][j][0], fb[0][j][1]);
      }
    }
  };

  float S[2][NT][4];                         // rows 32 mt + 16 i + g4 (+ 8), columns col0 + 8 j + c2
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = mt * 32 + i * 16 + g4 + 8 * h;
        const float2 x = S0 ? *reinterpret_cast<const float2*>(S0 + static_cast<long long>(bh) * GD * GD + r * GD + col0 + j * 8 + c2)
                            : make_float2(0.f, 0.f);
        S[i][j][2 * h] = x.x;
        S[i][j][2 * h + 1] = x.y;
        put(Ss, GD, r, nh * (DV / 2) + j * 8 + c2, x.x, x.y);
      }
  load_kq(0, 0);
  load_tp(0, 0);
  cp_commit();
  for (int ci = 0; ci < a.n; ++ci) {
    const int buf = ci & 1, t0 = (a.c0 + ci) * GC, n = min(GC, a.T - t0);
    const float* vf = vec + buf * VEC * GC;
    const uint32_t kqb = kq + buf * KQ;
    cp_wait<0>();
    __syncthreads();                         // k, q, factors and T are here, the state's pieces are written, P and the other buffer are free
    load_tp(ci, 1);
    cp_commit();
    if (ci + 1 < a.n) load_kq(ci + 1, buf ^ 1);
    cp_commit();
    uint32_t vv[2][NT];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int r = mt * 16 + g4 + 8 * h;
        vv[h][j] = r < n ? *reinterpret_cast<const uint32_t*>(a.v + b * a.v_bs + (t0 + r) * a.v_ts + hv * GD + col0 + j * 8 + c2) : 0u;
      }
    // k S and q S
    float xk[NT][4] = {}, xq[NT][4] = {}, lk[NT][4] = {}, lq[NT][4] = {};
#pragma unroll 2
    for (int s = 0; s < GD / 16; ++s) {
      uint32_t fk[4], fq[4], fb[3][NT][2];
      const int r = mt * 16 + (lane & 15), c = 2 * s + (lane >> 4);
      ldsm4(kqb + sw_off<256>(r, c), fk[0], fk[1], fk[2], fk[3]);
      ldsm4(kqb + sw_off<256>(GC + r, c), fq[0], fq[1], fq[2], fq[3]);
      load_b(Ss, GD, s * 16, fb);
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        mma16816(lk[j], fk, fb[2][j][0], fb[2][j][1]);
        mma16816(lq[j], fq, fb[2][j][0], fb[2][j][1]);
        mma16816(lk[j], fk, fb[1][j][0], fb[1][j][1]);
        mma16816(lq[j], fq, fb[1][j][0], fb[1][j][1]);
        mma16816(xk[j], fk, fb[0][j][0], fb[0][j][1]);
        mma16816(xq[j], fq, fb[0][j][0], fb[0][j][1]);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = mt * 16 + g4 + 8 * h;
      const float bt = vf[r], f1 = vf[GC + r], f2 = vf[2 * GC + r];
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const float x = bt * __uint_as_float(vv[h][j] << 16) - f1 * (xk[j][2 * h] + lk[j][2 * h]);
        const float y = bt * __uint_as_float(vv[h][j] & 0xFFFF0000u) - f1 * (xk[j][2 * h + 1] + lk[j][2 * h + 1]);
        put(Rs, GC, r, nh * (DV / 2) + j * 8 + c2, x, y);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          xq[j][2 * h + e] = f2 * (xq[j][2 * h + e] + lq[j][2 * h + e]);
          xk[j][2 * h + e] = lk[j][2 * h + e] = lq[j][2 * h + e] = 0.f;
        }
      }
    }
    __syncthreads();
    product6(Ts, Rs, xk, lk);                // Vn
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) xk[j][e] += lk[j][e];
    __syncthreads();                         // everyone has read R and T
    if (ci + 1 < a.n) load_tp(ci + 1, 0);
    cp_commit();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = mt * 16 + g4 + 8 * h;
      const float f3 = vf[3 * GC + r];
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int c = nh * (DV / 2) + j * 8 + c2;
        put(Vs, GC, r, c, xk[j][2 * h], xk[j][2 * h + 1]);
        put(Rs, GC, r, c, f3 * xk[j][2 * h], f3 * xk[j][2 * h + 1]);
      }
    }
    cp_wait<2>();                            // P; the next chunk's k, q and T may still be on their way
    __syncthreads();
    {                                        // the state: k^T (scaled Vn)
      float hi[2][NT][4] = {}, lo[2][NT][4] = {};
#pragma unroll
      for (int s = 0; s < GC / 16; ++s) {
        uint32_t fa[2][4], fb[3][NT][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)          // stored [token, key dim]: rows and columns of the fragment change places
          ldsm4t(kqb + sw_off<256>(s * 16 + (lane & 7) + ((lane >> 4) << 3), mt * 4 + 2 * i + ((lane >> 3) & 1)), fa[i][0], fa[i][1], fa[i][2], fa[i][3]);
        load_b(Rs, GC, s * 16, fb);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            mma16816(lo[i][j], fa[i], fb[2][j][0], fb[2][j][1]);
            mma16816(lo[i][j], fa[i], fb[1][j][0], fb[1][j][1]);
            mma16816(hi[i][j], fa[i], fb[0][j][0], fb[0][j][1]);
          }
      }
      const float gC = vf[4 * GC];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
#pragma unroll
          for (int e = 0; e < 4; ++e) S[i][j][e] = S[i][j][e] * gC + (hi[i][j][e] + lo[i][j][e]);
#pragma unroll
          for (int h = 0; h < 2; ++h)
            put(Ss, GD, mt * 32 + i * 16 + g4 + 8 * h, nh * (DV / 2) + j * 8 + c2, S[i][j][2 * h], S[i][j][2 * h + 1]);
        }
    }
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) xk[j][e] = 0.f;
    product6(Ps, Vs, xk, lq);                // O
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = mt * 16 + g4 + 8 * h;
      if (r < n) {
        __nv_bfloat16* o = out + ((static_cast<long long>(b) * a.T + t0 + r) * a.Hv + hv) * GD + col0 + c2;
#pragma unroll
        for (int j = 0; j < NT; ++j)
          *reinterpret_cast<uint32_t*>(o + j * 8) = pack_bf16(xq[j][2 * h] + (xk[j][2 * h] + lq[j][2 * h]),
                                                              xq[j][2 * h + 1] + (xk[j][2 * h + 1] + lq[j][2 * h + 1]));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float2*>(S_out + static_cast<long long>(bh) * GD * GD + (mt * 32 + i * 16 + g4 + 8 * h) * GD + col0 + j * 8 + c2) =
            make_float2(S[i][j][2 * h], S[i][j][2 * h + 1]);
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
                          bool l2norm, float eps, void* workspace, cudaStream_t stream) {
  if (KD != GD || VD != GD) return "gdn_chunk_fwd: key and value head dim must be 128";
  if (Hk <= 0 || Hv % Hk) return "gdn_chunk_fwd: value heads must be a multiple of key heads";
  if (B == 0 || T == 0) return nullptr;
  if (!FERRL_ONCE_PER_DEVICE(
          cudaFuncSetAttribute(gdn_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kPrepSmem)) == cudaSuccess &&
          cudaFuncSetAttribute(gdn_chunk_scan_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(scan_smem<64>())) == cudaSuccess &&
          cudaFuncSetAttribute(gdn_chunk_scan_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(scan_smem<32>())) == cudaSuccess))
    return "gdn_chunk_fwd: cannot reserve shared memory";
  const int round = chunk_round(B, T, Hv), chunks = (T + GC - 1) / GC;
  ChunkArgs a{static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v),
              q_bs, q_ts, k_bs, k_ts, v_bs, v_ts, g, beta, T, Hk, Hv, 0, 0, static_cast<__nv_bfloat16*>(workspace), nullptr};
  // One CTA fits an SM: narrow slices only where they all run at once.
  const bool narrow = static_cast<long long>(B) * Hv * 4 <= 148;
  for (int c0 = 0; c0 < chunks; c0 += round) {
    a.c0 = c0;
    a.n = std::min(round, chunks - c0);
    a.vec = reinterpret_cast<float*>(a.pieces + static_cast<long long>(B) * Hv * a.n * 6 * PIECE);
    const float* from = c0 == 0 ? S0 : S_out;
    gdn_chunk_prep_kernel<<<a.n * B * Hv, NTH, kPrepSmem, stream>>>(a, l2norm ? 1 : 0, eps);
    if (narrow) gdn_chunk_scan_kernel<32><<<B * Hv * 4, NTH, scan_smem<32>(), stream>>>(a, from, S_out, static_cast<__nv_bfloat16*>(out));
    else gdn_chunk_scan_kernel<64><<<B * Hv * 2, NTH, scan_smem<64>(), stream>>>(a, from, S_out, static_cast<__nv_bfloat16*>(out));
    count_launch(2);
  }
  return cudaGetLastError() == cudaSuccess ? nullptr : "gdn_chunk_fwd launch failed";
}

}  // namespace ferrl
