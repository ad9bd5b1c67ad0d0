// Adapter gradients: out[R, C] = U^T X with U [M, R] and X [M, C] bf16, fp32 result.
//
//   dA = (dy B)^T x        U = dy B  [tokens, R],  X = x   [tokens, K]
//   dB^T = t^T dy          U = x A^T [tokens, R],  X = dy  [tokens, N]
//
// The reduction runs over the token dimension, which is the strided one in both operands, so the
// TMA/tcgen05 GEMM (K-major operands) does not apply without materialising transposes of the
// activations.  Here both operands are streamed once, row-major, through a cp.async ring and the
// transposed fragments come out of ldmatrix.trans; the products run on mma.sync m16n8k16.
// Work is split over column tiles and token ranges; the per-range partial tiles are summed by the
// last CTA of each column tile in range order, so the result does not depend on scheduling.
// The reference forms these products with candle matmuls on transposed views
// (crates/ferrl/src/lora.rs backward of the adapter path).
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

constexpr int LG_COLS = 128;     // output columns per CTA
constexpr int LG_ROWS = 64;      // tokens per stage
constexpr int LG_STAGES = 3;
constexpr int LG_X_BYTES = LG_ROWS * 256;      // a stage's tile of X: rows of 128 bf16
// a stage's tile of U: rows of 128 bytes up to rank 64, of 256 above
template <int RT> constexpr int LG_U_ROW = RT <= 4 ? 128 : 256;
template <int RT> constexpr int LG_STAGE_BYTES = LG_X_BYTES + LG_ROWS * LG_U_ROW<RT>;

// Bound by reading X once.  In a chain of calls, us (bytes' time), before and now: 11392 tokens, rank 16 x 4096 columns 25 and 22 (14),
// 32 x 24576 114 and 90 (86), 48 x 6144 50 and 34 (22); 5119 tokens, 64 x 10240 54 and 32 (16); 4608 tokens, 32 x 43008 106 and 70 (61).  What
// the time was:
// two CTAs an SM, because a tile of U took as much shared memory as one of X; an address computed anew for every 16 bytes;
// the ranges' sums fetched one by one by the last CTA; ranges cut so that they filled waves and not so that they ended together.
constexpr int LG_CHAIN = 8;      // stages whose products are summed by the tensor cores alone

template <int RT>   // RT 16-row tiles of R (R <= 16*RT <= 128)
__global__ void __launch_bounds__(128, RT <= 4 ? 3 : 2)
lora_grad_kernel(const __nv_bfloat16* __restrict__ U, long long ldu, int R, const __nv_bfloat16* __restrict__ X,
                 long long ldx, int C, int M, int rows_per_split, float* __restrict__ partial,
                 int* __restrict__ counters, float* __restrict__ out, long long ldo) {
  extern __shared__ __align__(128) uint8_t lsm[];
  __shared__ int s_last;
  const int ct = blockIdx.x, split = blockIdx.y, n_splits = gridDim.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = ct * LG_COLS;
  const int m_begin = split * rows_per_split, m_end = min(M, m_begin + rows_per_split);
  const int n_stages = m_end > m_begin ? (m_end - m_begin + LG_ROWS - 1) / LG_ROWS : 0;
  constexpr int UR = LG_U_ROW<RT>;
  // this thread's 16 bytes of every eighth row of X, and of U rows a stage's worth apart
  const int xr = threadIdx.x >> 4, xc = threadIdx.x & 15;
  const bool x_ok = c0 + xc * 8 < C;
  const __nv_bfloat16* xp = X + static_cast<long long>(m_begin + xr) * ldx + (x_ok ? c0 + xc * 8 : 0);
  constexpr int UC = 2 * RT <= 8 ? 8 : 16;     // threads a row of U, those past 2 RT idle
  const int ur = threadIdx.x / UC, uc = threadIdx.x % UC;
  const bool u_ok = uc * 8 < R;
  const __nv_bfloat16* up = U + static_cast<long long>(m_begin + ur) * ldu + (u_ok ? uc * 8 : 0);

  auto issue = [&](int s) {
    if (s < n_stages) {
      const uint32_t xt = smem_addr(lsm + (s % LG_STAGES) * LG_STAGE_BYTES<RT>), ut = xt + LG_X_BYTES;
      const int left = m_end - m_begin - s * LG_ROWS;          // rows of this stage that there are
#pragma unroll
      for (int i = 0; i < LG_ROWS / 8; ++i) {
        const int r = i * 8 + xr;
        cp_async16(xt + sw_off<256>(r, xc), r < left ? xp + static_cast<long long>(i) * 8 * ldx : X, x_ok && r < left);
      }
      if (uc < 2 * RT) {
#pragma unroll
        for (int i = 0; i < LG_ROWS * UC / 128; ++i) {
          const int r = i * (128 / UC) + ur;
          cp_async16(ut + sw_off<UR>(r, uc), r < left ? up + static_cast<long long>(i) * (128 / UC) * ldu : U, u_ok && r < left);
        }
      }
      xp += LG_ROWS * ldx;
      up += LG_ROWS * ldu;
    }
    cp_commit();
  };

  float acc[RT][4][4];
#pragma unroll
  for (int a = 0; a < RT; ++a)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[a][n][e] = 0.f;

  // The tensor cores cut off where they add, so a long chain of sums drifts: up to rank 64 every LG_CHAIN stages join a total.
  constexpr bool kTotal = RT <= 4;
  float total[kTotal ? RT : 1][4][4];
#pragma unroll
  for (int a = 0; a < (kTotal ? RT : 1); ++a)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) total[a][n][e] = 0.f;
  auto join = [&]() {
    if constexpr (kTotal) {
#pragma unroll
      for (int a = 0; a < RT; ++a)
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            total[a][n][e] += acc[a][n][e];
            acc[a][n][e] = 0.f;
          }
    }
  };

#pragma unroll
  for (int s = 0; s < LG_STAGES - 1; ++s) issue(s);
  for (int s = 0; s < n_stages; ++s) {
    cp_wait<LG_STAGES - 2>();
    __syncthreads();
    issue(s + LG_STAGES - 1);
    const uint32_t xt = smem_addr(lsm + (s % LG_STAGES) * LG_STAGE_BYTES<RT>), ut = xt + LG_X_BYTES;
#pragma unroll
    for (int ks = 0; ks < LG_ROWS / 16; ++ks) {
      // B fragments: X[k = token][n = column], 4 n-tiles of this warp's 32 columns
      uint32_t b[8];
      {
        const int row = ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
        const int chunk = warp * 4 + (lane >> 4);
        ldsm4t(xt + sw_off<256>(row, chunk), b[0], b[1], b[2], b[3]);
        ldsm4t(xt + sw_off<256>(row, chunk + 2), b[4], b[5], b[6], b[7]);
      }
#pragma unroll
      for (int rt = 0; rt < RT; ++rt) {
        // A fragment: U^T[row = r][k = token] out of the [token][r] tile
        uint32_t a[4];
        const int mat = lane >> 3;
        const int row = ks * 16 + (lane & 7) + (mat >> 1) * 8;
        const int chunk = rt * 2 + (mat & 1);
        ldsm4t(ut + sw_off<UR>(row, chunk), a[0], a[1], a[2], a[3]);
#pragma unroll
        for (int n = 0; n < 4; ++n) mma16816(acc[rt][n], a, b[2 * n], b[2 * n + 1]);
      }
    }
    if (s % LG_CHAIN == LG_CHAIN - 1) join();
  }
  cp_wait<0>();
  if constexpr (kTotal) {
    join();
#pragma unroll
    for (int a = 0; a < RT; ++a)
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[a][n][e] = total[a][n][e];
  }

  // partial tile of this token range: [split][16*RT][C], fp32
  const int g = lane >> 2, t = lane & 3;
  float* part = partial + static_cast<long long>(split) * (16 * RT) * C;
#pragma unroll
  for (int rt = 0; rt < RT; ++rt)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int col = c0 + warp * 32 + n * 8 + 2 * t;
      if (col < C) {   // C % 8 == 0, so col + 1 < C as well
        *reinterpret_cast<float2*>(part + static_cast<long long>(rt * 16 + g) * C + col) = make_float2(acc[rt][n][0], acc[rt][n][1]);
        *reinterpret_cast<float2*>(part + static_cast<long long>(rt * 16 + g + 8) * C + col) = make_float2(acc[rt][n][2], acc[rt][n][3]);
      }
    }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const int seen = atomicAdd(&counters[ct], 1);
    s_last = (seen == n_splits - 1);
    if (s_last) counters[ct] = 0;     // ready for the next call on this stream
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // the last CTA of this column tile sums the ranges in order; four places of four ranges are on their way at a time (8192 tokens,
  // rank 128 x 1000 columns, 32 ranges: 48 us with one place as the compiler unrolls it, 55 with two of eight, 51 with four of four;
  // over 1008 shapes the last takes 0.92 times as long as two of eight)
  constexpr int NP = 4, NR = 4;
  const long long range = static_cast<long long>(16 * RT) * C;
  for (int i = threadIdx.x; i < R * (LG_COLS / 4); i += NP * 128) {
    const float* src[NP];
    bool ok[NP];
    float4 sum[NP];
#pragma unroll
    for (int h = 0; h < NP; ++h) {
      const int at = i + 128 * h, r = at / (LG_COLS / 4), c = c0 + (at % (LG_COLS / 4)) * 4;
      ok[h] = r < R && c < C;
      src[h] = partial + (ok[h] ? static_cast<long long>(r) * C + c : 0);
      sum[h] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    auto load = [&](int h, int s) { return __ldcg(reinterpret_cast<const float4*>(src[h] + s * range)); };
    auto add = [&](int h, const float4& v) {
      sum[h].x += v.x; sum[h].y += v.y; sum[h].z += v.z; sum[h].w += v.w;
    };
    int s = 0;
    for (; s + NR <= n_splits; s += NR) {
      float4 v[NP][NR];
#pragma unroll
      for (int j = 0; j < NR; ++j)
#pragma unroll
        for (int h = 0; h < NP; ++h) v[h][j] = load(h, s + j);
#pragma unroll
      for (int j = 0; j < NR; ++j)
#pragma unroll
        for (int h = 0; h < NP; ++h) add(h, v[h][j]);
    }
    for (; s < n_splits; ++s)
#pragma unroll
      for (int h = 0; h < NP; ++h) add(h, load(h, s));
#pragma unroll
    for (int h = 0; h < NP; ++h) {
      const int at = i + 128 * h;
      if (ok[h]) *reinterpret_cast<float4*>(out + static_cast<long long>(at / (LG_COLS / 4)) * ldo + c0 + (at % (LG_COLS / 4)) * 4) = sum[h];
    }
  }
}

}  // namespace

size_t lora_grad_workspace_floats(int R, int C, int n_splits) {
  const int rt = (R + 15) / 16;
  return static_cast<size_t>(n_splits) * rt * 16 * C;
}

int lora_grad_splits(int M, int R, int C, int num_sms) {
  // Three CTAs fit on an SM up to rank 64, two above.  Up to rank 64 the token split is the largest whose CTAs all run at once:
  // few long ranges, which end together (us by single calls, and with the rule below: 11392 tokens, rank 32 x 24576 columns 107 and 117,
  // 16 x 12288 64 and 68; 5119 tokens, 64 x 10240 39 and 50).  With more column tiles than that, and above rank 64, where a range is one chain
  // of sums, the split is chosen so that the grid fills whole waves: a grid of 1.08 waves takes as long as one of two.
  const int col_tiles = (C + LG_COLS - 1) / LG_COLS;
  const int slots = (R <= 64 ? 3 : 2) * num_sms;
  const int max_s = std::min(64, std::max(1, (M + 4 * LG_ROWS - 1) / (4 * LG_ROWS)));   // at least four stages per CTA
  if (R <= 64 && col_tiles <= slots) return std::min(max_s, slots / col_tiles);
  int best = 1;
  double best_eff = 0.0;
  for (int s = 1; s <= max_s; ++s) {
    const long long ctas = static_cast<long long>(col_tiles) * s;
    const long long waves = (ctas + slots - 1) / slots;
    const double eff = static_cast<double>(ctas) / static_cast<double>(waves * slots);
    if (eff > best_eff + 1e-9) {
      best_eff = eff;
      best = s;
    }
    if (eff >= 0.93 && ctas >= slots / 2) return s;      // smallest split that fills its waves
  }
  return best;
}

const char* lora_grad(const void* U, long long ldu, int R, const void* X, long long ldx, int C, int M, int n_splits,
                      float* partial, int* counters, float* out, long long ldo, cudaStream_t stream) {
  if (R <= 0 || R > 128 || (R % 8)) return "lora_grad: R must be a multiple of 8, at most 128";
  if ((C % 8) || (ldx % 8) || (ldu % 8) || (ldo % 4)) return "lora_grad: C, ldx, ldu must be multiples of 8 (ldo of 4)";
  if ((reinterpret_cast<uintptr_t>(U) & 15) || (reinterpret_cast<uintptr_t>(X) & 15) || (reinterpret_cast<uintptr_t>(out) & 15))
    return "lora_grad: operands must be 16-byte aligned";
  if (M <= 0 || C <= 0) return nullptr;
  const int rt = (R + 15) / 16;
  const int rows_per_split = ((M + n_splits - 1) / n_splits + LG_ROWS - 1) / LG_ROWS * LG_ROWS;
  dim3 grid((C + LG_COLS - 1) / LG_COLS, n_splits);
#define FERRL_LG(RTV)                                                                                                 \
  case RTV: {                                                                                                         \
    constexpr int smem = LG_STAGES * LG_STAGE_BYTES<RTV>;                                                             \
    if (!FERRL_ONCE_PER_DEVICE(cudaFuncSetAttribute(lora_grad_kernel<RTV>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                    smem) == cudaSuccess))                                            \
      return "lora_grad: cannot reserve shared memory";                                                               \
    lora_grad_kernel<RTV><<<grid, 128, smem, stream>>>(static_cast<const __nv_bfloat16*>(U), ldu, R,                  \
                                                       static_cast<const __nv_bfloat16*>(X), ldx, C, M, rows_per_split, \
                                                       partial, counters, out, ldo);                                  \
    break;                                                                                                            \
  }
  switch (rt) {
    FERRL_LG(1) FERRL_LG(2) FERRL_LG(3) FERRL_LG(4) FERRL_LG(5) FERRL_LG(6) FERRL_LG(7) FERRL_LG(8)
    default: return "lora_grad: unsupported rank";
  }
#undef FERRL_LG
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "lora_grad launch failed";
}


// The adapters of a fused projection as operands of its products: A_j [r, K] stacked, scale * B_j [rows_j, r] in the
// columns of its adapter and the rows of its part, 16 bits, zeros elsewhere.  One launch in place of a dozen small
// concatenations, products and casts.
namespace {

template <typename F>
__device__ __forceinline__ void each(long long n, F f) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += static_cast<long long>(gridDim.x) * blockDim.x) f(i);
}

__global__ void lora_pack_kernel(LoraParts p, __nv_bfloat16* __restrict__ a16, __nv_bfloat16* __restrict__ b16) {
  const long long na = static_cast<long long>(p.Rp) * p.K, nb = static_cast<long long>(p.N) * p.Rp;
  each(na + nb, [&](long long i) {
    if (i < na) {
      const int row = static_cast<int>(i / p.K), j = row / p.r;
      a16[i] = __float2bfloat16_rn(j < p.n ? p.A[j][i - static_cast<long long>(j) * p.r * p.K] : 0.f);
      return;
    }
    i -= na;
    const int n = static_cast<int>(i / p.Rp), c = static_cast<int>(i - static_cast<long long>(n) * p.Rp), j = c / p.r;
    const bool on = j < p.n && n >= p.start[j] && n < p.start[j] + p.rows[j];
    b16[i] = __float2bfloat16_rn(on ? p.B[j][static_cast<long long>(n - p.start[j]) * p.r + c - j * p.r] * p.scale : 0.f);
  });
}

// gradient of scale * B_j from the transposed gradient [R, N] of the stacked operand
__global__ void lora_unpack_kernel(const float* __restrict__ dbt, long long ld, LoraParts p, float* __restrict__ out) {
  const int j = blockIdx.y;
  float* o = out + p.off[j];
  each(static_cast<long long>(p.rows[j]) * p.r, [&](long long i) {
    const int c = static_cast<int>(i / p.rows[j]), row = static_cast<int>(i - static_cast<long long>(c) * p.rows[j]);
    o[static_cast<long long>(row) * p.r + c] = dbt[(static_cast<long long>(j) * p.r + c) * ld + p.start[j] + row] * p.scale;
  });
}

}  // namespace

const char* lora_pack(const LoraParts& p, void* a16, void* b16, cudaStream_t s) {
  const long long n = static_cast<long long>(p.Rp) * (p.K + p.N);
  if (n == 0) return nullptr;
  const long long blocks = (n + 255) / 256;
  lora_pack_kernel<<<static_cast<unsigned>(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, s>>>(p, static_cast<__nv_bfloat16*>(a16),
                                                                                               static_cast<__nv_bfloat16*>(b16));
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "lora_pack launch failed";
}

const char* lora_unpack(const float* dbt, long long ld, const LoraParts& p, float* out, cudaStream_t s) {
  long long most = 0;
  for (int j = 0; j < p.n; ++j) most = most < p.rows[j] ? p.rows[j] : most;
  if (p.n == 0 || most * p.r == 0) return nullptr;
  const long long blocks = (most * p.r + 255) / 256;
  lora_unpack_kernel<<<dim3(static_cast<unsigned>(blocks < 148 * 8 ? blocks : 148 * 8), p.n), 256, 0, s>>>(dbt, ld, p, out);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "lora_unpack launch failed";
}

}  // namespace ferrl
