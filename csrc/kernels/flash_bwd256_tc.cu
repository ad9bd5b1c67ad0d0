// Causal flash-attention backward at head dim 256 on the 5th-generation tensor cores (optional sliding window).
//
// dK and dV of 128 keys would take all 512 columns of tensor memory, so they are formed by CTAs of their own that each
// form the scores again; with dQ that makes three passes of one shape, 8 products instead of 7:
//
//            rows (resident)      streamed, 64 rows a step       scores                      W (16 bits, tensor memory)       result
//   dQ       128 queries: Q, dO   TA = K, TB = V                 S = Q K^T, dP = dO V^T      P o (dP - delta)                 dQ += W K
//   dK       128 keys: K, V       TA = Q, TB = dO, head by head  S^T = K Q^T, dP^T = V dO^T  P^T o (dP^T - delta)             dK += W Q
//   dV       128 keys: K          TA = Q, TB = dO, head by head  S^T = K Q^T                 P^T                              dV += W dO
//
// Tensor memory: result 256 columns, two score tiles of 64, two buffers of W of 32.  W is the A operand of the last product
// from there; its B operand is the streamed tile as it lies, read through an MN-major descriptor.  Shared memory holds the
// resident tiles (64 KB each) and three streamed ones (32 KB): two of TA and one of TB, or for dV two of TA and three of TB.
// No float atomics; every sum has a fixed order.
//
// What bounds it: a streamed tile of TA stays from its load through scores, softmax and last product, and two slots are all
// that fits, so a step takes about half of that life; the tensor cores need 1536 of its cycles.  All three kernels with the
// tensor maps' host time, against the warp-level kernels of flash_attn.cu: 5119 tokens, 24 and 4 heads 5974 -> 1523 us (529
// TFLOP/s, 32 % of measured); 4 x 1535, 16 and 2 heads 1732 -> 515; 1000, 8 and 2 heads 392 -> 95; 64, 8 and 2 heads 34 -> 22.
// Many rows of a tile or less are left to them (flash_bwd256_tc_better).
//
// dK and dV walk every query head of the group.  The first key tile sees all queries, so where key tiles are few a cluster
// of 2 or 4 CTAs takes the heads of a key tile in shares and adds the shares through distributed shared memory in rank order.
//
// Rows past a sequence's own length are read as zeros (4-D tensor maps), never as the next sequence's.
//
// Reference behaviour: the gradient of the eager GQA attention in crates/ferrl/src/dense.rs (candle autograd through
// softmax(QK^T)V).  Every wait is bounded.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "../api.h"
#include "../common.cuh"
#include "../gemm/tc_common.cuh"

namespace ferrl {
namespace {

using namespace tc;

constexpr int HD = 256;                    // head dim
constexpr int RT = 128;                    // resident rows
constexpr int KT = 64;                     // streamed rows a step
constexpr int R_ATOM = RT * 128;           // [128 rows x 64 columns]: 16 KB
constexpr int R_TILE = 4 * R_ATOM;         // 64 KB
constexpr int T_ATOM = KT * 128;           // [64 rows x 64 columns]: 8 KB
constexpr int T_TILE = 4 * T_ATOM;         // 32 KB
constexpr int TILES = 2 * R_TILE + 3 * T_TILE;
constexpr int STAT_SLOTS = 3;
constexpr int SMEM = TILES + STAT_SLOTS * KT * 8 + 256;
static_assert(SMEM <= 227 * 1024, "shared memory");
constexpr int THREADS = 320;               // TMA, MMA, eight softmax warps
constexpr uint32_t kBMajorMN = 1u << 16;   // instruction descriptor: B operand is MN-major
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kMaxShares = 4;

struct Bwd256Params {
  const float2* stats;      // [B, Hq, S_pad] per query row: {lse * log2(e), rowsum(O o dO)}, zeros for the padding rows
  int S_pad;                // S rounded up to 128
  __nv_bfloat16 *dq, *dk, *dv;
  long long dq_bs, dq_ts, dk_bs, dk_ts, dv_bs, dv_ts;
  int B, S, Hq, Hkv, window;      // window 0: plain causal; w > 0: query i sees keys (i - w, i]
  int shares;                     // CTAs of a cluster that share a key tile's heads
  float scale;
  int* status;
};

enum Mode { kDQ, kDK, kDV };

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void st_peer(uint32_t addr, uint32_t rank, float4 v) {      // addr: this CTA's view of the place
  uint32_t there;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(addr), "r"(rank));
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(there), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// One warp per row.  The padded, interleaved layout lets a step fetch the 64 rows of a query tile with one 512-byte copy.
__global__ void stats256_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o, const float* __restrict__ lse,
                                float2* __restrict__ stats, int B, int S, int S_pad, int Hq) {
  const long long w = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= static_cast<long long>(B) * S_pad * Hq) return;
  const int h = static_cast<int>(w % Hq);
  const long long bs = w / Hq;
  const int s = static_cast<int>(bs % S_pad), b = static_cast<int>(bs / S_pad);
  float2* dst = stats + (static_cast<long long>(b) * Hq + h) * S_pad + s;
  if (s >= S) {
    if (lane == 0) *dst = make_float2(0.f, 0.f);
    return;
  }
  const long long at = ((static_cast<long long>(b) * S + s) * Hq + h) * HD + lane * 8;
  const uint4 ov = *reinterpret_cast<const uint4*>(o + at), dv = *reinterpret_cast<const uint4*>(d_o + at);
  float acc = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 x = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&ov)[e]);
    const float2 y = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&dv)[e]);
    acc += x.x * y.x + x.y * y.y;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (lane == 0) *dst = make_float2(lse[(static_cast<long long>(b) * Hq + h) * S + s] * kLog2e, acc);
}

// R1, R2: resident operands; TA, TB: streamed ones.  `tile`: row tile; `head`: query head (dQ) or key head; `rank`: this
// CTA's share of the group's heads (dK, dV).
template <int MODE>
__device__ __forceinline__ void pass(const CUtensorMap* mR1, const CUtensorMap* mR2, const CUtensorMap* mTA, const CUtensorMap* mTB,
                                     const Bwd256Params& p, uint8_t* smem, int tile, int head, int b, int rank) {
  constexpr int TB_RING = MODE == kDV ? 3 : 1;
  uint8_t* sR1 = smem;
  uint8_t* sR2 = sR1 + R_TILE;                                     // not for dV
  uint8_t* sTA = sR1 + (MODE == kDV ? 1 : 2) * R_TILE;             // two tiles
  uint8_t* sTB = sTA + 2 * T_TILE;                                 // TB_RING tiles
  float2* sStat = reinterpret_cast<float2*>(smem + TILES);         // the step's query rows, a slot beside each of TA's (dK) or TB's (dV)
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + TILES + STAT_SLOTS * KT * 8);
  uint64_t* r_full = bars;            // [1]
  uint64_t* ta_full = bars + 1;       // [2]
  uint64_t* ta_empty = bars + 3;      // [2]
  uint64_t* tb_full = bars + 5;       // [3]
  uint64_t* tb_empty = bars + 8;      // [3]
  uint64_t* x1_full = bars + 11;      // S of the step is in tensor memory
  uint64_t* x2_full = bars + 12;      // dP too
  uint64_t* x_empty = bars + 13;      // the softmax warps hold both in registers
  uint64_t* w_full = bars + 14;       // [2] W is in tensor memory
  uint64_t* w_free = bars + 16;       // [2] the product reading W has retired
  uint64_t* out_full = bars + 18;     // [1] every product has retired
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.Hq / p.Hkv, row0 = tile * RT;
  // streamed tiles first .. first + cnt - 1, for every head of h0 .. h0 + n_heads - 1
  int first, cnt, h0 = 0, n_heads = 1;
  if (MODE == kDQ) {
    first = p.window > 0 ? max(0, row0 - p.window + 1) / KT : 0;
    cnt = (min(row0 + RT, p.S) - 1) / KT - first + 1;
  } else {
    first = row0 / KT;
    const int last = p.window > 0 ? min(p.S - 1, row0 + RT - 1 + p.window - 1) : p.S - 1;
    cnt = last / KT - first + 1;
    h0 = rank * G / p.shares;
    n_heads = (rank + 1) * G / p.shares - h0;
    h0 += head * G;
  }
  const int steps = n_heads * cnt;

  if (threadIdx.x == 0) {
    mbar_init(r_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ta_full[i], 1);
      mbar_init(&ta_empty[i], 1);
      mbar_init(&w_full[i], 8);
      mbar_init(&w_free[i], 1);
    }
    for (int i = 0; i < 3; ++i) {
      mbar_init(&tb_full[i], 1);
      mbar_init(&tb_empty[i], 1);
    }
    mbar_init(x1_full, 1);
    mbar_init(x2_full, 1);
    mbar_init(x_empty, 8);
    mbar_init(out_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tOut = tmem_base, tX1 = tmem_base + HD, tX2 = tX1 + KT, tW = tX2 + KT;     // W: two buffers of KT / 2 columns

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(r_full, (MODE == kDV ? 1 : 2) * R_TILE);
#pragma unroll
      for (int a = 0; a < 4; ++a) tma_load_4d(sR1 + a * R_ATOM, mR1, r_full, a * 64, head, row0, b);
      if (MODE != kDV) {
#pragma unroll
        for (int a = 0; a < 4; ++a) tma_load_4d(sR2 + a * R_ATOM, mR2, r_full, a * 64, head, row0, b);
      }
      for (int t = 0; t < steps; ++t) {
        const int h = MODE == kDQ ? head / G : h0 + t / cnt;
        const int r = (first + t % cnt) * KT;
        const int sa = t & 1, sb = t % TB_RING;
        auto stat = [&](int slot, uint64_t* bar) {
          bulk_load(sStat + slot * KT, p.stats + (static_cast<long long>(b) * p.Hq + h) * p.S_pad + r, KT * 8, bar);
        };
        if (!mbar_wait(&ta_empty[sa], ((t >> 1) & 1) ^ 1, abort_flag, p.status, kStatusWaitTimeoutProducer)) break;
        mbar_expect_tx(&ta_full[sa], T_TILE + (MODE == kDK ? KT * 8 : 0));
        if (MODE == kDK) stat(sa, &ta_full[sa]);
#pragma unroll
        for (int a = 0; a < 4; ++a) tma_load_4d(sTA + sa * T_TILE + a * T_ATOM, mTA, &ta_full[sa], a * 64, h, r, b);
        if (!mbar_wait(&tb_empty[sb], ((t / TB_RING) & 1) ^ 1, abort_flag, p.status, kStatusWaitTimeoutProducer)) break;
        mbar_expect_tx(&tb_full[sb], T_TILE + (MODE == kDV ? KT * 8 : 0));
        if (MODE == kDV) stat(sb, &tb_full[sb]);
#pragma unroll
        for (int a = 0; a < 4; ++a) tma_load_4d(sTB + sb * T_TILE + a * T_ATOM, mTB, &tb_full[sb], a * 64, h, r, b);
      }
      if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(10000);   // let copies in flight land before shared memory goes away
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA warp: all lanes walk the loop, one issues
    constexpr uint32_t idesc_x = make_idesc_bf16(RT, KT), idesc_out = make_idesc_bf16(RT, HD) | kBMajorMN;
    const uint64_t d1 = make_smem_desc(smem_u32(sR1)), d2 = make_smem_desc(smem_u32(sR2));
    auto scores = [&](uint32_t to, uint64_t a, uint64_t bt, uint64_t* full, uint64_t* freed) {
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks)
          umma(to, desc_adv(a, (ks >> 2) * R_ATOM + (ks & 3) * 32), desc_adv(bt, (ks >> 2) * T_ATOM + (ks & 3) * 32), idesc_x, ks > 0 ? 1u : 0u);
        umma_commit(full);
        if (freed) umma_commit(freed);
      }
      __syncwarp();
    };
    auto issue_x = [&](int t) -> bool {
      const int sa = t & 1;
      if (!mbar_wait_warp(&ta_full[sa], (t >> 1) & 1, abort_flag, p.status, kStatusWaitTimeoutMma)) return false;
      if (t > 0 && !mbar_wait_warp(x_empty, (t - 1) & 1, abort_flag, p.status, kStatusWaitTimeoutMma)) return false;
      tc_fence_after();
      scores(tX1, d1, make_smem_desc(smem_u32(sTA + sa * T_TILE)), x1_full, MODE == kDV ? &ta_empty[sa] : nullptr);
      if (MODE != kDV) {
        // TB has one slot, refilled while S is computed: wait for it only now
        if (!mbar_wait_warp(&tb_full[0], t & 1, abort_flag, p.status, kStatusWaitTimeoutMma)) return false;
        tc_fence_after();
        scores(tX2, d2, make_smem_desc(smem_u32(sTB)), x2_full, &tb_empty[0]);
      }
      return true;
    };
    bool ok = mbar_wait_warp(r_full, 0, abort_flag, p.status, kStatusWaitTimeoutMma);
    if (ok) ok = issue_x(0);
    for (int t = 0; t < steps && ok; ++t) {
      if (t + 1 < steps) ok = issue_x(t + 1);
      if (!ok) break;
      const int sa = t & 1, sb = t % TB_RING;
      if (!mbar_wait_warp(&w_full[sa], (t >> 1) & 1, abort_flag, p.status, kStatusWaitTimeoutMma) ||
          (MODE == kDV && !mbar_wait_warp(&tb_full[sb], (t / TB_RING) & 1, abort_flag, p.status, kStatusWaitTimeoutMma))) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint64_t bd = make_smem_desc_mn(smem_u32(MODE == kDV ? sTB + sb * T_TILE : sTA + sa * T_TILE), T_ATOM);
      const uint32_t acc0 = t > 0 ? 1u : 0u;
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < KT / 16; ++ks)            // contraction over the step's 64 rows
          umma_ts(tOut, tW + sa * (KT / 2) + ks * 8, desc_adv(bd, ks * 2048), idesc_out, ks > 0 ? 1u : acc0);
        umma_commit(&w_free[sa]);
        umma_commit(MODE == kDV ? &tb_empty[sb] : &ta_empty[sa]);
      }
      __syncwarp();
    }
    if (ok && elect_one()) umma_commit(out_full);
    __syncwarp();
  }

  // -------------------------------------------------------- softmax warps: thread = (resident row, half of the streamed ones)
  const int qd = warp & 3, half = (warp - 2) >> 2;
  const int r = qd * 32 + lane, row = row0 + r;
  const uint32_t lane_sel = static_cast<uint32_t>(qd * 32) << 16;
  bool ok = warp >= 2;
  if (warp >= 2) {
    const float c = p.scale * kLog2e;
    float2 mine = make_float2(0.f, 0.f);
    if (MODE == kDQ) mine = p.stats[(static_cast<long long>(b) * p.Hq + head) * p.S_pad + row];      // padded: no guard needed
    for (int t = 0; t < steps; ++t) {
      const int col0 = (first + t % cnt) * KT + half * 32;
      const int st = t & 1, slot = MODE == kDV ? t % TB_RING : st;
      if (!mbar_wait_warp(x1_full, t & 1, abort_flag, p.status, kStatusWaitTimeoutEpilogue) ||
          !mbar_wait_warp(MODE == kDV ? &tb_full[slot] : x2_full, MODE == kDV ? (t / TB_RING) & 1 : t & 1, abort_flag, p.status,
                          kStatusWaitTimeoutEpilogue)) {
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t sv[32], dv[32], w[16];
      tmem_ld32(tX1 + lane_sel + half * 32, sv);
      if (MODE != kDV) tmem_ld32(tX2 + lane_sel + half * 32, dv);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(x_empty);
      const float2* st_row = sStat + slot * KT + half * 32;
      // warp-uniform: every pair of this tile is a real query at or after a key inside its window
      const int q_lo = MODE == kDQ ? row0 : col0, q_hi = MODE == kDQ ? row0 + RT - 1 : col0 + 31;
      const int k_lo = MODE == kDQ ? col0 : row0, k_hi = MODE == kDQ ? col0 + 31 : row0 + RT - 1;
      const bool full = q_lo >= k_hi && q_hi < p.S && (p.window == 0 || q_hi - k_lo < p.window);
      auto weights = [&](auto masked, int lo, int hi) {
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float4 s4 = make_float4(mine.x, mine.y, mine.x, mine.y);
          if (MODE != kDQ) s4 = *reinterpret_cast<const float4*>(st_row + e);       // {lse, delta} of two queries (broadcast read)
          float p0 = exp2f(__uint_as_float(sv[e]) * c - s4.x), p1 = exp2f(__uint_as_float(sv[e + 1]) * c - s4.z);
          if (MODE != kDV) {
            p0 *= __uint_as_float(dv[e]) - s4.y;
            p1 *= __uint_as_float(dv[e + 1]) - s4.w;
          }
          if (decltype(masked)::value) {
            p0 = e >= lo && e < hi ? p0 : 0.f;
            p1 = e + 1 >= lo && e + 1 < hi ? p1 : 0.f;
          }
          w[e >> 1] = pack2(p0, p1);
        }
      };
      if (full) {
        weights(std::false_type{}, 0, 32);
      } else {      // the columns [lo, hi) of this row count
        int lo = 0, hi;
        if (MODE == kDQ) {
          hi = row < p.S ? row + 1 - col0 : 0;
          if (p.window > 0) lo = row - p.window + 1 - col0;
        } else {
          lo = row - col0;
          hi = p.S - col0;
          if (p.window > 0) hi = min(hi, row + p.window - col0);
        }
        weights(std::true_type{}, lo, hi);
      }
      if (t >= 2 && !mbar_wait_warp(&w_free[st], ((t >> 1) - 1) & 1, abort_flag, p.status, kStatusWaitTimeoutEpilogue)) {
        ok = false;
        break;
      }
      tc_fence_after();
      tmem_st16(tW + st * (KT / 2) + lane_sel + half * 16, w);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&w_full[st]);
    }
    if (ok && !mbar_wait_warp(out_full, 0, abort_flag, p.status, kStatusWaitTimeoutEpilogue)) ok = false;
    tc_fence_after();
  }

  // ---------------------------------------------------------------------------------------- result
  const int shares = MODE == kDQ ? 1 : p.shares, width = HD / shares;      // a CTA of a cluster stores its slice of the columns
  const long long bs = MODE == kDQ ? p.dq_bs : MODE == kDK ? p.dk_bs : p.dv_bs, ts = MODE == kDQ ? p.dq_ts : MODE == kDK ? p.dk_ts : p.dv_ts;
  __nv_bfloat16* out = (MODE == kDQ ? p.dq : MODE == kDK ? p.dk : p.dv) + b * bs + static_cast<long long>(row) * ts + head * HD;
  if (shares > 1) {
    // partial sums of the peers' slices into their (now idle) tiles: four columns of 128 rows at a time, row after row
    tc_fence_before();
    __syncthreads();
    cluster_sync();              // every CTA has done with its tiles
    tc_fence_after();
    if (ok) {
      for (int o = 1; o < shares; ++o) {
        const int peer = (rank + o) % shares;
        const int slot = rank < peer ? rank : rank - 1;
        for (int cc = half * (width / 2); cc < (half + 1) * (width / 2); cc += 32) {
          uint32_t v[32];
          tmem_ld32(tOut + lane_sel + peer * width + cc, v);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e += 4)
            st_peer(smem_u32(smem) + ((slot * (width / 4) + (cc + e) / 4) * RT + r) * 16, peer,
                    make_float4(__uint_as_float(v[e]), __uint_as_float(v[e + 1]), __uint_as_float(v[e + 2]), __uint_as_float(v[e + 3])));
        }
      }
    }
    __syncwarp();
    cluster_sync();
  }
  if (ok) {      // warp-uniform: the loads from tensor memory are warp-collective, only the stores are per row
    const float sc = MODE == kDV ? 1.f : p.scale;
    const int mine = shares > 1 ? rank * width : 0;
#pragma unroll 1
    for (int cc = half * (width / 2); cc < (half + 1) * (width / 2); cc += 32) {
      uint32_t v[32];
      __syncwarp();   // lanes that skipped the stores rejoin before the collective load
      tmem_ld32(tOut + lane_sel + mine + cc, v);
      tmem_ld_wait();
      if (row >= p.S) continue;
      if (shares > 1) {
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          float4 own = make_float4(__uint_as_float(v[e]), __uint_as_float(v[e + 1]), __uint_as_float(v[e + 2]), __uint_as_float(v[e + 3]));
          float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int s = 0; s < shares; ++s) {
            float4 x = own;
            if (s != rank) x = *reinterpret_cast<const float4*>(smem + (((s < rank ? s : s - 1) * (width / 4) + (cc + e) / 4) * RT + r) * 16);
            sum = make_float4(sum.x + x.x, sum.y + x.y, sum.z + x.z, sum.w + x.w);
          }
          v[e] = __float_as_uint(sum.x);
          v[e + 1] = __float_as_uint(sum.y);
          v[e + 2] = __float_as_uint(sum.z);
          v[e + 3] = __float_as_uint(sum.w);
        }
      }
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        uint4 x;
        x.x = pack2(__uint_as_float(v[ch * 8 + 0]) * sc, __uint_as_float(v[ch * 8 + 1]) * sc);
        x.y = pack2(__uint_as_float(v[ch * 8 + 2]) * sc, __uint_as_float(v[ch * 8 + 3]) * sc);
        x.z = pack2(__uint_as_float(v[ch * 8 + 4]) * sc, __uint_as_float(v[ch * 8 + 5]) * sc);
        x.w = pack2(__uint_as_float(v[ch * 8 + 6]) * sc, __uint_as_float(v[ch * 8 + 7]) * sc);
        reinterpret_cast<uint4*>(out + mine + cc)[ch] = x;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

// The tiles leave no room for alignment slack: the dynamic shared memory is declared 1024-byte aligned (the swizzled tiles need
// it) and a kernel refuses to run if it is not.
__device__ __forceinline__ bool aligned_tiles(const uint8_t* smem, int* status) {
  if ((smem_u32(smem) & 1023u) == 0) return true;
  if (threadIdx.x == 0) atomicCAS(status, kStatusOk, kStatusBadShape);
  return false;
}

__global__ void __launch_bounds__(THREADS, 1)
flash_bwd256_dq_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
                          const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, Bwd256Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if (!aligned_tiles(smem_raw, p.status)) return;
  pass<kDQ>(&tmQ, &tmdO, &tmK, &tmV, p, smem_raw, gridDim.z - 1 - blockIdx.z, blockIdx.x, blockIdx.y, 0);      // longest rows first
}

__global__ void __launch_bounds__(THREADS, 1)
flash_bwd256_dkv_tc_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                           const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO, Bwd256Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if (!aligned_tiles(smem_raw, p.status)) return;      // the same in every CTA of a cluster
  // key tile 0 has the most queries and comes first, dK (the longer pass) before dV
  const int heads = p.B * p.Hkv, at = blockIdx.y % heads;
  if (static_cast<int>(blockIdx.y) < heads)
    pass<kDK>(&tmK, &tmV, &tmQ, &tmdO, p, smem_raw, blockIdx.z, at % p.Hkv, at / p.Hkv, blockIdx.x);
  else
    pass<kDV>(&tmK, &tmV, &tmQ, &tmdO, p, smem_raw, blockIdx.z, at % p.Hkv, at / p.Hkv, blockIdx.x);
}

}  // namespace

// as many as it takes for about three CTAs a multiprocessor, since the first key tile is twice the mean
static int pick_shares(long long ctas, int G, int sms) {
  int shares = 1;
  while (2 * shares <= G && 2 * shares <= kMaxShares && ctas * shares < 3ll * sms) shares *= 2;
  return shares;
}

// Not where there are many short rows: a wave of these CTAs takes 10 us, whatever little it has to do, and the warp-level kernels take 6
// for each query head of a key head and one for 10 tokens or so (us, these and those, waves 3, 4, 6, 7: 4 rows of 8 tokens, 32 and 8
// heads 35, 29; 8 of 16, 24 and 4 43, 46; 8 of 64, 32 and 8 66, 45; 16 of 64, 24 and 4 80, 65; 16 of 96, 32 and 8 114, 174).
bool flash_bwd256_tc_better(int B, int S, int Hq, int Hkv, int sms) {
  if (S > 64 || Hkv < 1) return true;
  const int G = Hq / Hkv;
  const long long dq = static_cast<long long>(B) * Hq, dkv = 2ll * B * Hkv * pick_shares(2ll * B * Hkv, G, sms);
  const long long waves = (dq + sms - 1) / sms + (dkv + sms - 1) / sms;
  return waves < 3 || 64 * waves < 58 + 31 * G + S;
}

size_t flash_bwd256_tc_scratch_floats(const FlashArgs& a) {
  return static_cast<size_t>(a.B) * a.Hq * ((a.Sq + RT - 1) / RT * RT) * 2;
}

bool flash_bwd256_tc_supported(const FlashArgs& a) {
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return a.D == HD && a.causal && a.window >= 0 && a.q_offset == 0 && a.Sq == a.Sk && a.Sq >= 1 && a.Hkv > 0 && a.Hq % a.Hkv == 0 &&
         a.q_ts % 8 == 0 && a.k_ts % 8 == 0 && a.v_ts % 8 == 0 && a.do_ts == static_cast<long long>(a.Hq) * HD && a.q_bs % 8 == 0 &&
         a.k_bs % 8 == 0 && a.v_bs % 8 == 0 && a.q_ts > 0 && a.k_ts > 0 && a.v_ts > 0 && a.q_bs > 0 && a.k_bs > 0 && a.v_bs > 0 &&
         a.o_ts == a.do_ts && a.o_bs == a.do_bs && a.o_bs == a.o_ts * a.Sq && a.dq_ts % 8 == 0 && a.dk_ts % 8 == 0 && a.dv_ts % 8 == 0 &&
         al16(a.q) && al16(a.k) && al16(a.v) && al16(a.d_o) && al16(a.o) && al16(a.dq) && al16(a.dk) && al16(a.dv) &&
         a.B <= 65535 && static_cast<long long>(a.B) * a.Hkv * 2 <= 65535 && (a.Sq + RT - 1) / RT <= 65535;
}

// Needs a.lse from the forward and a.delta: fp32 scratch of flash_bwd256_tc_scratch_floats(a) elements, 16-byte aligned.
const char* flash_bwd256_tc(const FlashArgs& a, int* status, cudaStream_t stream) {
  if (!flash_bwd256_tc_supported(a)) return "flash_bwd256_tc: unsupported arguments";
  if (a.B == 0) return nullptr;
  const int n_t = (a.Sq + RT - 1) / RT, s_pad = n_t * RT, G = a.Hq / a.Hkv;
  const long long rows = static_cast<long long>(a.B) * s_pad * a.Hq;
  float2* stats = reinterpret_cast<float2*>(a.delta);
  stats256_kernel<<<static_cast<unsigned>((rows * 32 + 255) / 256), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(a.o), static_cast<const __nv_bfloat16*>(a.d_o), a.lse, stats, a.B, a.Sq, s_pad, a.Hq);
  count_launch();
  CUtensorMap mQ, mdO, mK, mV, mQt, mdOt, mKt, mVt;        // resident boxes, then the streamed ones
  auto maps = [&](CUtensorMap* res, CUtensorMap* str, const void* x, int heads, long long ts, long long bs) {
    return make_map_4d(res, x, a.B, a.Sq, heads, HD, HD, ts, bs, RT) && make_map_4d(str, x, a.B, a.Sq, heads, HD, HD, ts, bs, KT);
  };
  if (!maps(&mQ, &mQt, a.q, a.Hq, a.q_ts, a.q_bs) || !maps(&mdO, &mdOt, a.d_o, a.Hq, a.do_ts, a.do_bs) ||
      !maps(&mK, &mKt, a.k, a.Hkv, a.k_ts, a.k_bs) || !maps(&mV, &mVt, a.v, a.Hkv, a.v_ts, a.v_bs))
    return "flash_bwd256_tc: tensor map failed";
  Bwd256Params p{};
  p.stats = stats; p.S_pad = s_pad;
  p.dq = static_cast<__nv_bfloat16*>(a.dq); p.dq_bs = a.dq_bs; p.dq_ts = a.dq_ts;
  p.dk = static_cast<__nv_bfloat16*>(a.dk); p.dk_bs = a.dk_bs; p.dk_ts = a.dk_ts;
  p.dv = static_cast<__nv_bfloat16*>(a.dv); p.dv_bs = a.dv_bs; p.dv_ts = a.dv_ts;
  p.B = a.B; p.S = a.Sq; p.Hq = a.Hq; p.Hkv = a.Hkv; p.window = a.window; p.scale = a.scale; p.status = status;
  if (!FERRL_ONCE_PER_DEVICE(
          cudaFuncSetAttribute(flash_bwd256_dq_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) == cudaSuccess &&
          cudaFuncSetAttribute(flash_bwd256_dkv_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) == cudaSuccess))
    return "flash_bwd256_tc: cannot reserve shared memory";
  flash_bwd256_dq_tc_kernel<<<dim3(a.Hq, a.B, n_t), THREADS, SMEM, stream>>>(mQ, mdO, mKt, mVt, p);
  count_launch();
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  p.shares = pick_shares(2ll * a.B * a.Hkv * n_t, G, sms);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.shares, 2 * a.B * a.Hkv, n_t);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.shares;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, flash_bwd256_dkv_tc_kernel, mK, mV, mQt, mdOt, p) != cudaSuccess) return "flash_bwd256_tc launch failed";
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "flash_bwd256_tc launch failed";
}

}  // namespace ferrl
