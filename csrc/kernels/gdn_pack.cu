// What stands between a GatedDeltaNet layer's 16-bit activations and the chunk kernels of gdn_tc.cu, forward and backward.
//
// Reference: crates/ferrl/src/gdn.rs - l2norm :70 and the padding to whole chunks in gated_delta_rule_chunked :451-556.
//
//   gdn_pack          q, k, v, log decay, beta -> L2-normalised 32-bit rows (q also over sqrt(128)), zero rows up to whole chunks
//   gdn_pad           the output's gradient as 32-bit rows up to whole chunks
//   gdn_unpack_bwd    gradients of the raw q and k (sum over the value heads of a key head, then the L2 norm's backward) and of v,
//                     rounded to 16 bits once
//   gdn_decay_bwd     gradient of the log decays from that of their sums inside a chunk
//
// Elementwise passes over a few hundred MB, bound by HBM.  As about 60 tensor operations with 32-bit temporaries they took
// 1.15 ms of a layer's forward and backward (6140 tokens, 16 key and 16 value heads); a training step of three such layers
// fell from 33.1 to 30.6 ms with them.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../api.h"
#include "../common.cuh"
#include "vec.cuh"

namespace ferrl {
namespace {

constexpr int GD = 128;        // head dim: four entries a lane
constexpr int GC = 64;         // chunk length
constexpr int NTH = 256;

struct HeadRows {              // [B, T, H, 128] with packed heads
  const __nv_bfloat16* p;
  long long bs, ts;
  int H;
};

__device__ __forceinline__ float dot4(float4 a, float4 b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
__device__ __forceinline__ float4 scale4(float4 a, float s) { return make_float4(a.x * s, a.y * s, a.z * s, a.w * s); }

// One CTA per padded token, a warp per head.
__global__ void __launch_bounds__(NTH)
gdn_pack_kernel(HeadRows q, HeadRows k, HeadRows v, const float* __restrict__ g, const float* __restrict__ beta, int T, int Tp, float eps,
                float* __restrict__ qf, float* __restrict__ kf, float* __restrict__ vf, float* __restrict__ gp, float* __restrict__ bp) {
  const int b = blockIdx.x / Tp, t = blockIdx.x - b * Tp, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long row = blockIdx.x;
  const bool on = t < T;
  for (int h = warp; h < q.H + k.H + v.H; h += NTH / 32) {
    const int which = h < q.H ? 0 : h < q.H + k.H ? 1 : 2, hh = which == 0 ? h : which == 1 ? h - q.H : h - q.H - k.H;
    const HeadRows& s = which == 0 ? q : which == 1 ? k : v;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (on) {
      x = load4(s.p + b * s.bs + t * s.ts + hh * GD + lane * 4);
      if (which < 2) {
        const float r = rsqrtf(warp_sum(dot4(x, x)) + eps);
        x = scale4(x, r);
        if (which == 0) x = scale4(x, rsqrtf(static_cast<float>(GD)));
      }
    }
    store4((which == 0 ? qf : which == 1 ? kf : vf) + (row * s.H + hh) * GD + lane * 4, x);
  }
  for (int h = threadIdx.x; h < v.H; h += NTH) {          // beta = 0 and g = 0 leave the state as it is
    const long long at = (static_cast<long long>(b) * T + t) * v.H + h;
    gp[row * v.H + h] = on ? g[at] : 0.f;
    bp[row * v.H + h] = on ? beta[at] : 0.f;
  }
}

__global__ void __launch_bounds__(NTH)
gdn_pad_kernel(HeadRows s, int T, int Tp, float* __restrict__ out) {
  const int b = blockIdx.x / Tp, t = blockIdx.x - b * Tp;
  for (int i = threadIdx.x; i < s.H * (GD / 4); i += NTH)
    store4(out + (static_cast<long long>(blockIdx.x) * s.H * GD) + i * 4,
           t < T ? load4(s.p + b * s.bs + t * s.ts + i * 4) : make_float4(0.f, 0.f, 0.f, 0.f));
}

// One CTA per token.  y = x r, r = (|x|^2 + eps)^-1/2:  dx = r dy - x r^3 <x, dy>.
__global__ void __launch_bounds__(NTH)
gdn_unpack_bwd_kernel(HeadRows q, HeadRows k, const float* __restrict__ dqf, const float* __restrict__ dkf, const float* __restrict__ dvf, int Hv,
                      int T, int Tp, float eps, __nv_bfloat16* __restrict__ dq, __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv) {
  const int b = blockIdx.x / T, t = blockIdx.x - b * T, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long row = blockIdx.x, src = static_cast<long long>(b) * Tp + t;
  const int Hk = q.H, rep = Hv / Hk;
  for (int h = warp; h < 2 * Hk + Hv; h += NTH / 32) {
    if (h >= 2 * Hk) {
      const int hv = h - 2 * Hk;
      store4(dv + (row * Hv + hv) * GD + lane * 4, load4(dvf + (src * Hv + hv) * GD + lane * 4));
      continue;
    }
    const bool is_q = h < Hk;
    const int hk = is_q ? h : h - Hk;
    const HeadRows& s = is_q ? q : k;
    const float4 x = load4(s.p + b * s.bs + t * s.ts + hk * GD + lane * 4);
    const float* d = (is_q ? dqf : dkf) + (src * Hv + hk * rep) * GD + lane * 4;
    float4 y = load4(d);
    for (int j = 1; j < rep; ++j) {
      const float4 z = load4(d + j * GD);
      y.x += z.x; y.y += z.y; y.z += z.z; y.w += z.w;
    }
    if (is_q) y = scale4(y, rsqrtf(static_cast<float>(GD)));
    const float r = rsqrtf(warp_sum(dot4(x, x)) + eps), c = r * r * r * warp_sum(dot4(x, y));
    store4((is_q ? dq : dk) + (row * Hk + hk) * GD + lane * 4,
           make_float4(r * y.x - x.x * c, r * y.y - x.y * c, r * y.z - x.z * c, r * y.w - x.w * c));
  }
}

// dg_j = sum over i >= j of the chunk of dG_i; a thread per (chunk, head), [B, Tp, Hv] -> [B, T, Hv] with dbeta along
__global__ void gdn_decay_bwd_kernel(const float* __restrict__ dG, const float* __restrict__ dbp, long long n_chunks, int Hv, int T, int Tp,
                                     float* __restrict__ dg, float* __restrict__ dbeta) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n_chunks * Hv) return;
  const long long c = i / Hv;
  const int hv = static_cast<int>(i - c * Hv), per = Tp / GC;
  const long long b = c / per;
  const int t0 = static_cast<int>(c - b * per) * GC;
  float sum = 0.f;
#pragma unroll 8
  for (int j = GC - 1; j >= 0; --j) {
    const long long from = (b * Tp + t0 + j) * Hv + hv;
    sum += dG[from];
    if (t0 + j < T) {
      const long long to = (b * T + t0 + j) * Hv + hv;
      dg[to] = sum;
      dbeta[to] = dbp[from];
    }
  }
}

}  // namespace

const char* gdn_pack(const void* q, long long q_bs, long long q_ts, const void* k, long long k_bs, long long k_ts, const void* v,
                     long long v_bs, long long v_ts, const float* g, const float* beta, int B, int T, int Tp, int Hk, int Hv, float eps,
                     float* qf, float* kf, float* vf, float* gp, float* bp, cudaStream_t s) {
  if (B * Tp == 0) return nullptr;
  using N = const __nv_bfloat16*;
  gdn_pack_kernel<<<B * Tp, NTH, 0, s>>>({static_cast<N>(q), q_bs, q_ts, Hk}, {static_cast<N>(k), k_bs, k_ts, Hk},
                                         {static_cast<N>(v), v_bs, v_ts, Hv}, g, beta, T, Tp, eps, qf, kf, vf, gp, bp);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "gdn_pack launch failed";
}

const char* gdn_pad(const void* x, long long bs, long long ts, int B, int T, int Tp, int H, float* out, cudaStream_t s) {
  if (B * Tp == 0) return nullptr;
  gdn_pad_kernel<<<B * Tp, NTH, 0, s>>>({static_cast<const __nv_bfloat16*>(x), bs, ts, H}, T, Tp, out);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "gdn_pad launch failed";
}

const char* gdn_unpack_bwd(const void* q, long long q_bs, long long q_ts, const void* k, long long k_bs, long long k_ts, const float* dqf,
                           const float* dkf, const float* dvf, const float* dG, const float* dbp, int B, int T, int Tp, int Hk, int Hv,
                           float eps, void* dq, void* dk, void* dv, float* dg, float* dbeta, cudaStream_t s) {
  if (B * T == 0) return nullptr;
  using N = const __nv_bfloat16*;
  gdn_unpack_bwd_kernel<<<B * T, NTH, 0, s>>>({static_cast<N>(q), q_bs, q_ts, Hk}, {static_cast<N>(k), k_bs, k_ts, Hk}, dqf, dkf, dvf, Hv, T, Tp,
                                              eps, static_cast<__nv_bfloat16*>(dq), static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv));
  const long long chunks = static_cast<long long>(B) * (Tp / GC);
  gdn_decay_bwd_kernel<<<static_cast<unsigned>((chunks * Hv + 63) / 64), 64, 0, s>>>(dG, dbp, chunks, Hv, T, Tp, dg, dbeta);
  count_launch(2);
  return cudaGetLastError() == cudaSuccess ? nullptr : "gdn_unpack_bwd launch failed";
}

}  // namespace ferrl
