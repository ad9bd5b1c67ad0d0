// GatedDeltaNet kernels for sm_100a (Qwen3.5/3.6 linear-attention layers).
//
// Reference: crates/ferrl/src/gdn.rs - causal depthwise conv with left context :102-142, the
// single-step recurrent delta rule :286-317.  The reference composes both from tensor ops (a
// dozen launches per layer per token in decode); here each is one memory-bound kernel:
//
//   gdn_conv_fwd / gdn_conv_bwd  causal depthwise conv (+SiLU) over [B, L, C] without transposes,
//                                reading the K-1 tokens of left context from the carried state
//   gdn_conv_step                the one-token decode form; shifts the state in place
//   gdn_decode_step              L2-normalise q,k; S <- S*exp(g); delta rule update; o = S^T q,
//                                with the [kd, vd] fp32 state read and written exactly once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../api.h"
#include "../common.cuh"

namespace ferrl {

namespace {

constexpr int kMaxConvK = 8;

__device__ __forceinline__ float silu_f(float x) { return x / (1.f + __expf(-x)); }
__device__ __forceinline__ float dsilu_f(float x) {
  const float s = 1.f / (1.f + __expf(-x));
  return s * (1.f + x * (1.f - s));
}

// Causal depthwise convolution, forward and backward.  x [B, L, C] (row stride ldx), w [C, K], left [B, C, K-1] or null,
// y, dy, dx [B, L, C] contiguous.  A thread owns V neighbouring channels and walks `run` tokens with the last K - 1 inputs
// in registers, so a token is read once and not once per tap; the K - 1 tokens in front of a run are the only ones read
// twice.  Bound by instruction issue, the SiLU's exponential and reciprocal before all, and not by its bytes (210 MB
// forward, 315 MB backward at [5119, 10240], K = 4: 32 and 48 us).  So V = 4, one 8-byte access a token: eight channels
// took 126 and 188 registers, which left too few warps to hide the exponentials (72 and 148 us); four take 70 and 93
// (55 and 96 us).  The taps are read as whole words too: as V x K single values, a thread's own row apart from its
// neighbour's, they cost more cache accesses than the tokens of a run (94 and 145 us together with the eight channels).
// The next tokens are on their way while the present ones are worked on.  The taps are added in the order of the tap
// number whatever V is, so the results are the same bits.
template <int V> struct ConvRaw { using type = __nv_bfloat16; };      // V channels of a token as they lie
template <> struct ConvRaw<4> { using type = uint2; };
template <int V>
__device__ __forceinline__ void conv_unpack(const typename ConvRaw<V>::type& u, float (&f)[V]) {
  if constexpr (V > 1) {
    const uint32_t* h = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
    for (int e = 0; e < V / 2; ++e) {
      f[2 * e] = __uint_as_float(h[e] << 16);
      f[2 * e + 1] = __uint_as_float(h[e] & 0xffff0000u);
    }
  } else {
    f[0] = __bfloat162float(u);
  }
}
template <int V>
__device__ __forceinline__ void conv_load(const __nv_bfloat16* p, float (&f)[V]) {
  conv_unpack<V>(*reinterpret_cast<const typename ConvRaw<V>::type*>(p), f);
}
template <int V>
__device__ __forceinline__ void conv_store(__nv_bfloat16* p, const float (&f)[V]) {
  if constexpr (V > 1) {
    typename ConvRaw<V>::type u;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int e = 0; e < V / 2; ++e) h[e] = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
    *reinterpret_cast<typename ConvRaw<V>::type*>(p) = u;
  } else {
    p[0] = __float2bfloat16_rn(f[0]);
  }
}
// bf16 and back, two values a conversion
template <int V>
__device__ __forceinline__ void conv_round(float (&f)[V]) {
  if constexpr (V > 1) {
    typename ConvRaw<V>::type u;
    conv_store<V>(reinterpret_cast<__nv_bfloat16*>(&u), f);
    conv_unpack<V>(u, f);
  } else {
    f[0] = __bfloat162float(__float2bfloat16_rn(f[0]));
  }
}
// the K taps of V channels: V x K neighbouring values
template <int K, int V>
__device__ __forceinline__ void conv_taps(const __nv_bfloat16* w, float (&wv)[K][V]) {
  if constexpr (V > 1) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      float f[V];
      conv_unpack<V>(reinterpret_cast<const typename ConvRaw<V>::type*>(w)[i], f);
#pragma unroll
      for (int e = 0; e < V; ++e) wv[(i * V + e) % K][(i * V + e) / K] = f[e];
    }
  } else {
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
      for (int e = 0; e < V; ++e) wv[j][e] = __bfloat162float(w[e * K + j]);
  }
}
// channels c .. c+V-1 of x at token t of row b; the carried context where t < 0
template <int K, int V>
__device__ __forceinline__ void conv_input(const __nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ left,
                                           int b, int t, int c, int L, int C, float (&f)[V]) {
  if (t >= 0) {
    conv_load<V>(x + (static_cast<long long>(b) * L + t) * ldx + c, f);
  } else {
#pragma unroll
    for (int e = 0; e < V; ++e)
      f[e] = left ? __bfloat162float(left[(static_cast<long long>(b) * C + c + e) * (K - 1) + (K - 1 + t)]) : 0.f;
  }
}

template <int K, int V>
__global__ void __launch_bounds__(128)
gdn_conv_fwd_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ w,
                    const __nv_bfloat16* __restrict__ left, int L, int C, int runs, int run, int act, __nv_bfloat16* __restrict__ y) {
  const int c = (blockIdx.y * 128 + threadIdx.x) * V;
  if (c >= C) return;
  const int b = blockIdx.x / runs, t0 = (blockIdx.x - b * runs) * run, t1 = min(L, t0 + run);
  float wv[K][V], win[K][V];            // win[j]: the input that tap j meets
  conv_taps<K, V>(w + static_cast<long long>(c) * K, wv);
#pragma unroll
  for (int j = 1; j < K; ++j) conv_input<K, V>(x, ldx, left, b, t0 - K + j, c, L, C, win[j]);
  using Raw = typename ConvRaw<V>::type;
  const __nv_bfloat16* xp = x + static_cast<long long>(b) * L * ldx + c;
  __nv_bfloat16* yp = y + static_cast<long long>(b) * L * C + c;
  auto read = [&](int t) { return *reinterpret_cast<const Raw*>(xp + static_cast<long long>(t) * ldx); };
  auto token = [&](int t, const Raw& in) {
#pragma unroll
    for (int j = 0; j + 1 < K; ++j)
#pragma unroll
      for (int e = 0; e < V; ++e) win[j][e] = win[j + 1][e];
    conv_unpack<V>(in, win[K - 1]);
    float o[V];
#pragma unroll
    for (int e = 0; e < V; ++e) {
      o[e] = 0.f;
#pragma unroll
      for (int j = 0; j < K; ++j) o[e] += wv[j][e] * win[j][e];
    }
    if (act) {                           // the eager form rounds the conv output to the activation dtype before the SiLU
      conv_round<V>(o);
#pragma unroll
      for (int e = 0; e < V; ++e) o[e] = silu_f(o[e]);
    }
    conv_store<V>(yp + static_cast<long long>(t) * C, o);
  };
  if constexpr (V == 1) {                // short runs and many threads: nothing ahead (40 x 3072 2.8 us with, 2.5 without; 6000 x 1001 13.3, 11.5)
#pragma unroll 4
    for (int t = t0; t < t1; ++t) token(t, read(t));
  } else {                               // four tokens at a time, the next four on their way while these are worked on
    constexpr int U = 4;
    Raw now[U], next[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (t0 + u < t1) now[u] = read(t0 + u);
    for (int t = t0; t < t1; t += U) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (t + U + u < t1) next[u] = read(t + U + u);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (t + u >= t1) break;
        token(t + u, now[u]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) now[u] = next[u];
    }
  }
}

// dx[b,t,c] = sum_j w[c,j] * dpre[b, t + K-1-j, c], dpre = dy * silu'(pre); pre is recomputed, once for each output.
template <int K, int V>
__global__ void __launch_bounds__(128)
gdn_conv_bwd_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ w,
                    const __nv_bfloat16* __restrict__ left, const __nv_bfloat16* __restrict__ dy, int L, int C, int runs, int run,
                    int act, __nv_bfloat16* __restrict__ dx) {
  const int c = (blockIdx.y * 128 + threadIdx.x) * V;
  if (c >= C) return;
  const int b = blockIdx.x / runs, t0 = (blockIdx.x - b * runs) * run, t1 = min(L, t0 + run);
  float wv[K][V], win[K][V], d[K][V];   // d[j]: the gradient that tap j passes on, that of output t + K - 1 - j
  conv_taps<K, V>(w + static_cast<long long>(c) * K, wv);
#pragma unroll
  for (int j = 0; j < K; ++j)
#pragma unroll
    for (int e = 0; e < V; ++e) d[j][e] = 0.f;
#pragma unroll
  for (int j = 1; j < K; ++j) conv_input<K, V>(x, ldx, left, b, t0 - K + j, c, L, C, win[j]);
  using Raw = typename ConvRaw<V>::type;
  const __nv_bfloat16* xp = x + static_cast<long long>(b) * L * ldx + c;
  const __nv_bfloat16* gp = dy + static_cast<long long>(b) * L * C + c;
  auto read = [&](Raw& in, Raw& grad, int t) {
    in = *reinterpret_cast<const Raw*>(xp + static_cast<long long>(t) * ldx);
    grad = *reinterpret_cast<const Raw*>(gp + static_cast<long long>(t) * C);
  };
  auto token = [&](int to, const Raw& in, const Raw& grad) {
#pragma unroll
    for (int j = K - 1; j > 0; --j)
#pragma unroll
      for (int e = 0; e < V; ++e) d[j][e] = d[j - 1][e];
    if (to < L) {
#pragma unroll
      for (int j = 0; j + 1 < K; ++j)
#pragma unroll
        for (int e = 0; e < V; ++e) win[j][e] = win[j + 1][e];
      conv_unpack<V>(in, win[K - 1]);
      conv_unpack<V>(grad, d[0]);
      if (act) {
        float pre[V];
#pragma unroll
        for (int e = 0; e < V; ++e) {
          pre[e] = 0.f;
#pragma unroll
          for (int j = 0; j < K; ++j) pre[e] += wv[j][e] * win[j][e];
        }
        conv_round<V>(pre);
#pragma unroll
        for (int e = 0; e < V; ++e) d[0][e] *= dsilu_f(pre[e]);
      }
    } else {
#pragma unroll
      for (int e = 0; e < V; ++e) d[0][e] = 0.f;
    }
    const int t = to - (K - 1);
    if (t >= t0) {
      float o[V];
#pragma unroll
      for (int e = 0; e < V; ++e) {
        o[e] = 0.f;
#pragma unroll
        for (int j = 0; j < K; ++j) o[e] += wv[j][e] * d[j][e];
      }
      conv_store<V>(dx + (static_cast<long long>(b) * L + t) * C + c, o);
    }
  };
  const int t2 = min(L, t1 + K - 1);
  constexpr int U = 2;
  Raw now[2][U], next[2][U];
  auto fetch = [&](Raw (&r)[2][U], int t) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (t + u < t2) read(r[0][u], r[1][u], t + u);
  };
  fetch(now, t0);
  for (int tb = t0; tb < t1 + K - 1; tb += U) {
    fetch(next, tb + U);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (tb + u >= t1 + K - 1) break;
      token(tb + u, now[0][u], now[1][u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      now[0][u] = next[0][u];
      now[1][u] = next[1][u];
    }
  }
}

// Tokens per thread: long runs re-read less context (K - 1 tokens a run) and set out less often, but a short input wants
// threads: they shorten until there are 32768, to eight tokens (one where a thread has one channel).
int conv_run(long long rows_of_tokens, int L, int C, int V) {
  int run = V == 1 ? 16 : 32;
  while (run > (V == 1 ? 1 : 8) && rows_of_tokens * ((L + run - 1) / run) * (C / V) < (V == 1 ? 1LL << 16 : 1LL << 15)) run /= 2;
  return run;
}

// One token: y[b,c] = act(sum_j w[c,j] * ctx[j]), ctx = [state[b,c,:], x[b,c]]; state shifts left.
__global__ void gdn_conv_step_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ w,
                                     __nv_bfloat16* __restrict__ state, int B, int C, int K, int act,
                                     __nv_bfloat16* __restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B * C) return;
  const int c = i % C, b = i / C;
  __nv_bfloat16* st = state + static_cast<long long>(i) * (K - 1);
  const __nv_bfloat16 xv = x[static_cast<long long>(b) * ldx + c];
  float acc = __bfloat162float(w[c * K + K - 1]) * __bfloat162float(xv);
  for (int j = 0; j < K - 1; ++j) {
    const __nv_bfloat16 s = st[j];
    acc += __bfloat162float(w[c * K + j]) * __bfloat162float(s);
    if (j > 0) st[j - 1] = s;
  }
  if (K > 1) st[K - 2] = xv;
  acc = __bfloat162float(__float2bfloat16_rn(acc));
  y[i] = __float2bfloat16_rn(act ? silu_f(acc) : acc);
}

// One block per (b, value head); thread j owns column j of S [KD, VD] and keeps it in registers.
// q,k [B, Hk, KD] bf16 (row stride given), v [B, Hv, VD], g,beta [B, Hv] fp32, S [B, Hv, KD, VD] fp32.
template <int KD>
__global__ void gdn_decode_step_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                                       const __nv_bfloat16* __restrict__ v, long long ldq, long long ldk, long long ldv,
                                       const float* __restrict__ g, const float* __restrict__ beta,
                                       float* __restrict__ S, int Hk, int Hv, int VD, int l2norm, float eps,
                                       __nv_bfloat16* __restrict__ out, GdnRawGates raw) {
  __shared__ float qs[KD], ks[KD], red[32];
  const int b = blockIdx.x / Hv, hv = blockIdx.x % Hv;
  const int hk = hv / (Hv / Hk);
  const int tid = threadIdx.x;
  float qq = 0.f, kk = 0.f;
  for (int i = tid; i < KD; i += blockDim.x) {
    const float qv = __bfloat162float(q[static_cast<long long>(b) * ldq + hk * KD + i]);
    const float kv = __bfloat162float(k[static_cast<long long>(b) * ldk + hk * KD + i]);
    qs[i] = qv;
    ks[i] = kv;
    qq += qv * qv;
    kk += kv * kv;
  }
  float qn = 1.f, kn = 1.f;
  if (l2norm) {
    qn = rsqrtf(block_sum(qq, red) + eps);
    kn = rsqrtf(block_sum(kk, red) + eps);
  }
  __syncthreads();
  const float qscale = qn * rsqrtf(static_cast<float>(KD));
  const long long bh = static_cast<long long>(b) * Hv + hv;
  float eg, bt;
  if (raw.a) {
    // gates from the projection output: g = -exp(A_log) softplus(a + dt_bias), beta = sigmoid(b)
    const float x = __bfloat162float(raw.a[static_cast<long long>(b) * raw.lda + hv]) + raw.dt_bias[hv];
    const float sp = x > 20.f ? x : log1pf(__expf(x));
    eg = __expf(-__expf(raw.A_log[hv]) * sp);
    bt = 1.f / (1.f + __expf(-__bfloat162float(raw.b[static_cast<long long>(b) * raw.ldb + hv])));
  } else {
    eg = __expf(g[bh]);
    bt = beta[bh];
  }
  for (int j = tid; j < VD; j += blockDim.x) {
    float* Sc = S + bh * KD * VD + j;
    float col[KD];
    float kv = 0.f;
#pragma unroll
    for (int i = 0; i < KD; ++i) {
      col[i] = Sc[static_cast<long long>(i) * VD] * eg;
      kv += col[i] * (ks[i] * kn);
    }
    const float delta = (__bfloat162float(v[static_cast<long long>(b) * ldv + hv * VD + j]) - kv) * bt;
    float o = 0.f;
#pragma unroll
    for (int i = 0; i < KD; ++i) {
      col[i] += (ks[i] * kn) * delta;
      o += col[i] * (qs[i] * qscale);
      Sc[static_cast<long long>(i) * VD] = col[i];
    }
    out[bh * VD + j] = __float2bfloat16_rn(o);
  }
}

// The same step for KD x VD states that divide over 256 threads: thread (row group, column group) keeps RPT rows x 4
// columns of S in registers (16 x float4 at 128 x 128), so every load and store is a 16-byte access of a 512-byte row
// and all of a CTA's 64 KB are in flight at once; the two dot products (S^T k and S^T q) are finished across the row
// groups through shared memory in a fixed order.  (One column per thread, as above, needs KD registers per thread and
// spills at KD = 128.)
template <int KD, int VD>
__global__ void __launch_bounds__(256)
gdn_decode_step_tile_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                            const __nv_bfloat16* __restrict__ v, long long ldq, long long ldk, long long ldv,
                            const float* __restrict__ g, const float* __restrict__ beta, float* __restrict__ S, int Hk,
                            int Hv, int l2norm, float eps, __nv_bfloat16* __restrict__ out, GdnRawGates raw) {
  constexpr int CG = VD / 4, RG = 256 / CG, RPT = KD / RG;
  static_assert(VD % 4 == 0 && 256 % CG == 0 && KD % RG == 0 && RPT >= 1, "state does not divide over 256 threads");
  __shared__ float qs[KD], ks[KD], red[32];
  __shared__ __align__(16) float part[RG][VD];
  const int b = blockIdx.x / Hv, hv = blockIdx.x % Hv;
  const int hk = hv / (Hv / Hk);
  const int tid = threadIdx.x;
  const int cg = tid % CG, rg = tid / CG;
  const long long bh = static_cast<long long>(b) * Hv + hv;
  // the state does not depend on anything computed here: request it first
  float4* Sp = reinterpret_cast<float4*>(S + bh * KD * VD) + static_cast<long long>(rg) * RPT * CG + cg;
  float4 col[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) col[i] = Sp[i * CG];
  float qq = 0.f, kk = 0.f;
  for (int i = tid; i < KD; i += 256) {
    const float qv = __bfloat162float(q[static_cast<long long>(b) * ldq + hk * KD + i]);
    const float kv = __bfloat162float(k[static_cast<long long>(b) * ldk + hk * KD + i]);
    qs[i] = qv;
    ks[i] = kv;
    qq += qv * qv;
    kk += kv * kv;
  }
  float qn = 1.f, kn = 1.f;
  if (l2norm) {
    qn = rsqrtf(block_sum(qq, red) + eps);
    kn = rsqrtf(block_sum(kk, red) + eps);
  }
  __syncthreads();
  const float qscale = qn * rsqrtf(static_cast<float>(KD));
  float eg, bt;
  if (raw.a) {
    const float x = __bfloat162float(raw.a[static_cast<long long>(b) * raw.lda + hv]) + raw.dt_bias[hv];
    const float sp = x > 20.f ? x : log1pf(__expf(x));
    eg = __expf(-__expf(raw.A_log[hv]) * sp);
    bt = 1.f / (1.f + __expf(-__bfloat162float(raw.b[static_cast<long long>(b) * raw.ldb + hv])));
  } else {
    eg = __expf(g[bh]);
    bt = beta[bh];
  }
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const float kx = ks[rg * RPT + i] * kn;
    col[i].x *= eg; col[i].y *= eg; col[i].z *= eg; col[i].w *= eg;
    acc.x += col[i].x * kx; acc.y += col[i].y * kx; acc.z += col[i].z * kx; acc.w += col[i].w * kx;
  }
  *reinterpret_cast<float4*>(&part[rg][cg * 4]) = acc;
  __syncthreads();
  float4 kv = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int r = 0; r < RG; ++r) {
    const float4 t = *reinterpret_cast<const float4*>(&part[r][cg * 4]);
    kv.x += t.x; kv.y += t.y; kv.z += t.z; kv.w += t.w;
  }
  const __nv_bfloat16* vp = v + static_cast<long long>(b) * ldv + hv * VD + cg * 4;
  float4 delta;
  delta.x = (__bfloat162float(vp[0]) - kv.x) * bt;
  delta.y = (__bfloat162float(vp[1]) - kv.y) * bt;
  delta.z = (__bfloat162float(vp[2]) - kv.z) * bt;
  delta.w = (__bfloat162float(vp[3]) - kv.w) * bt;
  acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const float kx = ks[rg * RPT + i] * kn, qx = qs[rg * RPT + i] * qscale;
    col[i].x += kx * delta.x; col[i].y += kx * delta.y; col[i].z += kx * delta.z; col[i].w += kx * delta.w;
    acc.x += col[i].x * qx; acc.y += col[i].y * qx; acc.z += col[i].z * qx; acc.w += col[i].w * qx;
    Sp[i * CG] = col[i];
  }
  __syncthreads();                       // every thread has read the first sums
  *reinterpret_cast<float4*>(&part[rg][cg * 4]) = acc;
  __syncthreads();
  if (tid < VD) {
    float o = 0.f;
#pragma unroll
    for (int r = 0; r < RG; ++r) o += part[r][tid];
    out[bh * VD + tid] = __float2bfloat16_rn(o);
  }
}

}  // namespace

namespace {

constexpr int kConvV = 4;                // channels of a thread
// 8-byte accesses want whole groups of four channels on 8-byte boundaries; anything else goes channel by channel.
bool conv_vec(int C, long long ldx, const void* x, const void* w, const void* y, const void* z) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y) |
                       reinterpret_cast<uintptr_t>(z);
  return C % kConvV == 0 && ldx % kConvV == 0 && at % 8 == 0;
}

template <int K>
void conv_launch(bool bwd, const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* w, const __nv_bfloat16* left,
                 const __nv_bfloat16* dy, int B, int L, int C, int act, __nv_bfloat16* out, cudaStream_t stream) {
  // one channel and four a thread, us forward / backward: 130 tokens of 10240 5.0 / 7.9 and 4.1 / 6.0, 1000 of 3072 7.4 / 12.3
  // and 5.8 / 8.9, 5000 of 10240 86 / 136 and 48 / 89; below a million values one is as fast or faster
  const bool vec = conv_vec(C, ldx, x, w, out, dy) && static_cast<long long>(B) * L * C >= 1LL << 20;
  const int V = vec ? kConvV : 1, run = conv_run(B, L, C, V), runs = (L + run - 1) / run;
  const dim3 grid(B * runs, (C / V + 127) / 128);
  if (!bwd && vec) gdn_conv_fwd_kernel<K, kConvV><<<grid, 128, 0, stream>>>(x, ldx, w, left, L, C, runs, run, act, out);
  else if (!bwd) gdn_conv_fwd_kernel<K, 1><<<grid, 128, 0, stream>>>(x, ldx, w, left, L, C, runs, run, act, out);
  else if (vec) gdn_conv_bwd_kernel<K, kConvV><<<grid, 128, 0, stream>>>(x, ldx, w, left, dy, L, C, runs, run, act, out);
  else gdn_conv_bwd_kernel<K, 1><<<grid, 128, 0, stream>>>(x, ldx, w, left, dy, L, C, runs, run, act, out);
}

const char* conv_any(bool bwd, const void* x, long long ldx, const void* w, const void* left, const void* dy, int B, int L, int C,
                     int K, bool act, void* out, cudaStream_t stream) {
  if (K < 1 || K > kMaxConvK) return "gdn_conv: kernel width 1..8";
  if (static_cast<long long>(B) * L * C == 0) return nullptr;
  const auto* xp = static_cast<const __nv_bfloat16*>(x);
  const auto* wp = static_cast<const __nv_bfloat16*>(w);
  const auto* lp = static_cast<const __nv_bfloat16*>(left);
  const auto* dp = static_cast<const __nv_bfloat16*>(dy);
  auto* op = static_cast<__nv_bfloat16*>(out);
  switch (K) {
#define FERRL_CONV(KV) case KV: conv_launch<KV>(bwd, xp, ldx, wp, lp, dp, B, L, C, act ? 1 : 0, op, stream); break
    FERRL_CONV(1); FERRL_CONV(2); FERRL_CONV(3); FERRL_CONV(4); FERRL_CONV(5); FERRL_CONV(6); FERRL_CONV(7); FERRL_CONV(8);
#undef FERRL_CONV
  }
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : (bwd ? "gdn_conv_bwd launch failed" : "gdn_conv_fwd launch failed");
}

}  // namespace

const char* gdn_conv_fwd(const void* x, long long ldx, const void* w, const void* left, int B, int L, int C, int K,
                         bool act, void* y, cudaStream_t stream) {
  return conv_any(false, x, ldx, w, left, nullptr, B, L, C, K, act, y, stream);
}

const char* gdn_conv_bwd(const void* x, long long ldx, const void* w, const void* left, const void* dy, int B, int L,
                         int C, int K, bool act, void* dx, cudaStream_t stream) {
  return conv_any(true, x, ldx, w, left, dy, B, L, C, K, act, dx, stream);
}

const char* gdn_conv_step(const void* x, long long ldx, const void* w, void* state, int B, int C, int K, bool act,
                          void* y, cudaStream_t stream) {
  if (K < 1 || K > kMaxConvK) return "gdn_conv: kernel width 1..8";
  if (B * C == 0) return nullptr;
  gdn_conv_step_kernel<<<(B * C + 255) / 256, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(x), ldx,
                                                                static_cast<const __nv_bfloat16*>(w),
                                                                static_cast<__nv_bfloat16*>(state), B, C, K, act ? 1 : 0,
                                                                static_cast<__nv_bfloat16*>(y));
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "gdn_conv_step launch failed";
}

const char* gdn_decode_step(const void* q, const void* k, const void* v, long long ldq, long long ldk, long long ldv,
                            const float* g, const float* beta, float* S, int B, int Hk, int Hv, int KD, int VD,
                            bool l2norm, float eps, void* out, cudaStream_t stream, const GdnRawGates* raw_gates) {
  if (Hk <= 0 || Hv % Hk) return "gdn_decode_step: value heads must be a multiple of key heads";
  GdnRawGates raw{};
  if (raw_gates) raw = *raw_gates;
  if (!raw.a && (!g || !beta)) return "gdn_decode_step: either g and beta or the raw gate inputs are needed";
  if (raw.a && (!raw.b || !raw.A_log || !raw.dt_bias)) return "gdn_decode_step: incomplete raw gate inputs";
  if (B == 0) return nullptr;
  if (KD == 128 && VD == 128) {
    gdn_decode_step_tile_kernel<128, 128><<<B * Hv, 256, 0, stream>>>(
        static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v),
        ldq, ldk, ldv, g, beta, S, Hk, Hv, l2norm ? 1 : 0, eps, static_cast<__nv_bfloat16*>(out), raw);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? nullptr : "gdn_decode_step launch failed";
  }
  const int threads = std::min(256, (VD + 31) / 32 * 32);
#define FERRL_GDN_STEP(KDV)                                                                                        \
  gdn_decode_step_kernel<KDV><<<B * Hv, threads, 0, stream>>>(                                                     \
      static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v), \
      ldq, ldk, ldv, g, beta, S, Hk, Hv, VD, l2norm ? 1 : 0, eps, static_cast<__nv_bfloat16*>(out), raw)
  switch (KD) {
    case 16: FERRL_GDN_STEP(16); break;
    case 32: FERRL_GDN_STEP(32); break;
    case 64: FERRL_GDN_STEP(64); break;
    case 128: FERRL_GDN_STEP(128); break;
    default: return "gdn_decode_step: key dim must be 16, 32, 64 or 128";
  }
#undef FERRL_GDN_STEP
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "gdn_decode_step launch failed";
}

}  // namespace ferrl
