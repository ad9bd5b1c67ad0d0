// Small bandwidth-bound kernels: gated activation (SwiGLU / GeGLU) forward+backward,
// embedding gather, LoRA merge W + B*A, fused multi-tensor AdamW with global-norm clip,
// GRPO loss forward/backward.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../api.h"
#include "../common.cuh"
#include "vec.cuh"

namespace ferrl {
namespace {

__device__ __forceinline__ float act_fwd(float g, int act) {
  if (act == kActSilu) return g / (1.f + __expf(-g));
  // gelu, tanh form: (1 + tanh(u)) / 2 = 1 / (1 + exp(-2u)), which keeps fp32 accuracy under fast math
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return g / (1.f + __expf(-2.f * k0 * (g + k1 * g * g * g)));
}
__device__ __forceinline__ float act_grad(float g, int act) {
  if (act == kActSilu) {
    float s = 1.f / (1.f + __expf(-g));
    return s * (1.f + g * (1.f - s));
  }
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * (g + k1 * g * g * g);
  float t = tanhf(u);
  float du = k0 * (1.f + 3.f * k1 * g * g);
  return 0.5f * (1.f + t) + 0.5f * g * (1.f - t * t) * du;
}

// act(g) * u and its derivatives by g and u
__device__ __forceinline__ float glu_f(float g, float u, const GluAct& k) {
  if (k.act == kActClipped) {
    g = fminf(g, k.limit);
    u = fminf(fmaxf(u, -k.limit), k.limit);
    return g / (1.f + __expf(-k.alpha * g)) * (u + 1.f);
  }
  return act_fwd(g, k.act) * u;
}
__device__ __forceinline__ float2 glu_grad(float g, float u, const GluAct& k) {
  if (k.act == kActClipped) {
    const float gc = fminf(g, k.limit), uc = fminf(fmaxf(u, -k.limit), k.limit);
    const float s = 1.f / (1.f + __expf(-k.alpha * gc));
    return make_float2(g > k.limit ? 0.f : s * (1.f + k.alpha * gc * (1.f - s)) * (uc + 1.f), fabsf(u) > k.limit ? 0.f : gc * s);
  }
  return make_float2(u * act_grad(g, k.act), act_fwd(g, k.act));
}

// gate_up [rows, 2F] laid out [gate | up] -> out [rows, F]
template <typename T>
__global__ void glu_fwd_kernel(const T* __restrict__ gu, T* __restrict__ out, long long rows, int F, GluAct act) {
  pdl_trigger();   // a dependent GEMM may start streaming its weights while this kernel runs
  pdl_wait();      // launched as a programmatic dependent itself: nothing is read before the predecessor is done
  long long n = rows * F;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    long long r = i / F;
    int c = static_cast<int>(i - r * F);
    float g = to_f(gu[r * 2 * F + c]);
    float u = to_f(gu[r * 2 * F + F + c]);
    out[i] = from_f<T>(glu_f(g, u, act));
  }
}
// bf16 vector forms: 8 elements per thread per step, 16-byte loads and stores; F % 8 == 0
__global__ void glu_fwd_vec_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out, long long rows,
                                   int F, GluAct act, const int* __restrict__ token_of) {
  pdl_trigger();   // a dependent GEMM may start streaming its weights while this kernel runs
  pdl_wait();      // launched as a programmatic dependent itself: nothing is read before the predecessor is done
  const int chunks = F / 8;
  const long long n = rows * chunks;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / chunks;
    const int c = static_cast<int>(i - r * chunks);
    if (token_of && token_of[r & ~15LL] < 0) continue;       // padding behind an expert's tokens
    const uint4 gv = *reinterpret_cast<const uint4*>(gu + r * 2 * F + c * 8);
    const uint4 uv = *reinterpret_cast<const uint4*>(gu + r * 2 * F + F + c * 8);
    const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gv);
    const __nv_bfloat162* uh = reinterpret_cast<const __nv_bfloat162*>(&uv);
    uint4 o;
    __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 g = __bfloat1622float2(gh[e]), u = __bfloat1622float2(uh[e]);
      oh[e] = __floats2bfloat162_rn(glu_f(g.x, u.x, act), glu_f(g.y, u.y, act));
    }
    *reinterpret_cast<uint4*>(out + r * F + c * 8) = o;
  }
}
__global__ void glu_bwd_vec_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ dout,
                                   __nv_bfloat16* __restrict__ dgu, long long rows, int F, GluAct act) {
  const int chunks = F / 8;
  const long long n = rows * chunks;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / chunks;
    const int c = static_cast<int>(i - r * chunks);
    const uint4 gv = *reinterpret_cast<const uint4*>(gu + r * 2 * F + c * 8);
    const uint4 uv = *reinterpret_cast<const uint4*>(gu + r * 2 * F + F + c * 8);
    const uint4 dv = *reinterpret_cast<const uint4*>(dout + r * F + c * 8);
    const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gv);
    const __nv_bfloat162* uh = reinterpret_cast<const __nv_bfloat162*>(&uv);
    const __nv_bfloat162* dh = reinterpret_cast<const __nv_bfloat162*>(&dv);
    uint4 og, ou;
    __nv_bfloat162* ogh = reinterpret_cast<__nv_bfloat162*>(&og);
    __nv_bfloat162* ouh = reinterpret_cast<__nv_bfloat162*>(&ou);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 g = __bfloat1622float2(gh[e]), u = __bfloat1622float2(uh[e]), d = __bfloat1622float2(dh[e]);
      const float2 dx = glu_grad(g.x, u.x, act), dy = glu_grad(g.y, u.y, act);
      ogh[e] = __floats2bfloat162_rn(d.x * dx.x, d.y * dy.x);
      ouh[e] = __floats2bfloat162_rn(d.x * dx.y, d.y * dy.y);
    }
    *reinterpret_cast<uint4*>(dgu + r * 2 * F + c * 8) = og;
    *reinterpret_cast<uint4*>(dgu + r * 2 * F + F + c * 8) = ou;
  }
}

template <typename T>
__global__ void glu_bwd_kernel(const T* __restrict__ gu, const T* __restrict__ dout, T* __restrict__ dgu,
                               long long rows, int F, GluAct act) {
  long long n = rows * F;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    long long r = i / F;
    int c = static_cast<int>(i - r * F);
    float g = to_f(gu[r * 2 * F + c]);
    float u = to_f(gu[r * 2 * F + F + c]);
    float d = to_f(dout[i]);
    const float2 dd = glu_grad(g, u, act);
    dgu[r * 2 * F + c] = from_f<T>(d * dd.x);
    dgu[r * 2 * F + F + c] = from_f<T>(d * dd.y);
  }
}

// V entries an access (4 where width and addresses allow it): one entry a thread took 58 us for 8192 rows of 4096 bf16,
// now 23 (the bytes take 20)
template <typename T, int V>
__global__ void embedding_kernel(const long long* __restrict__ ids, const T* __restrict__ table, T* __restrict__ out,
                                 long long n_tok, int H, long long vocab, float scale) {
  long long tok = blockIdx.x;
  long long id = ids[tok];
  if (id < 0 || id >= vocab) id = 0;  // never index out of the table
  const T* src = table + id * H;
#pragma unroll 4
  for (int i = threadIdx.x * V; i < H; i += blockDim.x * V) {
    Vec<V> v = ld<V>(src + i);
    if (scale != 1.f) {
#pragma unroll
      for (int e = 0; e < V; ++e) v.v[e] *= scale;
    }
    st<V>(out + tok * H + i, v);
  }
}

// W'[o,i] = W[o,i] + sum_r B[o,r] A[r,i]   (A, B fp32; R small)
template <typename T>
__global__ void lora_merge_kernel(const T* __restrict__ w, const float* __restrict__ a, const float* __restrict__ b,
                                  T* __restrict__ out, int O, int I, int R) {
  extern __shared__ float sb[];  // B row for this output row
  int o = blockIdx.x;
  for (int r = threadIdx.x; r < R; r += blockDim.x) sb[r] = b[static_cast<long long>(o) * R + r];
  __syncthreads();
  for (int i = threadIdx.x; i < I; i += blockDim.x) {
    float acc = to_f(w[static_cast<long long>(o) * I + i]);
    for (int r = 0; r < R; ++r) acc += sb[r] * a[static_cast<long long>(r) * I + i];
    out[static_cast<long long>(o) * I + i] = from_f<T>(acc);
  }
}

// ------------------------------------------------------------------ AdamW
// Tensor table lives in device memory: one entry per tensor, chunked over blocks.
__global__ void sumsq_kernel(const AdamTensor* __restrict__ tab, const int* __restrict__ blk_tensor,
                             const long long* __restrict__ blk_off, double* __restrict__ out, int chunk) {
  __shared__ float red[32];
  const AdamTensor t = tab[blk_tensor[blockIdx.x]];
  long long off = blk_off[blockIdx.x];
  long long end = min(off + chunk, t.n);
  float s = 0.f;
  for (long long i = off + threadIdx.x; i < end; i += blockDim.x) {
    float g = t.g[i];
    s += g * g;
  }
  float tot = block_sum(s, red);
  if (threadIdx.x == 0) atomicAdd(out, static_cast<double>(tot));
}

// scalars[0] = sum of squares (double, already reduced). clip factor derived on device so no host sync is
// needed between the norm and the update.
__global__ void adamw_kernel(const AdamTensor* __restrict__ tab, const int* __restrict__ blk_tensor,
                             const long long* __restrict__ blk_off, const double* __restrict__ sumsq, int chunk,
                             float lr, float b1, float b2, float eps, float wd, float bc1_inv, float bc2_inv,
                             float max_norm, float pre_scale, float* __restrict__ norm_out) {
  const AdamTensor t = tab[blk_tensor[blockIdx.x]];
  long long off = blk_off[blockIdx.x];
  long long end = min(off + chunk, t.n);
  float gs = pre_scale;
  if (sumsq) {
    float norm = static_cast<float>(sqrt(*sumsq)) * pre_scale;
    if (blockIdx.x == 0 && threadIdx.x == 0 && norm_out) *norm_out = norm;
    if (norm == 0.f) return;  // all-zero gradient: leave parameters and moments untouched
    if (max_norm > 0.f && norm > max_norm) gs *= max_norm / norm;
  }
  for (long long i = off + threadIdx.x; i < end; i += blockDim.x) {
    float g = t.g[i] * gs;
    float m = b1 * t.m[i] + (1.f - b1) * g;
    float v = b2 * t.v[i] + (1.f - b2) * g * g;
    float p = t.p[i] * (1.f - lr * wd);
    p -= lr * (m * bc1_inv) / (sqrtf(v * bc2_inv) + eps);
    t.m[i] = m;
    t.v[i] = v;
    t.p[i] = p;
  }
}

// ------------------------------------------------------------------ GRPO loss
// One block per sequence row. Writes per-row partial sums; the host-side wrapper combines
// them according to the loss type. Also emits dL/dlogp given the upstream scale.
// mode bits: 1 = sequence-level ratio, 2 = has ref, 4 = has tis
__global__ void grpo_loss_kernel(const float* __restrict__ logp, const float* __restrict__ logp_old,
                                 const float* __restrict__ logp_ref, const float* __restrict__ adv,
                                 const float* __restrict__ mask, const float* __restrict__ tis,
                                 float* __restrict__ row_sum, float* __restrict__ row_cnt, float* __restrict__ dlogp,
                                 int L, float eps_lo, float eps_hi, float beta, int mode) {
  __shared__ float red[32];
  const int g = blockIdx.x;
  const float* lp = logp + static_cast<long long>(g) * L;
  const float* lo = logp_old + static_cast<long long>(g) * L;
  const float* lr_ = (mode & 2) ? logp_ref + static_cast<long long>(g) * L : nullptr;
  const float* mk = mask + static_cast<long long>(g) * L;
  const float* tw = (mode & 4) ? tis + static_cast<long long>(g) * L : nullptr;
  const float a = adv[g];
  const float CAP = 60.f;
  float cnt = 0.f, seq_num = 0.f;
  for (int t = threadIdx.x; t < L; t += blockDim.x) {
    float m = mk[t];
    if (m > 0.f) {
      cnt += m;
      seq_num += (lp[t] - lo[t]) * m;
    }
  }
  cnt = block_sum(cnt, red);
  float seq_lr = 0.f;
  bool seq_clamped = false;
  if (mode & 1) {
    seq_num = block_sum(seq_num, red);
    seq_lr = seq_num / fmaxf(cnt, 1.f);
    seq_clamped = (seq_lr < -CAP) || (seq_lr > CAP);
    seq_lr = fminf(fmaxf(seq_lr, -CAP), CAP);
  }
  float acc = 0.f;
  // For the sequence-level ratio every token's surrogate depends on every token's logp through the
  // mean; d(sum_t m_t surr_t)/d logp_u = m_u/cnt * sum_t m_t tis_t dsurr_t/dratio * ratio.
  float seq_coef = 0.f;
  for (int t = threadIdx.x; t < L; t += blockDim.x) {
    float m = mk[t];
    float val = 0.f, dval = 0.f;
    if (m > 0.f) {
      float d = lp[t] - lo[t];
      bool clamped = (mode & 1) ? seq_clamped : (d < -CAP || d > CAP);
      float ratio = __expf((mode & 1) ? seq_lr : fminf(fmaxf(d, -CAP), CAP));
      float un = ratio * a;
      float rc = fminf(fmaxf(ratio, 1.f - eps_lo), 1.f + eps_hi);
      float cl = rc * a;
      float surr = fminf(un, cl);
      // gradient flows through the unclipped branch when it is the minimum (ties go to unclipped)
      float dsurr_dratio = (un <= cl) ? a : ((ratio == rc) ? a : 0.f);
      if (a == 0.f) { surr = 0.f; dsurr_dratio = 0.f; }
      float w = tw ? tw[t] : 1.f;
      surr *= w;
      float dr = clamped ? 0.f : dsurr_dratio * w * ratio;  // d surr / d logp (token level)
      val = surr;
      if (mode & 1) seq_coef += m * dr; else dval = dr;
      if (lr_) {
        float dd = lr_[t] - lp[t];
        float e = __expf(dd);
        val -= beta * (e - dd - 1.f);
        dval += beta * (e - 1.f);  // d(-beta*k3)/dlogp = beta*(e - 1)
      }
      acc += val * m;
    }
    if (dlogp) dlogp[static_cast<long long>(g) * L + t] = dval * m;  // completed below for sequence level
  }
  acc = block_sum(acc, red);
  if (mode & 1) {
    seq_coef = block_sum(seq_coef, red);
    if (dlogp) {
      float per = seq_coef / fmaxf(cnt, 1.f);
      for (int t = threadIdx.x; t < L; t += blockDim.x) {
        float m = mk[t];
        if (m > 0.f) dlogp[static_cast<long long>(g) * L + t] += per * m;
      }
    }
  }
  if (threadIdx.x == 0) {
    row_sum[g] = acc;
    row_cnt[g] = cnt;
  }
}

// dlogp[g,t] *= -(upstream) * row_scale[g]
__global__ void grpo_scale_kernel(float* __restrict__ dlogp, const float* __restrict__ row_scale, long long n, int L) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    dlogp[i] *= row_scale[i / L];
}

inline unsigned grid_for(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  return static_cast<unsigned>(b < 1 ? 1 : (b > 148 * 16 ? 148 * 16 : b));
}

}  // namespace

const char* glu(int dtype, bool backward, const void* gu, const void* dout, void* out, long long rows, int F, GluAct act,
                cudaStream_t s, const int* token_of) {
  if (rows * F == 0) return nullptr;
  unsigned grid = grid_for(rows * F, 256);
  if (dtype == kF32) {
    if (backward)
      glu_bwd_kernel<float><<<grid, 256, 0, s>>>(static_cast<const float*>(gu), static_cast<const float*>(dout),
                                                 static_cast<float*>(out), rows, F, act);
    else
      glu_fwd_kernel<float><<<grid, 256, 0, s>>>(static_cast<const float*>(gu), static_cast<float*>(out), rows, F, act);
  } else if ((F % 8) == 0 && (reinterpret_cast<uintptr_t>(gu) & 15) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0 &&
             (reinterpret_cast<uintptr_t>(dout) & 15) == 0) {
    using B = __nv_bfloat16;
    const unsigned vgrid = grid_for(rows * (F / 8), 256);
    if (backward)
      glu_bwd_vec_kernel<<<vgrid, 256, 0, s>>>(static_cast<const B*>(gu), static_cast<const B*>(dout), static_cast<B*>(out),
                                               rows, F, act);
    else
      launch_pdl(glu_fwd_vec_kernel, dim3(vgrid), dim3(256), 0, s, static_cast<const B*>(gu), static_cast<B*>(out), rows, F, act, token_of);
  } else {
    using B = __nv_bfloat16;
    if (backward)
      glu_bwd_kernel<B><<<grid, 256, 0, s>>>(static_cast<const B*>(gu), static_cast<const B*>(dout),
                                             static_cast<B*>(out), rows, F, act);
    else
      glu_fwd_kernel<B><<<grid, 256, 0, s>>>(static_cast<const B*>(gu), static_cast<B*>(out), rows, F, act);
  }
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "glu launch failed";
}

const char* embedding(int dtype, const long long* ids, const void* table, void* out, long long n_tok, int H,
                      long long vocab, float scale, cudaStream_t s) {
  if (n_tok == 0) return nullptr;
  const bool vec = H % 4 == 0 && ((reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  const unsigned n = static_cast<unsigned>(n_tok);
#define FERRL_EMBED(T, V) \
  embedding_kernel<T, V><<<n, 256, 0, s>>>(ids, static_cast<const T*>(table), static_cast<T*>(out), n_tok, H, vocab, scale)
  if (dtype == kF32) {
    if (vec) FERRL_EMBED(float, 4); else FERRL_EMBED(float, 1);
  } else {
    if (vec) FERRL_EMBED(__nv_bfloat16, 4); else FERRL_EMBED(__nv_bfloat16, 1);
  }
#undef FERRL_EMBED
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "embedding launch failed";
}

namespace {
// Rows start[b] .. start[b] + L - 1 of x [B, S, W pieces], the last row again past the end, a warp per row.  Backward: every
// row's gradient is written, zeros outside the window; the last row's is a sum in the order of the window.  A negative start is
// reported and its sequence becomes NaNs in both directions, so that no result comes out of it.  Bound by the bytes: a gather by an index per element took 120 us for 8 x 1024 rows of 4096 out of
// 8 x 1423, its gradient a fill and an indexed sum 161; now 29 and 34 (134 and 160 MB: 20 and 24).
template <bool BWD>
__global__ void __launch_bounds__(256)
window_rows_kernel(const uint4* __restrict__ x, const long long* __restrict__ start, int B, int S, int L, int W, uint4* __restrict__ out, int* status) {
  const long long r = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31, rows = BWD ? S : L;
  if (r >= static_cast<long long>(B) * rows) return;
  const int b = static_cast<int>(r / rows), i = static_cast<int>(r - static_cast<long long>(b) * rows);
  const long long at = start[b];
  if (at < 0 && lane == 0) atomicCAS(status, kStatusOk, kStatusBadIndex);
  const uint32_t fill = at < 0 ? 0x7FFF7FFFu : 0u;
  const uint4* src = nullptr;
  if (at >= 0) {
    if (!BWD) src = x + (static_cast<long long>(b) * S + min(at + i, static_cast<long long>(S - 1))) * W;
    else if (i >= at && i - at < L) src = x + (static_cast<long long>(b) * L + (i - at)) * W;
  }
  if (BWD && i == S - 1 && at >= 0 && at + L > S) {          // the windows' rows past the end are this one
    for (int c = lane; c < W; c += 32) {
      float sum[8] = {};
      for (long long j = max(0LL, S - 1 - at); j < L; ++j) {
        const uint4 u = x[(static_cast<long long>(b) * L + j) * W + c];
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          sum[2 * e] += __uint_as_float(w[e] << 16);
          sum[2 * e + 1] += __uint_as_float(w[e] & 0xffff0000u);
        }
      }
      uint4 u;
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
      for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(sum[2 * e], sum[2 * e + 1]);
      out[r * W + c] = u;
    }
    return;
  }
#pragma unroll 4
  for (int c = lane; c < W; c += 32) out[r * W + c] = src ? src[c] : make_uint4(fill, fill, fill, fill);
}
}  // namespace

const char* window_rows(const void* x, const long long* start, int B, int S, int L, int width, bool backward, void* out, int* status, cudaStream_t s) {
  if (width % 8 || (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) % 16) return "window_rows: bf16 rows of whole 16-byte pieces";
  const long long rows = static_cast<long long>(B) * (backward ? S : L);
  if (rows == 0 || width == 0) return nullptr;
  const unsigned grid = static_cast<unsigned>((rows + 7) / 8);
  if (backward)
    window_rows_kernel<true><<<grid, 256, 0, s>>>(static_cast<const uint4*>(x), start, B, S, L, width / 8, static_cast<uint4*>(out), status);
  else
    window_rows_kernel<false><<<grid, 256, 0, s>>>(static_cast<const uint4*>(x), start, B, S, L, width / 8, static_cast<uint4*>(out), status);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "window_rows launch failed";
}

namespace {
// The sigmoid gate on an attention's output, bf16 rows of W pieces of eight, gate rows ldg pieces apart: out = a * s with s rounded
// as a tensor of the same type would be; da = dy * s, dgate = dy * a * s (1 - s).  Bound by the bytes: a conversion to float32, a
// sigmoid, a conversion back and a product took 220 us at 8188 rows of 4096 and their gradients 259; now 41 and 58 (201 and 335 MB:
// 31 and 51).
template <bool BWD>
__global__ void __launch_bounds__(256)
gate_mul_kernel(const uint4* __restrict__ a, const uint4* __restrict__ gate, long long ldg, const uint4* __restrict__ dy, long long n, int W,
                uint4* __restrict__ out, uint4* __restrict__ dgate) {
  auto unpack = [](const uint4& u, float (&f)[8]) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      f[2 * e] = __uint_as_float(w[e] << 16);
      f[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
    }
  };
  auto pack = [](const float (&f)[8]) {
    uint4 u;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
    return u;
  };
  const long long step = static_cast<long long>(gridDim.x) * 256;
#pragma unroll 2
  for (long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x; i < n; i += step) {
    const long long row = i / W;
    float x[8], g[8], d[8], s16[8];
    unpack(a[i], x);
    unpack(gate[row * ldg + (i - row * W)], g);
    if (BWD) unpack(dy[i], d);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      g[e] = 1.f / (1.f + __expf(-g[e]));
      s16[e] = __bfloat162float(__float2bfloat16_rn(g[e]));
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (BWD) {
        x[e] = d[e] * x[e] * g[e] * (1.f - g[e]);
        d[e] *= s16[e];
      } else {
        x[e] *= s16[e];
      }
    }
    out[i] = pack(BWD ? d : x);
    if (BWD) dgate[i] = pack(x);
  }
}
}  // namespace

// backward where dy is given: out = da
const char* gate_mul(const void* a, const void* gate, long long ldg, const void* dy, long long rows, int width, void* out, void* dgate, cudaStream_t s) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(dy) |
                       reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dgate);
  if (width % 8 || ldg % 8 || at % 16) return "gate_mul: rows of whole 16-byte pieces";
  const long long n = rows * (width / 8);
  if (n == 0) return nullptr;
  const unsigned grid = static_cast<unsigned>(std::min<long long>((n + 511) / 512, 148 * 64));
#define FERRL_GATE(BWD)                                                                                                        \
  gate_mul_kernel<BWD><<<grid, 256, 0, s>>>(static_cast<const uint4*>(a), static_cast<const uint4*>(gate), ldg / 8,            \
                                            static_cast<const uint4*>(dy), n, width / 8, static_cast<uint4*>(out), static_cast<uint4*>(dgate))
  if (dy) FERRL_GATE(true); else FERRL_GATE(false);
#undef FERRL_GATE
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "gate_mul launch failed";
}

const char* lora_merge(int dtype, const void* w, const float* a, const float* b, void* out, int O, int I, int R,
                       cudaStream_t s) {
  if (O == 0 || I == 0) return nullptr;
  size_t sm = static_cast<size_t>(R) * sizeof(float);
  if (dtype == kF32)
    lora_merge_kernel<float><<<O, 256, sm, s>>>(static_cast<const float*>(w), a, b, static_cast<float*>(out), O, I, R);
  else
    lora_merge_kernel<__nv_bfloat16><<<O, 256, sm, s>>>(static_cast<const __nv_bfloat16*>(w), a, b,
                                                        static_cast<__nv_bfloat16*>(out), O, I, R);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "lora_merge launch failed";
}

const char* adamw_multi(const AdamTensor* tab_dev, const int* blk_tensor_dev, const long long* blk_off_dev,
                        int n_blocks, int chunk, double* sumsq_dev, bool compute_norm, float lr, float b1, float b2,
                        float eps, float wd, float bc1_inv, float bc2_inv, float max_norm, float pre_scale,
                        float* norm_out_dev, cudaStream_t s) {
  if (n_blocks == 0) return nullptr;
  if (compute_norm) {
    cudaMemsetAsync(sumsq_dev, 0, sizeof(double), s);
    sumsq_kernel<<<n_blocks, 256, 0, s>>>(tab_dev, blk_tensor_dev, blk_off_dev, sumsq_dev, chunk);
    count_launch();
  }
  adamw_kernel<<<n_blocks, 256, 0, s>>>(tab_dev, blk_tensor_dev, blk_off_dev, compute_norm ? sumsq_dev : nullptr, chunk, lr, b1, b2, eps, wd,
                                        bc1_inv, bc2_inv, max_norm, pre_scale, norm_out_dev);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "adamw launch failed";
}

const char* grpo_loss_rows(const float* logp, const float* logp_old, const float* logp_ref, const float* adv,
                           const float* mask, const float* tis, float* row_sum, float* row_cnt, float* dlogp, int G,
                           int L, float eps_lo, float eps_hi, float beta, int mode, cudaStream_t s) {
  if (G == 0) return nullptr;
  grpo_loss_kernel<<<G, 256, 0, s>>>(logp, logp_old, logp_ref, adv, mask, tis, row_sum, row_cnt, dlogp, L, eps_lo,
                                     eps_hi, beta, mode);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "grpo_loss launch failed";
}

const char* grpo_scale_rows(float* dlogp, const float* row_scale, int G, int L, cudaStream_t s) {
  long long n = static_cast<long long>(G) * L;
  if (n == 0) return nullptr;
  grpo_scale_kernel<<<grid_for(n, 256), 256, 0, s>>>(dlogp, row_scale, n, L);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "grpo_scale launch failed";
}

}  // namespace ferrl
