// Vocabulary-wide row kernels for sm_100a.
//
//   logprob_rows      per row: log_softmax(f(logit)/T)[target] with an online (single read) max/sum;
//                     f = identity or cap*tanh(x/cap); keeps the row's log-sum-exp for backward
//   logprob_rows_bwd  overwrites the logits row in place with d(loss)/d(logit)
//                     = dlp * (onehot - softmax) * f'(x) / T, ready to feed the dX GEMM
//   sample_rows       temperature + nucleus (top-p) sampling, one cluster per row, counter RNG keyed by
//                     (seed, global row, draw); returns token and behaviour log-prob
//
// sample_rows does all probability mass arithmetic in 2^-40 fixed point with integer atomics, so
// the nucleus threshold and the drawn token do not depend on the order in which threads add
// (bit-reproducible across runs).  The nucleus threshold is found by narrowing the range of keys that
// holds it - no sort, no host copy of the row.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../api.h"
#include "../common.cuh"

namespace ferrl {
namespace {

namespace cg = cooperative_groups;

__device__ __forceinline__ float capf(float x, float cap) { return cap > 0.f ? cap * tanhf(x / cap) : x; }

template <typename T>
__global__ void logprob_rows_kernel(const T* __restrict__ logits, long long ld, const long long* __restrict__ targets,
                                    float* __restrict__ lp, float* __restrict__ lse, int V, float inv_t, float cap) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const T* x = logits + row * ld;
  float m = -INFINITY, s = 0.f;
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    float z = capf(to_f(x[i]), cap) * inv_t;
    if (z > m) {
      s = s * __expf(m - z) + 1.f;
      m = z;
    } else {
      s += __expf(z - m);
    }
  }
  float gm = block_max(m, red);
  float part = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
  float tot = block_sum(part, red);
  if (threadIdx.x == 0) {
    float l = gm + logf(tot);
    long long t = targets[row];
    float zt = (t >= 0 && t < V) ? capf(to_f(x[t]), cap) * inv_t : -INFINITY;
    lp[row] = zt - l;
    lse[row] = l;
  }
}

template <typename T>
__global__ void logprob_rows_bwd_kernel(T* __restrict__ logits, long long ld, const long long* __restrict__ targets,
                                        const float* __restrict__ lse, const float* __restrict__ dlp, int V,
                                        float inv_t, float cap) {
  const long long row = blockIdx.x;
  T* x = logits + row * ld;
  const float l = lse[row], g = dlp[row];
  const long long t = targets[row];
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    float raw = to_f(x[i]);
    float y = capf(raw, cap);
    float p = __expf(y * inv_t - l);
    float d = g * ((i == t ? 1.f : 0.f) - p) * inv_t;
    if (cap > 0.f) {
      float th = y / cap;
      d *= (1.f - th * th);
    }
    x[i] = from_f<T>(d);
  }
}

// bf16 vector forms: 8 logits per 16-byte access, so a thread keeps eight times the bytes in flight
// (the scalar kernels above run at a fifth of the copy bandwidth because they are latency-bound).
__global__ void logprob_rows_vec_kernel(const __nv_bfloat16* __restrict__ logits, long long ld,
                                        const long long* __restrict__ targets, float* __restrict__ lp,
                                        float* __restrict__ lse, int V, float inv_t, float cap) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const __nv_bfloat16* x = logits + row * ld;
  float m = -INFINITY, s = 0.f;
  for (int i = threadIdx.x * 8; i < V; i += blockDim.x * 8) {
    const uint4 raw = *reinterpret_cast<const uint4*>(x + i);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
    float z[8];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __bfloat1622float2(h[e]);
      z[2 * e] = capf(f.x, cap) * inv_t;
      z[2 * e + 1] = capf(f.y, cap) * inv_t;
    }
    float zm = z[0];
#pragma unroll
    for (int e = 1; e < 8; ++e) zm = fmaxf(zm, z[e]);
    if (zm > m) {
      s *= __expf(m - zm);
      m = zm;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) s += __expf(z[e] - m);
  }
  const float gm = block_max(m, red);
  const float part = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
  const float tot = block_sum(part, red);
  if (threadIdx.x == 0) {
    const float l = gm + logf(tot);
    const long long t = targets[row];
    const float zt = (t >= 0 && t < V) ? capf(__bfloat162float(x[t]), cap) * inv_t : -INFINITY;
    lp[row] = zt - l;
    lse[row] = l;
  }
}

__global__ void logprob_rows_bwd_vec_kernel(__nv_bfloat16* __restrict__ logits, long long ld,
                                            const long long* __restrict__ targets, const float* __restrict__ lse,
                                            const float* __restrict__ dlp, int V, float inv_t, float cap) {
  const long long row = blockIdx.x;
  __nv_bfloat16* x = logits + row * ld;
  const float l = lse[row], g = dlp[row];
  const long long t = targets[row];
  for (int i = threadIdx.x * 8; i < V; i += blockDim.x * 8) {
    uint4 raw = *reinterpret_cast<const uint4*>(x + i);
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __bfloat1622float2(h[e]);
      float d[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float rawv = k == 0 ? f.x : f.y;
        const float y = capf(rawv, cap);
        const float p = __expf(y * inv_t - l);
        float dd = g * (((i + 2 * e + k) == t ? 1.f : 0.f) - p) * inv_t;
        if (cap > 0.f) {
          const float th = y / cap;
          dd *= (1.f - th * th);
        }
        d[k] = dd;
      }
      h[e] = __floats2bfloat162_rn(d[0], d[1]);
    }
    *reinterpret_cast<uint4*>(x + i) = raw;
  }
}

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

constexpr int ST = 512;        // threads of a CTA
constexpr int SW = ST / 32;    // warps of a CTA
constexpr int SRES = 3;        // CTAs on an SM
constexpr int SCL = 8;         // CTAs of a cluster at most
constexpr int SEG = 8;         // segments of the general cut
constexpr int BINS = 256;      // bins of a refinement
constexpr int AHEAD = 4;       // groups of a lane in flight in the last walk
constexpr int KN = 18 * 128;   // 16-bit magnitudes that have counters: 18 octaves
constexpr int NC = 2 * KN + 2; // counters: negative values, -0, +0, positive values, in the order of their keys
constexpr int TINY = 1024;     // values without a counter that a CTA lists

// A cluster of CTAs draws a row's token, one contiguous slice of the vocabulary each.
//
// 16-bit logits that are cut have few distinct values, so one pass over HBM counts them (one shared atomic per element, and
// neighbouring bins are spread over the banks); masses, the total, the nucleus cut and each CTA's share of the kept
// mass then come from the counts alone, and only the CTA that the draw falls into walks its slice again.  The 18 octaves that
// have counters end an octave above the largest of 4096 sampled magnitudes, which every CTA finds for itself; the sample's
// maximum also tells which values are too small to have a mass (masks, finite ones too), and those are skipped.  What else
// lies outside the octaves is listed, and the cut may lie among it.  A row that overflows a list (many values of another
// order of magnitude) takes the general path, as 32-bit rows and rows without a cut do:
//
//   1. maximum of the row
//   2. masses of SEG segments of the row by distance from the maximum, in columns of shared memory that belong to
//      one thread (plain adds, no atomics); their sum is the total mass, one of them holds the cut
//   3. key range of that segment, then BINS bins of it at a time until a bin is one key: the few elements inside
//      go to histograms of four 32-bit pieces of the mass (10 and 11 bits, so that 2^21 elements of a CTA cannot
//      overflow one; a 64-bit shared atomic is a compare-and-swap loop)
//
// Every sum is an integer sum, so neither the cluster size, the path nor the order of the adds shows in the result.
// 128 rows of 151936 bf16 logits, top-p 0.95: 178 -> 76 us (one CTA of 1024 threads per row, three shared atomics per
// element and digit before; shared atomics still bound it, 17 cycles a warp, the bytes would take 6 us; half the row masked 120 ->
// 74, half zeros 248 -> 76; a row of two scales by the general path 201 -> 193).  Without a cut 53 -> 38.  float32: 339 -> 165,
// half masked 327 -> 150.  One row of 151936: 167 -> 30 us.
template <typename T, bool VEC, bool CUT>
__global__ void __launch_bounds__(ST, SRES)
sample_rows_kernel(const T* __restrict__ logits, long long ld, const long long* __restrict__ global_rows,
                   uint64_t seed, const int* __restrict__ draw_dev, int draw_host, long long* __restrict__ tok_out,
                   float* __restrict__ lp_out, int V, float inv_t, float top_p) {
  using u64 = unsigned long long;
  constexpr bool K16 = sizeof(T) == 2;
  constexpr int EPT = 16 / sizeof(T);       // elements of a group: one 16-byte access
  extern __shared__ __align__(16) u64 priv[];   // [SEG][ST]; counters and the list of small values before that
  __shared__ unsigned int planes[4][BINS];
  __shared__ u64 bins[2][BINS];             // this CTA's masses of a refinement; two, read by the others in turn
  __shared__ u64 segs[SEG];
  __shared__ u64 kept_sh, wmass[SW], wlist[SW][4], sel_u64[2];
  __shared__ float row_max, red[32];
  __shared__ unsigned int range_sh[2], sel_u32, n_tiny;
  unsigned int* counts = reinterpret_cast<unsigned int*>(priv);             // [NC], ascending keys
  unsigned int* tiny = counts + NC;                                     // [TINY]
  unsigned int* merged = tiny + TINY;                                       // [NC], the counts of the whole row
  cg::cluster_group cluster = cg::this_cluster();
  const int CL = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const long long row = blockIdx.x / CL;
  const T* x = logits + row * ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float FIX = 1099511627776.f;  // 2^40

  const int Gt = (V + EPT - 1) / EPT, gpc = (Gt + CL - 1) / CL;
  const int g0 = min(Gt, rank * gpc), G = min(gpc, Gt - g0);               // this CTA's groups
  auto load = [&](int g) -> uint4 {                                        // group g of the slice, -inf past the row's end
    if (VEC) return *(reinterpret_cast<const uint4*>(x) + g0 + g);
    uint4 raw;
    T* e = reinterpret_cast<T*>(&raw);
    const int i0 = (g0 + g) * EPT;
#pragma unroll
    for (int k = 0; k < EPT; ++k) e[k] = i0 + k < V ? x[i0 + k] : from_f<T>(-INFINITY);
    return raw;
  };
  auto group = [&](int g, float* v) {
    const uint4 raw = load(g);
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int k = 0; k < EPT; ++k) v[k] = to_f(e[k]);
  };
  // Combines one value of every CTA; the loads of other CTAs' shared memory are all in flight at once.
  auto gather = [&](auto* at, auto combine) {
    auto v = *at;
    decltype(v) o[SCL];
#pragma unroll
    for (int r = 0; r < SCL; ++r) o[r] = r < CL && r != rank ? *cluster.map_shared_rank(at, r) : v;
#pragma unroll
    for (int r = 0; r < SCL; ++r)
      if (r < CL && r != rank) v = combine(v, o[r]);
    return v;
  };
  auto plus = [](u64 a, u64 b) { return a + b; };

  unsigned int *counts_top = counts + KN - 1, *counts_mid = counts + KN + 2;     // of the least magnitudes that have counters
  constexpr bool counted = K16 && CUT;      // without a cut the sum of the masses is all that is wanted

  // 1. the row's maximum, and for 16-bit logits that are cut the counts of their values
  unsigned int klo = 0;                     // the least magnitude with a counter
  float least = -INFINITY;                  // the least value that may have a mass
  if (counted) {
    float v[EPT], top = -INFINITY, mag = 0.f;
    const uint4 sample = load(static_cast<int>(static_cast<long long>(tid) * Gt / ST) - g0);
#pragma unroll
    for (int u = 0; u < 4; ++u)             // on their way meanwhile
      if (VEC && tid + u * ST < G) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint4*>(x) + g0 + tid + u * ST));
    for (int i = tid; i < NC; i += ST) counts[i] = 0;
    if (tid == 0) n_tiny = 0;
#pragma unroll
    for (int k = 0; k < EPT; ++k) {
      v[k] = to_f(reinterpret_cast<const T*>(&sample)[k]);
      top = fmaxf(top, v[k]);
    }
    auto block = [&](float x, float* at) {
      x = warp_max(x);
      if (lane == 0) at[warp] = x;
      __syncthreads();
      return warp_max(at[lane % SW]);
    };
    least = block(top, red) - 28.f / inv_t;                 // e^-28 < 2^-40
#pragma unroll
    for (int k = 0; k < EPT; ++k)
      if (v[k] >= least && fabsf(v[k]) < INFINITY) mag = fmaxf(mag, fabsf(v[k]));
    const int octave = static_cast<int>(__float_as_uint(block(mag, red + SW)) >> 23);
    klo = static_cast<unsigned int>(min(max(1, (octave - 16) * 128), 0x7F80 - KN));
  }
  float m = -INFINITY;
  unsigned int zeros = 0;                   // +0 in the lower half, -0 in the upper
  __nv_bfloat162 m2 = __float2bfloat162_rn(-INFINITY);
  for (int gb = tid; gb < G; gb += 4 * ST) {
    uint4 raw[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (gb + u * ST < G) raw[u] = load(gb + u * ST);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (gb + u * ST < G) {
        if (!counted) {
          const T* e = reinterpret_cast<const T*>(&raw[u]);
#pragma unroll
          for (int k = 0; k < EPT; ++k) m = fmaxf(m, to_f(e[k]));
          continue;
        }
        // half the pass is instruction issue: two values a word, the rare ones set aside in a loop of their own
        const unsigned int words[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
        bool odd = false;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const unsigned int w = words[k >> 1];
          if (!(k & 1)) m2 = __hmax2(m2, *reinterpret_cast<const __nv_bfloat162*>(&w));
          const unsigned int at = ((k & 1 ? w >> 16 : w) & 0x7FFFu) - klo;
          const bool neg = (k & 1 ? w : w << 16) & 0x80000000u;
          if (at < KN) atomicAdd(neg ? counts_top - at : counts_mid + at, 1u);
          odd |= at >= KN;
        }
        if (odd) {
          for (int k = 0; k < 8; ++k) {
            const unsigned int bits = (k & 1 ? words[k >> 1] >> 16 : words[k >> 1]) & 0xFFFFu, mag = bits & 0x7FFFu;
            if (mag == 0) {
              zeros += bits ? 0x10000u : 1u;
            } else if (mag - klo >= KN && mag < 0x7F80u && __uint_as_float(bits << 16) >= least) {
              const unsigned int i = atomicAdd(&n_tiny, 1u);
              if (i < TINY) tiny[i] = bits;
            }
          }
        }
      }
  }
  if (counted) {
    m = fmaxf(__low2float(m2), __high2float(m2));
    if (zeros & 0xFFFFu) atomicAdd(&counts[KN + 1], zeros & 0xFFFFu);
    if (zeros >> 16) atomicAdd(&counts[KN], zeros >> 16);
  }
  m = block_max(m, red);
  if (tid == 0) row_max = m;
  cluster.sync();
  m = gather(&row_max, [](float a, float b) { return fmaxf(a, b); });

  auto e_val = [&](float xv) -> float { return __expf((xv - m) * inv_t); };   // exp(-inf) = 0 for padding
  auto fix_of = [&](float e) -> u64 { return static_cast<u64>(fmaxf(e, 0.f) * FIX); };    // NaN has no mass
  constexpr float kLeast = 9.094947017729282e-13f;      // 2^-40, the least with a mass: masked entries cost no more than their load
  // The order of the cut: for 16-bit logits the sortable pattern of the logit itself (it orders as the probability
  // does), for 32-bit ones the pattern of the unnormalised probability.
  auto key_of = [&](float xv, float e) -> unsigned int {
    if (K16) {
      const unsigned int u = __float_as_uint(xv) >> 16;
      return (u & 0x8000u) ? (~u & 0xFFFFu) : (u | 0x8000u);
    }
    return __float_as_uint(e);
  };
  // Segments fall with the key: a unit of the exponent each for 16 bits, an octave of the probability for 32.
  auto seg_of = [&](float xv, float e) -> unsigned int {
    const unsigned int s = K16 ? __float2uint_rz((m - xv) * inv_t) : (0x3FFFFFFFu - __float_as_uint(e)) >> 23;
    return min(s, static_cast<unsigned int>(SEG - 1));
  };
  auto warp_total = [&](u64 v) -> u64 {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  const int gpw = ((G + SW - 1) / SW + 31) / 32 * 32;                      // groups of a warp, in vocabulary order
  const int w0 = min(G, warp * gpw), w1 = min(G, w0 + gpw);

  unsigned int thresh_key = 0;              // keep everything
  u64 Z = 0, kept_mass = 0;
  u64 mine = 0;                             // kept mass of this CTA
  bool general = !counted;
  // a cut to narrow down: keys lo .. hi, the masses above them and those to keep, of the listed values or of the row
  bool narrow = false, listed = false;
  unsigned int lo = 0, hi = 0;
  u64 target = 0, above = 0;
  auto value = [&](int s) {                 // of counter s
    const unsigned int b = s >= KN + 2 ? s - (KN + 2) + klo : s >= KN ? (KN + 1 - s) << 15 : (0x8000u | (KN - 1 - s + klo));
    return __uint_as_float(b << 16);
  };
  if (counted) {
    general = gather(&n_tiny, [](unsigned int a, unsigned int b) { return max(a, b); }) > TINY;
    if (!general) {
      // This CTA merges one part of the counters, in descending order of the values: other CTAs' shared memory is read
      // a warp's width at a time, and each counter by one CTA only (64 rows of
      // 50264: 35 us; 43 with all counters merged by every CTA, 117 with a thread's strided counters read one by one).
      const int part = (NC + CL - 1) / CL, per = (part + ST - 1) / ST;
      const int p0 = min(NC, rank * part), pn = min(NC - p0, part);
      for (int i = tid; i < pn; i += ST)
        merged[i] = gather(&counts[NC - 1 - p0 - i], [](unsigned int a, unsigned int b) { return a + b; });
      // The listed values are of four classes, each between counters: large positive ones before them all, small positive
      // ones before the zeros, small negative ones behind those, large negative ones behind all.
      u64 sum = 0;
      {
        u64 f[4] = {};
        for (unsigned int i = tid; i < n_tiny; i += ST) {
          const unsigned int bits = tiny[i], far = (bits & 0x7FFFu) >= klo, c = bits & 0x8000u ? 2 + far : 1 - far;
          const u64 t = fix_of(e_val(__uint_as_float(bits << 16)));
#pragma unroll
          for (int j = 0; j < 4; ++j) f[j] += c == j ? t : 0;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const u64 t = warp_total(f[j]);
          if (lane == 0) wlist[warp][j] = t;
        }
      }
      __syncthreads();
      const int i0 = min(pn, tid * per), i1 = min(pn, i0 + per);
      auto mass_at = [&](int i) -> u64 {
        return merged[i] ? merged[i] * fix_of(e_val(value(NC - 1 - p0 - i))) : 0;
      };
      for (int i = i0; i < i1; ++i) sum += mass_at(i);
      u64 incl = sum;
      for (int o = 1; o < 32; o <<= 1) {
        const u64 p = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += p;
      }
      if (lane == 31) wmass[warp] = incl;
      __syncthreads();
      u64 whole = 0;
#pragma unroll
      for (int w = 0; w < SW; ++w) {
        if (w < warp) incl += wmass[w];
        whole += wmass[w];
      }
      if (tid < 4) {
        u64 t = 0;
#pragma unroll
        for (int w = 0; w < SW; ++w) t += wlist[w][tid];
        segs[1 + tid] = t;
      }
      if (tid == 0) {
        segs[0] = whole;
        sel_u32 = 0;
        sel_u64[0] = 0;
      }
      cluster.sync();
      const u64 parts = lane < CL ? *cluster.map_shared_rank(&segs[0], lane) : 0;
      u64 of_class = lane < 4 * CL ? *cluster.map_shared_rank(&segs[1 + (lane & 3)], lane >> 2) : 0;
      for (int o = 4; o < 32; o <<= 1) of_class += __shfl_xor_sync(0xffffffffu, of_class, o);
      u64 l[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) l[j] = __shfl_sync(0xffffffffu, of_class, j);
      Z = warp_total(parts) + l[0] + l[1] + l[2] + l[3];
      target = max(static_cast<u64>(static_cast<double>(Z) * static_cast<double>(top_p)), u64(1));
      u64 cum = warp_total(lane < rank ? parts : 0) + incl - sum + l[0];
      if (cum + sum + l[1] + l[2] >= target)
        for (int i = i0; i < i1; ++i) {
          const int d = p0 + i;
          const u64 c = cum + (d >= KN ? l[1] : 0) + (d >= KN + 2 ? l[2] : 0), f = mass_at(i);
          const u64 before = d == KN ? l[1] : d == KN + 2 ? l[2] : 0;            // the listed class between counter d and the last
          if (c < target ? c + f >= target : c - before < target && before) {    // in one thread of the cluster at most
            sel_u64[0] = c < target ? c + f : c - before;
            sel_u32 = c < target ? key_of(value(NC - 1 - d), 0.f) : d == KN ? 1 : 2;    // no key of a finite value is 1 or 2
          }
          cum += f;
        }
      cluster.sync();
      thresh_key = gather(&sel_u32, [](unsigned int a, unsigned int b) { return max(a, b); });
      kept_mass = gather(&sel_u64[0], [](u64 a, u64 b) { return max(a, b); });
      if (Z > 0 && (target <= l[0] || target > Z - l[3] || thresh_key < 3)) {
        const unsigned int end = klo + KN;
        narrow = listed = true;
        above = target <= l[0] ? 0 : target > Z - l[3] ? Z - l[3] : kept_mass;
        lo = target <= l[0] ? 0x8000u | end : target > Z - l[3] ? 0x0080u : thresh_key == 1 ? 0x8001u : 0x8000u - klo;
        hi = target <= l[0] ? 0xFF7Fu : target > Z - l[3] ? 0x7FFFu - end : thresh_key == 1 ? 0x7FFFu + klo : 0x7FFEu;
      }
    } else {
      cluster.sync();                       // the counters give way to the columns below
    }
  }
  if (general) {
    // 2. masses by segment, of a row that is not cut by warp
    if (CUT) {
#pragma unroll
      for (int s = 0; s < SEG; ++s) priv[s * ST + tid] = 0;
      for (int g = w0 + lane; g < w1; g += 32) {
        float v[EPT];
        group(g, v);
#pragma unroll
        for (int k = 0; k < EPT; ++k) {
          const float e = e_val(v[k]);
          priv[seg_of(v[k], e) * ST + tid] += fix_of(e);
        }
      }
      __syncthreads();
      for (int s = warp; s < SEG; s += SW) {
        u64 t = 0;
#pragma unroll
        for (int i = 0; i < ST / 32; ++i) t += priv[s * ST + i * 32 + lane];
        t = warp_total(t);
        if (lane == 0) segs[s] = t;
      }
    } else {
      u64 t = 0;
#pragma unroll 4
      for (int g = w0 + lane; g < w1; g += 32) {
        float v[EPT];
        group(g, v);
#pragma unroll
        for (int k = 0; k < EPT; ++k) t += fix_of(e_val(v[k]));
      }
      t = warp_total(t);
      if (lane == 0) wmass[warp] = t;
      __syncthreads();
      if (tid < SEG) {
        t = 0;
        for (int w = 0; w < SW; ++w) t += tid == 0 ? wmass[w] : 0;
        segs[tid] = t;
      }
    }
    if (tid < 2) range_sh[tid] = tid == 0 ? 0xFFFFFFFFu : 0u;
    cluster.sync();
    int cut = SEG;
    {
      const u64 t = lane < SEG ? gather(&segs[lane], plus) : 0;
      Z = warp_total(t);                      // every warp computes the same
      u64 incl = t;
      for (int o = 1; o < 32; o <<= 1) {
        const u64 p = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += p;
      }
      if (CUT) {
        target = static_cast<u64>(static_cast<double>(Z) * static_cast<double>(top_p));
        const unsigned int hit = __ballot_sync(0xffffffffu, t > 0 && incl >= target);
        cut = hit ? __ffs(hit) - 1 : SEG;
        if (cut < SEG) above = __shfl_sync(0xffffffffu, incl - t, cut);
      }
      for (int s = 0; s < cut; ++s) mine += segs[s];
    }

    // 3. the cut inside its segment
    kept_mass = Z;
    if (cut < SEG) {
      lo = 0xFFFFFFFFu;
      hi = 0;
      for (int g = w0 + lane; g < w1; g += 32) {
        float v[EPT];
        group(g, v);
#pragma unroll
        for (int k = 0; k < EPT; ++k) {
          const float e = e_val(v[k]);
          if (e >= kLeast && seg_of(v[k], e) == static_cast<unsigned int>(cut)) {
            const unsigned int key = key_of(v[k], e);
            lo = min(lo, key);
            hi = max(hi, key);
          }
        }
      }
      lo = __reduce_min_sync(0xffffffffu, lo);
      hi = __reduce_max_sync(0xffffffffu, hi);
      if (lane == 0) {
        atomicMin(&range_sh[0], lo);
        atomicMax(&range_sh[1], hi);
      }
      cluster.sync();
      lo = gather(&range_sh[0], [](unsigned int a, unsigned int b) { return min(a, b); });
      hi = gather(&range_sh[1], [](unsigned int a, unsigned int b) { return max(a, b); });
      thresh_key = lo;
      narrow = lo < hi;
      if (!narrow) {                          // a segment of one key, as in a flat row
        kept_mass = above + gather(&segs[cut], plus);
        mine += segs[cut];
      }
    }
  }
  if (narrow) {
    for (int it = 0;; ++it) {
      const int shift = max(0, 24 - __clz(hi - lo));                         // BINS bins cover hi - lo
      for (int i = tid; i < 4 * BINS; i += ST) planes[0][i] = 0;
      __syncthreads();
      auto add = [&](float xv) {
        float e = K16 ? 0.f : e_val(xv);
        const unsigned int at = key_of(xv, e) - lo;
        if (at > hi - lo) return;
        if (K16) e = e_val(xv);
        const u64 f = fix_of(e);
        if (f == 0) return;
        const unsigned int b = at >> shift;
        atomicAdd(&planes[0][b], static_cast<unsigned int>(f & 0x7FFu));
        atomicAdd(&planes[1][b], static_cast<unsigned int>((f >> 11) & 0x3FFu));
        atomicAdd(&planes[2][b], static_cast<unsigned int>((f >> 21) & 0x3FFu));
        atomicAdd(&planes[3][b], static_cast<unsigned int>(f >> 31));
      };
      if (listed) {
        for (unsigned int i = tid; i < n_tiny; i += ST) add(__uint_as_float(tiny[i] << 16));
      } else {
        for (int g = w0 + lane; g < w1; g += 32) {
          float v[EPT];
          group(g, v);
#pragma unroll
          for (int k = 0; k < EPT; ++k) add(v[k]);
        }
      }
      __syncthreads();
      u64* own = bins[it & 1];
      if (tid < BINS)
        own[tid] = static_cast<u64>(planes[0][tid]) + (static_cast<u64>(planes[1][tid]) << 11) +
                   (static_cast<u64>(planes[2][tid]) << 21) + (static_cast<u64>(planes[3][tid]) << 31);
      cluster.sync();
      u64* total = reinterpret_cast<u64*>(merged);      // done with, as are the columns of the mass pass
      if (tid < BINS) total[tid] = gather(&own[tid], plus);
      __syncthreads();
      if (warp == 0) {                      // from the highest key down, eight bins to a lane
        constexpr int PER = BINS / 32;
        u64 t[PER], s = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) s += t[i] = total[BINS - 1 - lane * PER - i];
        u64 incl = s;
        for (int o = 1; o < 32; o <<= 1) {
          const u64 p = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += p;
        }
        u64 cum = above + incl - s;
        int b = -1;
#pragma unroll
        for (int i = 0; i < PER; ++i)
          if (b < 0) {
            if (t[i] > 0 && cum + t[i] >= target) b = BINS - 1 - lane * PER - i;
            else cum += t[i];
          }
        const unsigned int hit = __ballot_sync(0xffffffffu, b >= 0);
        const int src = hit ? __ffs(hit) - 1 : 31;
        b = max(0, __shfl_sync(0xffffffffu, b, src));
        u64 kept = 0;                       // of this CTA, above bin b
        for (int i = b + 1 + lane; i < BINS; i += 32) kept += own[i];
        kept = warp_total(kept);
        if (lane == src) {
          sel_u64[0] = cum;
          sel_u32 = static_cast<unsigned int>(b);
        }
        if (lane == 0) sel_u64[1] = kept;
      }
      __syncthreads();
      above = sel_u64[0];
      mine += sel_u64[1];
      const unsigned int b = sel_u32;
      lo += b << shift;
      if (shift == 0) {
        kept_mass = above + total[b];
        mine += own[b];
        break;
      }
      hi = min(hi, lo + (1u << shift) - 1);
      __syncthreads();
    }
    thresh_key = lo;
  }
  if (counted && !general) {                // from the counters and the list instead
    mine = 0;
#pragma unroll
    for (int i = 0; i < (NC + ST - 1) / ST; ++i) {
      const int s = tid + i * ST;
      const unsigned int n = s < NC ? counts[s] : 0;
      const float xv = value(s);
      if (n && key_of(xv, 0.f) >= thresh_key) mine += n * fix_of(e_val(xv));
    }
    for (unsigned int i = tid; i < n_tiny; i += ST) {
      const float xv = __uint_as_float(tiny[i] << 16);
      if (key_of(xv, 0.f) >= thresh_key) mine += fix_of(e_val(xv));
    }
    mine = warp_total(mine);
    __syncthreads();
    if (lane == 0) wmass[warp] = mine;
    __syncthreads();
    mine = 0;
#pragma unroll
    for (int w = 0; w < SW; ++w) mine += wmass[w];
  }

  // 4. the draw
  if (tid == 0) kept_sh = mine;
  cluster.sync();
  const int draw = draw_dev ? *draw_dev : draw_host;
  const uint64_t key = mix64(seed + static_cast<uint64_t>(global_rows[row]) * 0x9E3779B97F4A7C15ull);
  const uint64_t bits = mix64(key + static_cast<uint64_t>(draw + 1) * 0x9E3779B97F4A7C15ull);
  const u64 u24 = bits >> 40;
  const u64 point = (kept_mass >> 24) * u24 + (((kept_mass & 0xFFFFFFull) * u24) >> 24);
  u64 before = 0, all = 0;
  {
    const u64 t = lane < CL ? *cluster.map_shared_rank(&kept_sh, lane) : 0;
    before = warp_total(lane < rank ? t : 0);
    all = warp_total(t);
  }
  cluster.sync();                           // nobody reads this CTA's shared memory from here on
  auto emit = [&](int pick) {
    tok_out[row] = pick;
    const float le = (to_f(x[pick]) - m) * inv_t;
    const float lmass = logf(static_cast<float>(static_cast<double>(kept_mass) / 1099511627776.0));
    lp_out[row] = fminf(le - lmass, 0.f);
  };
  if (point >= all) {
    // degenerate row (all mass rounded to zero): fall back to the arg-max element
    if (rank == 0 && tid == 0) {
      int pick = 0;
      float best = -INFINITY;
      for (int i = 0; i < V; ++i) {
        const float v = to_f(x[i]);
        if (v > best) { best = v; pick = i; }
      }
      emit(pick);
    }
    return;
  }
  if (point < before || point >= before + mine) return;
  auto group_mass = [&](int g, float* v) -> u64 {
    u64 t = 0;
    group(g, v);
#pragma unroll
    for (int k = 0; k < EPT; ++k) {
      const float e = e_val(v[k]);
      if (key_of(v[k], e) >= thresh_key) t += fix_of(e);
    }
    return t;
  };
  float v[EPT];
  if (CUT) {                            // those of a row that is not cut are known
    u64 t = 0;
#pragma unroll 4
    for (int g = w0 + lane; g < w1; g += 32) t += group_mass(g, v);
    t = warp_total(t);
    if (lane == 0) wmass[warp] = t;
    __syncthreads();
  }
  for (int w = 0; w < warp; ++w) before += wmass[w];
  if (point < before || point >= before + wmass[warp]) return;
  for (int gb = w0; gb < w1; gb += 32 * AHEAD) {       // one warp is left; a step is 32 neighbouring groups, AHEAD of them loaded at a time
    u64 t[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) t[u] = gb + 32 * u + lane < w1 ? group_mass(gb + 32 * u + lane, v) : 0;
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      u64 incl = t[u];
      for (int o = 1; o < 32; o <<= 1) {
        const u64 p = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += p;
      }
      const unsigned int hit = __ballot_sync(0xffffffffu, before + incl > point);
      if (hit) {
        if (lane == __ffs(hit) - 1) {
          u64 cum = before + incl - t[u];
          int pick = -1;
          group(gb + 32 * u + lane, v);
#pragma unroll
          for (int k = 0; k < EPT; ++k) {
            const float e = e_val(v[k]);
            if (pick < 0 && key_of(v[k], e) >= thresh_key) {
              cum += fix_of(e);
              if (cum > point) pick = (g0 + gb + 32 * u + lane) * EPT + k;
            }
          }
          emit(pick);
        }
        return;
      }
      before += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
}

}  // namespace

// Combine the per-tile (max, sum exp) pairs of the head GEMM's log-prob epilogue: lse = log sum exp over the
// vocabulary, lp = target logit - lse.  One thread per row; the tile-major layout keeps the reads coalesced.
__global__ void logprob_finalize_kernel(const float2* __restrict__ ws, const float* __restrict__ tl, int n_tiles, int M,
                                        float* __restrict__ lp, float* __restrict__ lse) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= M) return;
  float m = -INFINITY;
  for (int t = 0; t < n_tiles; ++t) m = fmaxf(m, ws[static_cast<long long>(t) * M + row].x);
  float s = 0.f;
  for (int t = 0; t < n_tiles; ++t) {
    const float2 v = ws[static_cast<long long>(t) * M + row];
    s += v.y * __expf(v.x - m);
  }
  const float l = m + __logf(s);
  lse[row] = l;
  lp[row] = tl[row] - l;
}

// Vocabulary-sharded form: the same combine, but the result stays a partial (max, sum exp, target logit) per row,
// to be merged with the other shards' partials (tensor-parallel head).  stats [M, 3].
__global__ void logprob_shard_stats_kernel(const float2* __restrict__ ws, const float* __restrict__ tl, int n_tiles, int M,
                                           float* __restrict__ stats) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= M) return;
  float m = -INFINITY;
  for (int t = 0; t < n_tiles; ++t) m = fmaxf(m, ws[static_cast<long long>(t) * M + row].x);
  float s = 0.f;
  for (int t = 0; t < n_tiles; ++t) {
    const float2 v = ws[static_cast<long long>(t) * M + row];
    s += v.y * __expf(v.x - m);
  }
  stats[3 * row] = m;
  stats[3 * row + 1] = s;
  stats[3 * row + 2] = tl[row];
}

const char* logprob_shard_stats(const float* ws, const float* tl, int n_tiles, int M, float* stats, cudaStream_t s) {
  if (M == 0) return nullptr;
  logprob_shard_stats_kernel<<<(M + 127) / 128, 128, 0, s>>>(reinterpret_cast<const float2*>(ws), tl, n_tiles, M, stats);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "logprob_shard_stats launch failed";
}

const char* logprob_finalize(const float* ws, const float* tl, int n_tiles, int M, float* lp, float* lse, cudaStream_t s) {
  if (M == 0) return nullptr;
  logprob_finalize_kernel<<<(M + 127) / 128, 128, 0, s>>>(reinterpret_cast<const float2*>(ws), tl, n_tiles, M, lp, lse);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "logprob_finalize launch failed";
}

const char* logprob_rows(int dtype, const void* logits, long long ld, const long long* targets, float* lp, float* lse,
                         long long rows, int V, float temperature, float softcap, cudaStream_t s) {
  if (rows == 0) return nullptr;
  float inv_t = 1.f / temperature;
  if (dtype == kF32)
    logprob_rows_kernel<float><<<static_cast<unsigned>(rows), 1024, 0, s>>>(static_cast<const float*>(logits), ld,
                                                                           targets, lp, lse, V, inv_t, softcap);
  else if ((V % 8) == 0 && (ld % 8) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0)
    logprob_rows_vec_kernel<<<static_cast<unsigned>(rows), 512, 0, s>>>(static_cast<const __nv_bfloat16*>(logits), ld,
                                                                       targets, lp, lse, V, inv_t, softcap);
  else
    logprob_rows_kernel<__nv_bfloat16><<<static_cast<unsigned>(rows), 1024, 0, s>>>(
        static_cast<const __nv_bfloat16*>(logits), ld, targets, lp, lse, V, inv_t, softcap);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "logprob_rows launch failed";
}

const char* logprob_rows_bwd(int dtype, void* logits, long long ld, const long long* targets, const float* lse,
                             const float* dlp, long long rows, int V, float temperature, float softcap,
                             cudaStream_t s) {
  if (rows == 0) return nullptr;
  float inv_t = 1.f / temperature;
  if (dtype == kF32)
    logprob_rows_bwd_kernel<float><<<static_cast<unsigned>(rows), 1024, 0, s>>>(static_cast<float*>(logits), ld,
                                                                               targets, lse, dlp, V, inv_t, softcap);
  else if ((V % 8) == 0 && (ld % 8) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0)
    logprob_rows_bwd_vec_kernel<<<static_cast<unsigned>(rows), 512, 0, s>>>(static_cast<__nv_bfloat16*>(logits), ld,
                                                                           targets, lse, dlp, V, inv_t, softcap);
  else
    logprob_rows_bwd_kernel<__nv_bfloat16><<<static_cast<unsigned>(rows), 1024, 0, s>>>(
        static_cast<__nv_bfloat16*>(logits), ld, targets, lse, dlp, V, inv_t, softcap);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "logprob_rows_bwd launch failed";
}

namespace {
template <typename T, bool VEC, bool CUT>
const char* sample_launch(const void* logits, long long ld, const long long* global_rows, unsigned long long seed, const int* draw_dev,
                          int draw_host, long long* tok_out, float* lp_out, int rows, int V, float inv_t, float top_p, cudaStream_t s) {
  constexpr size_t kDyn = std::max(SEG * ST * sizeof(unsigned long long), (2 * NC + TINY) * sizeof(unsigned int));
  if (!FERRL_ONCE_PER_DEVICE(cudaFuncSetAttribute(sample_rows_kernel<T, VEC, CUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  static_cast<int>(kDyn)) == cudaSuccess))
    return "sample_rows: cannot reserve shared memory";
  // Clusters that give each SM two or three CTAs (one alone waits on its own barriers: 128 rows of 151936 bf16 logits take
  // 107 us with one CTA, 76, 74, 80 and 90 with 2, 3, 4 and 8), down to slices of 16384 elements (256 rows of 32768: 48 us
  // with one CTA, 53 with two; 32 rows of 50264: 47 with one, 29 with three, 27 with six).
  // And enough of them that a CTA's slice stays within the 2^21 elements that its 32-bit histograms hold.
  const int cl = std::max({1, std::min({SCL, (384 + rows - 1) / rows, V / 16384}), V > 1 << 21 ? std::min(SCL, (V >> 20) + 1) : 1});
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(rows) * cl);
  cfg.blockDim = dim3(ST);
  cfg.dynamicSmemBytes = kDyn;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cl;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, sample_rows_kernel<T, VEC, CUT>, static_cast<const T*>(logits), ld, global_rows,
                                           static_cast<uint64_t>(seed), draw_dev, draw_host, tok_out, lp_out, V, inv_t, top_p);
  count_launch();
  return e == cudaSuccess ? nullptr : "sample_rows launch failed";
}
}  // namespace

const char* sample_rows(int dtype, const void* logits, long long ld, const long long* global_rows,
                        unsigned long long seed, const int* draw_dev, int draw_host, long long* tok_out, float* lp_out,
                        int rows, int V, float temperature, float top_p, cudaStream_t s) {
  if (rows == 0) return nullptr;
  const float inv_t = 1.f / temperature;
  const int per = dtype == kF32 ? 4 : 8;
  const bool vec = V % per == 0 && ld % per == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0;
  const bool cut = top_p > 0.f && top_p < 1.f;          // rows without a cut want no more than their sum
#define FERRL_SAMPLE(T, VEC, CUT) \
  sample_launch<T, VEC, CUT>(logits, ld, global_rows, seed, draw_dev, draw_host, tok_out, lp_out, rows, V, inv_t, top_p, s)
  if (dtype == kF32) {
    if (vec) return cut ? FERRL_SAMPLE(float, true, true) : FERRL_SAMPLE(float, true, false);
    return cut ? FERRL_SAMPLE(float, false, true) : FERRL_SAMPLE(float, false, false);
  }
  if (vec) return cut ? FERRL_SAMPLE(__nv_bfloat16, true, true) : FERRL_SAMPLE(__nv_bfloat16, true, false);
  return cut ? FERRL_SAMPLE(__nv_bfloat16, false, true) : FERRL_SAMPLE(__nv_bfloat16, false, false);
#undef FERRL_SAMPLE
}

}  // namespace ferrl
