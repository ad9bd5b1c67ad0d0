// Products of at most 16 rows: out[M, N] = X[M, K] W[N, K]^T (+ residual), or act(gate) * up of a weight whose
// rows come in groups of eight gate and eight up rows.  One token of a few sequences streams every weight once and does
// nothing else, so the kernel is a stream of W with as little around it as possible:
//
//   * a CTA owns 16 rows of W, its eight warps 128 of every 1024 columns each; warp-level tensor products (m16n8k16) take W as
//     the operand of 16 rows and X as the one of 8.  The order of k inside a product is free as long as both operands
//     agree, so a lane loads 16 bytes of its two rows at a time, straight into the fragments of two products.
//   * launched as a programmatic dependent W is nothing that an earlier kernel writes: the first loads are under way before the
//     wait for the stream predecessor.
//   * the warps' sums meet in shared memory and are added in warp order.
//
// Nothing hides the few rows' latency in the tiled kernels of tcgen05_gemm.cu: barriers, tensor memory and a cluster's exchange.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../api.h"
#include "../common.cuh"
#include "../kernels/mma_sync.cuh"

namespace ferrl {
namespace {

constexpr int WARPS = 8;
constexpr int KW = 128;        // columns of W that a warp takes at a time

struct FewArgs {
  const __nv_bfloat16 *x, *w, *res;
  __nv_bfloat16* out;
  long long ldx, ldw, ldr, ldo;
  int M, N, K, act;
  float alpha, limit;
};

__device__ __forceinline__ uint4 load_w(const __nv_bfloat16* p) {      // volatile: stays in front of the wait
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float glu(int act, float gate, float up, float alpha, float limit) {
  if (act == kActClipped) {
    const float g = fminf(gate, limit), u = fminf(fmaxf(up, -limit), limit);
    return g / (1.f + __expf(-alpha * g)) * (u + 1.f);
  }
  if (act == kActSilu) return gate / (1.f + __expf(-gate)) * up;
  return 0.5f * gate * (1.f + tanhf(0.7978845608028654f * (gate + 0.044715f * gate * gate * gate))) * up;
}

// H: groups of eight rows of W in a tile (with one, half of a product's rows are zeros); NT: groups of eight rows of X
template <int H, int NT, bool GLU>
__global__ void __launch_bounds__(WARPS * 32, 2) few_rows_kernel(FewArgs a) {
  constexpr int R = 8 * NT, COLS = 8 * H;
  __shared__ float red[2][WARPS][COLS * R];
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int tiles = (a.N + COLS - 1) / COLS, chunks = (a.K + KW - 1) / KW;
  const int per = warp < chunks ? (chunks - warp + WARPS - 1) / WARPS : 0;      // this warp's chunks of a tile
  const uint4 zero = make_uint4(0, 0, 0, 0);
  auto fetch = [&](int tile, int i, uint4 (&w)[4 * H]) {
    const int k0 = (warp + i * WARPS) * KW + t * 8;
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int row = tile * COLS + h * 8 + g;
      const __nv_bfloat16* p = a.w + row * a.ldw + k0;
#pragma unroll
      for (int j = 0; j < 4; ++j) w[h * 4 + j] = row < a.N && k0 + j * 32 < a.K ? load_w(p + j * 32) : zero;
    }
  };
  uint4 w[4 * H], next[4 * H];
  int tile = blockIdx.x;
  if (per > 0 && tile < tiles) fetch(tile, 0, w);
  pdl_wait();
  for (int buf = 0; tile < tiles; tile += gridDim.x, buf ^= 1) {
    float acc[2][NT][4];
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[s][n][e] = 0.f;
    for (int i = 0; i < per; ++i) {
      const int k0 = (warp + i * WARPS) * KW + t * 8;
      uint4 x[NT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int row = n * 8 + g;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          x[n][j] = row < a.M && k0 + j * 32 < a.K ? *reinterpret_cast<const uint4*>(a.x + row * a.ldx + k0 + j * 32) : zero;
      }
      if (i + 1 < per) fetch(tile, i + 1, next);
      else if (tile + static_cast<int>(gridDim.x) < tiles) fetch(tile + gridDim.x, 0, next);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint4 low = H == 2 ? w[4 * (H - 1) + j] : zero;
        const uint32_t lo[4] = {w[j].x, low.x, w[j].y, low.y}, hi[4] = {w[j].z, low.z, w[j].w, low.w};
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          mmah::mma16816(acc[0][n], lo, x[n][j].x, x[n][j].y);
          mmah::mma16816(acc[1][n], hi, x[n][j].z, x[n][j].w);
        }
      }
#pragma unroll
      for (int j = 0; j < 4 * H; ++j) w[j] = next[j];
    }
    float* mine = red[buf][warp];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int h = 0; h < H; ++h)
        *reinterpret_cast<float2*>(mine + (h * 8 + g) * R + n * 8 + 2 * t) =
            make_float2(acc[0][n][2 * h] + acc[1][n][2 * h], acc[0][n][2 * h + 1] + acc[1][n][2 * h + 1]);
    __syncthreads();                            // the other buffer is free too: its readers have come here
    const int id = threadIdx.x, row = id % R, col = id / R;
    auto sum = [&](int c) {
      float s = 0.f;
#pragma unroll
      for (int v = 0; v < WARPS; ++v) s += red[buf][v][c * R + row];
      return s;
    };
    if (GLU) {
      if (col < 8 && row < a.M && tile * COLS + 8 + col < a.N)
        a.out[row * a.ldo + tile * 8 + col] = __float2bfloat16_rn(glu(a.act, sum(col), sum(col + 8), a.alpha, a.limit));
    } else if (col < COLS && row < a.M && tile * COLS + col < a.N) {
      float s = sum(col);
      if (a.res) s += __bfloat162float(a.res[row * a.ldr + tile * COLS + col]);
      a.out[row * a.ldo + tile * COLS + col] = __float2bfloat16_rn(s);
    }
  }
}

}  // namespace

bool gemm_few_rows_supported(const GemmArgs& a) {
  return a.M >= 1 && a.M <= 16 && a.N >= 1 && a.K >= 8 && a.K % 8 == 0 && a.lda % 8 == 0 && a.ldb % 8 == 0 && a.K2 == 0 && !a.out_f32 && !a.b_mn &&
         (!a.glu_act || (a.N % 16 == 0 && !a.residual)) && (reinterpret_cast<uintptr_t>(a.A) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.B) & 15) == 0 &&
         !a.tile_expert && a.ar_world <= 1 && !a.ss_in && !a.ss_out && !a.lp_mode;
}

// Against the tiled kernels in a chain of launches, weights from HBM, as both are launched (us, tiled and this one; 1 to 8 rows; * this
// one early, see below): 256 x 1024* 3.6, 1.5; 1536 x 1024* 4.2, 1.9; 1024 x 3072* 5.3, 4.0; 4096 x 1024 5.7, 3.5; 4096 x 4096 9.8, 8.5;
// 6144 x 4096 13.8, 12.7; 4096 x 12288 20.5, 18.5; 12288 x 4096 23.4, 20.6.  The lines:
//   * long sums of few columns leave multiprocessors idle, which the tiled kernels' k-splits do not (512 x 8192* 7.3, 8.0; 1024 x 8192*
//     8.9, 8.7; 1536 x 8192 9.3, 9.8; 1024 x 16384* 12.7, 15.7; 2560 x 9728 15.2, 13.4);
//   * beyond 52 million entries, 34 where rows are short and many, the stream is all that counts and the tiled kernels' copies have
//     the edge (24576 x 4096 34.2, 37.1; 24576 x 2048 19.0, 19.7; 49152 x 1024 19.3, 20.0; a tie at 32768 x 1024 14.3, 14.1 and 16384 x
//     2048 13.7, 13.9), and from 20 million where the eight warps' shares of k do not come out even (32768 x 1280 16.4, 19.8; 16384 x
//     1280 9.9, 11.5);
//   * 9 to 16 rows read X twice as often: up to 20 million entries (4096 x 4096 9.9, 9.0; 2048 x 8192 11.2, 11.1; 16384 x 2048 13.8, 15.6;
//     1344 x 5376 7.4, 8.2).
bool gemm_few_rows_better(const GemmArgs& a) {
  if (!gemm_few_rows_supported(a)) return false;
  const long long entries = static_cast<long long>(a.N) * a.K, round = WARPS * KW;
  if (a.K > 4096 && a.N < (a.M <= 8 && a.K <= 8192 ? 1024 : 2048)) return false;
  return entries <= 20000000 || (a.M <= 8 && entries <= (a.N <= 20480 ? 52000000 : 34000000) && a.K * 100ll >= (a.K + round - 1) / round * round * 85);
}

const char* gemm_few_rows(const GemmArgs& a, cudaStream_t stream, int rows_of_w) {
  if (!gemm_few_rows_supported(a)) return "few rows: at most 16, bf16, 16-byte rows, no side operand";
  FewArgs f{};
  f.x = static_cast<const __nv_bfloat16*>(a.A); f.w = static_cast<const __nv_bfloat16*>(a.B); f.res = static_cast<const __nv_bfloat16*>(a.residual);
  f.out = static_cast<__nv_bfloat16*>(a.out);
  f.ldx = a.lda; f.ldw = a.ldb; f.ldr = a.ldr; f.ldo = a.ldo;
  f.M = a.M; f.N = a.N; f.K = a.K; f.act = a.glu_act - 1; f.alpha = a.glu_alpha; f.limit = a.glu_limit;
  // Tiles of 8 rows of W while each has a place of its own on the chip and enough columns to share out, but not where only tiles of 16
  // are few enough to be launched early (us, 8 and 16: 1024 x 3072 3.6, 4.0; 1024 x 8192 8.4, 9.2; 2048 x 2048 3.8, 3.2; 2048 x 4096 6.3,
  // 5.9; 2368 x 4096 6.4, 6.8; 2496 x 1664 5.2, 4.0).
  const int early = a.num_sms * 7 / 8;
  const bool narrow = a.N <= 16 * a.num_sms && a.K >= 2048 && a.M <= 8 && !(a.pdl && a.N > 8 * early && a.N <= 16 * early);
  const bool wide = a.glu_act || (rows_of_w ? rows_of_w == 16 : !narrow);
  const int tiles = (a.N + (wide ? 15 : 7)) / (wide ? 16 : 8);
  const dim3 grid(std::min(tiles, 2 * a.num_sms));
  void (*kern)(FewArgs);
  if (a.M <= 8) kern = a.glu_act ? few_rows_kernel<2, 1, true> : wide ? few_rows_kernel<2, 1, false> : few_rows_kernel<1, 1, false>;
  else kern = a.glu_act ? few_rows_kernel<2, 2, true> : wide ? few_rows_kernel<2, 2, false> : few_rows_kernel<1, 2, false>;
  // CTAs that are resident early share the chip with whatever runs there: with more of them than its left-over places the rest
  // waits for a second wave (a decode step of 8 rows, 3712 wide, 522 us, and 410 with such grids launched in stream order).  The line
  // lies where one on every multiprocessor still has a place (12 rows, 2176 wide, 136 CTAs: 213 and 175 us; 1024 wide, up to 128: 236 and
  // 252 without any early launch).
  if (a.pdl && static_cast<int>(grid.x) <= early) launch_pdl(kern, grid, dim3(WARPS * 32), 0, stream, f);
  else kern<<<grid, WARPS * 32, 0, stream>>>(f);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? nullptr : "few rows: launch failed";
}

}  // namespace ferrl
