// Projections of decode steps: out[M, N] = x[M, K] W[N, K]^T for M <= 64 rows, bf16 in, fp32 accumulation.
//
// Such a product reads every weight once and does almost no arithmetic, so it is bound by weight bytes and, for the sizes of
// one layer, by latency. A CTA owns eight weight rows per tile and two tiles (one gate and one up tile in the gated form); its eight
// or sixteen warps take every eighth or sixteenth slice of K and meet in shared memory. Weights and activations go straight from global
// memory into warp-level MMA fragments: a lane loads eight or sixteen consecutive k of a row and both operands read them in the same permuted
// order, which a dot product does not notice. (A 128-row tcgen05 tile would be mostly padding here, and its tensor-memory set-up
// and drain cost more than the whole product.) A warp keeps a ring of slices in registers; a CTA of eight warps 64 KB up to 32 rows and
// 32 KB above (the accumulators of four row tiles take the rest), two of them an SM; a CTA of sixteen 128 KB. It is filled before the
// kernel waits for the previous one (resident weights; others are multiplied by a plainly launched kernel) and refilled across tiles, so
// that the weights never stop flowing.
//
// SILU: W holds gate rows [0, N) and up rows [half, half + N); the output is silu(gate) * up.
// cap > 0 (plain form): the output is cap * tanh(out / cap), the soft limit of logits.
#include "sm100_common.cuh"
#include "inv_api.h"

namespace inv {

__device__ __forceinline__ void sg_mma(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// P 16-byte pieces of a weight row: used once, keep them out of L1
template <int P>
__device__ __forceinline__ void sg_load_stream(const __nv_bfloat16* p, uint4* v) {
  if (P == 1)
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w) : "l"(p));
  else
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w), "=r"(v[P - 1].x), "=r"(v[P - 1].y), "=r"(v[P - 1].z), "=r"(v[P - 1].w)
                 : "l"(p));
}
// Eight values of a row of which only the first `n` exist (n <= 0: none); used for the last slice of K.
__device__ __forceinline__ uint4 sg_mask(uint4 v, int n) {
  uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) u[j] = n >= 2 * j + 2 ? u[j] : n == 2 * j + 1 ? (u[j] & 0xffffu) : 0u;
  return make_uint4(u[0], u[1], u[2], u[3]);
}

// MT: 16-row tiles of x. P: 16-byte pieces per lane and slice (two where rows allow it: whole lines instead of halves). SG_WARPS: 8, two CTAs an
// SM, or 16.
template <int MT, int P, bool SILU, int SG_WARPS>
__global__ void __launch_bounds__(SG_WARPS * 32, SG_WARPS == 8 ? 2 : 1)
    skinny_gemm_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const __nv_bfloat16* __restrict__ W, int ldw, int M, int N, int K, int half,
                       void* __restrict__ out, int ldo, int out_f32, float cap, int n_tiles) {
  constexpr int SG_THREADS = 32 * SG_WARPS;
  constexpr int WT = 2;                      // weight tiles of eight rows: neighbours, or gate and up
  constexpr int COLS = SILU ? 8 : 16;        // output columns of a CTA's tile
  constexpr int SL = 32 * P;                 // k of a slice
  constexpr int UN = (MT >= 4 ? 4 : 8) / P;  // slices in flight
  constexpr int PL = WT * 8 + 4;
  extern __shared__ float sg_part[];         // [SG_WARPS][MT * 16][PL]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tig = lane & 3;
  const int slices = (K + SL - 1) / SL;
  release_next();
  uint4 ring[UN][WT][P];
  // slice s of a tile; columns past N read the last row and are not stored, k past K are zeros
  auto fetch = [&](int tile, int s, uint4 (&r)[WT][P]) {
    const int left = K - s * SL - tig * 8 * P;   // elements of this lane's that exist
#pragma unroll
    for (int t = 0; t < WT; ++t) {
      const int row = SILU ? min(tile * 8 + g, N - 1) + t * half : min(tile * 16 + t * 8 + g, N - 1);
      if (left > 0) {
        sg_load_stream<P>(W + (size_t)row * ldw + s * SL + tig * 8 * P, r[t]);
        if (P == 1 && left < 8) r[t][0] = sg_mask(r[t][0], left);
      } else {
#pragma unroll
        for (int i = 0; i < P; ++i) r[t][i] = make_uint4(0, 0, 0, 0);
      }
    }
  };
  int tile = blockIdx.x;
#pragma unroll
  for (int u = 0; u < UN; ++u)
    if (warp + u * SG_WARPS < slices) fetch(tile, warp + u * SG_WARPS, ring[u]);
  wait_previous();
  const __nv_bfloat16* xp[2 * MT];
#pragma unroll
  for (int m = 0; m < 2 * MT; ++m) xp[m] = x + (size_t)min(m * 8 + g, M - 1) * ldx + tig * 8 * P;
  for (; tile < n_tiles; tile += gridDim.x) {
    float acc[MT][WT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int t = 0; t < WT; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[m][t][i] = 0.f;
    for (int s0 = warp; s0 < slices; s0 += UN * SG_WARPS) {
#pragma unroll
      for (int u = 0; u < UN; ++u) {
        const int s = s0 + u * SG_WARPS;
        if (s >= slices) break;
#pragma unroll
        for (int i = 0; i < P; ++i) {
          uint4 a[2 * MT];
          const int left = K - s * SL - tig * 8 * P - 8 * i;
#pragma unroll
          for (int m = 0; m < 2 * MT; ++m) {
            a[m] = left > 0 ? *reinterpret_cast<const uint4*>(xp[m] + s * SL + 8 * i) : make_uint4(0, 0, 0, 0);
            if (P == 1 && left < 8) a[m] = sg_mask(a[m], left);
          }
#pragma unroll
          for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int t = 0; t < WT; ++t) {
              const uint4 w = ring[u][t][i];
              sg_mma(acc[m][t], a[2 * m].x, a[2 * m + 1].x, a[2 * m].y, a[2 * m + 1].y, w.x, w.y);
              sg_mma(acc[m][t], a[2 * m].z, a[2 * m + 1].z, a[2 * m].w, a[2 * m + 1].w, w.z, w.w);
            }
        }
        const int next = s + UN * SG_WARPS;    // the slot is free: a later slice of this tile or one of the next tile's first
        if (next < slices) fetch(tile, next, ring[u]);
        else if (tile + (int)gridDim.x < n_tiles) fetch(tile + gridDim.x, warp + u * SG_WARPS, ring[u]);
      }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int t = 0; t < WT; ++t) {
        float* p = sg_part + (size_t)(warp * MT * 16 + m * 16 + g) * PL + t * 8 + 2 * tig;
        *reinterpret_cast<float2*>(p) = make_float2(acc[m][t][0], acc[m][t][1]);
        *reinterpret_cast<float2*>(p + 8 * PL) = make_float2(acc[m][t][2], acc[m][t][3]);
      }
    __syncthreads();
    const int n0 = tile * COLS;
    for (int i = tid; i < MT * 16 * COLS; i += SG_THREADS) {
      const int r = i / COLS, c = i % COLS;
      if (r >= M || n0 + c >= N) continue;
      float a = 0.f, b = 0.f;
#pragma unroll
      for (int w = 0; w < SG_WARPS; ++w) {
        a += sg_part[(size_t)(w * MT * 16 + r) * PL + c];
        if (SILU) b += sg_part[(size_t)(w * MT * 16 + r) * PL + 8 + c];
      }
      if (SILU) a = a / (1.0f + expf(-a)) * b;
      else if (cap > 0.f) a = cap * tanhf(a / cap);
      if (out_f32) static_cast<float*>(out)[(size_t)r * ldo + n0 + c] = a;
      else static_cast<__nv_bfloat16*>(out)[(size_t)r * ldo + n0 + c] = __float2bfloat16_rn(a);
    }
    __syncthreads();
  }
}

template <int MT, int P, bool SILU, int SG_WARPS>
static int launch_skinny(const void* x, int ldx, const void* W, int ldw, int M, int N, int K, int half, void* out, int ldo, int out_f32, float cap, int tiles,
                         bool early, cudaStream_t st) {
  constexpr int bytes = SG_WARPS * MT * 16 * (2 * 8 + 4) * 4, ctas = 148 * (SG_WARPS == 8 ? 2 : 1);
  launch_step(early, skinny_gemm_kernel<MT, P, SILU, SG_WARPS>, dim3(tiles < ctas ? tiles : ctas), SG_WARPS * 32, bytes, st, (const __nv_bfloat16*)x, ldx,
               (const __nv_bfloat16*)W, ldw, M, N, K, half, out, ldo, out_f32, cap, tiles);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}
// Sixteen warps: where every tile has an SM to itself and a row has more slices than eight warps keep in flight (K > 2048): a second CTA would find
// no tile, so eight warps left half of the SM's loads unissued and walked a chain of slices twice as long. Back to back, 2048 x 5632: one row
// 9.7 -> 6.5 us, 16 rows 10.1 -> 7.0, 32 rows 14.1 -> 9.9; 1024 x 2816, 16 rows: 3.9 -> 3.0. Shorter rows (2048 x 2048, 3.2 us) fit in the eight
// warps' rings. With more tiles, where single CTAs take an odd number of rounds, which two CTAs an SM round up to an even one:
//   three rounds of long rows: 5632 x 3072, 16 rows 11.2 -> 8.4, 32 rows 17.5 -> 15.2; of 2048 (weights in whole lines) only if the last one is filled
//     by a quarter: 5920 x 2048 7.7 -> 6.5, 4752 x 2048 (one tile in it) 5.5 -> 6.1; in halves of lines 7104 x 1032 6.1 -> 6.6, 7104 x 2056 alike;
//   five rounds of 2048 likewise (gated 5632 x 2048, 16 rows: 10.3 -> 9.7, 32 rows 16.4 -> 14.6), seven and more: one row 5 % slower;
//   up to 16 rows any number of rounds of long rows: 21312 x 3072 26.8 -> 23.2, 54464 x 4096 86 -> 80; 17 to 32 rows 21312 x 3072 41.3 -> 45.8.
// Above 32 rows the accumulators of four row tiles take the registers.
template <int MT, int P, bool SILU>
static int launch_skinny(const void* x, int ldx, const void* W, int ldw, int M, int N, int K, int half, void* out, int ldo, int out_f32, float cap,
                         bool early, cudaStream_t st) {
  const int tiles = SILU ? (N + 7) / 8 : (N + 15) / 16, slices = (K + 32 * P - 1) / (32 * P);
  if constexpr (MT <= 2) {
    const int rounds = (tiles + 147) / 148, last = tiles - 148 * (rounds - 1);
    const bool rows_long = slices >= (P == 2 ? 48 : 96), worth = rows_long || (P == 2 && slices >= 32 && last >= 37);
    const bool wide = rounds == 1 ? slices > 8 * (8 / P)
                                  : rounds % 2 == 1 && worth && (rounds == 3 || (P == 2 && (rows_long ? MT == 1 : rounds == 5)));
    if (wide) return launch_skinny<MT, P, SILU, 16>(x, ldx, W, ldw, M, N, K, half, out, ldo, out_f32, cap, tiles, early, st);
  }
  return launch_skinny<MT, P, SILU, 8>(x, ldx, W, ldw, M, N, K, half, out, ldo, out_f32, cap, tiles, early, st);
}

}  // namespace inv

using namespace inv;

// ldx and ldw are multiples of 8 and at least K rounded up to 8; M <= 64. silu_half > 0: the gated form above. early: W is resident
// (launch_step).
extern "C" int inv_skinny_gemm(const void* x, int ldx, const void* W, int ldw, int M, int N, int K, int silu_half, void* out, int ldo, int out_f32,
                               float cap, int early, void* stream) {
  const int k8 = (K + 7) & ~7;
  if (M > 64 || (ldx % 8) || (ldw % 8) || ldx < k8 || ldw < k8 || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(W) & 15))
    return -ERR_BAD_ARG;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  const bool pairs = K % 16 == 0 && ldw % 16 == 0 && (reinterpret_cast<uintptr_t>(W) & 31) == 0;   // 32-byte pieces of weight rows
#define INV_SGP(MT, P)                                                                                                                \
  (silu_half > 0 ? launch_skinny<MT, P, true>(x, ldx, W, ldw, M, N, K, silu_half, out, ldo, out_f32, cap, early != 0, st)                             \
                 : launch_skinny<MT, P, false>(x, ldx, W, ldw, M, N, K, 0, out, ldo, out_f32, cap, early != 0, st))
#define INV_SG(MT) (pairs ? INV_SGP(MT, 2) : INV_SGP(MT, 1))
  if (M <= 16) return INV_SG(1);
  if (M <= 32) return INV_SG(2);
  return INV_SG(4);
#undef INV_SG
#undef INV_SGP
}
