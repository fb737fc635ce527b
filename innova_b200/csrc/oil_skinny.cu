// Products of a few tokens with packed block-32 weights: y[M, N] = x[M, K] dequant(W)[N, K]^T for M <= 16, in one kernel with what
// surrounds it: an RMSNorm of x in front, and bias, residual or SwiGLU behind.
//
// At a handful of tokens such a product is bound by latency: the weights of a layer of width 2048 are 25 MB, four microseconds. The
// tcgen05 kernel (oil_gemm.cu) pays for tensor memory, two barrier rings, reductions into a cleared accumulator and a finish
// kernel of its own, 9 us a projection however small it is. Here a CTA owns 16 weight rows (8 gate and 8 up rows in the gated
// form) and its eight or sixteen warps take every eighth or sixteenth 256-wide slice of K straight from memory into registers: a lane loads two blocks of 32
// codes of a row (one whole 32-byte sector of the 4-bit format) with their scales, expands them through the lookup table and feeds
// warp-level MMA fragments (weights are the 16-row side, tokens the 8-column side; both read k in the same permuted order, which a
// dot product does not notice). Sums meet in shared memory, in one fixed order. Resident weights are requested before the
// kernel waits for the previous grid; others are multiplied by a plainly launched kernel. The rows of x stay in shared memory in
// fragment order; the host entry states the limits.
#include "oil_expand.cuh"
#include "inv_api.h"

namespace inv {

namespace os {
constexpr int ROWS = 16, SLICE = 256;
enum Mode { PLAIN = 0, SWIGLU = 1, SUMS = 2 };   // bf16 with bias and residual; silu(gate) * up; fp32 sums
}  // namespace os

struct OilSkinnyParams {
  const __nv_bfloat16* x;
  int ldx;
  const uint8_t* idx;
  const __nv_bfloat16* scales;
  const float* codebook;
  const __nv_bfloat16* norm_w;     // optional: x is rms_norm(x) * norm_w, rounded to bf16
  float eps;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  int ld_res;
  void* out;
  int ldo;
  int M, N, K, mode, n_tiles;
};

__device__ __forceinline__ void os_mma(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float2 os_pair(uint32_t v) { return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); }

// The codes of two blocks of 32 weights: 2 * BITS words, read once.
template <int BITS>
__device__ __forceinline__ void os_load(const uint8_t* p, uint32_t* w) {
  if (BITS == 2) {
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "l"(p));
  } else {
#pragma unroll
    for (int i = 0; i < BITS / 4; ++i)
      asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(w[8 * i]), "=r"(w[8 * i + 1]), "=r"(w[8 * i + 2]), "=r"(w[8 * i + 3]), "=r"(w[8 * i + 4]), "=r"(w[8 * i + 5]),
                     "=r"(w[8 * i + 6]), "=r"(w[8 * i + 7])
                   : "l"(p + 32 * i));
  }
}

// MT: 8-token tiles; WARPS: 8, two CTAs an SM, or 16.
template <int BITS, int MT, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 2 : 1) oil_skinny_kernel(const OilSkinnyParams p) {
  using namespace os;
  constexpr int THREADS = 32 * WARPS;
  constexpr int UN = BITS == 8 ? 1 : 2;              // slices whose codes are in flight together
  constexpr int PL = MT * 8 + 1;                     // pitch of a row's partial sums
  extern __shared__ uint4 os_smem[];
  uint4* sx = os_smem;                               // x in fragment order: [slice][block of a lane][4] rows of [token][lane's quarter] x 8 values
  const int slices = (p.K + SLICE - 1) / SLICE;
  const int pitch = p.M * 4 + 1;                     // one piece more than a row needs: neighbouring rows start in other banks
  float* part = reinterpret_cast<float*>(sx + (size_t)slices * 8 * pitch);     // [WARPS][ROWS][PL]
  __shared__ __align__(128) uint32_t lut[BITS == 2 ? 32 : 256 * 32];
  __shared__ float s_cb[BITS == 8 ? 256 : 16];
  __shared__ float s_red[WARPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tig = lane & 3;
  release_next();
  if (tid < (BITS == 8 ? 256 : 1 << BITS)) s_cb[tid] = p.codebook[tid];

  const int half = p.N / 2;
  const size_t row_bytes = (size_t)p.K * BITS / 8;
  const int nsp = p.K / 64;                          // pairs of blocks per row
  uint32_t raw[UN][2][2 * BITS], sc[UN][2];
  // codes and scales of slice s; rows past N read the last row and are not stored
  auto fetch = [&](int tile, int s, uint32_t (&r)[2][2 * BITS], uint32_t (&c)[2]) {
    const int r0 = p.mode == SWIGLU ? min(tile * 8 + g, half - 1) : min(tile * ROWS + g, p.N - 1);
    const int r1 = p.mode == SWIGLU ? r0 + half : min(tile * ROWS + g + 8, p.N - 1);
    const int pair = s * 4 + tig;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const size_t row = h ? r1 : r0;
      if (pair < nsp) {
        os_load<BITS>(p.idx + row * row_bytes + (size_t)pair * (8 * BITS), r[h]);
        c[h] = __ldg(reinterpret_cast<const uint32_t*>(p.scales) + row * nsp + pair);
      } else {
#pragma unroll
        for (int k = 0; k < 2 * BITS; ++k) r[h][k] = 0;
        c[h] = 0;                                    // zero weights
      }
    }
  };
  int tile = blockIdx.x;
#pragma unroll
  for (int u = 0; u < UN; ++u)
    if (warp + u * WARPS < slices) fetch(tile, warp + u * WARPS, raw[u], sc[u]);
  __syncthreads();
  if (BITS != 2) oil_lut_fill<BITS>(lut, s_cb, tid, THREADS);
  wait_previous();

  // x into shared memory, P threads per token; what lies behind K is zero
  {
    int P = THREADS;
    while (P * p.M > THREADS && P > 1) P >>= 1;
    const int token = tid / P, t = tid % P;
    const bool have = token < p.M;
    const int k8s = slices * 32, k8_real = p.K / 8;
    const uint4* src = reinterpret_cast<const uint4*>(p.x + (size_t)(have ? token : 0) * p.ldx);
    constexpr int UX = 4;                            // loads in flight together
    float rstd = 0.f;
    if (p.norm_w) {
      float ss = 0.f;
      for (int k0 = t; have && k0 < k8_real; k0 += UX * P) {
        uint4 v[UX];
#pragma unroll
        for (int i = 0; i < UX; ++i) v[i] = k0 + i * P < k8_real ? src[k0 + i * P] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < UX; ++i) {
          const float2 a = os_pair(v[i].x), b = os_pair(v[i].y), c = os_pair(v[i].z), d = os_pair(v[i].w);
          ss += a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y + c.x * c.x + c.y * c.y + d.x * d.x + d.y * d.y;
        }
      }
      for (int o = min(P, 32) >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (P > 32) {
        if (lane == 0) s_red[warp] = ss;
        __syncthreads();
        ss = 0.f;
        for (int w = 0; w < P / 32; ++w) ss += s_red[(warp & ~(P / 32 - 1)) + w];
      }
      rstd = rsqrtf(ss / p.K + p.eps);
    }
    const uint4* wn = reinterpret_cast<const uint4*>(p.norm_w);
    for (int k0 = t; have && k0 < k8s; k0 += UX * P) {
      uint4 v[UX], w[UX];
#pragma unroll
      for (int i = 0; i < UX; ++i) {
        const bool in = k0 + i * P < k8_real;
        v[i] = in ? src[k0 + i * P] : make_uint4(0, 0, 0, 0);
        if (p.norm_w) w[i] = in ? __ldg(wn + k0 + i * P) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int i = 0; i < UX; ++i) {
        const int k8 = k0 + i * P;
        if (p.norm_w) {
          const float2 a = os_pair(v[i].x), b = os_pair(v[i].y), c = os_pair(v[i].z), d = os_pair(v[i].w);
          const float2 wa = os_pair(w[i].x), wb = os_pair(w[i].y), wc = os_pair(w[i].z), wd = os_pair(w[i].w);
          v[i] = make_uint4(pack_bf16x2(a.x * rstd * wa.x, a.y * rstd * wa.y), pack_bf16x2(b.x * rstd * wb.x, b.y * rstd * wb.y),
                            pack_bf16x2(c.x * rstd * wc.x, c.y * rstd * wc.y), pack_bf16x2(d.x * rstd * wd.x, d.y * rstd * wd.y));
        }
        if (k8 < k8s) sx[((k8 >> 5) * 8 + (k8 & 7)) * pitch + token * 4 + ((k8 >> 3) & 3)] = v[i];
      }
    }
    __syncthreads();
  }

  for (; tile < p.n_tiles; tile += gridDim.x) {
    float acc[MT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
    for (int s0 = warp; s0 < slices; s0 += UN * WARPS) {
#pragma unroll
      for (int u = 0; u < UN; ++u) {
        const int slice = s0 + u * WARPS;
        if (slice >= slices) break;
#pragma unroll
        for (int b = 0; b < 2; ++b) {                // the lane's two blocks of the slice
          uint32_t w0[16], w1[16];
          const __nv_bfloat16_raw r0{(unsigned short)(sc[u][0] >> (16 * b))}, r1{(unsigned short)(sc[u][1] >> (16 * b))};
          expand_block<BITS>(raw[u][0] + b * BITS, __nv_bfloat16(r0), lut, s_cb, lane, w0);
          expand_block<BITS>(raw[u][1] + b * BITS, __nv_bfloat16(r1), lut, s_cb, lane, w1);
          if (b == 1) {                              // the slot is free: the next slice of this tile or the first ones of the next
            const int next = slice + UN * WARPS;
            if (next < slices) fetch(tile, next, raw[u], sc[u]);
            else if (tile + (int)gridDim.x < p.n_tiles) fetch(tile + gridDim.x, warp + u * WARPS, raw[u], sc[u]);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int m = 0; m < MT; ++m) {
              const int token = m * 8 + g;
              const uint4 v = token < p.M ? sx[(slice * 8 + b * 4 + q) * pitch + token * 4 + tig] : make_uint4(0, 0, 0, 0);
              os_mma(acc[m], w0[4 * q], w1[4 * q], w0[4 * q + 1], w1[4 * q + 1], v.x, v.y);
              os_mma(acc[m], w0[4 * q + 2], w1[4 * q + 2], w0[4 * q + 3], w1[4 * q + 3], v.z, v.w);
            }
        }
      }
    }
    float* mine = part + (size_t)warp * ROWS * PL;
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      mine[g * PL + m * 8 + 2 * tig] = acc[m][0];
      mine[g * PL + m * 8 + 2 * tig + 1] = acc[m][1];
      mine[(g + 8) * PL + m * 8 + 2 * tig] = acc[m][2];
      mine[(g + 8) * PL + m * 8 + 2 * tig + 1] = acc[m][3];
    }
    __syncthreads();
    const int cols = p.mode == SWIGLU ? 8 : ROWS, n_out = p.mode == SWIGLU ? half : p.N;
    for (int i = tid; i < cols * p.M; i += THREADS) {
      const int c = i % cols, m = i / cols, n = tile * cols + c;
      if (n >= n_out) continue;
      float a = 0.f, b = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        a += part[((size_t)w * ROWS + c) * PL + m];
        if (p.mode == SWIGLU) b += part[((size_t)w * ROWS + c + 8) * PL + m];
      }
      if (p.mode == SUMS) {
        static_cast<float*>(p.out)[(size_t)m * p.ldo + n] = a;
        continue;
      }
      if (p.bias) {
        a += __bfloat162float(p.bias[n]);
        if (p.mode == SWIGLU) b += __bfloat162float(p.bias[half + n]);
      }
      if (p.mode == SWIGLU) {                        // the projection is rounded to bf16 before the activation
        a = __bfloat162float(__float2bfloat16_rn(a));
        b = __bfloat162float(__float2bfloat16_rn(b));
        a = a / (1.f + __expf(-a)) * b;
      } else if (p.residual) {
        a += __bfloat162float(p.residual[(size_t)m * p.ld_res + n]);
      }
      static_cast<__nv_bfloat16*>(p.out)[(size_t)m * p.ldo + n] = __float2bfloat16_rn(a);
    }
    __syncthreads();
  }
}

template <int BITS, int MT, int WARPS>
static int launch_oil_skinny(const OilSkinnyParams& p, bool early, int smem, cudaStream_t st) {
  static int limit = 0;
  if (limit == 0) {
    const cudaError_t e = cudaFuncSetAttribute(oil_skinny_kernel<BITS, MT, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 190 * 1024);
    if (e != cudaSuccess) return -(int)e;
    limit = 190 * 1024;
  }
  if (smem > limit) return -ERR_BAD_ARG;
  const int per_sm = WARPS == 8 && 2 * (smem + (BITS == 2 ? 3 : 35) * 1024) <= 226 * 1024 ? 2 : 1;
  launch_step(early, oil_skinny_kernel<BITS, MT, WARPS>, dim3(p.n_tiles < 148 * per_sm ? p.n_tiles : 148 * per_sm), WARPS * 32, smem, st, p);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}
// Sixteen warps where a tile has an SM to itself and more slices than eight warps: all of its weights are then in flight at once and the
// expansion, which is bound by instruction issue, has four warps a scheduler (2048 x 5632: eight tokens 6.6 -> 5.8 us, three 6.3 -> 5.0; one token back
// to back 4.5 with eight and 4.65 with sixteen, but behind the attention and gate/up products of a decode step, whose end its loads overlap,
// sixteen take 1 us a layer less: generate of one sequence, 8 layers, 64 steps: 18.05 -> 17.5 ms).
// With several tiles an SM two CTAs of eight warps do the same and overlap their reductions.
template <int BITS, int MT>
static int launch_oil_skinny(const OilSkinnyParams& p, bool early, cudaStream_t st) {
  using namespace os;
  const int slices = (p.K + SLICE - 1) / SLICE;
  const int x = slices * 128 * (4 * p.M + 1), sums = ROWS * (MT * 8 + 1) * 4;
  if (p.n_tiles <= 148 && slices > 8 && x + 16 * sums <= 190 * 1024) return launch_oil_skinny<BITS, MT, 16>(p, early, x + 16 * sums, st);
  return launch_oil_skinny<BITS, MT, 8>(p, early, x + 8 * sums, st);
}

}  // namespace inv

using namespace inv;

// M <= 16 tokens, K % 64 == 0, and x (M * K rounded up to 256, 2 bytes each, and a little) within 180 KB of shared memory. x and norm_w on 16
// bytes, the codes on 32, the scales on 4, ldx % 8 == 0. mode 0: out bf16 [M, N] = product + bias + residual. mode 1: out bf16
// [M, N / 2] = silu(gate + bias) * (up + bias), gate rows [0, N / 2), up rows behind them. mode 2: out fp32 [M, N] = product. norm_w
// (optional): x is rms_norm(x) * norm_w, as its own kernel would round it. early: codes, scales and codebook are
// resident (launch_step).
extern "C" int inv_oil_skinny(const void* x, int ldx, const void* idx, const void* scales, const float* codebook, int bits, const void* norm_w,
                              float eps, const void* bias, const void* residual, int ld_res, void* out, int ldo, int M, int N, int K, int mode,
                              int early, void* stream) {
  if ((bits != 2 && bits != 4 && bits != 8) || M < 1 || M > 16 || (K % 64) || K < 64 || (ldx % 8) || N < 1 || mode < 0 || mode > 2 ||
      (mode == 1 && (N % 2)) || ((uintptr_t)x | (uintptr_t)norm_w) % 16 || (uintptr_t)idx % 32 || (uintptr_t)scales % 4 ||
      (long)((K + 255) / 256) * 128 * (4 * M + 1) > 180 * 1024)
    return -ERR_BAD_ARG;
  OilSkinnyParams p{(const __nv_bfloat16*)x, ldx, (const uint8_t*)idx, (const __nv_bfloat16*)scales, codebook, (const __nv_bfloat16*)norm_w, eps,
                    (const __nv_bfloat16*)bias, (const __nv_bfloat16*)residual, ld_res, out, ldo, M, N, K, mode,
                    mode == 1 ? (N / 2 + 7) / 8 : (N + 15) / 16};
  cudaStream_t st = (cudaStream_t)stream;
  const bool pdl = early != 0;
#define INV_OS(B) (M <= 8 ? launch_oil_skinny<B, 1>(p, pdl, st) : launch_oil_skinny<B, 2>(p, pdl, st))
  return bits == 2 ? INV_OS(2) : bits == 4 ? INV_OS(4) : INV_OS(8);
#undef INV_OS
}
