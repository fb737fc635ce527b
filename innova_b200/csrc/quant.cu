// Train-in-format quantisation kernels: block-wise codebook quantise / dequantise and the
// straight-through fake-quant forward.
//
// Compute format (the reference's in-memory engines, src/oil_engines_oil8.cpp:42-140,
// src/oil_engines_core.cpp:15-160, used by STEQuantizer, src/ste_quantizer.cpp:19-66,145-202):
// weights are cut into blocks of 32 consecutive values; a block stores its abs-max as scale, and every
// value stores the index of the nearest entry of a shared codebook over the normalised range [-1, 1]
// (256 entries for OIL8, 16 for OIL4). SPARK is ternary {-s, 0, +s} with a 0.5*max dead zone, OIL1 is
// sign times the block's mean magnitude.
//
// Four lanes own one block, eight consecutive values each: 16- or 32-byte loads, a block's abs-max in two shuffles. Modes:
// 0 OIL8, 1 OIL4, 2 SPARK, 3 OIL1.
#include "sm100_common.cuh"
#include "inv_api.h"

namespace inv {

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_add(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Index of the codebook entry nearest to x; cb is sorted ascending, K is a power of two.
__device__ __forceinline__ int nearest_sorted(const float* cb, int K, float x) {
  int lo = 0;
  for (int step = K >> 1; step > 0; step >>= 1)
    if (cb[lo + step] <= x) lo += step;
  if (lo + 1 < K && (cb[lo + 1] - x) < (x - cb[lo])) ++lo;
  return lo;
}

__device__ __forceinline__ void load8(const float* p, float* v) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float* v) {
  const uint4 r = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ void store8(float* p, const float* v) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float* v) {
  *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}
// Sum over a block whose lane l (of four) holds elements 8 l .. 8 l + 7, in the order of a butterfly over 32 lanes.
__device__ __forceinline__ float block_add(const float* x) {
  float v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = x[i] + __shfl_xor_sync(0xffffffffu, x[i], 2);
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], 1);
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] += v[i + 4];
  return (v[0] + v[2]) + (v[1] + v[3]);
}

enum CodeForm { CODES_NONE = 0, CODES_BYTE = 1, CODES_NIBBLE = 2, CODES_TWO_BIT = 3 };
struct QuantOut {
  void* q;              // dequantised values, optional
  int q_bf16;
  uint8_t* codes;       // one byte per value, or packed (low bits first)
  int form;
  void* scales;         // one per block, optional
  int scales_bf16;
};

// The decision "(cb[lo + 1] - x) < (x - cb[lo])" is monotone in x, so the code of x is the number of thresholds T[1..K-1] at or
// below x, T[j] being the smallest float that takes entry j. Found by bisection over the float order.
__device__ __forceinline__ int float_order(float f) {
  const int i = __float_as_int(f);
  return i >= 0 ? i : (int)0x80000000 - i;
}
__device__ __forceinline__ float order_float(int o) { return __int_as_float(o >= 0 ? o : (int)0x80000000 - o); }
__device__ __forceinline__ float code_threshold(float c0, float c1) {
  if (!(c0 < c1)) return c1;
  long long lo = float_order(c0), hi = float_order(c1);
  while (hi - lo > 1) {
    const long long mid = lo + (hi - lo) / 2;
    const float x = order_float((int)mid);
    if ((c1 - x) < (x - c0)) hi = mid;
    else lo = mid;
  }
  return order_float((int)hi);
}

// Whole blocks of 32 values, 16-byte aligned. One read of a table entry gives a value's code: x falls into one of BUCKETS buckets of
// [-1, 1] (the bits of x * BUCKETS / 2 + 2^23 + BUCKETS / 2), which knows the thresholds below it and the one inside it. Codebooks with
// several thresholds in a bucket walk on from there; the next block's values are requested before this one is coded. Bound by the table:
// each lane reads an entry of eight bytes at a place of its own, which takes a warp 5.8 passes for Gaussian blocks where 2 would do (simulated on
// the bucket rule), 30 us of shared memory for 11008 x 4096; then by issue and, from fp32, by memory: 11008 x 4096 fp32 to packed nibbles and
// bf16 scales in 55 us, 3.8 TB/s (one warp per block with a binary search per value, then a packing and a rounding launch: 270 us); 20 M
// values bf16 to bf16 through 256 entries in 33 us (107 us).
template <typename TIn, int MODE>
__global__ void __launch_bounds__(256) block_quant8_kernel(const TIn* __restrict__ in, QuantOut out, const float* __restrict__ codebook,
                                                           long nblocks) {
  constexpr int K = MODE == 0 ? 256 : 16;                 // table sizes; a 256-entry codebook takes the MODE 0 instance
  constexpr int BUCKETS = MODE == 0 ? 1024 : 256;
  struct Entry { float thr; int base; };
  __shared__ Entry s_entry[MODE <= 1 ? BUCKETS + 2 : 1];
  __shared__ float s_cb[MODE <= 1 ? K : 1], s_thr[MODE <= 1 ? K + 1 : 1];
  __shared__ int s_walk;
  if (MODE <= 1) {
    if (threadIdx.x == 0) s_walk = 0;
    for (int i = threadIdx.x; i < K; i += blockDim.x) s_cb[i] = codebook[i];
    __syncthreads();
    for (int i = threadIdx.x; i <= K; i += blockDim.x)
      s_thr[i] = i == 0 ? -INFINITY : i == K ? INFINITY : code_threshold(s_cb[i - 1], s_cb[i]);
    __syncthreads();
    constexpr int PER = (BUCKETS + 2 + 255) / 256;         // neighbouring buckets per thread: one search, then steps
    int base = 0;
    for (int i = 0; i < PER; ++i) {
      const int b = threadIdx.x * PER + i;
      if (b > BUCKETS + 1) break;
      // bucket b holds the x that round to b after scaling; the margin covers the rounding of the product
      const float low = ((float)b - 0.5f) * (2.f / BUCKETS) - 1.f - 1e-6f, high = ((float)b + 0.5f) * (2.f / BUCKETS) - 1.f + 1e-6f;
      if (i == 0) {
        for (int step = K >> 1; step > 0; step >>= 1)
          if (s_thr[base + step] <= low) base += step;
      } else {
        while (s_thr[base + 1] <= low) ++base;
      }
      const bool none = b == BUCKETS + 1;                  // what is no number
      if (!none && base + 2 <= K && s_thr[base + 2] <= high) s_walk = 1;
      s_entry[b] = Entry{none ? INFINITY : s_thr[base + 1], none ? 0 : base};
    }
    __syncthreads();
  }
  [[maybe_unused]] const bool walk = MODE <= 1 && s_walk != 0;
  const int lane = threadIdx.x & 31, sub = lane & 3;
  const long stride = (long)gridDim.x * (blockDim.x >> 5) * 8;
  const long first = (blockIdx.x * (long)(blockDim.x >> 5) + (threadIdx.x >> 5)) * 8;
  float next[8];
  if (first < nblocks) load8(in + min(first + (lane >> 2), nblocks - 1) * 32 + sub * 8, next);
  for (long b0 = first; b0 < nblocks; b0 += stride) {
    const long b = b0 + (lane >> 2);
    const bool ok = b < nblocks;
    const long i = (ok ? b : nblocks - 1) * 32 + sub * 8;
    float w[8], a[8], q[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) w[k] = next[k];
    if (b0 + stride < nblocks) load8(in + min(b + stride, nblocks - 1) * 32 + sub * 8, next);   // in flight while this one is coded
    float amax = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      a[k] = fabsf(w[k]);
      amax = fmaxf(amax, a[k]);
    }
    float scale;
    uint32_t code[8];
    if (MODE <= 2) {
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    }
    if (MODE <= 1) {
      const bool dead = amax < 1e-10f;  // an all-zero block keeps scale 0, so that it dequantises to exactly zero
      scale = dead ? 1.f : amax;
      const float inv = 1.f / scale;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float x = w[k] * inv;
        const Entry e = s_entry[min(__float_as_int(fmaf(x, BUCKETS / 2, 8388608.f + BUCKETS / 2)) & (2 * BUCKETS - 1), BUCKETS + 1)];
        code[k] = e.base + (x >= e.thr ? 1 : 0);
        if (walk)
          while (x >= s_thr[code[k] + 1]) ++code[k];
      }
      if (dead) scale = 0.f;
      if (out.q)
#pragma unroll
        for (int k = 0; k < 8; ++k) q[k] = s_cb[code[k]] * scale;
    } else if (MODE == 2) {
      float kept[8], ones = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const bool keep = a[k] > 0.5f * amax && amax > 0.f;
        kept[k] = keep ? a[k] : 0.f;
        ones += keep ? 1.f : 0.f;
        code[k] = keep ? (w[k] > 0.f ? 1 : 2) : 0;
      }
      ones += __shfl_xor_sync(0xffffffffu, ones, 1);
      ones += __shfl_xor_sync(0xffffffffu, ones, 2);
      const float mag = block_add(kept);
      scale = ones > 0.f ? mag / ones : 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) q[k] = code[k] ? copysignf(scale, w[k]) : 0.f;
    } else {
      scale = block_add(a) / 32.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        code[k] = w[k] >= 0.f ? 1 : 0;
        q[k] = w[k] >= 0.f ? scale : -scale;
      }
    }
    if (!ok) continue;
    if (out.q) {
      if (out.q_bf16) store8((__nv_bfloat16*)out.q + i, q);
      else store8((float*)out.q + i, q);
    }
    if (out.form == CODES_BYTE) {
      uint32_t p[2] = {0, 0};
#pragma unroll
      for (int k = 0; k < 8; ++k) p[k >> 2] |= code[k] << (8 * (k & 3));
      *reinterpret_cast<uint2*>(out.codes + i) = make_uint2(p[0], p[1]);
    } else if (out.form == CODES_NIBBLE) {
      uint32_t p = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) p |= (code[k] & 15u) << (4 * k);
      *reinterpret_cast<uint32_t*>(out.codes + (i >> 1)) = p;
    } else if (out.form == CODES_TWO_BIT) {
      uint32_t p = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) p |= code[k] << (2 * k);
      *reinterpret_cast<uint16_t*>(out.codes + (i >> 2)) = (uint16_t)p;
    }
    if (out.scales && sub == 0) {
      if (out.scales_bf16) ((__nv_bfloat16*)out.scales)[b] = __float2bfloat16_rn(scale);
      else ((float*)out.scales)[b] = scale;
    }
  }
}

// The values that are not a whole block, and addresses off 16 bytes: one warp per block, a value per lane, one byte per code.
// in: fp32 or bf16 weights (n values). out_q (bf16 or fp32, optional): dequantised values.
// idx (optional): one byte per value. scales (optional): one float per block of 32.
template <typename TIn, typename TOut>
__global__ void __launch_bounds__(256) block_quant_kernel(const TIn* __restrict__ in, TOut* __restrict__ out_q, uint8_t* __restrict__ idx,
                                                          float* __restrict__ scales, const float* __restrict__ codebook, int K, long n,
                                                          int mode) {
  __shared__ float cb[256];
  for (int i = threadIdx.x; i < K; i += blockDim.x) cb[i] = codebook ? codebook[i] : 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const long nblocks = (n + 31) / 32;
  for (long b = blockIdx.x * (long)(blockDim.x >> 5) + (threadIdx.x >> 5); b < nblocks; b += (long)gridDim.x * (blockDim.x >> 5)) {
    const long i = b * 32 + lane;
    const bool ok = i < n;
    const float w = ok ? (float)in[i] : 0.f;
    const float amax = warp_max(fabsf(w));
    const bool dead = amax < 1e-10f;  // an all-zero block keeps scale 0, so that it dequantises to exactly zero
    float scale = dead ? 1.f : amax;
    float q;
    int code;
    if (mode <= 1) {
      code = nearest_sorted(cb, K, w / scale);
      if (dead) scale = 0.f;
      q = cb[code] * scale;
    } else if (mode == 2) {
      const bool keep = fabsf(w) > 0.5f * amax && amax > 0.f;
      const float cnt = warp_add(keep ? 1.f : 0.f);
      const float mag = warp_add(keep ? fabsf(w) : 0.f);
      scale = cnt > 0.f ? mag / cnt : 0.f;
      code = keep ? (w > 0.f ? 1 : 2) : 0;
      q = keep ? copysignf(scale, w) : 0.f;
    } else {
      const int cntn = (int)min(32L, n - b * 32);
      scale = warp_add(fabsf(w)) / (float)cntn;
      code = w >= 0.f ? 1 : 0;
      q = w >= 0.f ? scale : -scale;
    }
    if (ok) {
      if (out_q) out_q[i] = (TOut)q;
      if (idx) idx[i] = (uint8_t)code;
    }
    if (scales && lane == 0) scales[b] = scale;
  }
}

// A packed weight matrix -> bf16: bf16(codebook[code]) * scale in one rounding, the same value that the GEMM expands. Eight values
// per thread and step, 16-byte stores. Bound by the stores: 11008 x 4096 in 19 us, 6.1 TB/s (a chain of eight library kernels took
// 540 us).
template <int BITS>
__global__ void __launch_bounds__(256) weight_dequant_kernel(const uint8_t* __restrict__ codes, const __nv_bfloat16* __restrict__ scales,
                                                             const float* __restrict__ codebook, __nv_bfloat16* __restrict__ out, long n8) {
  __shared__ uint32_t lut[256];   // 4 bits: the pair of values of a byte; 8 bits: the value; 2 bits: the pair of values of a nibble
  {
    const int e = threadIdx.x;
    if (BITS == 4) lut[e] = pack_bf16x2(codebook[e & 15], codebook[e >> 4]);
    else if (BITS == 8) lut[e] = pack_bf16x2(codebook[e], 0.f);
    else if (e < 16) lut[e] = pack_bf16x2(codebook[e & 3], codebook[e >> 2]);
  }
  __syncthreads();
  constexpr int UNROLL = 4;
  for (long g0 = blockIdx.x * 256L * UNROLL + threadIdx.x; g0 < n8; g0 += (long)gridDim.x * 256 * UNROLL) {
    uint2 raw[UNROLL];
    __nv_bfloat16 s[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const long g = g0 + u * 256L;
      if (g >= n8) break;
      if (BITS == 8) raw[u] = reinterpret_cast<const uint2*>(codes)[g];
      else if (BITS == 4) raw[u].x = reinterpret_cast<const uint32_t*>(codes)[g];
      else raw[u].x = reinterpret_cast<const uint16_t*>(codes)[g];
      s[u] = scales[g >> 2];
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const long g = g0 + u * 256L;
      if (g >= n8) break;
      const __nv_bfloat162 s2 = __halves2bfloat162(s[u], s[u]);
      uint32_t o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t pair;
        if (BITS == 8) {
          const uint32_t two = (k < 2 ? raw[u].x : raw[u].y) >> (16 * (k & 1));
          pair = lut[two & 255] | (lut[(two >> 8) & 255] << 16);
        } else if (BITS == 4) {
          pair = lut[(raw[u].x >> (8 * k)) & 255];
        } else {
          pair = lut[(raw[u].x >> (4 * k)) & 15];
        }
        const __nv_bfloat162 v = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&pair), s2);
        o[k] = *reinterpret_cast<const uint32_t*>(&v);
      }
      reinterpret_cast<uint4*>(out)[g] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// out[i] = codebook[idx[i]] * scales[i / 32]   (OIL8 / OIL4 compute format -> bf16)
__global__ void block_dequant_kernel(const uint8_t* __restrict__ idx, const float* __restrict__ scales, const float* __restrict__ codebook, int K,
                                     __nv_bfloat16* __restrict__ out, long n) {
  __shared__ float cb[256];
  for (int i = threadIdx.x; i < K; i += blockDim.x) cb[i] = codebook[i];
  __syncthreads();
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16_rn(cb[idx[i] & (K - 1)] * scales[i >> 5]);
}

// Packs one-byte OIL4 indices into nibbles: out[i] = idx[2i] | idx[2i+1] << 4.
__global__ void pack_nibbles_kernel(const uint8_t* __restrict__ idx, uint8_t* __restrict__ out, long n2) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n2; i += (long)gridDim.x * blockDim.x)
    out[i] = (uint8_t)((idx[2 * i] & 15) | (idx[2 * i + 1] << 4));
}

}  // namespace inv

using namespace inv;

template <typename TIn>
static void quant8(const TIn* in, const QuantOut& out, const float* codebook, int K, long nblocks, int mode, cudaStream_t st) {
  long blocks = (nblocks + 63) / 64;
  if (blocks > 148 * 8) blocks = 148 * 8;
  const int g = (int)blocks;
  if (mode <= 1 && K == 256) block_quant8_kernel<TIn, 0><<<g, 256, 0, st>>>(in, out, codebook, nblocks);
  else if (mode <= 1) block_quant8_kernel<TIn, 1><<<g, 256, 0, st>>>(in, out, codebook, nblocks);
  else if (mode == 2) block_quant8_kernel<TIn, 2><<<g, 256, 0, st>>>(in, out, codebook, nblocks);
  else block_quant8_kernel<TIn, 3><<<g, 256, 0, st>>>(in, out, codebook, nblocks);
}

// in_dtype / out_dtype: 0 = fp32, 1 = bf16. Any of out_q, idx, scales may be null.
extern "C" int inv_block_quant(const void* in, int in_dtype, void* out_q, int out_dtype, uint8_t* idx, float* scales, const float* codebook,
                               int K, long n, int mode, void* stream) {
  if (n <= 0) return 0;
  if (mode < 0 || mode > 3 || (mode <= 1 && (codebook == nullptr || (K != 16 && K != 256)))) return -ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  long whole = n / 32;
  if (((uintptr_t)in | (uintptr_t)out_q) & 15 || (uintptr_t)idx & 7) whole = 0;
  if (whole > 0) {
    const QuantOut o{out_q, out_dtype, idx, idx ? CODES_BYTE : CODES_NONE, scales, 0};
    if (in_dtype == 0) quant8((const float*)in, o, codebook, K, whole, mode, st);
    else quant8((const __nv_bfloat16*)in, o, codebook, K, whole, mode, st);
    const long at = whole * 32;
    in = (const char*)in + at * (in_dtype == 0 ? 4 : 2);
    if (out_q) out_q = (char*)out_q + at * (out_dtype == 0 ? 4 : 2);
    if (idx) idx += at;
    if (scales) scales += whole;
    n -= at;
  }
  if (n > 0) {
    long blocks = ((n + 31) / 32 + 7) / 8;
    if (blocks > 148 * 16) blocks = 148 * 16;
    const int g = (int)blocks;
    if (in_dtype == 0 && out_dtype == 0)
      block_quant_kernel<float, float><<<g, 256, 0, st>>>((const float*)in, (float*)out_q, idx, scales, codebook, K, n, mode);
    else if (in_dtype == 0 && out_dtype == 1)
      block_quant_kernel<float, __nv_bfloat16><<<g, 256, 0, st>>>((const float*)in, (__nv_bfloat16*)out_q, idx, scales, codebook, K, n, mode);
    else if (in_dtype == 1 && out_dtype == 1)
      block_quant_kernel<__nv_bfloat16, __nv_bfloat16><<<g, 256, 0, st>>>((const __nv_bfloat16*)in, (__nv_bfloat16*)out_q, idx, scales, codebook,
                                                                         K, n, mode);
    else
      block_quant_kernel<__nv_bfloat16, float><<<g, 256, 0, st>>>((const __nv_bfloat16*)in, (float*)out_q, idx, scales, codebook, K, n, mode);
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}

// n weights (a multiple of 32, 16-byte aligned) -> packed codes (mode 0: a byte, 1: a nibble, 2 and 3: two bits each, low bits first)
// and one bf16 scale per block of 32.
extern "C" int inv_quantize_weight(const void* in, int in_dtype, uint8_t* codes, void* scales, const float* codebook, int K, long n, int mode,
                                   void* stream) {
  if (n <= 0) return 0;
  if (mode < 0 || mode > 3 || (mode <= 1 && (codebook == nullptr || (K != 16 && K != 256))) || n % 32 || ((uintptr_t)in & 15) || ((uintptr_t)codes & 7))
    return -ERR_BAD_ARG;
  const QuantOut o{nullptr, 0, codes, mode == 0 ? CODES_BYTE : mode == 1 ? CODES_NIBBLE : CODES_TWO_BIT, scales, 1};
  if (in_dtype == 0) quant8((const float*)in, o, codebook, K, n / 32, mode, (cudaStream_t)stream);
  else quant8((const __nv_bfloat16*)in, o, codebook, K, n / 32, mode, (cudaStream_t)stream);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}

// The other way: n values (a multiple of 32) from packed codes of 2, 4 or 8 bits with a codebook of 4, 16 or 256 entries.
extern "C" int inv_weight_dequant(const uint8_t* codes, const void* scales, const float* codebook, int bits, void* out, long n, void* stream) {
  if (n <= 0) return 0;
  if ((bits != 2 && bits != 4 && bits != 8) || n % 32 || ((uintptr_t)out & 15) || ((uintptr_t)codes & 7)) return -ERR_BAD_ARG;
  const long n8 = n / 8;
  long g = (n8 + 1023) / 1024;
  if (g > 148 * 8) g = 148 * 8;
  cudaStream_t st = (cudaStream_t)stream;
  const __nv_bfloat16* sc = (const __nv_bfloat16*)scales;
  if (bits == 2) weight_dequant_kernel<2><<<(int)g, 256, 0, st>>>(codes, sc, codebook, (__nv_bfloat16*)out, n8);
  else if (bits == 4) weight_dequant_kernel<4><<<(int)g, 256, 0, st>>>(codes, sc, codebook, (__nv_bfloat16*)out, n8);
  else weight_dequant_kernel<8><<<(int)g, 256, 0, st>>>(codes, sc, codebook, (__nv_bfloat16*)out, n8);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}

extern "C" int inv_block_dequant(const uint8_t* idx, const float* scales, const float* codebook, int K, void* out, long n, void* stream) {
  if (n <= 0) return 0;
  if (K != 16 && K != 256) return -ERR_BAD_ARG;
  long g = (n + 255) / 256;
  if (g > 148 * 16) g = 148 * 16;
  block_dequant_kernel<<<(int)g, 256, 0, (cudaStream_t)stream>>>(idx, scales, codebook, K, (__nv_bfloat16*)out, n);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}

extern "C" int inv_pack_nibbles(const uint8_t* idx, uint8_t* out, long n, void* stream) {
  if (n <= 0) return 0;
  if (n & 1) return -ERR_BAD_ARG;
  long g = (n / 2 + 255) / 256;
  if (g > 148 * 16) g = 148 * 16;
  pack_nibbles_kernel<<<(int)g, 256, 0, (cudaStream_t)stream>>>(idx, out, n / 2);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}
