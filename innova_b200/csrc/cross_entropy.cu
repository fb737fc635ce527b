// Fused softmax cross-entropy over bf16 logits: one pass for the statistics, one pass that
// overwrites the logits with their gradient. Nothing of size [T, V] is allocated.
//
// Replaces the reference's cross_entropy_loss / cross_entropy_grad (src/autograd_grad.cpp:220-271:
// mean over positions of logsumexp - logit[target], grad = (softmax - onehot) / count) and the
// vk_cross_entropy pair (src/gpu_compute_vulkan.cpp:1156-1202). Label smoothing follows the
// reference trainer's option (src/trainer_core.cpp:408-474).
#include "sm100_common.cuh"
#include "inv_api.h"

namespace inv {

constexpr int CE_THREADS = 512;
constexpr float kL2E = 1.4426950408889634f, CE_FLOOR = -131072.f, CE_LARGE = 91000.f;

// The maximum in powers of two. No bf16 value lies within 300 of CE_FLOOR below it: what is held there adds nothing at all.
__device__ __forceinline__ float ce_log2(float m) { return fmaxf(__fmul_rn(m, kL2E), CE_FLOOR); }
// What a sum relative to the maximum m becomes relative to the maximum mn >= m.
__device__ __forceinline__ float ce_ratio(float m, float mn) {
  return exp2f(ce_log2(m) - ce_log2(mn));
}

// logits: [T, ld] bf16, columns [V, ld) are padding. labels < 0 are ignored.
// loss[t] = (1-eps)*nll + eps*(lse - mean(x));  if grad != 0: logits <- dloss/dlogits * gscale.
__global__ void __launch_bounds__(CE_THREADS) cross_entropy_kernel(__nv_bfloat16* __restrict__ logits, const int64_t* __restrict__ labels,
                                                                   float* __restrict__ loss, float* __restrict__ lse_out, int V, int ld,
                                                                   float gscale, float smoothing, int write_grad) {
  __shared__ float sm_m[CE_THREADS / 32], sm_s[CE_THREADS / 32], sm_x[CE_THREADS / 32];
  __shared__ float bc[3];
  const int row = blockIdx.x;
  __nv_bfloat16* x = logits + (size_t)row * ld;
  const long label = labels[row];
  const int nvec = ld / 8, whole = V / 8;  // vectors of eight columns, those without padding
  // m is the maximum and mc = m * log2(e) as rounded: s sums 2^(x log2(e) - mc), and the logarithm below counts with the same mc.
  // Far from zero (masked logits) what the rounding takes is no longer small, nor the product finite: mc is held at CE_FLOOR, and
  // columns below it add nothing. A row whose maximum is that large counts its maxima afterwards: bf16 values of that size lie at
  // least 256 apart. (To sum them right as they come costs the loop its shape, with any test in it: 607 -> 625 us at the size below.)
  float m = -INFINITY, mc = 0.f, s = 0.f, sx = 0.f;
  // A thread's vectors are read two at a time. Maximum on packed pairs, one fused multiply-add, one exponential and one addition per
  // value: 16384 x 50257 in 610 us (a test per column and a sum of the logits nobody asked for: 740 us; the rows of the resident
  // CTAs stay in L2 for the second pass, so 500 us is what the bytes take).
  auto raise = [&](float to) {
    const float c = ce_log2(to);
    s = m == -INFINITY ? 0.f : s * exp2f(mc - c);
    m = to;
    mc = c;
  };
  auto add = [&](const uint4& v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(w);
    const __nv_bfloat162 h2 = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
    const float lm = fmaxf(__low2float(h2), __high2float(h2));
    if (lm > m) raise(lm);
    float t = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float lo = __uint_as_float(w[j] << 16), hi = __uint_as_float(w[j] & 0xffff0000u);
      t += exp2f(fmaf(lo, kL2E, -mc)) + exp2f(fmaf(hi, kL2E, -mc));
      if (smoothing != 0.f) sx += lo + hi;
    }
    s += t;
  };
  int i = threadIdx.x;
  for (; i + CE_THREADS < whole; i += 2 * CE_THREADS) {
    const uint4 a = *reinterpret_cast<const uint4*>(x + i * 8), b = *reinterpret_cast<const uint4*>(x + (i + CE_THREADS) * 8);
    add(a);
    add(b);
  }
  if (i < whole) add(*reinterpret_cast<const uint4*>(x + i * 8));
  if (threadIdx.x < V - whole * 8) {  // the columns before the padding, one per thread
    const float f = __bfloat162float(x[whole * 8 + threadIdx.x]);
    if (f > m) raise(f);
    s += exp2f(fmaf(f, kL2E, -mc));
    if (smoothing != 0.f) sx += f;
  }
  // warp then block reduction of (m, s) pairs
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float m2 = __shfl_xor_sync(0xffffffffu, m, o);
    float s2 = __shfl_xor_sync(0xffffffffu, s, o);
    sx += __shfl_xor_sync(0xffffffffu, sx, o);
    float mn = fmaxf(m, m2);
    s = (m == -INFINITY ? 0.f : s * ce_ratio(m, mn)) + (m2 == -INFINITY ? 0.f : s2 * ce_ratio(m2, mn));
    m = mn;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    sm_m[warp] = m;
    sm_s[warp] = s;
    sm_x[warp] = sx;
  }
  __syncthreads();
  if (warp == 0) {
    m = lane < CE_THREADS / 32 ? sm_m[lane] : -INFINITY;
    s = lane < CE_THREADS / 32 ? sm_s[lane] : 0.f;
    sx = lane < CE_THREADS / 32 ? sm_x[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float m2 = __shfl_xor_sync(0xffffffffu, m, o);
      float s2 = __shfl_xor_sync(0xffffffffu, s, o);
      sx += __shfl_xor_sync(0xffffffffu, sx, o);
      float mn = fmaxf(m, m2);
      s = (m == -INFINITY ? 0.f : s * ce_ratio(m, mn)) + (m2 == -INFINITY ? 0.f : s2 * ce_ratio(m2, mn));
      m = mn;
    }
    if (lane == 0) {
      bc[0] = m;
      bc[1] = s;
      bc[2] = sx;
    }
  }
  __syncthreads();
  m = bc[0];
  s = bc[1];
  sx = bc[2];
  mc = __fmul_rn(m, kL2E);
  const bool large = fabsf(m) >= CE_LARGE;
  if (large && fabsf(m) < INFINITY) {   // the same for all threads of the row
    float n = 0.f;
    for (int c = threadIdx.x; c < V; c += CE_THREADS) {
      const float f = __bfloat162float(x[c]);
      n += f == m ? 1.f : f < m ? 0.f : f;   // what is no number stays none
    }
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (lane == 0) sm_s[warp] = n;
    __syncthreads();
    s = 0.f;
    for (int w = 0; w < CE_THREADS / 32; ++w) s += sm_s[w];
  }
  // the bracket gives back what the rounding of mc took, so that m is rounded once, in the last addition
  const float lse = m + 0.6931471805599453f * (__log2f(s) + (large ? 0.f : fmaf(-m, kL2E, mc)));
  const bool valid = label >= 0 && label < V;
  if (threadIdx.x == 0) {
    float l = 0.f;
    if (valid) {
      const float xl = __bfloat162float(x[label]);
      l = (1.f - smoothing) * (lse - xl) + smoothing * (lse - sx / V);
    }
    loss[row] = l;
    if (lse_out) lse_out[row] = lse;
  }
  if (!write_grad) return;
  // Second pass: p = exp2(x * log2(e) - (m * log2(e) + log2(s))) with the packed bf16x2 exponential: two results per
  // MUFU instruction, and the result is stored as bf16 anyway. (With one fp32 exponential per element in each pass the
  // kernel was bound by the special-function unit, not by memory.) The label's column is rewritten in fp32 afterwards.
  const float g = valid ? gscale : 0.f;
  const float c = -(mc + __log2f(s));
  const uint32_t g2 = pack_bf16x2(g, g);
  const uint32_t ug2 = pack_bf16x2(-g * smoothing / V, -g * smoothing / V);
  const float xl = valid ? __bfloat162float(x[label]) : 0.f;
  __syncthreads();  // x[label] has been read by every thread before anyone overwrites it
  for (int i = threadIdx.x; i < nvec; i += CE_THREADS) {
    uint4 v = *reinterpret_cast<const uint4*>(x + i * 8);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 t = __bfloat1622float2(h[j]);
      const uint32_t e = ex2_bf16x2(pack_bf16x2_int(fmaf(t.x, kL2E, c), fmaf(t.y, kL2E, c)));
      asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(o[j]) : "r"(e), "r"(g2), "r"(ug2));
    }
    if (i * 8 + 8 > V) {  // the vector that straddles the end of the vocabulary, and the padding behind it
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (i * 8 + 2 * j >= V) o[j] = 0u;
        else if (i * 8 + 2 * j + 1 >= V) o[j] &= 0x0000ffffu;
      }
    }
    *reinterpret_cast<uint4*>(x + i * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  if (valid) {
    __syncthreads();
    if (threadIdx.x == 0) {
      const float pl = exp2f(large ? xl - m : fmaf(xl, kL2E, -mc)) / s;
      x[label] = __float2bfloat16((pl - smoothing / V - (1.f - smoothing)) * g);
    }
  }
}

// out[0] = number of labels >= 0, at least 1; out[1] = scale / out[0]. One CTA.
__global__ void __launch_bounds__(1024) ce_count_kernel(const int64_t* __restrict__ labels, int T, float scale, float* __restrict__ out) {
  __shared__ int red[32];
  int n = 0;
#pragma unroll 8
  for (int i = threadIdx.x; i < T; i += 1024) n += labels[i] >= 0 ? 1 : 0;
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = n;
  __syncthreads();
  if (threadIdx.x < 32) {
    n = __reduce_add_sync(0xffffffffu, red[threadIdx.x]);
    if (threadIdx.x == 0) {
      const float f = (float)(n < 1 ? 1 : n);
      out[0] = f;
      out[1] = __fdiv_rn(scale, f);
    }
  }
}

// out = sum(loss) / count. One CTA, one fixed order.
__global__ void __launch_bounds__(1024) ce_mean_kernel(const float* __restrict__ loss, int T, const float* __restrict__ count, float* __restrict__ out) {
  __shared__ float red[32];
  float s = 0.f;
#pragma unroll 8
  for (int i = threadIdx.x; i < T; i += 1024) s += loss[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = red[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) *out = __fdiv_rn(s, *count);
  }
}

// out = bf16(x * *scale), the factor in fp32 on the device. Bound by memory: 65536 x 768 in 31 us, 6.4 TB/s (widening, multiplying and
// rounding as three library kernels: 310 us).
__global__ void __launch_bounds__(256) scale_bf16_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ scale,
                                                         __nv_bfloat16* __restrict__ out, long n) {
  const float f = *scale;
  const long n8 = n / 8, stride = (long)gridDim.x * 256;
  for (long i = blockIdx.x * 256L + threadIdx.x; i < n8; i += stride) {
    const uint4 v = reinterpret_cast<const uint4*>(x)[i];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = pack_bf16x2(__uint_as_float(w[j] << 16) * f, __uint_as_float(w[j] & 0xffff0000u) * f);
    reinterpret_cast<uint4*>(out)[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
  if (blockIdx.x == 0 && threadIdx.x < n - n8 * 8) {
    const long i = n8 * 8 + threadIdx.x;
    out[i] = __float2bfloat16_rn(__bfloat162float(x[i]) * f);
  }
}

}  // namespace inv

using namespace inv;

extern "C" int inv_ce_count(const int64_t* labels, int T, float scale, float* out, void* stream) {
  ce_count_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(labels, T, scale, out);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}

extern "C" int inv_ce_mean(const float* loss, int T, const float* count, float* out, void* stream) {
  ce_mean_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(loss, T, count, out);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}

// x and out on 16 bytes, dense.
extern "C" int inv_scale_bf16(const void* x, const float* scale, void* out, long n, void* stream) {
  if (((uintptr_t)x | (uintptr_t)out) & 15) return -ERR_BAD_ARG;
  if (n <= 0) return 0;
  long g = (n / 8 + 255) / 256;
  g = g < 1 ? 1 : g > 148 * 16 ? 148 * 16 : g;
  scale_bf16_kernel<<<(int)g, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, scale, (__nv_bfloat16*)out, n);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}

extern "C" int inv_cross_entropy(void* logits, const int64_t* labels, float* loss, float* lse, int T, int V, int ld, float gscale,
                                 float smoothing, int write_grad, void* stream) {
  if (ld % 8 || V > ld) return -ERR_BAD_ARG;
  if (T <= 0) return 0;
  cross_entropy_kernel<<<T, CE_THREADS, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)logits, labels, loss, lse, V, ld, gscale, smoothing,
                                                                   write_grad);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}
