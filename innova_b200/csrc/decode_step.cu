// The two ends of a greedy decode step. As operations of the framework around it they are a gather, a copy and an increment in front, an arg-max
// and two copies behind, 3 to 7 us each with their gaps: 33 of the 290 us of a step of one sequence (8 layers of width 2048).
#include "sm100_common.cuh"
#include "inv_api.h"

namespace inv {

// x[b, :] = emb[tokens[b], :], pos[b] = lens[b], lens[b] += 1. A token below zero counts from the end of the table, one outside it reads row 0
// and leaves ERR_BAD_ARG in *status. grid (pieces of a row, B); one thread a sequence moves its length.
__global__ void __launch_bounds__(256) step_begin_kernel(const int64_t* __restrict__ tokens, const uint4* __restrict__ emb, int row, int rows,
                                                         uint4* __restrict__ x, int* __restrict__ lens, int* __restrict__ pos, int* status) {
  const int b = blockIdx.y, i = blockIdx.x * 256 + threadIdx.x;
  if (i < row) {
    int64_t id = tokens[b];
    if (id < 0) id += rows;
    if (id < 0 || id >= rows) {
      if (i == 0 && status) atomicCAS(status, 0, ERR_BAD_ARG);
      id = 0;
    }
    x[(size_t)b * row + i] = emb[(size_t)id * row + i];
  }
  if (i == 0) {
    const int n = lens[b];
    pos[b] = n;
    lens[b] = n + 1;
  }
}

// The index of a row's largest value, the first of several, a NaN above all numbers (as torch.argmax), to next[b] and to out[b, lens[b] - base].
// One CTA a row: 8192 values in 2.6 us.
__global__ void __launch_bounds__(1024) step_next_kernel(const float* __restrict__ logits, long ld, int V, int64_t* __restrict__ next, int64_t* __restrict__ out,
                                                         int ld_out, const int* __restrict__ lens, int base) {
  __shared__ float s_v[32];
  __shared__ int s_i[32];
  const float* row = logits + blockIdx.x * ld;
  auto above = [](float a, int ia, float b, int ib) {      // (a, ia) is to be taken before (b, ib)
    const bool na = a != a, nb = b != b;
    if (na != nb) return na;
    return (!na && a != b) ? a > b : ia < ib;
  };
  float best = -INFINITY;
  int at = 0x7fffffff;
  for (int i0 = threadIdx.x; i0 < V; i0 += 4096) {
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = i0 + k * 1024 < V ? row[i0 + k * 1024] : -INFINITY;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = i0 + k * 1024;
      if (i < V && above(v[k], i, best, at)) {
        best = v[k];
        at = i;
      }
    }
  }
  auto fold = [&](int lanes) {
    for (int o = lanes >> 1; o > 0; o >>= 1) {
      const float v = __shfl_xor_sync(0xffffffffu, best, o);
      const int i = __shfl_xor_sync(0xffffffffu, at, o);
      if (above(v, i, best, at)) {
        best = v;
        at = i;
      }
    }
  };
  fold(32);
  if ((threadIdx.x & 31) == 0) {
    s_v[threadIdx.x >> 5] = best;
    s_i[threadIdx.x >> 5] = at;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  best = s_v[threadIdx.x];
  at = s_i[threadIdx.x];
  fold(32);
  if (threadIdx.x == 0) {
    next[blockIdx.x] = at;
    const int col = lens[blockIdx.x] - base;
    if (out && col >= 0 && col < ld_out) out[(size_t)blockIdx.x * ld_out + col] = at;
  }
}

}  // namespace inv

using namespace inv;

// emb: rows of row_bytes bytes (a multiple of 16) on 16 bytes; tokens int64 [B]; status may be null. Plainly launched.
extern "C" int inv_step_begin_checked(const void* tokens, const void* emb, int row_bytes, int rows, void* x, int* lens, int* pos, int B, int* status,
                                      void* stream) {
  if (row_bytes < 16 || row_bytes % 16 || rows < 1 || ((uintptr_t)emb | (uintptr_t)x) % 16) return -ERR_BAD_ARG;
  if (B <= 0) return 0;
  const int row = row_bytes / 16;
  for (int b0 = 0; b0 < B; b0 += 65535) {
    const int n = B - b0 < 65535 ? B - b0 : 65535;
    step_begin_kernel<<<dim3((row + 255) / 256, n), 256, 0, (cudaStream_t)stream>>>((const int64_t*)tokens + b0, (const uint4*)emb, row, rows,
                                                                                    (uint4*)x + (size_t)b0 * row, lens + b0, pos + b0, status);
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}
extern "C" int inv_step_begin(const void* tokens, const void* emb, int row_bytes, int rows, void* x, int* lens, int* pos, int B, void* stream) {
  return inv_step_begin_checked(tokens, emb, row_bytes, rows, x, lens, pos, B, nullptr, stream);
}

// logits fp32 [B, ld], V of each row; next int64 [B]; out int64 [B, ld_out] or null.
extern "C" int inv_step_next(const float* logits, long ld, int V, void* next, void* out, int ld_out, const int* lens, int base, int B, void* stream) {
  if (V < 1 || ld < V) return -ERR_BAD_ARG;
  if (B <= 0) return 0;
  step_next_kernel<<<B, 1024, 0, (cudaStream_t)stream>>>(logits, ld, V, (int64_t*)next, (int64_t*)out, ld_out, lens, base);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}
