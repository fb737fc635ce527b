// Expansion of the packed block-32 weight formats into bf16 pairs, shared by the tile and the skinny product.
#pragma once
#include "sm100_common.cuh"

namespace inv {

// Lookup table of the 4- and 8-bit formats in shared memory, 256 entries x 32 bank copies: entry e of lane l lives at
// lut[e * 32 + l], so that every lane reads its own bank whatever the indices are. OIL4: the bf16 pair (codebook[low nibble],
// codebook[high nibble]) of a byte; OIL8: one bf16. `t` of `n` threads (multiples of 8): eight write the 32 copies of an entry.
template <int BITS>
__device__ __forceinline__ void oil_lut_fill(uint32_t* lut, const float* cb, int t, int n) {
  for (int e = t >> 3; e < 256; e += n >> 3) {
    const uint32_t v = (BITS == 4) ? pack_bf16x2(cb[e & 15], cb[e >> 4]) : pack_bf16x2(cb[e], 0.f);
    *reinterpret_cast<uint4*>(lut + e * 32 + (t & 7) * 4) = make_uint4(v, v, v, v);
  }
}

// Entry `(w >> SHIFT) & 255` of lane `lane4 / 4`: the byte moves straight to its place in the address (128 bytes an entry), so that a
// lookup is a shift, a masked merge and the load where the table stands at a fixed address (22016 x 4096 at one token through the
// tile kernel: 37.6 -> 33.3 us).
template <int SHIFT>
__device__ __forceinline__ uint32_t oil_lookup(const uint32_t* lut, uint32_t w, uint32_t lane4) {
  const uint32_t at = ((SHIFT >= 7 ? w >> (SHIFT >= 7 ? SHIFT - 7 : 0) : w << (SHIFT < 7 ? 7 - SHIFT : 0)) & 0x7f80u) | lane4;
  return *reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(lut) + at);
}

// Expands one block of 32 weights (BITS words of indices) into 16 packed bf16 pairs, times the block's scale.
template <int BITS>
__device__ __forceinline__ void expand_block(const uint32_t* w, __nv_bfloat16 s, const uint32_t* lut, const float* cb, int lane, uint32_t* o) {
  const __nv_bfloat162 sc2 = __halves2bfloat162(s, s);
  const uint32_t lane4 = lane * 4;
  auto scaled = [&](uint32_t pair) {
    const __nv_bfloat162 v = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&pair), sc2);
    return *reinterpret_cast<const uint32_t*>(&v);
  };
  if (BITS == 2) {
    // 4-entry codebook (ternary {-1, 0, +1, 0} for SPARK / OIL1 weights, or the OIL2 levels): the four scaled
    // entries sit in one 64-bit register and every 2-bit code selects 16 bits of it
    const __nv_bfloat162 e01 = __hmul2(__floats2bfloat162_rn(cb[0], cb[1]), sc2);
    const __nv_bfloat162 e23 = __hmul2(__floats2bfloat162_rn(cb[2], cb[3]), sc2);
    const uint64_t tbl = (uint64_t)(*reinterpret_cast<const uint32_t*>(&e01)) | ((uint64_t)(*reinterpret_cast<const uint32_t*>(&e23)) << 32);
#pragma unroll
    for (int j = 0; j < 2; ++j) {  // a 32-bit word = 16 codes = 8 output pairs
      const uint32_t codes = w[j];
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const uint32_t lo = (uint32_t)(tbl >> (16 * ((codes >> (4 * b)) & 3))) & 0xffffu;
        const uint32_t hi = (uint32_t)(tbl >> (16 * ((codes >> (4 * b + 2)) & 3))) << 16;
        o[j * 8 + b] = lo | hi;
      }
    }
  } else if (BITS == 4) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o[j * 4] = scaled(oil_lookup<0>(lut, w[j], lane4));
      o[j * 4 + 1] = scaled(oil_lookup<8>(lut, w[j], lane4));
      o[j * 4 + 2] = scaled(oil_lookup<16>(lut, w[j], lane4));
      o[j * 4 + 3] = scaled(oil_lookup<24>(lut, w[j], lane4));
    }
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o[j * 2] = scaled(__byte_perm(oil_lookup<0>(lut, w[j], lane4), oil_lookup<8>(lut, w[j], lane4), 0x5410));
      o[j * 2 + 1] = scaled(__byte_perm(oil_lookup<16>(lut, w[j], lane4), oil_lookup<24>(lut, w[j], lane4), 0x5410));
    }
  }
}

}  // namespace inv
