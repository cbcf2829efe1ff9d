// Warp-level pieces of the token-major activation quantisers (quantize.cu, rmsnorm.cu).
#pragma once

#include "common.cuh"

namespace b200moe {
namespace {

__device__ __forceinline__ void unpack8_bf16(const uint4& raw, float* out) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    out[2 * i] = __uint_as_float(w[i] << 16);
    out[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

// Up to 128 entries of a token's position list from entry k0 on, four per lane, fetched together; -1 = no position.
__device__ __forceinline__ void load_positions(const int32_t* __restrict__ map, int K, int k0, int lane, int64_t n_pos,
                                               int (&cand)[4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int k = k0 + c * 32 + lane;
    cand[c] = k < K ? map[k] : -1;
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
    if (cand[c] >= n_pos) cand[c] = -1;
}

// A warp quantises 256 columns, eight per lane (`raw`): the lane's eight code bytes and, in the lanes of each half
// warp, the four scale bytes of its 128 columns.  The four lanes l & ~3 .. l | 3 hold one 32-element block.  In packed
// order lane q of a block holds elements p * 4 + q (p = 0..7) and stores bytes 8q .. 8q + 7, i.e. byte pair
// (2q, 2q + 1) of every lane of its group.
__device__ __forceinline__ void quantize_quarter(const uint4& raw, int packed, int lane, bool inside, uint32_t& w0,
                                                 uint32_t& w1, uint32_t& cell) {
  float v[8];
  unpack8_bf16(raw, v);
  uint32_t mx = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) mx = max(mx, __float_as_uint(v[j]) & 0x7fffffffu);
  mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
  mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
  float f1, f2;
  mx_block_factors(mx, f1, f2);
  w0 = pack4_e4m3(v[0] * f1 * f2, v[1] * f1 * f2, v[2] * f1 * f2, v[3] * f1 * f2);
  w1 = pack4_e4m3(v[4] * f1 * f2, v[5] * f1 * f2, v[6] * f1 * f2, v[7] * f1 * f2);
  if (packed) {
    const int q = lane & 3;
    uint32_t o0 = 0, o1 = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const uint32_t a0 = __shfl_sync(0xffffffffu, w0, (lane & ~3) + s);
      const uint32_t a1 = __shfl_sync(0xffffffffu, w1, (lane & ~3) + s);
      const uint32_t x = ((q >= 2 ? a1 : a0) >> (16 * (q & 1))) & 0xffffu;
      o0 |= (x & 0xffu) << (8 * s);
      o1 |= (x >> 8) << (8 * s);
    }
    w0 = o0;
    w1 = o1;
  }
  cell = inside ? static_cast<uint32_t>(mx_block_scale_byte(mx)) << (8 * ((lane >> 2) & 3)) : 0u;
  cell |= __shfl_xor_sync(0xffffffffu, cell, 4);
  cell |= __shfl_xor_sync(0xffffffffu, cell, 8);
}

}  // namespace
}  // namespace b200moe
