// RMSNorm (optionally with a fused residual add) feeding the decode MoE block: one CTA per token row, fp32
// statistics, bf16 in and out.
#include "common.cuh"
#include "quantize_row.cuh"

namespace b200moe {
namespace {

struct NormArgs {
  const __nv_bfloat16* inp;
  const __nv_bfloat16* residual;
  const void* gamma;
  int gamma_dtype, H;
  float inv_count, eps;
  __nv_bfloat16* out;
  __nv_bfloat16* residual_out;
};

__device__ __forceinline__ uint32_t pack2_bf16(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Eight columns from `at` on (`n` of them exist) of bf16(inp + residual), inp alone without a residual; `vec` = 16-byte
// accesses.
__device__ __forceinline__ uint4 load_sum8(const NormArgs& a, int64_t at, int n, bool vec) {
  float x[8], r[8];
  if (vec) {
    const uint4 raw = *reinterpret_cast<const uint4*>(a.inp + at);
    if (a.residual == nullptr) return raw;
    unpack8_bf16(raw, x);
    unpack8_bf16(*reinterpret_cast<const uint4*>(a.residual + at), r);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      x[j] = j < n ? __bfloat162float(a.inp[at + j]) : 0.f;
      r[j] = j < n && a.residual != nullptr ? __bfloat162float(a.residual[at + j]) : 0.f;
    }
  }
  if (a.residual != nullptr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] += r[j];
  }
  return make_uint4(pack2_bf16(x[0], x[1]), pack2_bf16(x[2], x[3]), pack2_bf16(x[4], x[5]), pack2_bf16(x[6], x[7]));
}

// 1 / rms of a row, the same bits in every thread of the CTA: thread i sums the squares of columns 8 (i + blockDim j)
// .. + 7, then its warp, then the warps in order.  Both kernels below take it from here, so that the fused one writes
// the bytes the separate one does.
__device__ __forceinline__ float row_rinv(const NormArgs& a, int64_t base, bool vec) {
  __shared__ float s_part[32];
  float ss = 0.f;
  for (int h = threadIdx.x * 8; h < a.H; h += blockDim.x * 8) {
    float v[8];
    unpack8_bf16(load_sum8(a, base + h, a.H - h, vec), v);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = ss;
  __syncthreads();
  float total = 0.f;
  for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) total += s_part[w];
  return 1.0f / sqrtf(total * a.inv_count + a.eps);
}

// Normalises the eight columns from `h` on (the second read of the row comes from L1 / L2) and stores them, with the
// residual sum where it is asked for; returns the bf16 values.
__device__ __forceinline__ uint4 normalise8(const NormArgs& a, int64_t base, int h, float rinv, bool vec) {
  const int n = a.H - h;
  const uint4 sum = load_sum8(a, base + h, n, vec);
  float v[8];
  unpack8_bf16(sum, v);
  if (a.residual != nullptr && a.residual_out != nullptr) {
    if (vec) {
      *reinterpret_cast<uint4*>(a.residual_out + base + h) = sum;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < n) a.residual_out[base + h + j] = __float2bfloat16_rn(v[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] *= rinv;
    if (a.gamma != nullptr && j < n) v[j] *= load_as_float(a.gamma, h + j, a.gamma_dtype);
  }
  const uint4 o = make_uint4(pack2_bf16(v[0], v[1]), pack2_bf16(v[2], v[3]), pack2_bf16(v[4], v[5]), pack2_bf16(v[6], v[7]));
  if (vec) {
    *reinterpret_cast<uint4*>(a.out + base + h) = o;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < n) a.out[base + h + j] = __float2bfloat16_rn(v[j]);
  }
  return o;
}

// 16-byte accesses need every row of every tensor to start on a 16-byte boundary.
__device__ __forceinline__ bool rows_aligned(const NormArgs& a) {
  const uintptr_t bits = reinterpret_cast<uintptr_t>(a.inp) | reinterpret_cast<uintptr_t>(a.residual) |
                         reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.residual_out);
  return (bits & 15) == 0 && a.H % 8 == 0;
}

__global__ void __launch_bounds__(512) rmsnorm_kernel(NormArgs a) {
  grid_enter();
  const int64_t base = static_cast<int64_t>(blockIdx.x) * a.H;
  const bool vec = rows_aligned(a);
  const float rinv = row_rinv(a, base, vec);
  for (int h = threadIdx.x * 8; h < a.H; h += blockDim.x * 8) normalise8(a, base, h, rinv, vec);
}

// RMSNorm (+ residual) fused with the MXFP8 activation quantisation, for callers that know where every token's
// row goes before the router has run (all-expert decode: token t sits at position e * T_pad + t of every local
// expert e).  One CTA per token: the row's statistics, then each warp takes 256 columns at a time, writes the bf16
// row the router reads and quantises the same values to every position in the token's list -- the arithmetic and the
// stores of scatter_quantize_kernel, without the round trip of the normalised rows through HBM.
//
// A decode batch has few rows, so latency bounds it: a warp per token with 2-byte accesses kept 16 CTAs busy for
// 56 us at 128 tokens x 3072 columns and 16 positions each; a CTA per token with 16-byte accesses takes 8.8.
__global__ void __launch_bounds__(512) rmsnorm_quantize_kernel(NormArgs a, const int32_t* __restrict__ table, int K,
                                                               int64_t n_pos, int packed, uint8_t* __restrict__ codes,
                                                               uint8_t* __restrict__ sf,
                                                               int32_t* __restrict__ tile_flags) {
  grid_enter(table);
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x, H = a.H;
  const int64_t base = static_cast<int64_t>(t) * H;
  const int64_t k_atoms = (H + 127) >> 7;
  const int32_t* my_map = table + static_cast<int64_t>(t) * K;
  const bool vec = rows_aligned(a);
  int first[4];
  load_positions(my_map, K, 0, lane, n_pos, first);
  if (tile_flags != nullptr)
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
      const int p = my_map[k];
      if (p >= 0 && p < n_pos) atomicMax(&tile_flags[p >> 7], (p & 127) + 1);
    }
  const float rinv = row_rinv(a, base, vec);
  const int blk = lane >> 2, q = lane & 3;
  for (int c0 = (threadIdx.x >> 5) * 256; c0 < H; c0 += (blockDim.x >> 5) * 256) {
    const int col = c0 + lane * 8;  // position along the contraction axis the codes are stored at
    // packed order (reference-format weights): contraction position k' = t*512 + p*4 + q holds hidden column
    // q*(H/4) + t*128 + p; lane (blk, q) takes eight consecutive p of one q and the four lanes of a block trade
    // bytes afterwards, exactly as the stand-alone quantiser does
    const int kb = (c0 >> 5) + blk;
    const int src = packed ? q * (H >> 2) + (kb >> 4) * 128 + (kb & 15) * 8 : col;
    uint4 row = make_uint4(0, 0, 0, 0);
    if (col < H) row = normalise8(a, base, src, rinv, vec);
    uint32_t w0, w1, cell;
    quantize_quarter(row, packed, lane, col < H, w0, w1, cell);
    for (int k0 = 0; k0 < K; k0 += 128) {
      int cand[4] = {first[0], first[1], first[2], first[3]};
      if (k0 > 0) load_positions(my_map, K, k0, lane, n_pos, cand);
#pragma unroll
      for (int c = 0; c < 4; ++c)
        for (uint32_t left = __ballot_sync(0xffffffffu, cand[c] >= 0); left != 0u; left &= left - 1u) {
          const int64_t p = __shfl_sync(0xffffffffu, cand[c], __ffs(left) - 1);
          if (col >= H) continue;
          *reinterpret_cast<uint2*>(codes + p * H + col) = make_uint2(w0, w1);
          if ((lane & 15) == 0) *reinterpret_cast<uint32_t*>(sf + sf_atom_offset(p, col >> 5, k_atoms)) = cell;
        }
    }
  }
}

// A thread per eight columns, up to 16 warps.
int norm_threads(int H) {
  const int warps = (H + 255) / 256;
  return 32 * (warps < 16 ? warps : 16);
}

}  // namespace
}  // namespace b200moe

using namespace b200moe;

extern "C" int b200moe_rmsnorm_quantize_mxfp8(const void* inp_bf16, const void* residual_bf16, const void* gamma,
                                              int gamma_dtype, int T, int H, int hidden_actual, float eps,
                                              void* out_bf16, void* residual_out_bf16, const int32_t* table, int K,
                                              int64_t n_pos, int h_packed_order, uint8_t* codes, uint8_t* sf_atoms,
                                              int32_t* tile_flags, b200moe_stream_t stream) {
  B200MOE_REQUIRE(!h_packed_order || H % 512 == 0, B200MOE_ERR_INVALID,
                  "rmsnorm_quantize: the packed hidden order needs H %% 512 == 0, got %d", H);
  B200MOE_REQUIRE(inp_bf16 && out_bf16 && table && codes && sf_atoms && T > 0 && n_pos > 0 && K >= 1,
                  B200MOE_ERR_INVALID, "rmsnorm_quantize: bad arguments");
  B200MOE_REQUIRE(H > 0 && H % 128 == 0, B200MOE_ERR_INVALID,
                  "rmsnorm_quantize: H must be a positive multiple of 128, got %d", H);
  B200MOE_REQUIRE(gamma == nullptr || gamma_dtype == B200MOE_F32 || gamma_dtype == B200MOE_BF16, B200MOE_ERR_INVALID,
                  "rmsnorm_quantize: gamma must be fp32 or bf16");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (tile_flags != nullptr)
    B200MOE_CUDA_OK(cudaMemsetAsync(tile_flags, 0, static_cast<size_t>(ceil_div64(n_pos, 128)) * 4, st));
  const float inv_count = 1.0f / static_cast<float>(hidden_actual > 0 ? hidden_actual : H);
  const NormArgs a{static_cast<const __nv_bfloat16*>(inp_bf16), static_cast<const __nv_bfloat16*>(residual_bf16), gamma,
                   gamma_dtype, H, inv_count, eps, static_cast<__nv_bfloat16*>(out_bf16),
                   static_cast<__nv_bfloat16*>(residual_out_bf16)};
  B200MOE_CUDA_OK(launch_overlapped(rmsnorm_quantize_kernel, dim3(T), norm_threads(H), 0, st, a, table, K, n_pos,
                                    h_packed_order, codes, sf_atoms, tile_flags));
  B200MOE_LAUNCH_OK("rmsnorm_quantize_kernel");
  return B200MOE_OK;
}

extern "C" int b200moe_rmsnorm(const void* inp_bf16, const void* residual_bf16, const void* gamma, int gamma_dtype,
                               int T, int H, int hidden_actual, float eps, void* out_bf16, void* residual_out_bf16,
                               b200moe_stream_t stream) {
  B200MOE_REQUIRE(inp_bf16 && out_bf16 && T > 0 && H > 0, B200MOE_ERR_INVALID, "rmsnorm: bad arguments");
  B200MOE_REQUIRE(gamma == nullptr || gamma_dtype == B200MOE_F32 || gamma_dtype == B200MOE_BF16, B200MOE_ERR_INVALID,
                  "rmsnorm: gamma must be fp32 or bf16");
  const float inv_count = 1.0f / static_cast<float>(hidden_actual > 0 ? hidden_actual : H);
  const NormArgs a{static_cast<const __nv_bfloat16*>(inp_bf16), static_cast<const __nv_bfloat16*>(residual_bf16), gamma,
                   gamma_dtype, H, inv_count, eps, static_cast<__nv_bfloat16*>(out_bf16),
                   static_cast<__nv_bfloat16*>(residual_out_bf16)};
  B200MOE_CUDA_OK(launch_overlapped(rmsnorm_kernel, dim3(T), norm_threads(H), 0, static_cast<cudaStream_t>(stream), a));
  B200MOE_LAUNCH_OK("rmsnorm_kernel");
  return B200MOE_OK;
}
