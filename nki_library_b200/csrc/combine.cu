// Combine: out[t, :] = sum of the rows of y_pos that belong to token t, in a
// fixed (table) order, fp32 accumulation, one bf16 rounding.  Deterministic
// replacement for the reference's per-block read-modify-write of the output.
#include "common.cuh"

namespace b200moe {
namespace {

constexpr int kMaxCandidates = 8192;  // table width limit: the row list of one token lives in shared memory

// Bound by the y_pos rows it reads (32768 tokens x 4096 columns, top-8: 2.4 GB in 366 us, the copy rate).  A decode batch
// has too few tokens for that and sees the latency of a chain of loads instead: the list is fetched 128 entries at a time,
// ROWS rows are on their way before the first is added, and blockIdx.y spreads a token's columns over several CTAs when
// there are few tokens (cold caches; 3 tokens x 3072 columns, top-8: 10.4 -> 3.7 us; 128 tokens, 16 rows each:
// 17.4 -> 6.0 us).
template <int ROWS>
__global__ void __launch_bounds__(128) combine_kernel(const __nv_bfloat16* __restrict__ y_pos,
                                                      const int32_t* __restrict__ table, int T, int n_cand, int H,
                                                      __nv_bfloat16* __restrict__ out) {
  extern __shared__ int32_t s_rows[];  // n_cand entries: every candidate may be valid (all-expert decode)
  __shared__ int s_n;
  grid_enter(y_pos, table);
  const int t = blockIdx.x;
  if (threadIdx.x < 32) {
    int base = 0;
    for (int c0 = 0; c0 < n_cand; c0 += 128) {
      int32_t p[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = c0 + j * 32 + threadIdx.x;
        p[j] = c < n_cand ? table[static_cast<int64_t>(t) * n_cand + c] : -1;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned m = __ballot_sync(0xffffffffu, p[j] >= 0);
        if (p[j] >= 0) s_rows[base + __popc(m & ((1u << threadIdx.x) - 1u))] = p[j];
        base += __popc(m);
      }
    }
    if (threadIdx.x == 0) s_n = base;
  }
  __syncthreads();
  const int n = s_n;
  for (int h = (blockIdx.y * blockDim.x + threadIdx.x) * 8; h < H; h += gridDim.y * blockDim.x * 8) {
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int r0 = 0; r0 < n; r0 += ROWS) {
      uint4 raw[ROWS];
#pragma unroll
      for (int j = 0; j < ROWS; ++j)
        if (r0 + j < n) raw[j] = __ldg(reinterpret_cast<const uint4*>(y_pos + static_cast<int64_t>(s_rows[r0 + j]) * H + h));
#pragma unroll
      for (int j = 0; j < ROWS; ++j) {
        if (r0 + j >= n) break;
        const uint32_t w[4] = {raw[j].x, raw[j].y, raw[j].z, raw[j].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[2 * i] += __uint_as_float(w[i] << 16);
          acc[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
        }
      }
    }
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 v = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
      o[i] = *reinterpret_cast<const uint32_t*>(&v);
    }
    *reinterpret_cast<uint4*>(out + static_cast<int64_t>(t) * H + h) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

}  // namespace
}  // namespace b200moe

using namespace b200moe;

extern "C" int b200moe_combine(const void* y_pos_bf16, const int32_t* table, int T, int n_cand, int H, void* out_bf16,
                               b200moe_stream_t stream) {
  B200MOE_REQUIRE(y_pos_bf16 && table && out_bf16, B200MOE_ERR_INVALID, "combine: null pointer argument");
  B200MOE_REQUIRE(T > 0 && n_cand > 0 && H > 0 && H % 8 == 0, B200MOE_ERR_INVALID,
                  "combine: need T, n_cand > 0 and H %% 8 == 0");
  B200MOE_REQUIRE(n_cand <= kMaxCandidates, B200MOE_ERR_INVALID, "combine: at most %d candidates per row, got %d",
                  kMaxCandidates, n_cand);
  // A CTA covers 1024 columns at a time: one per token once the tokens alone give every SM several.  Then occupancy hides
  // the latency as well as loads in flight do, which cost registers (cold L2, 4096 tokens of two rows: 24.6 us with one
  // row at a time, 26.0 with four, 30.7 with eight; 2531 tokens of four rows of 64: 25.6 with two, 21.5 with four, 22.5
  // with eight; 32768 tokens of eight: 396, 366, 360).
  const bool many = T >= 8 * sm_count();
  const auto kernel = !many ? combine_kernel<8> : (n_cand <= 2 ? combine_kernel<1> : combine_kernel<4>);
  B200MOE_CUDA_OK(launch_overlapped(kernel, dim3(T, many ? 1 : (H + 1023) / 1024), 128,
                                    static_cast<size_t>(n_cand) * sizeof(int32_t), static_cast<cudaStream_t>(stream),
                                    static_cast<const __nv_bfloat16*>(y_pos_bf16), table, T, n_cand, H,
                                    static_cast<__nv_bfloat16*>(out_bf16)));
  B200MOE_LAUNCH_OK("combine_kernel");
  return B200MOE_OK;
}
