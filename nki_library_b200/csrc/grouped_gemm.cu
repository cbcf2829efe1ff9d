// Grouped MXFP8 expert contractions on the sm_100a tensor cores.
//
// The weights are the M operand and the tokens the N operand of every MMA: a tile is 128 weight rows (256 on a CTA
// pair, tcgen05 cta_group::2) times N tokens of one expert, N any multiple of 16 (32 on a pair) up to 128 (256).  An
// expert's tokens are therefore cut into tiles of nearly equal width without padding them to 128, and one launch
// covers every expert whatever its load.  With tokens as M (the earlier form of this kernel) an expert's last tile
// cost a full 128 or 256 rows, odd tiles needed a second launch that streamed the weights again, and the output rows
// left as 32-byte pieces.  Eager passes of the whole layer in a stream, earlier form -> this one: 4096 tokens, 8 experts of
// 4096 x 14336, top-2: 1544 -> 1411 us; 8192 tokens, 256 experts of 7168 x 2048, top-8, skewed: 4568 -> 4410; 2531 tokens,
// 64 experts of 3072 x 1536, top-4 (160 tokens per expert): 522 -> 351; 64 tokens on the first layer: 302 -> 287.
//
// What bounds it: with many tokens the L2 -> SM feed (a pair's tile of 256 x 256 needs 64 bytes per SM and tensor-pipe
// clock; about 48 arrive) and the power cap; with few tokens the stream of weights from HBM.
//
// Warp roles of a persistent CTA (512 threads):
//   warps 0, 3, 2  TMA producers: per 128-byte K slab the weight rows (0), the token rows (3; both 128B-swizzled) and
//               their UE8M0 scale atoms (2)
//   warp 1      allocates TMEM, issues four tcgen05.mma.kind::mxf8f6f4.block_scale (K = 32 each) per slab
//   warps 4..7  move each slab's scale atoms shared memory -> registers -> TMEM (tcgen05.st, one TMEM lane quadrant
//               per warp, one TMEM slot per pipeline stage); the same bytes through tcgen05.cp cost the tensor pipe
//               about 20 % of its cycles
//   warps 8..15 epilogue: two groups of four warps take alternate chunks of 32 tokens.  Each thread owns one weight
//               row (TMEM lane), pulls its part of the accumulator into registers, hands the TMEM buffer back, then
//               EPI 0: + bias, clamp per row; the chunk is turned around in shared memory so that a thread holds 16
//                      intermediates of one token: act(gate) * up in fp32, MXFP8 re-quantisation, codes + scales out
//               EPI 1: (+ bias) x routing affinity to bf16, turned around in shared memory likewise so that every
//                      token's 128 outputs leave as one 256-byte copy
// Tiles are walked expert by expert, weight tile by weight tile, token tile fastest: CTAs that run side by side share
// a weight tile in L2.  Blocks run up to the first zero in `conditions`.  Every mbarrier wait is bounded: on expiry
// the kernel records a code in `status`, stops issuing work and tears down.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "tcgen05_ptx.cuh"

namespace b200moe {
namespace {

constexpr int kBlockK = 128;  // bytes per pipeline slab (128 8-bit elements, 64 bf16)
constexpr int kGroupM = 16;
constexpr int kMaxExperts = 512;
constexpr int kThreads = 512;

struct GemmParams {
  const uint8_t* x_sf;
  const uint8_t* w_sf;
  int64_t w_sf_expert_stride;
  int w_row_atoms;  // scale atoms along the weight-row axis per expert
  const int32_t* block_to_expert;
  const int32_t* conditions;
  const int32_t* tile_flags;  // per 128-position tile: leading rows that can hold a token (NULL = all)
  const int32_t* tpi;
  int hidden_rows, n_blocks, B, E;
  int m_tiles_total, k_blocks;
  int n_total;  // weight rows per expert
  int max_n;    // tokens per tile at most
  const float* bias;
  int act;
  float gate_lo, gate_hi, up_lo, up_hi;
  uint8_t* m_codes;
  uint8_t* m_sf;
  int I;
  const void* aff;
  int aff_dtype;
  int aff_per_row;  // 0: table [rows, E] addressed tok*E + e; 1: vector [rows] addressed tok
  __nv_bfloat16* y_pos;
  int H_out;
  // expert parallelism: when row_src is set, row r of the result goes to row (row_src[r] & 0xffffff) of the buffer
  // peer_out[row_src[r] >> 24] (the GPU the token came from, over NVLink) instead of y_pos
  const int32_t* row_src;
  int64_t peer_rows;
  void* peer_out[8];
  int32_t* status;
  unsigned long long* clock_probe;  // optional: CTA 0 writes {SM cycles, nanoseconds} spent in the kernel
  const float* col_scale;  // dense (bf16) variant: per-expert, per-weight-row dequantisation factors [E, n_total]
                           // of fp8-row weights (NULL = none), applied to the accumulator before the bias
  int w_format;            // element format of the weight operand (B200MOE_W_*); activations are e4m3
  int w_slab_bytes;        // bytes of a weight row per slab that a copy reports (64 for 4-bit weights)
  int chained;             // launched while the kernel in front of it drains (see launch_tc)
};

// Per-CTA tile schedule, built once in shared memory.
struct Sched {
  int start[kMaxExperts + 1];  // token tiles before expert e
  int first_row[kMaxExperts];  // first position of expert e
  int rows[kMaxExperts];       // positions from there to its last token; negative: an inner 128-row tile is not full,
                               // and the expert is walked in windows of 128 positions instead
  int n_active;                // blocks before the first zero condition
  int contiguous;              // every expert's blocks are adjacent
  int h, w_tiles;              // weight rows per tile, tiles per expert
  int n_full, parts;           // tiles [0, n_full) are whole; each later index is one of `parts` equal row ranges of a
                               // tile that would not fill a last round of CTAs
  int total;                   // number of tiles to walk
  int stages, x_bytes;         // single CTA: pipeline depth and bytes of token rows per slab
};

__device__ __forceinline__ int round_up(int v, int m) { return (v + m - 1) / m * m; }

__device__ __forceinline__ int token_tiles(const GemmParams& p, int rows) {
  return rows < 0 ? (-rows + 127) >> 7 : (rows + p.max_n - 1) / p.max_n;
}

// CTAS 2: 256 weight rows per tile.  CTAS 1: 128, or fewer where that spreads the rows more evenly over the CTAs
// (a decode launch is bound by streaming weights, so its time is the largest number of rows any CTA gets): e.g. 8
// experts x 4096 rows on 148 CTAs are 1.73 rounds of 128-row tiles, but exactly two rounds of 112-row tiles.
//
// Everything read from global memory here is fetched at once into `scratch` (shared memory the pipeline will use
// later, `scratch_ints` long; larger problems read global memory again): the prologue costs one memory latency, which
// is what a decode launch of a few tens of microseconds notices.  (A chained launch reads before it waits: past L1.)
template <int CTAS, int EPI>
__device__ __forceinline__ void build_sched(const GemmParams& p, Sched& s, int n_units, int* scratch, int scratch_ints,
                                            int ring_bytes, int slab_fixed_bytes, int max_stages) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int sub = p.B >> 7;
  if (tid == 0) { s.n_active = p.n_blocks; s.contiguous = 1; }
  for (int e = tid; e < p.E; e += nthr) { s.first_row[e] = 0; s.rows[e] = 0; s.start[e] = 0; }
  __syncthreads();
  const bool staged = p.n_blocks + p.m_tiles_total <= scratch_ints;
  for (int b = tid; b < p.n_blocks; b += nthr) {
    const int e = staged ? __ldcg(p.block_to_expert + b) : 0;
    const int run = p.conditions != nullptr ? __ldcg(p.conditions + b) : 1;
    if (staged) scratch[b] = e;
    if (run == 0) atomicMin(&s.n_active, b);
  }
  const bool have_flags = p.tile_flags != nullptr;
  if (staged && have_flags)
    for (int t = tid; t < p.m_tiles_total; t += nthr) scratch[p.n_blocks + t] = __ldcg(p.tile_flags + t);
  const auto b2e = [&](int b) { return staged ? scratch[b] : __ldcg(p.block_to_expert + b); };
  const auto flags = [&](int t) { return staged ? scratch[p.n_blocks + t] : __ldcg(p.tile_flags + t); };
  __syncthreads();
  const int n_active = s.n_active;
  // start[] counts an expert's separate runs of blocks here, rows[] its 128-row tiles
  for (int b = tid; b < n_active; b += nthr) {
    const int e = b2e(b);
    if (e < 0 || e >= p.E) continue;
    if (b == 0 || b2e(b - 1) != e) {
      s.first_row[e] = b * p.B;
      if (atomicAdd(&s.start[e], 1) > 0) s.contiguous = 0;
    }
    atomicAdd(&s.rows[e], sub);
  }
  __syncthreads();
  const bool contiguous = s.contiguous;
  for (int e = tid; e < p.E && contiguous; e += nthr) {
    int live = s.rows[e], last = 128;
    if (have_flags && live > 0) {
      const int t0 = s.first_row[e] >> 7;
      while (live > 0 && (last = flags(t0 + live - 1)) == 0) --live;
    }
    s.rows[e] = live > 0 ? (live - 1) * 128 + last : 0;
  }
  __syncthreads();
  if (have_flags && contiguous) {
    for (int t = tid; t < n_active * sub; t += nthr) {
      if (flags(t) >= 128) continue;
      const int e = b2e(t / sub);
      if (e < 0 || e >= p.E) continue;
      const int r = s.rows[e], end = s.first_row[e] + (r < 0 ? -r : r);
      if ((t + 1) * 128 < end && r > 0) atomicMin(&s.rows[e], -r);
    }
    __syncthreads();
  }
  if (tid < 32) {
    int run = 0, widest = 0;
    for (int e0 = 0; e0 < p.E; e0 += 32) {
      const int e = e0 + tid;
      const int rows = e < p.E ? s.rows[e] : 0;
      const int own = token_tiles(p, rows);
      if (rows != 0) widest = max(widest, rows < 0 ? 128 : (rows + own - 1) / own);
      int v = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (tid >= o) v += u;
      }
      if (e < p.E) s.start[e] = run + v - own;
      run += __shfl_sync(0xffffffffu, v, 31);
    }
    widest = contiguous ? static_cast<int>(__reduce_max_sync(0xffffffffu, static_cast<uint32_t>(widest))) : 128;
    const int tok_tiles = contiguous ? run : n_active * sub;
    int h = 128 * CTAS, parts = 1, stages = max_stages, x_bytes = 0;
    if constexpr (CTAS == 1) {
      // one candidate height per lane: 128, 128 - kGran, ... (MX blocks of 32 intermediates need whole groups of 32
      // gate and 32 up rows).  Heights under 96 keep too few bytes in flight and are only taken when they leave
      // far fewer rows on the fullest CTA.
      constexpr int kGran = EPI == 0 ? 64 : 16;
      const int c = 128 - tid * kGran;
      uint32_t key = 0xffffffffu;
      if (c >= (EPI == 0 ? 64 : 32)) {
        const int tiles = tok_tiles * ((p.n_total + c - 1) / c);
        const int whole = tiles / n_units, rest = tiles - whole * n_units;
        int cut = 1;
        if (rest > 0)
          for (int q = 2; q * kGran <= c && rest * q <= n_units; ++q)
            if (c % (q * kGran) == 0) cut = q;
        const int cost = whole * max(c, 88) + (rest > 0 ? c / cut : 0);
        key = (static_cast<uint32_t>(min(cost, 0x3fffff)) << 10) | static_cast<uint32_t>(tid << 5) | static_cast<uint32_t>(cut);
      }
      key = __reduce_min_sync(0xffffffffu, key);
      h = 128 - static_cast<int>((key >> 5) & 31) * kGran;
      parts = static_cast<int>(key & 31);
      // narrow token tiles leave room for a deeper ring of weight slabs
      x_bytes = max(round_up(widest, 16), 16) * kBlockK;
      stages = min(max_stages, ring_bytes / (x_bytes + slab_fixed_bytes));
    }
    if (tid == 0) {
      s.start[p.E] = run;
      s.h = h;
      s.w_tiles = (p.n_total + h - 1) / h;
      s.parts = parts;
      s.stages = stages;
      s.x_bytes = x_bytes;
      const int tiles = tok_tiles * s.w_tiles;
      s.n_full = parts > 1 ? tiles / n_units * n_units : tiles;
      s.total = s.n_full + (tiles - s.n_full) * parts;
    }
  }
  __syncthreads();
}

// A tile: token rows [row0, row0 + n) of the position axis, weight rows [w_row0, w_row0 + w_rows) of `expert`.
struct TileRec {
  int row0, w_row0, expert;
  int shape;  // bits 0-9 n, bits 10-19 w_rows; 0 = nothing to do
  __device__ __forceinline__ int n() const { return shape & 1023; }
  __device__ __forceinline__ int w_rows() const { return shape >> 10; }
};

template <int CTAS>
__device__ __forceinline__ TileRec decode_tile(const GemmParams& p, const Sched& s, int tile) {
  constexpr int kStepN = CTAS == 2 ? 32 : 16;
  int sub_part = 0;
  bool cut = false;
  if (tile >= s.n_full) {
    cut = true;
    sub_part = (tile - s.n_full) % s.parts;
    tile = s.n_full + (tile - s.n_full) / s.parts;
  }
  int e, w_tile, row0, n;
  if (s.contiguous) {
    int lo = 0, hi = p.E;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s.start[mid] * s.w_tiles <= tile) lo = mid; else hi = mid;
    }
    e = lo;
    const int local = tile - s.start[e] * s.w_tiles;
    const int cnt = s.start[e + 1] - s.start[e];
    const int t = local % cnt;
    w_tile = local / cnt;
    const int rows = s.rows[e];
    if (rows < 0) {
      row0 = s.first_row[e] + t * 128;
      n = __ldcg(p.tile_flags + (row0 >> 7));
      if (n > p.max_n) n = p.max_n;  // (max_n is at least 128)
    } else {
      const int width = round_up((rows + cnt - 1) / cnt, kStepN);
      row0 = s.first_row[e] + t * width;
      n = min(width, rows - t * width);
    }
  } else {
    // scattered blocks: one tile per 128 positions, in the given order
    const int units = s.n_active * (p.B >> 7);
    const int per_group = kGroupM * s.w_tiles;
    const int g = tile / per_group;
    const int first = g * kGroupM;
    const int gs = min(kGroupM, units - first);
    const int within = tile - g * per_group;
    const int m_tile = first + within % gs;
    w_tile = within / gs;
    e = __ldcg(p.block_to_expert + m_tile / (p.B >> 7));
    row0 = m_tile * 128;
    n = (e < 0 || e >= p.E) ? 0 : (p.tile_flags ? __ldcg(p.tile_flags + m_tile) : 128);
  }
  const int h = cut ? s.h / s.parts : s.h;
  const int w_row0 = w_tile * s.h + sub_part * h;
  const int w_rows = min(h, p.n_total - w_row0);
  if (n <= 0 || w_rows <= 0) return TileRec{0, 0, 0, 0};
  return TileRec{row0, w_row0, e, round_up(n, kStepN) | (w_rows << 10)};
}

// A CTA's own tiles, decoded once in the prologue by all threads (the decode -- a search over the experts, divisions,
// tile_flags reads -- costs about a thousand clocks, which the MMA-issuing thread would otherwise spend at every tile
// boundary with the tensor pipe idle); tiles past the table are decoded on the spot.
constexpr int kTileTable = 256;

template <int CTAS>
__device__ __forceinline__ TileRec fetch_tile(const GemmParams& p, const Sched& s, const TileRec* table, int it, int tile) {
  if (it < kTileTable) {
    const int4 r = *reinterpret_cast<const int4*>(table + it);
    return TileRec{r.x, r.y, r.z, r.w};
  }
  return decode_tile<CTAS>(p, s, tile);
}

// Chunk buffer of the gate/up epilogue: 32 tokens x 128 weight rows of fp32, token-major.  Rows 64.. sit 8 words
// further on and a token's row is 140 words, so that the 16-byte reads of eight neighbouring threads (two tokens x
// four row ranges) touch 32 different banks, as do the 4-byte writes of 32 neighbouring rows.
constexpr int kTurnPitch = 140;
constexpr int kTurnBytes = 32 * kTurnPitch * 4;
// The down epilogue's: 32 tokens x 128 output columns of bf16, a token's row 272 bytes so that the eight 16-byte rows of
// a transposing matrix store touch 32 different banks; two buffers, so that one is filled while the other is copied out.
constexpr int kRowPitch = 272;
constexpr int kRowBytes = 32 * kRowPitch;

template <int EPI, int CTAS>
struct SmemLayout {
  static constexpr int kMaxN = CTAS == 2 ? 256 : 128;
  static constexpr int kMaxStages = CTAS == 2 ? 5 : 8;
  static constexpr int kW = 128 * kBlockK;
  static constexpr int kX = (kMaxN / CTAS) * kBlockK;  // a CTA pair splits the token rows
  static constexpr int kSfwAtoms = CTAS == 2 ? 1 : 2;  // weight rows of a single CTA may start inside an atom
  static constexpr int kSfxAtoms = kMaxN / 128 + 1;    // so may token rows
  static constexpr int kSf = (kSfwAtoms + kSfxAtoms) * 512;
  static constexpr int kRing = CTAS == 2 ? kMaxStages * (kW + kX + kSf) : 180 * 1024;
  // per epilogue group: the chunk buffer(s); EPI 1 also the affinity and the destination row of each of its tokens
  static constexpr int kGroup = EPI == 0 ? kTurnBytes : 2 * kRowBytes + (kMaxN / 2) * 8;
  static constexpr int kOffEpi = kRing;
  static constexpr int kOffBar = kOffEpi + 2 * kGroup;
  static constexpr int kOffSched = kOffBar + 384;
  static constexpr int kOffTiles = (kOffSched + static_cast<int>(sizeof(Sched)) + 15) & ~15;
  static constexpr int kBytes = kOffTiles + kTileTable * static_cast<int>(sizeof(TileRec)) + 1024;  // + alignment slack
  static_assert(kGroup % 16 == 0 && kRing % 1024 == 0, "alignment of the epilogue buffers");
};

// Two accumulators of 224 columns (single CTA: 128), used in turn, so that a tile's MMAs run while the epilogue drains
// the one before; a tile of more than 224 tokens takes both.  The MMA issuer and the epilogue walk the same sequence.
struct AccCursor {
  uint32_t taken[2] = {0, 0}, filled[2] = {0, 0};  // phase parities of tmem_empty / tmem_full
  int next = 0;
  __device__ __forceinline__ int begin(bool wide) { return wide ? 0 : next; }
  __device__ __forceinline__ void end(bool wide) {
    if (wide) {
      taken[0] ^= 1u;
      taken[1] ^= 1u;
      filled[0] ^= 1u;
      next = 0;
    } else {
      if (next == 0) { taken[0] ^= 1u; filled[0] ^= 1u; }
      else { taken[1] ^= 1u; filled[1] ^= 1u; }
      next ^= 1;
    }
  }
};

__device__ __forceinline__ void group_barrier(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }
// All 128 threads of an epilogue group agree whether the wait succeeded.
__device__ __forceinline__ bool group_all(int id, bool ok) {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.b32 p, %1, 0;\n"
      "bar.red.and.pred q, %2, 128, p;\n"
      "selp.u32 %0, 1, 0, q;\n"
      "}\n"
      : "=r"(r)
      : "r"(ok ? 1 : 0), "r"(id)
      : "memory");
  return r != 0;
}

constexpr float kLog2E = 1.4426950408889634f;
__device__ __forceinline__ float ex2_approx_ftz(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_approx_ftz(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// The largest magnitude of three; a NaN among them gives a NaN, whose exponent is the largest there is.
__device__ __forceinline__ float max3_abs_nan(float a, float b, float c) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// Two products / sums in one instruction, each rounded as the single ones are.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(r))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(r))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return r;
}

// act(gate) * up for 16 intermediates of one token; returns the largest |product| as bits.
//
// With short contractions the gate/up launch is bound by this epilogue: two warps per scheduler, waiting for one another at
// every turn of a chunk.  So SiLU, gate * 1 / (1 + 2^(-gate log2 e)), works in pairs (Blackwell's two-wide fp32 products) on
// the flush-to-zero forms of the two approximations; what they flush vanishes beside the 1 or is 0 either way: the quotient has the same bits as __fdividef(gate, 1 + __expf(-gate)) for all 2^32 gates.  It also has
// kernels of its own: with the other activations' code between its own in the unrolled chunks it ran 20 % longer.
// 512 hidden columns, 64 experts of 4096 intermediates, 16384 tokens, top-4, gate/up launch: 754 us with single products,
// the four activations in one kernel and bias and clamp applied whether there are any or not, 512 like this.
template <bool SILU>
__device__ __forceinline__ uint32_t swiglu16(float (&g)[16], const float (&u)[16], int act) {
  const auto each = [&](auto f) {
#pragma unroll
    for (int j = 0; j < 16; ++j) g[j] = f(g[j]) * u[j];
  };
  if constexpr (SILU) {
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      const float2 x = make_float2(g[j], g[j + 1]);
      const float2 y = mul2(x, make_float2(-kLog2E, -kLog2E));
      const float2 d = add2(make_float2(1.0f, 1.0f), make_float2(ex2_approx_ftz(y.x), ex2_approx_ftz(y.y)));
      const float2 m = mul2(mul2(x, make_float2(rcp_approx_ftz(d.x), rcp_approx_ftz(d.y))), make_float2(u[j], u[j + 1]));
      g[j] = m.x;
      g[j + 1] = m.y;
    }
  } else if (act == B200MOE_ACT_SWISH) each([](float x) { return apply_act(x, B200MOE_ACT_SWISH); });
  else if (act == B200MOE_ACT_GELU) each([](float x) { return apply_act(x, B200MOE_ACT_GELU); });
  else each([](float x) { return apply_act(x, B200MOE_ACT_GELU_TANH); });
  float mx = max3_abs_nan(0.0f, g[0], g[1]);
#pragma unroll
  for (int j = 2; j < 16; j += 2) mx = max3_abs_nan(mx, g[j], g[j + 1]);
  return __float_as_uint(mx);
}

// KIND 0: MXFP8 activations x MX weights, block-scaled MMAs (kind::mxf8f6f4.block_scale).
// KIND 1: bf16 activations x bf16 weights (kind::f16), the reference's non-MX variants: no scale atoms travel, the
//         four scale-mover warps idle, the gate/up epilogue writes bf16 intermediates instead of MX codes.  Operand
//         rows are addressed in bytes, so a 128-byte slab is 64 bf16 elements = four K = 16 MMAs.
// CTAS 2: the two CTAs of a cluster form one tcgen05 cta_group::2 unit.  Each loads its own 128 weight rows and half of
//         the token rows; the even CTA issues M = 256 MMAs that read both CTAs' shared memory and write both CTAs'
//         TMEM, so a token row crosses L2 -> SM once per 256 weight rows.
struct WeightMaps { CUtensorMap rows128, rows64, rows32, rows16; };
struct TokenMaps { CUtensorMap rows128, rows64, rows32, rows16; };

template <int EPI, int CTAS, int KIND, bool SILU>
__global__ void __launch_bounds__(kThreads, 1)
grouped_mxfp8_gemm_kernel(const __grid_constant__ WeightMaps wmap, const __grid_constant__ TokenMaps xmap,
                          const __grid_constant__ CUtensorMap sfw_map, const __grid_constant__ CUtensorMap sfx_map,
                          const GemmParams p) {
  using L = SmemLayout<EPI, CTAS>;
  constexpr int kMaxStages = L::kMaxStages;
  constexpr int kChunks = L::kMaxN / 64;   // 32-token chunks per epilogue group
  constexpr int kAccStride = CTAS == 2 ? 224 : 128;
  constexpr int kSfCol = 448;              // TMEM columns: accumulators, then per stage 4 of weight and 4 / 8 of token scales
  constexpr int kSfSlot = CTAS == 2 ? 12 : 8;
  static_assert(kSfCol + kMaxStages * kSfSlot <= 512, "scale slots exceed TMEM");
  constexpr uint32_t kTmemCols = 512;
  // M is fixed; N is or-ed in per tile
  const uint32_t idesc_base = KIND == 0 ? (make_idesc(128 * CTAS, 0) | (static_cast<uint32_t>(p.w_format) << 7))
                                        : make_idesc_bf16(128 * CTAS, 0);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* full = bars;
  uint64_t* empty = bars + kMaxStages;
  uint64_t* sf_full = bars + 2 * kMaxStages;   // scale atoms of a stage landed (per CTA)
  uint64_t* sf_ready = bars + 3 * kMaxStages;  // ... and sit in their TMEM slot (pair leader)
  uint64_t* tmem_full = bars + 4 * kMaxStages;
  uint64_t* tmem_empty = bars + 4 * kMaxStages + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + 4 * kMaxStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);
  Sched& sched = *reinterpret_cast<Sched*>(smem + L::kOffSched);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // warp-uniform to the compiler
  const int lane = threadIdx.x & 31;
  long long probe_c0 = 0;
  unsigned long long probe_t0 = 0;
  if (p.clock_probe != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
    probe_c0 = clock64();
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(probe_t0));
  }
  const int cta_rank = CTAS == 2 ? static_cast<int>(cluster_cta_rank()) : 0;
  const int unit = blockIdx.x / CTAS, n_units = gridDim.x / CTAS;
  // cleared here and not by a memset node in front of every launch: a wait that reports expires after seconds
  if (blockIdx.x == 0 && threadIdx.x == 0) *p.status = 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
      mbar_init(&sf_full[s], 1);
      mbar_init(&sf_ready[s], 4 * CTAS);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], 8 * CTAS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    if constexpr (CTAS == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr)),
                   "r"(kTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr)),
                   "r"(kTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  build_sched<CTAS, EPI>(p, sched, n_units, reinterpret_cast<int*>(smem), L::kRing / 4, L::kRing, L::kW + L::kSf, kMaxStages);
  const int total_tiles = sched.total;
  const int stages = CTAS == 2 ? kMaxStages : sched.stages;
  const int x_stage = CTAS == 2 ? L::kX : sched.x_bytes;
  const int off_x = stages * L::kW, off_sf = off_x + stages * x_stage;
  TileRec* tile_table = reinterpret_cast<TileRec*>(smem + L::kOffTiles);
  for (int i = threadIdx.x; i < kTileTable; i += kThreads) {
    const int tile = unit + i * n_units;
    if (tile < total_tiles) tile_table[i] = decode_tile<CTAS>(p, sched, tile);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the prologue's scratch becomes the copies' target
  tc_fence_before();
  __syncthreads();
  if constexpr (CTAS == 2) cluster_sync_all();  // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;

  // Register budget per warpgroup (4 warps): the epilogue warps hold up to 128 accumulator values per thread,
  // everyone else needs few.  512 threads x 128 at launch = 2 x 128 x 64 + 2 x 128 x 192.
  if (warp < 4) {
    reg_dec<64>();
    // Each of these warps walks its loop as a whole, with warp-uniform values, and one elected lane issues: a lone
    // thread pays about a hundred clocks per copy for moving the operands of one instruction into uniform registers,
    // and three copies' worth per slab more than the slab's MMAs take, which is why the copies have three warps.
    const bool leader = elect_one();
    if (warp != 1) {
      // ---------------------------------------------------------- TMA producers
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      // weights do not depend on the launch in front, the token rows and their scales do
      if (p.chained && warp != 0) grid_wait();
      // not before the launch in front is complete: the next one reads more than this one before it waits
      if (warp == 3) grid_launch_dependents();
      for (int tile = unit, it = 0; tile < total_tiles && ok; tile += n_units, ++it) {
        const TileRec r = fetch_tile<CTAS>(p, sched, tile_table, it, tile);
        if (r.shape == 0 || (KIND != 0 && warp == 2)) continue;
        const int w_row0 = r.w_row0 + cta_rank * 128;
        // a pair always copies 2 x 128 weight rows (rows past the end read as zero)
        const int w_copy = CTAS == 2 ? 128 : round_up(r.w_rows(), 16);
        if (warp == 0) {
          // weight rows; the even CTA's barrier counts both CTAs' operand bytes of a pair
          const uint32_t stage_bytes = static_cast<uint32_t>(CTAS * w_copy * p.w_slab_bytes + r.n() * kBlockK);
          for (int kb = 0; kb < p.k_blocks; ++kb) {
            if (!mbar_wait(&empty[stage], phase ^ 1u, abort_flag, p.status, 1)) { ok = false; break; }
            uint8_t* ws = smem + stage * L::kW;
            if (leader) {
              if (cta_rank == 0) mbar_expect_tx(&full[stage], stage_bytes);
              if constexpr (CTAS == 2) {
                tma2_load_3d(ws, &wmap.rows128, kb * kBlockK, w_row0, r.expert, &full[stage]);
              } else if (w_copy == 128) {
                tma_load_3d(ws, &wmap.rows128, kb * kBlockK, w_row0, r.expert, &full[stage]);
              } else {
                int at = 0;
                if (w_copy & 64) { tma_load_3d(ws, &wmap.rows64, kb * kBlockK, w_row0, r.expert, &full[stage]); at = 64; }
                if (w_copy & 32) { tma_load_3d(ws + at * kBlockK, &wmap.rows32, kb * kBlockK, w_row0 + at, r.expert, &full[stage]); at += 32; }
                if (w_copy & 16) tma_load_3d(ws + at * kBlockK, &wmap.rows16, kb * kBlockK, w_row0 + at, r.expert, &full[stage]);
              }
            }
            if (++stage == stages) { stage = 0; phase ^= 1u; }
          }
        } else if (warp == 3) {
          // token rows
          const int n_cta = r.n() / CTAS, x_row0 = r.row0 + cta_rank * n_cta;
          for (int kb = 0; kb < p.k_blocks; ++kb) {
            if (!mbar_wait(&empty[stage], phase ^ 1u, abort_flag, p.status, 1)) { ok = false; break; }
            uint8_t* xs = smem + off_x + stage * x_stage;
            if (leader) {
              auto load_x = [&](const CUtensorMap& map, int at) {
                if constexpr (CTAS == 2) tma2_load_2d(xs + at * kBlockK, &map, kb * kBlockK, x_row0 + at, &full[stage]);
                else tma_load_2d(xs + at * kBlockK, &map, kb * kBlockK, x_row0 + at, &full[stage]);
              };
              int at = 0;
              if (n_cta & 128) { load_x(xmap.rows128, 0); at = 128; }
              if (n_cta & 64) { load_x(xmap.rows64, at); at += 64; }
              if (n_cta & 32) { load_x(xmap.rows32, at); at += 32; }
              if (n_cta & 16) load_x(xmap.rows16, at);
            }
            if (++stage == stages) { stage = 0; phase ^= 1u; }
          }
        } else {
          // scale atoms of this CTA's weight rows and of all the tile's tokens -> this CTA's own barrier
          // (atoms past the end of the table read as zero and still count their bytes)
          const int x_atom0 = r.row0 >> 7, x_atoms = ((r.row0 + r.n() - 1) >> 7) - x_atom0 + 1;
          const int w_atom0 = w_row0 >> 7;
          const int w_atoms = CTAS == 2 ? 1 : ((w_row0 + w_copy - 1) >> 7) - w_atom0 + 1;
          const int w_first = (r.expert * p.w_row_atoms + w_atom0) * p.k_blocks, x_first = x_atom0 * p.k_blocks;
          for (int kb = 0; kb < p.k_blocks; ++kb) {
            if (!mbar_wait(&empty[stage], phase ^ 1u, abort_flag, p.status, 1)) { ok = false; break; }
            uint8_t* sf = smem + off_sf + stage * L::kSf;
            if (leader) {
              mbar_expect_tx(&sf_full[stage], static_cast<uint32_t>(w_atoms + x_atoms) * 512);
              tma_load_2d(sf, &sfw_map, 0, w_first + kb, &sf_full[stage]);
              if (L::kSfwAtoms > 1 && w_atoms > 1) tma_load_2d(sf + 512, &sfw_map, 0, w_first + p.k_blocks + kb, &sf_full[stage]);
              sf += L::kSfwAtoms * 512;
              tma_load_2d(sf, &sfx_map, 0, x_first + kb, &sf_full[stage]);
              if (x_atoms > 1) tma_load_2d(sf + 512, &sfx_map, 0, x_first + p.k_blocks + kb, &sf_full[stage]);
              if (L::kSfxAtoms > 2 && x_atoms > 2)
                tma_load_2d(sf + 1024, &sfx_map, 0, x_first + 2 * p.k_blocks + kb, &sf_full[stage]);
            }
            if (++stage == stages) { stage = 0; phase ^= 1u; }
          }
        }
      }
      if (!ok) {
        // let copies already in flight land before the CTA retires
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
      }
    } else if (cta_rank == 0) {
      // ---------------------------------------------------------- MMA issuer (even CTA only when paired)
      int stage = 0;
      uint32_t phase = 0;
      AccCursor cur;
      bool ok = true;
      for (int tile = unit, it = 0; tile < total_tiles && ok; tile += n_units, ++it) {
        const TileRec r = fetch_tile<CTAS>(p, sched, tile_table, it, tile);
        if (r.shape == 0) continue;
        const bool wide = r.n() > kAccStride;
        const int acc = cur.begin(wide);
        if (!mbar_wait(&tmem_empty[acc], (acc ? cur.taken[1] : cur.taken[0]) ^ 1u, abort_flag, p.status, 2)) break;
        if (wide && !mbar_wait(&tmem_empty[1], cur.taken[1] ^ 1u, abort_flag, p.status, 2)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * kAccStride;
        const uint32_t idesc_tile = idesc_base | (static_cast<uint32_t>(r.n() >> 3) << 17);
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!mbar_wait(&full[stage], phase, abort_flag, p.status, 3)) { ok = false; break; }
          if constexpr (KIND == 0)
            if (!mbar_wait(&sf_ready[stage], phase, abort_flag, p.status, 5)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sfw_tmem = tmem_base + kSfCol + stage * kSfSlot;
          const uint32_t sfx_tmem = sfw_tmem + 4;
          const uint64_t w_desc = desc_sw128(smem_u32(smem + stage * L::kW));
          const uint64_t x_desc = desc_sw128(smem_u32(smem + off_x + stage * x_stage));
          if (leader) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint32_t accumulate = (kb | k) != 0 ? 1u : 0u;
              if constexpr (KIND == 0) {
                const uint32_t idesc = idesc_tile | (static_cast<uint32_t>(k) << 29) | (static_cast<uint32_t>(k) << 4);
                if constexpr (CTAS == 2) tc2_mma_mxf8(d_tmem, w_desc + 2 * k, x_desc + 2 * k, idesc, sfw_tmem, sfx_tmem, accumulate);
                else tc_mma_mxf8(d_tmem, w_desc + 2 * k, x_desc + 2 * k, idesc, sfw_tmem, sfx_tmem, accumulate);
              } else {
                if constexpr (CTAS == 2) tc2_mma_bf16(d_tmem, w_desc + 2 * k, x_desc + 2 * k, idesc_tile, accumulate);
                else tc_mma_bf16(d_tmem, w_desc + 2 * k, x_desc + 2 * k, idesc_tile, accumulate);
              }
            }
            if constexpr (CTAS == 2) tc2_commit_pair(&empty[stage]);
            else tc_commit(&empty[stage]);
          }
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        if (ok && leader) {
          if constexpr (CTAS == 2) tc2_commit_pair(&tmem_full[acc]);
          else tc_commit(&tmem_full[acc]);
        }
        cur.end(wide);
      }
    }
  } else if (warp < 8) {
    reg_dec<64>();
    // ------------------------------------------------------------ scale-factor movers (one TMEM lane quadrant each)
    // Row r of an atom sits at byte (r % 32) * 16 + (r / 32) * 4 and belongs in TMEM lane r % 32, column r / 32: for
    // rows that start on an atom boundary the 16 bytes at lane * 16 are a lane's four columns.  Token rows start at
    // any multiple of 32 (columns shift), on a single CTA any multiple of 16, like its weight rows (lanes turn too).
    const int q = warp & 3;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = unit, it = 0; KIND == 0 && tile < total_tiles && ok; tile += n_units, ++it) {
      const TileRec r = fetch_tile<CTAS>(p, sched, tile_table, it, tile);
      if (r.shape == 0) continue;
      const int x_off = r.row0 & 127, w_off = CTAS == 2 ? 0 : r.w_row0 & 127;
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        if (!mbar_wait(&sf_full[stage], phase, abort_flag, p.status, 6)) { ok = false; break; }
        const uint8_t* sf = smem + off_sf + stage * L::kSf;
        const uint8_t* sfx = sf + L::kSfwAtoms * 512;
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + kSfCol + stage * kSfSlot;
        auto turned = [&](const uint8_t* atoms, int off, int group) {  // four columns from row off + 32 * group
          uint32_t v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int row = off + lane + 32 * (group + j);
            v[j] = *reinterpret_cast<const uint32_t*>(atoms + (row >> 7) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4);
          }
          return make_uint4(v[0], v[1], v[2], v[3]);
        };
        if (w_off == 0) tc_st4(taddr, *reinterpret_cast<const uint4*>(sf + lane * 16));
        else tc_st4(taddr, turned(sf, w_off, 0));
        if (x_off == 0) {
          tc_st4(taddr + 4, *reinterpret_cast<const uint4*>(sfx + lane * 16));
          if constexpr (CTAS == 2) tc_st4(taddr + 8, *reinterpret_cast<const uint4*>(sfx + 512 + lane * 16));
        } else {
          tc_st4(taddr + 4, turned(sfx, x_off, 0));
          if constexpr (CTAS == 2) tc_st4(taddr + 8, turned(sfx, x_off, 4));
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (CTAS == 2 && cta_rank != 0) mbar_arrive_leader_relaxed(&sf_ready[stage]);
          else mbar_arrive(&sf_ready[stage]);
        }
        if (++stage == stages) { stage = 0; phase ^= 1u; }
      }
    }
  } else {
    reg_inc<192>();
    // ------------------------------------------------------------ epilogue (every CTA drains its own TMEM)
    const int q = warp & 3;
    const int group = (warp - 8) >> 2;
    const int row = q * 32 + lane;  // weight row within this CTA's 128
    AccCursor cur;
    const bool clamp = (p.gate_lo == p.gate_lo) || (p.gate_hi == p.gate_hi) || (p.up_lo == p.up_lo) ||
                       (p.up_hi == p.up_hi);
    const bool as_is = !clamp && p.bias == nullptr && (KIND == 0 || p.col_scale == nullptr);  // nothing to do per weight row
    const float lo_limit = (q & 1) ? p.up_lo : p.gate_lo, hi_limit = (q & 1) ? p.up_hi : p.gate_hi;
    const float c_lo = lo_limit == lo_limit ? lo_limit : -INFINITY, c_hi = hi_limit == hi_limit ? hi_limit : INFINITY;
    uint8_t* const group_smem = smem + L::kOffEpi + group * L::kGroup;
    float* const turn = reinterpret_cast<float*>(group_smem);
    float* const tok_aff = reinterpret_cast<float*>(group_smem + 2 * kRowBytes);
    int* const tok_dst = reinterpret_cast<int*>(tok_aff + L::kMaxN / 2);
    const int tg = threadIdx.x & 127;
    int out_buf = 0;  // EPI 1: which of the group's two chunk buffers is next
    for (int tile = unit, it = 0; tile < total_tiles; tile += n_units, ++it) {
      const TileRec r = fetch_tile<CTAS>(p, sched, tile_table, it, tile);
      if (r.shape == 0) continue;
      const int n = r.n();
      const int w_row0 = r.w_row0 + cta_rank * 128;
      const int w_rows = min(128, r.w_rows() - cta_rank * 128);  // rows of this CTA that exist (may be <= 0)
      const int64_t w_index = static_cast<int64_t>(r.expert) * p.n_total + w_row0;
      // EPI 0: the thread's TMEM lane is its row; EPI 1: rows lane / 4 + 8 i of the warp's 32
      constexpr int kOwn = EPI == 0 ? 1 : 4;
      float bias[kOwn], factor[kOwn];
#pragma unroll
      for (int i = 0; i < kOwn; ++i) {
        const int own = EPI == 0 ? row : q * 32 + (lane >> 2) + 8 * i;
        bias[i] = p.bias != nullptr && own < w_rows ? p.bias[w_index + own] : 0.0f;
        factor[i] = KIND == 1 && p.col_scale != nullptr && own < w_rows ? p.col_scale[w_index + own] : 1.0f;
      }
      if constexpr (EPI == 1) {
        // where each of the group's tokens goes and what it is scaled by, one token per thread, while the MMAs are
        // still running
        const int col = (group + 2 * (tg >> 5)) * 32 + lane;
        if (tg < L::kMaxN / 2) {
          int dst = -1;
          float aff = 1.0f;
          if (col < n) {
            const int pos = r.row0 + col;
            const int tok = p.tpi ? __ldcg(p.tpi + pos) : pos;
            if (tok >= 0 && tok < p.hidden_rows) {
              dst = pos;
              if (p.row_src != nullptr) {
                dst = p.row_src[pos] & 0x7fffffff;
                if ((dst >> 24) >= 8 || (dst & 0xffffff) >= p.peer_rows || p.peer_out[dst >> 24] == nullptr) dst = -1;
              }
              if (p.aff != nullptr)
                aff = load_as_float<true>(p.aff, p.aff_per_row ? static_cast<int64_t>(tok) : static_cast<int64_t>(tok) * p.E + r.expert,
                                          p.aff_dtype);
            }
          }
          tok_aff[tg] = aff;
          tok_dst[tg] = dst;
        }
      }
      const bool wide = n > kAccStride;
      const int acc = cur.begin(wide);
      bool ok = mbar_wait(&tmem_full[acc], acc ? cur.filled[1] : cur.filled[0], abort_flag, p.status, 4);
      ok = group_all(1 + group, ok);  // the group meets at barriers below: leave together
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * kAccStride;
      uint32_t raw[kChunks][32];
#pragma unroll
      for (int l = 0; l < kChunks; ++l)
        if ((group + 2 * l) * 32 < n) {
          if constexpr (EPI == 0) {
            tc_ld32_nowait(taddr + (group + 2 * l) * 32, raw[l]);
          } else {
            tc_ld16x256_nowait(taddr + (group + 2 * l) * 32, raw[l]);
            tc_ld16x256_nowait(taddr + (16u << 16) + (group + 2 * l) * 32, raw[l] + 16);
          }
        }
      tc_wait_ld();
      // the accumulator now lives in registers: give the TMEM buffer back before doing the math
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        // relaxed: the accumulator is in registers (wait::ld above); a releasing arrive would first wait for this
        // thread's global stores of the previous tile to become visible and hold the next tile's MMAs back
        for (int a = acc; a <= (wide ? 1 : acc); ++a) {
          if (CTAS == 2 && cta_rank != 0) mbar_arrive_leader_relaxed(&tmem_empty[a]);
          else mbar_arrive_relaxed(&tmem_empty[a]);
        }
      }
      cur.end(wide);
      if (w_rows <= 0) continue;  // uniform across the CTA: the pair's second half lies past the last weight row

      if constexpr (EPI == 0) {
        const int tok_in_chunk = tg >> 2, part = tg & 3;
        const int blk = part >> 1;  // which 32 intermediates; the thread takes half of them
        const float* mine = turn + tok_in_chunk * kTurnPitch + blk * 72 + (part & 1) * 16;
        float* column = turn + row + (q >= 2 ? 8 : 0);
        const int i0 = (w_row0 >> 1) + blk * 32;
        const bool have = blk * 64 < w_rows;
#pragma unroll
        for (int l = 0; l < kChunks; ++l) {
          const int col0 = (group + 2 * l) * 32;
          if (col0 >= n) break;
          if (as_is) {
#pragma unroll
            for (int j = 0; j < 32; ++j) column[j * kTurnPitch] = __uint_as_float(raw[l][j]);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              float v = __uint_as_float(raw[l][j]);
              if constexpr (KIND == 1) v = __fmul_rn(v, factor[0]);  // rounded before the bias, never one fused step
              v += bias[0];
              if (clamp) v = fminf(fmaxf(v, c_lo), c_hi);
              column[j * kTurnPitch] = v;
            }
          }
          group_barrier(1 + group);
          float g[16], u[16];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float4 a = *reinterpret_cast<const float4*>(mine + 4 * j);
            const float4 b = *reinterpret_cast<const float4*>(mine + 32 + 4 * j);
            g[4 * j] = a.x; g[4 * j + 1] = a.y; g[4 * j + 2] = a.z; g[4 * j + 3] = a.w;
            u[4 * j] = b.x; u[4 * j + 1] = b.y; u[4 * j + 2] = b.z; u[4 * j + 3] = b.w;
          }
          uint32_t mx = swiglu16<SILU>(g, u, p.act);
          const int64_t pos = r.row0 + col0 + tok_in_chunk;
          const bool store = have && col0 + tok_in_chunk < n;
          if constexpr (KIND == 1) {
            // dense variant: the intermediate stays bf16 (the next contraction's operand type)
            uint32_t o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const __nv_bfloat162 b2 = __floats2bfloat162_rn(g[2 * j], g[2 * j + 1]);
              o[j] = *reinterpret_cast<const uint32_t*>(&b2);
            }
            if (store)
              st_global_256(reinterpret_cast<__nv_bfloat16*>(p.m_codes) + pos * p.I + i0 + (part & 1) * 16, o[0], o[1], o[2],
                            o[3], o[4], o[5], o[6], o[7]);
          } else {
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            uint32_t w[4];
            const int e_max = static_cast<int>(mx >> 23);
            if (e_max >= 9) {  // one exact power-of-two factor
              const float f = __uint_as_float(static_cast<uint32_t>(135 - e_max + 127) << 23);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 lo = mul2(make_float2(g[4 * j], g[4 * j + 1]), make_float2(f, f));
                const float2 hi = mul2(make_float2(g[4 * j + 2], g[4 * j + 3]), make_float2(f, f));
                w[j] = pack4_e4m3(lo.x, lo.y, hi.x, hi.y);
              }
            } else {
              float f1, f2;
              mx_block_factors(mx, f1, f2);
#pragma unroll
              for (int j = 0; j < 4; ++j)
                w[j] = pack4_e4m3(g[4 * j] * f1 * f2, g[4 * j + 1] * f1 * f2, g[4 * j + 2] * f1 * f2, g[4 * j + 3] * f1 * f2);
            }
            if (store) {
              *reinterpret_cast<uint4*>(p.m_codes + pos * p.I + i0 + (part & 1) * 16) = make_uint4(w[0], w[1], w[2], w[3]);
              if ((part & 1) == 0) p.m_sf[sf_atom_offset(pos, i0 >> 5, (p.I + 127) >> 7)] = mx_block_scale_byte(mx);
            }
          }
          group_barrier(1 + group);  // the chunk buffer is free again
        }
      } else {
        // A thread holds, of every 8 tokens, tokens 2 (lane % 4) and + 1 of four weight rows (lane / 4 + 8 i): packed to
        // bf16 pairs these are the fragments of four 8 x 8 matrices, which the transposing matrix store turns into
        // 16-byte pieces of token rows.  A bulk copy per token then moves 256 contiguous bytes to global memory: the
        // stores cost no registers and no L1 write slots (with 4-byte stores from registers the short contractions
        // ran at half the speed).
        const float2* const aff2 = reinterpret_cast<const float2*>(tok_aff) + (lane & 3);
        const uint32_t row_bytes = static_cast<uint32_t>(w_rows) * 2;
#pragma unroll
        for (int l = 0; l < kChunks; ++l) {
          if ((group + 2 * l) * 32 >= n) break;
          uint8_t* const buf = group_smem + out_buf * kRowBytes;
          out_buf ^= 1;
          // the copies out of this buffer two chunks ago (issued by lanes of these warps) have read it
          asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          group_barrier(1 + group);
          const uint32_t to = smem_u32(buf) + (lane & 7) * kRowPitch + (q * 32 + (lane >> 3) * 8) * 2;
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const float2 a = aff2[l * 16 + g * 4];
            uint32_t m[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float v0 = __uint_as_float(raw[l][(i >> 1) * 16 + g * 4 + (i & 1) * 2]);
              float v1 = __uint_as_float(raw[l][(i >> 1) * 16 + g * 4 + (i & 1) * 2 + 1]);
              if constexpr (KIND == 1) {
                v0 = __fmul_rn(v0, factor[i]);
                v1 = __fmul_rn(v1, factor[i]);
              }
              const __nv_bfloat162 b2 = __floats2bfloat162_rn((v0 + bias[i]) * a.x, (v1 + bias[i]) * a.y);
              m[i] = *reinterpret_cast<const uint32_t*>(&b2);
            }
            stmatrix_x4_trans(to + g * 8 * kRowPitch, m[0], m[1], m[2], m[3]);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          group_barrier(1 + group);
          const int c = q * 8 + (lane & 7);
          const int dst = tok_dst[l * 32 + c];
          if (p.row_src == nullptr) {
            if (lane < 8 && dst >= 0)
              bulk_store(p.y_pos + static_cast<int64_t>(dst) * p.H_out + w_row0, buf + c * kRowPitch, row_bytes);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          } else if (dst >= 0) {
            // to the GPU the token came from: four lanes per row, 16 bytes each at a time
            __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.peer_out[dst >> 24]) +
                                 static_cast<int64_t>(dst & 0xffffff) * p.H_out + w_row0;
            for (int b = (lane >> 3) * 8; b < w_rows; b += 32)
              *reinterpret_cast<uint4*>(out + b) = *reinterpret_cast<const uint4*>(buf + c * kRowPitch + b * 2);
          }
        }
        // the token list may change once every thread of the group is past its reads of it
        group_barrier(1 + group);
      }
    }
    // copies read this CTA's shared memory and must be complete before the grid is
    if constexpr (EPI == 1) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  // a CTA without tiles must not let this grid complete before the one in front either
  if (p.chained) grid_wait();
  tc_fence_before();
  __syncthreads();
  if (p.clock_probe != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
    unsigned long long t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
    p.clock_probe[0] = static_cast<unsigned long long>(clock64() - probe_c0);
    p.clock_probe[1] = t1 - probe_t0;
  }
  if constexpr (CTAS == 2) cluster_sync_all();  // the peer may still read this CTA's shared memory until here
  if (warp == 1) {
    tc_fence_after();
    if constexpr (CTAS == 2)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// ------------------------------------------------------------------ validation kernels (CUDA cores)
__device__ __forceinline__ float e4m3_to_float(uint8_t c) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(c), __NV_E4M3);
  return __half2float(*reinterpret_cast<const __half*>(&h));
}

__device__ __forceinline__ int64_t weight_offset(int64_t rows, int K, int w_format) {
  return w_format == B200MOE_W_E2M1 ? rows * K / 2 : rows * K;
}
// Weight element k of a row of K elements in any of the supported formats.
__device__ __forceinline__ float weight_to_float(const uint8_t* row, int k, int w_format) {
  if (w_format == B200MOE_W_E2M1) {
    const uint32_t nib = (row[k >> 1] >> ((k & 1) * 4)) & 0xFu;
    const uint32_t ex = (nib >> 1) & 3u, man = nib & 1u;
    const float mag = ex == 0 ? 0.5f * man : (1.0f + 0.5f * man) * static_cast<float>(1u << (ex - 1));
    return (nib & 8u) ? -mag : mag;
  }
  if (w_format == B200MOE_W_E5M2) {
    const __half_raw h = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(row[k]), __NV_E5M2);
    return __half2float(*reinterpret_cast<const __half*>(&h));
  }
  return e4m3_to_float(row[k]);
}

__device__ float mx_dot(const uint8_t* a, const uint8_t* a_sf, int64_t a_row, const uint8_t* b, const uint8_t* b_sf,
                        int64_t b_row, int K, int w_format) {
  const int64_t k_atoms = (K + 127) >> 7;
  const uint8_t* brow = b + b_row * (w_format == B200MOE_W_E2M1 ? K / 2 : K);
  float acc = 0.f;
  for (int kb = 0; kb < K / 32; ++kb) {
    float part = 0.f;
    for (int j = 0; j < 32; ++j)
      part += e4m3_to_float(a[a_row * K + kb * 32 + j]) * weight_to_float(brow, kb * 32 + j, w_format);
    const int sa = a_sf[sf_atom_offset(a_row, kb, k_atoms)], sb = b_sf[sf_atom_offset(b_row, kb, k_atoms)];
    acc += part * exp2f(static_cast<float>(sa - 127)) * exp2f(static_cast<float>(sb - 127));
  }
  return acc;
}

__device__ bool block_is_active(const GemmParams& p, int block) {
  if (p.conditions == nullptr) return true;
  for (int b = 0; b <= block; ++b)
    if (p.conditions[b] == 0) return false;
  return true;
}

__global__ void simt_gemm1_kernel(const uint8_t* x, const uint8_t* w, GemmParams p, int K) {
  // one thread per (position, 32-block of intermediates)
  const int blocks_i = p.I / 32;
  const int64_t total = static_cast<int64_t>(p.m_tiles_total) * 128 * blocks_i;
  for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int ib = static_cast<int>(idx % blocks_i);
    const int64_t row = idx / blocks_i;
    const int m_tile = static_cast<int>(row >> 7);
    const int block = m_tile / (p.B >> 7);
    if (!block_is_active(p, block)) continue;
    if (p.tile_flags && p.tile_flags[m_tile] == 0) continue;
    const int e = p.block_to_expert[block];
    if (e < 0 || e >= p.E) continue;
    const uint8_t* we = w + weight_offset(static_cast<int64_t>(e) * p.n_total, K, p.w_format);
    const uint8_t* wsf = p.w_sf + static_cast<int64_t>(e) * p.w_sf_expert_stride;
    const float* bias = p.bias ? p.bias + static_cast<int64_t>(e) * p.n_total : nullptr;
    float m[32];
    uint32_t mx = 0;
    for (int j = 0; j < 32; ++j) {
      const int n_g = ib * 64 + j, n_u = n_g + 32;
      float gv = mx_dot(x, p.x_sf, row, we, wsf, n_g, K, p.w_format);
      float uv = mx_dot(x, p.x_sf, row, we, wsf, n_u, K, p.w_format);
      if (bias) { gv += bias[n_g]; uv += bias[n_u]; }
      if (p.gate_lo == p.gate_lo) gv = fmaxf(gv, p.gate_lo);
      if (p.gate_hi == p.gate_hi) gv = fminf(gv, p.gate_hi);
      if (p.up_lo == p.up_lo) uv = fmaxf(uv, p.up_lo);
      if (p.up_hi == p.up_hi) uv = fminf(uv, p.up_hi);
      m[j] = apply_act(gv, p.act) * uv;
      mx = max(mx, __float_as_uint(m[j]) & 0x7fffffffu);
    }
    float f1, f2;
    mx_block_factors(mx, f1, f2);
    uint32_t* dst = reinterpret_cast<uint32_t*>(p.m_codes + row * p.I + ib * 32);
    for (int j = 0; j < 8; ++j)
      dst[j] = pack4_e4m3(m[4 * j] * f1 * f2, m[4 * j + 1] * f1 * f2, m[4 * j + 2] * f1 * f2, m[4 * j + 3] * f1 * f2);
    p.m_sf[sf_atom_offset(row, ib, (p.I + 127) >> 7)] = mx_block_scale_byte(mx);
  }
}

__global__ void simt_gemm2_kernel(const uint8_t* m, const uint8_t* w, GemmParams p, int K) {
  const int64_t total = static_cast<int64_t>(p.m_tiles_total) * 128 * p.H_out;
  for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int h = static_cast<int>(idx % p.H_out);
    const int64_t row = idx / p.H_out;
    const int m_tile = static_cast<int>(row >> 7);
    const int block = m_tile / (p.B >> 7);
    if (!block_is_active(p, block)) continue;
    if (p.tile_flags && p.tile_flags[m_tile] == 0) continue;
    const int e = p.block_to_expert[block];
    if (e < 0 || e >= p.E) continue;
    const int tok = p.tpi ? p.tpi[row] : static_cast<int>(row);
    if (tok < 0 || tok >= p.hidden_rows) continue;
    float y = mx_dot(m, p.x_sf, row, w + weight_offset(static_cast<int64_t>(e) * p.n_total, K, p.w_format),
                     p.w_sf + static_cast<int64_t>(e) * p.w_sf_expert_stride, h, K, p.w_format);
    if (p.bias) y += p.bias[static_cast<int64_t>(e) * p.H_out + h];
    if (p.aff)
      y *= load_as_float(p.aff, p.aff_per_row ? static_cast<int64_t>(tok) : static_cast<int64_t>(tok) * p.E + e,
                         p.aff_dtype);
    __nv_bfloat16* out_row = p.y_pos + row * p.H_out;
    if (p.row_src != nullptr) {
      const int32_t src = p.row_src[row];
      const int dst_rank = (src >> 24) & 0x7f;
      const int64_t dst_row = src & 0xffffff;
      if (dst_rank >= 8 || dst_row >= p.peer_rows || p.peer_out[dst_rank] == nullptr) continue;
      out_row = static_cast<__nv_bfloat16*>(p.peer_out[dst_rank]) + dst_row * p.H_out;
    }
    out_row[h] = __float2bfloat16_rn(y);
  }
}

// Dense (bf16 x bf16) counterparts of the two validation kernels: one thread per output element.
__device__ float dense_dot(const __nv_bfloat16* a, const __nv_bfloat16* b, int K) {
  float acc = 0.f;
  for (int k = 0; k < K; ++k) acc += __bfloat162float(a[k]) * __bfloat162float(b[k]);
  return acc;
}

__global__ void simt_dense_gemm1_kernel(const __nv_bfloat16* x, const __nv_bfloat16* w, GemmParams p, int K) {
  const int64_t total = static_cast<int64_t>(p.m_tiles_total) * 128 * p.I;
  for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(idx % p.I);
    const int64_t row = idx / p.I;
    const int m_tile = static_cast<int>(row >> 7);
    const int block = m_tile / (p.B >> 7);
    if (!block_is_active(p, block)) continue;
    if (p.tile_flags && p.tile_flags[m_tile] == 0) continue;
    const int e = p.block_to_expert[block];
    if (e < 0 || e >= p.E) continue;
    const int n_g = (i >> 5) * 64 + (i & 31), n_u = n_g + 32;
    const __nv_bfloat16* we = w + static_cast<int64_t>(e) * p.n_total * K;
    float gv = dense_dot(x + row * K, we + static_cast<int64_t>(n_g) * K, K);
    float uv = dense_dot(x + row * K, we + static_cast<int64_t>(n_u) * K, K);
    if (p.col_scale) {
      gv *= p.col_scale[static_cast<int64_t>(e) * p.n_total + n_g];
      uv *= p.col_scale[static_cast<int64_t>(e) * p.n_total + n_u];
    }
    if (p.bias) { gv += p.bias[static_cast<int64_t>(e) * p.n_total + n_g]; uv += p.bias[static_cast<int64_t>(e) * p.n_total + n_u]; }
    if (p.gate_lo == p.gate_lo) gv = fmaxf(gv, p.gate_lo);
    if (p.gate_hi == p.gate_hi) gv = fminf(gv, p.gate_hi);
    if (p.up_lo == p.up_lo) uv = fmaxf(uv, p.up_lo);
    if (p.up_hi == p.up_hi) uv = fminf(uv, p.up_hi);
    reinterpret_cast<__nv_bfloat16*>(p.m_codes)[row * p.I + i] = __float2bfloat16_rn(apply_act(gv, p.act) * uv);
  }
}

__global__ void simt_dense_gemm2_kernel(const __nv_bfloat16* m, const __nv_bfloat16* w, GemmParams p, int K) {
  const int64_t total = static_cast<int64_t>(p.m_tiles_total) * 128 * p.H_out;
  for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int h = static_cast<int>(idx % p.H_out);
    const int64_t row = idx / p.H_out;
    const int m_tile = static_cast<int>(row >> 7);
    const int block = m_tile / (p.B >> 7);
    if (!block_is_active(p, block)) continue;
    if (p.tile_flags && p.tile_flags[m_tile] == 0) continue;
    const int e = p.block_to_expert[block];
    if (e < 0 || e >= p.E) continue;
    const int tok = p.tpi ? p.tpi[row] : static_cast<int>(row);
    if (tok < 0 || tok >= p.hidden_rows) continue;
    float y = dense_dot(m + row * K, w + (static_cast<int64_t>(e) * p.n_total + h) * K, K);
    if (p.col_scale) y *= p.col_scale[static_cast<int64_t>(e) * p.H_out + h];
    if (p.bias) y += p.bias[static_cast<int64_t>(e) * p.H_out + h];
    if (p.aff)
      y *= load_as_float(p.aff, p.aff_per_row ? static_cast<int64_t>(tok) : static_cast<int64_t>(tok) * p.E + e,
                         p.aff_dtype);
    p.y_pos[row * p.H_out + h] = __float2bfloat16_rn(y);
  }
}

// ------------------------------------------------------------------ host side
// Rows of K elements, one byte each, or (nibbles) two per byte: the 4-bit map type expands every 8 packed
// bytes to a 16-byte shared-memory chunk, which is the padded form the f8f6f4 MMA reads 4-bit operands in,
// so a 128-element slab still occupies a 128-byte swizzled row.
int make_rows_map(CUtensorMap* map, const void* base, int64_t K, int64_t rows, int64_t batch, int box_rows,
                  bool nibbles = false) {
  EncodeTiledFn enc = get_encode_fn();
  B200MOE_REQUIRE(enc != nullptr, B200MOE_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint32_t rank = batch > 0 ? 3 : 2;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(batch > 0 ? batch : 1)};
  const cuuint64_t pitch = static_cast<cuuint64_t>(nibbles ? K / 2 : K);
  cuuint64_t strides[2] = {pitch, pitch * static_cast<cuuint64_t>(rows)};
  cuuint32_t box[3] = {static_cast<cuuint32_t>(kBlockK), static_cast<cuuint32_t>(box_rows), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(map, nibbles ? CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B : CU_TENSOR_MAP_DATA_TYPE_UINT8, rank,
                         const_cast<void*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  B200MOE_REQUIRE(r == CUDA_SUCCESS, B200MOE_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", static_cast<int>(r));
  return B200MOE_OK;
}

int make_atoms_map(CUtensorMap* map, const void* base, int64_t n_atoms) {
  // scale atoms as rows of 128 32-bit words, one atom per TMA box
  EncodeTiledFn enc = get_encode_fn();
  B200MOE_REQUIRE(enc != nullptr, B200MOE_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[2] = {128, static_cast<cuuint64_t>(n_atoms)};
  cuuint64_t strides[1] = {512};
  cuuint32_t box[2] = {128, 1};
  cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  B200MOE_REQUIRE(r == CUDA_SUCCESS, B200MOE_ERR_CUDA, "cuTensorMapEncodeTiled (scale atoms) failed with code %d",
                  static_cast<int>(r));
  return B200MOE_OK;
}

template <int EPI, int CTAS, int KIND, bool SILU>
int launch_tc(const WeightMaps& wm, const TokenMaps& xm, const CUtensorMap& sfw, const CUtensorMap& sfx,
              const GemmParams& p, cudaStream_t st) {
  using L = SmemLayout<EPI, CTAS>;
  auto kern = grouped_mxfp8_gemm_kernel<EPI, CTAS, KIND, SILU>;
  static_assert(L::kBytes <= 227 * 1024, "shared memory of the contraction kernel");
  B200MOE_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(kern), L::kBytes));
  // only sizes the grid: at most one token tile per 128 positions; a single CTA may cut its 128 weight rows further
  const int64_t total = static_cast<int64_t>(p.m_tiles_total) * ceil_div64(p.n_total, CTAS == 2 ? 256 : (EPI == 0 ? 64 : 16));
  const int units = sm_count() / CTAS;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>((total < units ? total : units) * CTAS));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = L::kBytes;
  cfg.stream = st;
  // A chained contraction is scheduled as the CTAs of the launch in front exit, so that its prologue and the first
  // weight slabs (a ring full per SM) overlap that launch's tail.  Only on the caller's word: before it waits it reads
  // the block list, conditions, tile flags and weights (a down contraction also token ids and affinities), which must
  // have been complete when the launch in front was made.  Between an unchained pair of contractions 7.5 us passed
  // from the last CTA's end to the first one's start, and 8 to 10 more to the first slab in shared memory.
  // 64-token decode of 8 experts of 4096 x 14336: 274 -> 264 us, 16 tokens on 128 experts of 4096 x 1536, top-8,
  // captured: 285 -> 273 us.
  cudaLaunchAttribute attr[2];
  if (CTAS == 2) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = CTAS;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  if (p.chained) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  B200MOE_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, wm, xm, sfw, sfx, p));
  B200MOE_LAUNCH_OK("grouped_mxfp8_gemm_kernel");
  return B200MOE_OK;
}

// `impl` is the per-call variant word of the entry points: bit 0 selects the CUDA-core validation kernels, the
// B200MOE_GEMM_* bits restrict the tile shapes the tensor-core path may pick.  Nothing here is process state.
// `kind`: 0 = MX (x and w are element codes, K counts elements = bytes, or nibbles for e2m1 weights); 1 = dense
// bf16 operands (K counts bf16 elements; the copies address rows in bytes).
int run_gemm(int epi, const uint8_t* x, const uint8_t* w, GemmParams& p, int K, int impl, void* clock_probe,
             cudaStream_t st, int kind = 0) {
  B200MOE_REQUIRE((impl & ~(B200MOE_IMPL_SIMT | B200MOE_GEMM_TILE_N128 | B200MOE_GEMM_NO_PAIR | B200MOE_GEMM_FORCE_PAIR |
                            B200MOE_GEMM_NO_SPLIT | B200MOE_GEMM_NO_OVERLAP | B200MOE_GEMM_CHAINED)) == 0,
                  B200MOE_ERR_INVALID, "unknown bits in the variant word 0x%x", impl);
  B200MOE_REQUIRE(clock_probe == nullptr || (reinterpret_cast<uintptr_t>(clock_probe) & 7) == 0, B200MOE_ERR_INVALID,
                  "the clock probe buffer must be 8-byte aligned");
  B200MOE_REQUIRE(p.B > 0 && p.B % 128 == 0, B200MOE_ERR_INVALID, "block size must be a multiple of 128, got %d", p.B);
  B200MOE_REQUIRE(K % 32 == 0 && K >= 32, B200MOE_ERR_INVALID, "contraction length must be a multiple of 32, got %d", K);
  B200MOE_REQUIRE(kind == 0 || !(impl & B200MOE_GEMM_TILE_N128), B200MOE_ERR_INVALID,
                  "TILE_N128 is an option of the MX contractions only; use NO_PAIR");
  B200MOE_REQUIRE(p.n_blocks > 0 && p.E > 0 && p.E <= kMaxExperts, B200MOE_ERR_INVALID,
                  "need at least one block and between 1 and %d experts", kMaxExperts);
  B200MOE_REQUIRE(p.status != nullptr, B200MOE_ERR_INVALID, "status pointer must not be null");
  B200MOE_REQUIRE(p.w_format == B200MOE_W_E4M3 || p.w_format == B200MOE_W_E5M2 || p.w_format == B200MOE_W_E2M1,
                  B200MOE_ERR_INVALID, "unknown weight format %d", p.w_format);
  const bool nibbles = p.w_format == B200MOE_W_E2M1;
  B200MOE_REQUIRE(!nibbles || K % 128 == 0, B200MOE_ERR_INVALID,
                  "e2m1 weights need a contraction length that is a multiple of 128, got %d", K);
  p.m_tiles_total = p.n_blocks * (p.B / 128);
  p.clock_probe = static_cast<unsigned long long*>(clock_probe);
  const int Kb = kind == 1 ? 2 * K : K;  // row pitch the copies see, in element-code bytes
  p.k_blocks = (Kb + kBlockK - 1) / kBlockK;
  p.w_row_atoms = (p.n_total + 127) / 128;
  p.w_sf_expert_stride = static_cast<int64_t>(p.w_row_atoms) * p.k_blocks * 512;
  if (impl & B200MOE_IMPL_SIMT) {
    B200MOE_CUDA_OK(cudaMemsetAsync(p.status, 0, 4, st));
    const int64_t work = epi == 0 ? static_cast<int64_t>(p.m_tiles_total) * 128 * (p.I / 32)
                                  : static_cast<int64_t>(p.m_tiles_total) * 128 * p.H_out;
    const int64_t cap = static_cast<int64_t>(sm_count()) * 32;
    const int grid = static_cast<int>(ceil_div64(work, 128) < cap ? ceil_div64(work, 128) : cap);
    if (kind == 1) {
      const auto* ab = reinterpret_cast<const __nv_bfloat16*>(x);
      const auto* bb = reinterpret_cast<const __nv_bfloat16*>(w);
      if (epi == 0) simt_dense_gemm1_kernel<<<grid, 128, 0, st>>>(ab, bb, p, K);
      else simt_dense_gemm2_kernel<<<grid, 128, 0, st>>>(ab, bb, p, K);
    } else if (epi == 0) simt_gemm1_kernel<<<grid, 128, 0, st>>>(x, w, p, K);
    else simt_gemm2_kernel<<<grid, 128, 0, st>>>(x, w, p, K);
    B200MOE_LAUNCH_OK("simt_gemm_kernel");
    return B200MOE_OK;
  }
  // CTA pairs (256 weight rows, up to 256 tokens per tile; each CTA copies half of the token rows) when the block list has
  // room for two 128-row tiles per expert, and for blocks of a multiple of 256 positions.  The host knows the list's
  // length, not how many tokens an expert got, so the rule is a guess where the list is mostly padding: with few tokens per
  // expert a launch is bound by streaming the weights, which single CTAs (128 weight rows or fewer) spread over the SMs in
  // finer pieces.  Captured layers in us, blocks of 128 (which choose by length) / of 256 (always pairs): 8 experts of
  // 4096 x 4096, top-2, 1 token per expert 66 / 104, 64 tokens 108 / 111, 128 tokens 136 / 125, 192 tokens 133 / 132;
  // 64 experts of 3072 x 1536, top-4: 126 / 153, 211 / 216, 275 / 247, 282 / 295.
  // Tiles of up to 256 tokens although only 224 leave room for a second accumulator: the 8192-token layer above took 7 %
  // longer with tiles of at most 224, the 4096-token one 1 % -- fewer operand bytes per MMA outweigh the drain at a tile's
  // end.
  const bool pair = !(impl & (B200MOE_GEMM_NO_PAIR | B200MOE_GEMM_TILE_N128)) && (sm_count() % 2 == 0) &&
                    (p.B % 256 == 0 || (impl & B200MOE_GEMM_FORCE_PAIR) || p.m_tiles_total >= 2 * p.E);
  p.max_n = pair ? 256 : 128;
  p.w_slab_bytes = nibbles ? kBlockK / 2 : kBlockK;
  // (a gate/up launch that has to clear scale atoms first follows a memset, not a kernel; a probed launch must not count
  // the drain of the one in front)
  p.chained = (impl & B200MOE_GEMM_CHAINED) != 0 && clock_probe == nullptr && (epi == 1 || kind == 1 || p.I % 128 == 0);
  WeightMaps wm;
  TokenMaps xm;
  CUtensorMap* const w_maps[4] = {&wm.rows128, &wm.rows64, &wm.rows32, &wm.rows16};
  CUtensorMap* const x_maps[4] = {&xm.rows128, &xm.rows64, &xm.rows32, &xm.rows16};
  CUtensorMap sfx, sfw;
  // weight boxes: a pair copies 128 rows at a time, a single CTA's gate/up tiles have 128 or 64, its down tiles any
  // multiple of 16
  const int n_w_maps = pair ? 1 : (epi == 0 ? 2 : 4);
  for (int i = 0; i < 4; ++i) {
    int rc = make_rows_map(x_maps[i], x, Kb, static_cast<int64_t>(p.m_tiles_total) * 128, 0, 128 >> i);
    if (rc != B200MOE_OK) return rc;
    if (i < n_w_maps) {
      rc = make_rows_map(w_maps[i], w, Kb, p.n_total, p.E, 128 >> i, nibbles);
      if (rc != B200MOE_OK) return rc;
    } else {
      *w_maps[i] = wm.rows128;  // never used
    }
  }
  if (kind == 0) {
    int rc = make_atoms_map(&sfx, p.x_sf, static_cast<int64_t>(p.m_tiles_total) * p.k_blocks);
    if (rc != B200MOE_OK) return rc;
    rc = make_atoms_map(&sfw, p.w_sf, static_cast<int64_t>(p.E) * p.w_row_atoms * p.k_blocks);
    if (rc != B200MOE_OK) return rc;
  } else {
    sfx = sfw = xm.rows128;  // never dereferenced by the dense kernel
  }
  const bool silu = p.act == B200MOE_ACT_SILU;
  const auto launch = [&](auto ctas, auto dense) {
    constexpr int C = decltype(ctas)::value, D = decltype(dense)::value;
    if (epi == 1) return launch_tc<1, C, D, false>(wm, xm, sfw, sfx, p, st);
    return silu ? launch_tc<0, C, D, true>(wm, xm, sfw, sfx, p, st) : launch_tc<0, C, D, false>(wm, xm, sfw, sfx, p, st);
  };
  const std::integral_constant<int, 0> zero;
  const std::integral_constant<int, 1> one;
  const std::integral_constant<int, 2> two;
  if (pair) return kind == 1 ? launch(two, one) : launch(two, zero);
  return kind == 1 ? launch(one, one) : launch(one, zero);
}

}  // namespace
}  // namespace b200moe

using namespace b200moe;

extern "C" int b200moe_grouped_gemm1_swiglu(const uint8_t* x_codes, const uint8_t* x_sf, const uint8_t* w1_dev,
                                            const uint8_t* w1_sf, int w_format, const float* bias_gu_dev,
                                            const int32_t* block_to_expert, const int32_t* conditions,
                                            const int32_t* tile_flags, int n_blocks, int B, int E, int H, int I,
                                            int act_fn, float gate_lo, float gate_hi, float up_lo, float up_hi,
                                            uint8_t* m_codes, uint8_t* m_sf, int32_t* status, int impl,
                                            void* clock_probe, b200moe_stream_t stream) {
  B200MOE_REQUIRE(x_codes && x_sf && w1_dev && w1_sf && block_to_expert && m_codes && m_sf, B200MOE_ERR_INVALID,
                  "grouped_gemm1: null pointer argument");
  B200MOE_REQUIRE(I % 32 == 0 && I > 0, B200MOE_ERR_INVALID, "grouped_gemm1: I must be a positive multiple of 32, got %d", I);
  B200MOE_REQUIRE(act_fn >= 0 && act_fn <= 3, B200MOE_ERR_INVALID, "grouped_gemm1: unknown activation %d", act_fn);
  B200MOE_REQUIRE((reinterpret_cast<uintptr_t>(m_codes) & 31) == 0, B200MOE_ERR_INVALID,
                  "grouped_gemm1: m_codes must be 32-byte aligned (the epilogue stores 32 bytes at a time)");
  GemmParams p{};
  p.x_sf = x_sf;
  p.w_sf = w1_sf;
  p.w_format = w_format;
  p.block_to_expert = block_to_expert;
  p.conditions = conditions;
  p.tile_flags = tile_flags;
  p.n_blocks = n_blocks;
  p.B = B;
  p.E = E;
  p.n_total = 2 * I;
  p.bias = bias_gu_dev;
  p.act = act_fn;
  p.gate_lo = gate_lo;
  p.gate_hi = gate_hi;
  p.up_lo = up_lo;
  p.up_hi = up_hi;
  p.m_codes = m_codes;
  p.m_sf = m_sf;
  p.I = I;
  p.status = status;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (I % 128 != 0)  // partially filled scale atoms along I must read as zero
    B200MOE_CUDA_OK(cudaMemsetAsync(m_sf, 0, b200moe_sf_bytes(static_cast<int64_t>(n_blocks) * B, I), st));
  return run_gemm(0, x_codes, w1_dev, p, H, impl, clock_probe, st);
}

namespace {
int gemm2_impl(const uint8_t* m_codes, const uint8_t* m_sf, const uint8_t* w2_dev, const uint8_t* w2_sf, int w_format,
               const float* bias_d, const int32_t* block_to_expert, const int32_t* conditions,
               const int32_t* tile_flags, const int32_t* token_position_to_id, int hidden_rows, int n_blocks, int B,
               int E, int H, int I, const void* affinities, int aff_dtype, int aff_per_row, void* y_pos_bf16,
               const int32_t* row_src, void* const* peer_out, int world, int64_t peer_rows, int32_t* status, int impl,
               void* clock_probe, b200moe_stream_t stream) {
  B200MOE_REQUIRE(m_codes && m_sf && w2_dev && w2_sf && block_to_expert && (y_pos_bf16 || row_src),
                  B200MOE_ERR_INVALID, "grouped_gemm2: null pointer argument");
  B200MOE_REQUIRE(H % 32 == 0 && H > 0, B200MOE_ERR_INVALID, "grouped_gemm2: H must be a positive multiple of 32, got %d", H);
  B200MOE_REQUIRE(aff_dtype == B200MOE_F32 || aff_dtype == B200MOE_BF16, B200MOE_ERR_INVALID,
                  "grouped_gemm2: affinities must be fp32 or bf16");
  GemmParams p{};
  p.x_sf = m_sf;
  p.w_sf = w2_sf;
  p.w_format = w_format;
  p.block_to_expert = block_to_expert;
  p.conditions = conditions;
  p.tile_flags = tile_flags;
  p.tpi = token_position_to_id;
  p.hidden_rows = hidden_rows;
  p.n_blocks = n_blocks;
  p.B = B;
  p.E = E;
  p.n_total = H;
  p.bias = bias_d;
  p.aff = affinities;
  p.aff_dtype = aff_dtype;
  p.aff_per_row = aff_per_row;
  p.y_pos = static_cast<__nv_bfloat16*>(y_pos_bf16);
  p.H_out = H;
  p.I = I;
  p.status = status;
  if (row_src != nullptr) {
    B200MOE_REQUIRE(peer_out != nullptr && world >= 1 && world <= 8 && token_position_to_id != nullptr,
                    B200MOE_ERR_INVALID, "grouped_gemm2: peer output needs 1..8 peer buffers and the row validity list");
    p.row_src = row_src;
    p.peer_rows = peer_rows;
    for (int i = 0; i < 8; ++i) p.peer_out[i] = i < world ? peer_out[i] : nullptr;
    for (int i = 0; i < world; ++i)
      B200MOE_REQUIRE(p.peer_out[i] != nullptr && (reinterpret_cast<uintptr_t>(p.peer_out[i]) & 31) == 0,
                      B200MOE_ERR_INVALID, "grouped_gemm2: peer buffer %d is null or not 32-byte aligned", i);
  } else {
    B200MOE_REQUIRE((reinterpret_cast<uintptr_t>(y_pos_bf16) & 31) == 0, B200MOE_ERR_INVALID,
                    "grouped_gemm2: y_pos must be 32-byte aligned (the epilogue stores 32 bytes at a time)");
  }
  return run_gemm(1, m_codes, w2_dev, p, I, impl, clock_probe, static_cast<cudaStream_t>(stream));
}
}  // namespace

extern "C" int b200moe_grouped_gemm2_scale(const uint8_t* m_codes, const uint8_t* m_sf, const uint8_t* w2_dev,
                                           const uint8_t* w2_sf, int w_format, const float* bias_d,
                                           const int32_t* block_to_expert, const int32_t* conditions,
                                           const int32_t* tile_flags, const int32_t* token_position_to_id,
                                           int hidden_rows, int n_blocks, int B, int E, int H, int I,
                                           const void* affinities, int aff_dtype, int aff_per_row, void* y_pos_bf16,
                                           int32_t* status, int impl, void* clock_probe,
                                           b200moe_stream_t stream) {
  return gemm2_impl(m_codes, m_sf, w2_dev, w2_sf, w_format, bias_d, block_to_expert, conditions, tile_flags,
                    token_position_to_id, hidden_rows, n_blocks, B, E, H, I, affinities, aff_dtype, aff_per_row,
                    y_pos_bf16, nullptr, nullptr, 0, 0, status, impl, clock_probe, stream);
}

extern "C" int b200moe_ep_gemm2_scale_return(const uint8_t* m_codes, const uint8_t* m_sf, const uint8_t* w2_dev,
                                             const uint8_t* w2_sf, int w_format, const float* bias_d,
                                             const int32_t* block_to_expert, const int32_t* conditions,
                                             const int32_t* tile_flags, const int32_t* row_valid, int64_t cap_rows,
                                             int n_blocks, int B, int E_local, int H, int I, const float* row_affinity,
                                             const int32_t* row_src, void* const* back_peers, int world,
                                             int64_t back_rows, int32_t* status, int impl, b200moe_stream_t stream) {
  B200MOE_REQUIRE(row_valid && row_src && back_peers, B200MOE_ERR_INVALID, "ep_gemm2_scale_return: null pointer argument");
  return gemm2_impl(m_codes, m_sf, w2_dev, w2_sf, w_format, bias_d, block_to_expert, conditions, tile_flags, row_valid,
                    static_cast<int>(cap_rows), n_blocks, B, E_local, H, I, row_affinity, B200MOE_F32, 1, nullptr,
                    row_src, back_peers, world, back_rows, status, impl, nullptr, stream);
}


// ---- dense (bf16) variants: the reference's non-MX expert kernels ------------------------------------------------
extern "C" int b200moe_dense_gemm1_swiglu(const void* x_bf16, const void* w1_bf16, const float* w1_col_scale,
                                          const float* bias_gu_dev, const int32_t* block_to_expert,
                                          const int32_t* conditions, const int32_t* tile_flags, int n_blocks, int B,
                                          int E, int H, int I, int act_fn, float gate_lo, float gate_hi, float up_lo,
                                          float up_hi, void* m_bf16, int32_t* status, int impl,
                                          b200moe_stream_t stream) {
  B200MOE_REQUIRE(x_bf16 && w1_bf16 && block_to_expert && m_bf16, B200MOE_ERR_INVALID,
                  "dense_gemm1: null pointer argument");
  B200MOE_REQUIRE(I % 32 == 0 && I > 0 && H % 32 == 0 && H > 0, B200MOE_ERR_INVALID,
                  "dense_gemm1: H and I must be positive multiples of 32 (H = %d, I = %d)", H, I);
  B200MOE_REQUIRE(act_fn >= 0 && act_fn <= 3, B200MOE_ERR_INVALID, "dense_gemm1: unknown activation %d", act_fn);
  B200MOE_REQUIRE((reinterpret_cast<uintptr_t>(m_bf16) & 31) == 0, B200MOE_ERR_INVALID,
                  "dense_gemm1: the intermediate buffer must be 32-byte aligned");
  GemmParams p{};
  p.block_to_expert = block_to_expert;
  p.conditions = conditions;
  p.tile_flags = tile_flags;
  p.n_blocks = n_blocks;
  p.B = B;
  p.E = E;
  p.n_total = 2 * I;
  p.bias = bias_gu_dev;
  p.col_scale = w1_col_scale;
  p.act = act_fn;
  p.gate_lo = gate_lo;
  p.gate_hi = gate_hi;
  p.up_lo = up_lo;
  p.up_hi = up_hi;
  p.m_codes = static_cast<uint8_t*>(m_bf16);
  p.I = I;
  p.status = status;
  return run_gemm(0, static_cast<const uint8_t*>(x_bf16), static_cast<const uint8_t*>(w1_bf16), p, H, impl, nullptr,
                  static_cast<cudaStream_t>(stream), 1);
}

extern "C" int b200moe_dense_gemm2_scale(const void* m_bf16, const void* w2_bf16, const float* w2_col_scale,
                                         const float* bias_d, const int32_t* block_to_expert,
                                         const int32_t* conditions, const int32_t* tile_flags,
                                         const int32_t* token_position_to_id, int hidden_rows, int n_blocks, int B,
                                         int E, int H, int I, const void* affinities, int aff_dtype, int aff_per_row,
                                         void* y_pos_bf16, int32_t* status, int impl, b200moe_stream_t stream) {
  B200MOE_REQUIRE(m_bf16 && w2_bf16 && block_to_expert && y_pos_bf16, B200MOE_ERR_INVALID,
                  "dense_gemm2: null pointer argument");
  B200MOE_REQUIRE(H % 32 == 0 && H > 0 && I % 32 == 0 && I > 0, B200MOE_ERR_INVALID,
                  "dense_gemm2: H and I must be positive multiples of 32 (H = %d, I = %d)", H, I);
  B200MOE_REQUIRE(aff_dtype == B200MOE_F32 || aff_dtype == B200MOE_BF16, B200MOE_ERR_INVALID,
                  "dense_gemm2: affinities must be fp32 or bf16");
  B200MOE_REQUIRE((reinterpret_cast<uintptr_t>(y_pos_bf16) & 31) == 0, B200MOE_ERR_INVALID,
                  "dense_gemm2: y_pos must be 32-byte aligned");
  GemmParams p{};
  p.block_to_expert = block_to_expert;
  p.conditions = conditions;
  p.tile_flags = tile_flags;
  p.tpi = token_position_to_id;
  p.hidden_rows = hidden_rows;
  p.n_blocks = n_blocks;
  p.B = B;
  p.E = E;
  p.n_total = H;
  p.bias = bias_d;
  p.col_scale = w2_col_scale;
  p.aff = affinities;
  p.aff_dtype = aff_dtype;
  p.aff_per_row = aff_per_row;
  p.y_pos = static_cast<__nv_bfloat16*>(y_pos_bf16);
  p.H_out = H;
  p.I = I;
  p.status = status;
  return run_gemm(1, static_cast<const uint8_t*>(m_bf16), static_cast<const uint8_t*>(w2_bf16), p, I, impl, nullptr,
                  static_cast<cudaStream_t>(stream), 1);
}
