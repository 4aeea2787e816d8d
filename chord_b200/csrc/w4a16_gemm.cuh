// W4A16 grouped GEMM for sm_100a: BF16 activations x INT4 weights with one
// BF16 scale per 32-element K group, FP32 accumulation in tensor memory.
//
// One kernel serves the three operators of the reference library
// (chord_kernels/ops.py:8-90): `indexed` (routed rows named by sorted_ids /
// expert_ids / num_tokens_padded), `contiguous` (128-row expert runs named by
// m_indices) and `masked` (per-group valid-row counts).  They differ only in
// how a tile finds its expert, its activation rows and its output rows.
//
// Orientation ("swap-AB"): the 128 weight rows of a tile are the MMA's M
// dimension and the tile's tokens (16..256) are its N dimension, so
//     D[128 weight rows, tokens] += Wdeq[128, 16] * X[tokens, 16]^T
// per K16 step.  The dequantised weights never touch shared memory: dequant
// warps read the packed words the TMA brought in, expand them to BF16 in
// registers and store them straight into tensor memory, from where
// tcgen05.mma takes its A operand.  Activations arrive K-major with the
// 128-byte swizzle: one tiled TMA box per K half where a tile's rows are
// consecutive, a cp.async gather by two helper warps (or, selectable, TMA
// tile::gather4) where sorted_ids names them.
//
// Two shared-memory rings decouple the HBM stream from the token side: a
// weight/scale stage is free again as soon as the dequant warps have read it
// into registers (its content lives on in tensor memory), so that ring can be
// deep enough (20+ stages of 9 KB) to cover HBM latency, while an activation
// stage stays until the MMAs that read it have completed.
//
// The issue loops (TMA: one thread, MMA: a warp with an elected lane) are kept free of
// divisions and descriptor rebuilds: each is one chain of dependent instructions, of which
// a warp retires one only every few cycles, and at decode sizes a K16 MMA has roughly 45
// cycles of HBM time to hide behind.
//
// Warp roles (one CTA per SM, persistent):
//   warp 0            producer: TMA for packed weights
//   warp 1            producer: TMA for scales
//   warps 2-3         activations: tiled TMA (one thread), cp.async gather (64 threads)
//                     or TMA gather4 (one warp); warp 2 also allocates tensor memory
//   warps 4-7         MMA issuers; issuer i takes the stages with index = i modulo the
//                     issuer count and owns one accumulator
//   warps 8..8+4G-1   G dequant groups of four warps (one per TMEM lane quarter)
//   last four warps   epilogue: TMEM -> registers -> BF16 -> global, plus the
//                     stream-K reduction through `locks` and the FP32 workspace
// Where the activation rows are consecutive and at most two issuers run (`tiled_roles`), warp 0
// loads weights and scales, warps 1 and 3 issue, and warps 4-7 are a second group of
// epilogue warps.
//
// Why several issuers: an issuer's chain per K16 (its share of the waits, an MMA, its share of
// the commits) is longer than the ~45 cycles in which a 128x16 tile of packed weights
// arrives from HBM per SM.  With small token tiles (decode) the stages are therefore
// dealt to 2 or 4 issuers in different warps, each accumulating into its own
// TMEM columns; the epilogue adds the accumulators in issuer order, so the
// result does not depend on timing.  Large token tiles use a single issuer, tiles of two
// weight blocks one per block.
//
// Scheduling follows the reference's scheme (humming/scheduler.cuh:73-101):
// whole tiles are dealt round-robin to the CTAs while full waves last; the
// remaining tiles are flattened into (tile, k-block) units and split evenly
// over the grid (stream-K).  A tile split this way is finished by the CTA that
// holds its k=0 slice: the other slices write FP32 partials to their workspace
// slot and bump the owner's lock word; the owner waits for the count, adds the
// partials in CTA order (deterministic), rounds once to BF16 and resets the
// lock to zero (reference protocol: humming/epilogue/pipeline.cuh:132-163).
//
// Numerics match the reference's kernels (humming/arith/mainloop_arith.cuh:66-101,
// deep_gemm/ptx/ld_st.cuh:15-40): weight = RN_bf16((code - 8) * scale), products
// and sums in FP32, one rounding to BF16 at the end.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "ptx.cuh"
#include "ring.h"

namespace chord {

enum GemmMode : int32_t { kModeIndexed = 0, kModeContiguous = 1, kModeMasked = 2 };
// How activation rows reach shared memory.  Consecutive rows (contiguous,
// masked) always use one tiled TMA box per 64-wide K half; the routed rows of
// `indexed` are gathered by two helper warps with cp.async (default) or by the
// producer with TMA tile::gather4.
enum XLoadMode : int32_t { kXLoadCpAsync = 0, kXLoadGather4 = 1, kXLoadTiled = 2 };

// Device status bits (OR-ed into *status by a kernel that gave up on a wait).
enum StatusBits : int32_t {
  kStatusProducerTimeout = 1,
  kStatusMmaTimeout = 2,
  kStatusDequantTimeout = 4,
  kStatusEpilogueTimeout = 8,
  kStatusLockTimeout = 16,
};

constexpr int kBlockN = 128;      // weight rows per tile (MMA M)
constexpr int kBlockK = 128;      // K elements per pipeline stage (two 64-wide swizzle atoms)
constexpr int kMaxWStages = 24;   // ring of packed-weight + scale stages
constexpr int kMaxXStages = 8;    // ring of activation stages
// Tensor-memory ring for the dequantised A operand: `a_stages` stages of 64 columns,
// each handed over in two halves of one 64-wide K half (32 columns), so that the
// MMAs of a stage's first half are issued while its second half is still being
// dequantised.  The ring takes the columns the accumulators leave free (4 stages next
// to 256 accumulator columns, 6 next to 128): the deeper it is, the further the
// dequant warps run ahead of the MMA issuers, which hides the barrier round trips
// between them.
constexpr int kMaxAStages = 8;
constexpr int kAColsPerStage = kBlockK / 2;
constexpr int kHelperThreads = 64;  // warps 2-3: activation gather for `indexed`
constexpr int kTmemCols = 512;
constexpr int kMaxTileTokens = 256;
constexpr int kMaxGroups = 512;   // masked: prefix table capacity
constexpr int kMaxMTiles = 2048;  // contiguous: 128-row blocks of the activation tensor
constexpr int kWStageBytes = (kBlockK / 16) * 1024;
constexpr int kSStageBytes = (kBlockK / 32) * 256;

struct GemmParams {
  int32_t mode;
  int32_t x_load;
  int32_t n;            // weight rows per expert
  int32_t k;
  int32_t num_experts;
  int32_t x_rows;       // rows of the activation tensor
  int32_t out_rows;     // rows of the output tensor
  int32_t tile_tokens;  // indexed: block_m; contiguous: 128; masked: tokens per M tile
  int32_t mma_n;        // tile_tokens rounded up to 16
  int32_t top_k;        // indexed
  int32_t max_m;        // masked
  int32_t m_blocks;     // contiguous: m / 128
  int32_t run_part;     // contiguous: 0 = every block; 1 = only the blocks left over when each expert's run of consecutive 128-row blocks is cut into pairs (single-block experts, last block of an odd run); 2 = only the pairs
  int32_t x_box_rows;   // tiled activation loads: rows per TMA box
  int32_t sorted_len;   // indexed: capacity of sorted_ids
  int32_t expert_len;   // indexed: capacity of expert_ids
  int32_t w_stages;     // depth of the weight/scale ring
  int32_t x_stages;     // depth of the activation ring
  int32_t issuers;      // 1, 2 or 4 MMA issuers (and accumulators)
  int32_t ksplit;       // single-issuer layouts: a second issuer takes the second K half of tiles of <= 128 tokens
  int32_t fuse_silu;    // 1 = gate_up with SiLU*mul in the epilogue: a tile is gate block j and up block j (row N/2 + 128 j), out is [rows, N/2]
  int32_t npair;        // 1 = a tile is two neighbouring 128-row weight blocks sharing one activation stage (tiles of <= 128 tokens)
  int32_t pair;         // 1 = launched as clusters of two CTAs: a tile is two neighbouring 128-row weight blocks, one per CTA, multiplied by one tcgen05.mma.cta_group::2 stream; each CTA loads half of the tile's token rows
  int32_t a_stages;     // depth of the TMEM A ring; accumulators start at column 64 * a_stages
  int32_t num_locks;
  int32_t slot_ordered; // host side only (indexed): row s of x is the row of routing slot s, so the rows load as consecutive boxes without a copy
  int32_t pdl;          // host side only: launch with the programmatic stream-serialization attribute
  int32_t lock_spins;   // polls (64 ns apart) a stream-K owner spends on its lock word before it gives up
  const int32_t* sorted_ids;
  const int32_t* expert_ids;
  const int32_t* num_tokens_padded;
  const int32_t* m_indices;
  const int32_t* masked_m;
  const __nv_bfloat16* x;
  __nv_bfloat16* out;
  void* const* out_row_ptr;  // optional (indexed): out_row_ptr[id] = address of the row that receives routed id's result
  float* workspace;     // grid * 128 * mma_n floats
  int32_t* locks;
  int32_t* status;
};

struct TileInfo {
  int32_t n0;      // first weight row
  int32_t expert;
  int32_t ntok;    // token slots of the tile that carry a row (one past the last one)
  int32_t rows;    // token slots whose output rows the tile writes (contiguous: whole blocks)
  int32_t base;    // indexed: first sorted_ids slot; contiguous: first row; masked: first row of the group
  int32_t m0;      // masked: first row inside the group
  int32_t limit;   // masked: masked_m of the group
  int32_t mma_n;   // MMA N of this tile: ntok rounded up to 16
  bool valid;
};

enum SegType : int32_t { kSegFull = 0, kSegOwner = 1, kSegContrib = 2 };

struct Segment {
  int32_t tile;
  int32_t kb, ke;  // k-block range [kb, ke)
  int32_t type;
  int32_t peer;    // owner: number of contributors; contributor: owner CTA
};

// Shortest stream-K slice in K steps.  A finer split costs more in partial sums and per-slice
// set-up than the extra parallelism returns.
constexpr int32_t kMinSlice = 8;

// Enumerates the work of one CTA; every warp role walks the same sequence.
struct SegmentIterator {
  int32_t grid, cta, ki;
  int32_t dp_waves, dp_tiles, wave;
  int64_t units, u0, u1;
  int32_t geff;

  // `whole_short_tiles` (decode kernels, whose workers commonly outnumber the tiles): tiles
  // shorter than kMinSlice are dealt out whole instead of several to a worker (8 experts of 1024 x
  // 512, four steps per tile: 12.8 us with slices of eight, 8.7 us with whole tiles).  Longer tiles
  // keep slices of eight: with four, 64 experts of 1024 x 1024 (512 tiles of eight steps, 592
  // workers) were cut up instead of taken whole, 17.9 us against 14.0 us with 1 row per expert.
  __host__ __device__ void init(int32_t tiles, int32_t k_iters, int32_t grid_, int32_t cta_,
                                bool whole_short_tiles = false) {
    grid = grid_;
    cta = cta_;
    ki = k_iters;
    dp_waves = tiles / grid;
    int32_t sk_tiles = tiles - dp_waves * grid;
    // A tail of less than kMinSlice steps per CTA would be cut into slivers: fold one full wave into it.
    if (dp_waves > 0 && sk_tiles > 0 && static_cast<int64_t>(sk_tiles) * ki < static_cast<int64_t>(kMinSlice) * grid) {
      dp_waves -= 1;
      sk_tiles += grid;
    }
    dp_tiles = dp_waves * grid;
    wave = 0;
    units = static_cast<int64_t>(sk_tiles) * ki;
    // No slice shorter than kMinSlice (unless the whole tail is).
    int64_t slices = units / kMinSlice > 0 ? units / kMinSlice : (units > 0 ? 1 : 0);
    if (whole_short_tiles && ki < kMinSlice) slices = sk_tiles;
    geff = slices < grid ? static_cast<int32_t>(slices) : grid;
    if (cta < geff) {
      u0 = cta * units / geff;
      u1 = (cta + 1) * units / geff;
    } else {
      u0 = u1 = 0;
    }
  }

  __host__ __device__ int32_t cta_of_unit(int64_t u) const {
    return static_cast<int32_t>(((u + 1) * geff - 1) / units);
  }

  __host__ __device__ bool next(Segment& s) {
    if (wave < dp_waves) {
      s.tile = wave * grid + cta;
      s.kb = 0;
      s.ke = ki;
      s.type = kSegFull;
      s.peer = 0;
      ++wave;
      return true;
    }
    if (u0 >= u1) return false;
    const int64_t t = u0 / ki;
    const int32_t kb = static_cast<int32_t>(u0 - t * ki);
    const int64_t room = u1 - u0;
    const int32_t ke = (ki - kb) < room ? ki : static_cast<int32_t>(kb + room);
    s.tile = dp_tiles + static_cast<int32_t>(t);
    s.kb = kb;
    s.ke = ke;
    if (kb == 0 && ke == ki) {
      s.type = kSegFull;
      s.peer = 0;
    } else if (kb == 0) {
      s.type = kSegOwner;
      s.peer = cta_of_unit(t * ki + ki - 1) - cta;
    } else {
      s.type = kSegContrib;
      s.peer = cta_of_unit(t * ki);
    }
    u0 += ke - kb;
    return true;
  }
};

struct __align__(16) GemmShared {
  uint64_t wfull[kMaxWStages];   // weights + scales landed        (2 producer arrivals + bytes)
  uint64_t wempty[kMaxWStages];  // dequant warps have read them   (4 arrivals)
  uint64_t xfull[kMaxXStages];   // activations landed
  uint64_t xempty[kMaxXStages];  // the stage's MMAs have completed (1 commit)
  uint64_t afull[2 * kMaxAStages];   // per K half: dequantised operand stored (4 arrivals)
  uint64_t aempty[2 * kMaxAStages];  // per K half: its MMAs have completed (1 commit)
  uint64_t dfull[2];
  uint64_t dempty[2];
  uint64_t mma_done;             // all MMAs issued have completed (one commit per issuer, at the end)
  uint32_t tmem_base;
  uint32_t abort_flag;
  int32_t m_blocks;
  volatile uint32_t epilogue_failed;
  int32_t x_slots;                   // helpers: token slots of the current tile that carry a row
  int32_t out_row[kMaxTileTokens];   // epilogue: output row per token slot, -1 = skip
  __align__(16) __nv_bfloat16 stage[8][16][32];  // epilogue: per-warp transpose buffer (second set: the pair kernel's second epilogue group)
  int32_t x_row[kMaxTileTokens];     // producer (cp.async variant): activation row per slot
  int32_t group_prefix[kMaxGroups + 1];  // masked: first M tile of each group
  // contiguous: M tiles after merging neighbouring 128-row blocks of one expert:
  // expert | first block << 15 | (256 rows ? 1 : 0) << 31
  uint32_t mtile[kMaxMTiles];
  // contiguous, indexed: token slots of each M tile that carry a row (padding rows at
  // the end of an expert's run, sentinels at the end of a routing block, do not): the
  // tile's MMA runs with N = that count rounded up to 16, not with the full block.
  uint16_t tile_rows[kMaxMTiles];
  int32_t have_tile_rows;
};

__device__ __forceinline__ TileInfo decode_tile(const GemmParams& p, const GemmShared& sh,
                                                int32_t tile, uint32_t rank = 0) {
  TileInfo t;
  // With `npair` a tile spans two neighbouring 128-row weight blocks (n0 and n0 + 128).
  // With fused SiLU*mul the two blocks are gate block n0 and up block N/2 + n0.
  // With `pair` the two blocks belong to the two CTAs of the cluster: n0 is this CTA's.
  const int32_t wide = p.npair | p.pair;
  const int32_t n_blocks = p.fuse_silu ? (p.n >> 1) / kBlockN : p.n / (kBlockN << wide);
  const int32_t mb = tile / n_blocks;
  t.n0 = (tile - mb * n_blocks) * (p.fuse_silu ? kBlockN : (kBlockN << wide)) +
         static_cast<int32_t>(rank) * kBlockN;
  t.m0 = 0;
  t.limit = 0;
  t.mma_n = p.mma_n;
  if (p.mode == kModeIndexed) {
    t.expert = __ldg(p.expert_ids + mb);
    t.ntok = sh.have_tile_rows ? static_cast<int32_t>(sh.tile_rows[mb]) : p.tile_tokens;
    t.rows = t.ntok;
    t.base = mb * p.tile_tokens;
  } else if (p.mode == kModeContiguous) {
    const uint32_t info = sh.mtile[mb];
    t.expert = static_cast<int32_t>(info & 0x7FFFu);
    t.rows = (info >> 31) ? 256 : 128;
    t.ntok = static_cast<int32_t>(sh.tile_rows[mb]);
    t.base = static_cast<int32_t>((info >> 15) & 0xFFFFu) * 128;
  } else {
    // Largest g with group_prefix[g] <= mb.
    int32_t lo = 0, hi = p.num_experts;
    while (hi - lo > 1) {
      const int32_t mid = (lo + hi) >> 1;
      if (sh.group_prefix[mid] <= mb) lo = mid; else hi = mid;
    }
    t.expert = lo;
    t.m0 = (mb - sh.group_prefix[lo]) * p.tile_tokens;
    int32_t mm = __ldg(p.masked_m + lo);
    mm = mm < 0 ? 0 : (mm > p.max_m ? p.max_m : mm);
    t.limit = mm;
    const int32_t left = mm - t.m0;
    t.ntok = left < p.tile_tokens ? left : p.tile_tokens;
    t.rows = t.ntok;
    t.base = lo * p.max_m;
  }
  t.mma_n = (t.ntok + 15) & ~15;
  t.valid = t.expert >= 0 && t.expert < p.num_experts && t.ntok > 0;
  return t;
}

// Activation row feeding token slot `slot` of a tile; `p.x_rows` (one past the
// end) for a slot that carries no token, which the TMA reads as zeros.
__device__ __forceinline__ int32_t x_row_of(const GemmParams& p, const TileInfo& t, int32_t slot) {
  if (p.mode == kModeIndexed) {
    const int32_t id = __ldg(p.sorted_ids + t.base + slot);
    const int32_t row = id / p.top_k;
    return (id >= 0 && row < p.x_rows) ? row : p.x_rows;
  }
  if (p.mode == kModeContiguous) return t.base + slot;
  return (t.m0 + slot < t.limit) ? t.base + t.m0 + slot : p.x_rows;
}

// Output row written by token slot `slot`, or -1.
__device__ __forceinline__ int32_t out_row_of(const GemmParams& p, const TileInfo& t, int32_t slot) {
  if (slot >= t.rows) return -1;
  if (p.mode == kModeIndexed) {
    const int32_t id = __ldg(p.sorted_ids + t.base + slot);
    return (id >= 0 && id < p.out_rows) ? id : -1;
  }
  if (p.mode == kModeContiguous) return t.base + slot;
  return (t.m0 + slot < t.limit) ? t.base + t.m0 + slot : -1;
}

// Dequantisation.  A packed word (rows r and r+8, K offsets {2q, 2q+1, 2q+8, 2q+9} of a K16
// block; humming/kernel/repack.cuh:8-33) becomes four BF16 pairs in the order of
// tcgen05.st.16x128b, which is also that of the A fragment of mma.m16n8k16:
//   d0 = (row r,   K 2q..2q+1)     d1 = (row r+8, K 2q..2q+1)
//   d2 = (row r,   K 2q+8..2q+9)   d3 = (row r+8, K 2q+8..2q+9)
// each RN_bf16((code - 8) * scale), the reference's weight, subnormal ones included.
//
// One mask and one fused multiply-add per pair: a BF16 bit pattern below 0x100 is the number
// pattern * 2^-133 (subnormals and the first binade have the same spacing), so a nibble in bits
// 0-3 of a half is code * 2^-133 and one in bits 4-7 is code * 2^-129 as it stands; no exponent
// has to be put in and its 128 taken out again.  Then code * 2^-133 * (scale * 2^133) - scale * 8 =
// (code - 8) * scale, rounded once; both factors are exact in BF16 as long as scale * 2^133 stays
// finite, which is |scale| < 2^-5 (weights of up to 1/4).  A warp that meets another scale in a
// 128-wide stage takes dequant_fragment_any for that stage: 128 + code, minus 136, times the scale.
//
// Per word that is one shift, four masks and four multiply-adds, and four operations per pair of
// scales (shared by two words), against three shifts, four masks, four
// subtractions and four multiplications: the decode kernel is bound by the instructions of its
// warps.  48 experts of 4096 x 7168, replayed graph in a burst, us, a build with dequant_fragment_any
// alone (without the later changes to both kernels) / scales of 2^-5 and more now / scales below
// 2^-5 now: 5 rows each 155 / 158 / 137, 20 rows 276 / 235 / 215, 28 rows 280 / 276 / 261; general kernel, 60 rows
// 279 / 292 / 256, 85 rows 305 / 317 / 290.
constexpr uint32_t kSmallScaleEnd = 0x3D00u;  // 2^-5 as BF16

struct ScaleFactors {
  uint32_t lo, hi, off;  // scale * 2^133, scale * 2^129, scale * -8; low half row r, high half row r+8
};

// 2^127 is BF16's largest power of two; the rest is multiplied too, or added to the exponents (scale *
// 2^127 is a normal number below 2^122, or zero, which becomes 2^-121, whose products with a code's
// 2^-129 vanish in the rounding).  The decode kernel adds, the general one multiplies: 48 experts of
// 4096 x 7168, us, multiplying / adding: 5 rows 140 / 138, 20 rows 217 / 214, 28 rows 258 / 261 there, 40 rows 256 /
// 260, fused 85 rows 316 / 319 here.
template <bool kAddExponents>
__device__ __forceinline__ ScaleFactors scale_factors(uint32_t scales) {
  ScaleFactors f;
  uint32_t t;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(t) : "r"(scales), "r"(0x7F007F00u));
  if constexpr (kAddExponents) {
    f.lo = t + 0x03000300u;
    f.hi = t + 0x01000100u;
  } else {
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(f.lo) : "r"(t), "r"(0x42804280u));
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(f.hi) : "r"(t), "r"(0x40804080u));
  }
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(f.off) : "r"(scales), "r"(0xC100C100u));
  return f;
}

// Scales are broadcast with mov.b32 unpack/pack, which the assembler folds into the operand
// selectors of the arithmetic (a byte-permute per broadcast takes a slot of the half-rate integer
// pipe each).
__device__ __forceinline__ void dequant_fragment(uint32_t w, const ScaleFactors& f, uint32_t& d0, uint32_t& d1,
                                                 uint32_t& d2, uint32_t& d3) {
  asm("{\n\t"
      ".reg .b32 v0, v1, v2, v3, u, l0, l1, h0, h1, o0, o1;\n\t"
      ".reg .b16 a, b;\n\t"
      "mov.b32 {a, b}, %5;\n\t"
      "mov.b32 l0, {a, a};\n\t"
      "mov.b32 l1, {b, b};\n\t"
      "mov.b32 {a, b}, %6;\n\t"
      "mov.b32 h0, {a, a};\n\t"
      "mov.b32 h1, {b, b};\n\t"
      "mov.b32 {a, b}, %7;\n\t"
      "mov.b32 o0, {a, a};\n\t"
      "mov.b32 o1, {b, b};\n\t"
      "shr.u32 u, %4, 8;\n\t"
      "and.b32 v0, %4, 0x000F000F;\n\t"
      "and.b32 v1, u, 0x000F000F;\n\t"
      "and.b32 v2, %4, 0x00F000F0;\n\t"
      "and.b32 v3, u, 0x00F000F0;\n\t"
      "fma.rn.bf16x2 %0, v0, l0, o0;\n\t"
      "fma.rn.bf16x2 %1, v1, l1, o1;\n\t"
      "fma.rn.bf16x2 %2, v2, h0, o0;\n\t"
      "fma.rn.bf16x2 %3, v3, h1, o1;\n\t"
      "}\n"
      : "=&r"(d0), "=&r"(d1), "=&r"(d2), "=&r"(d3)
      : "r"(w), "r"(f.lo), "r"(f.hi), "r"(f.off));
}

// For any scale, infinite and NaN ones too.
__device__ __forceinline__ void dequant_fragment_any(uint32_t w, uint32_t scales, uint32_t& d0, uint32_t& d1,
                                                     uint32_t& d2, uint32_t& d3) {
  asm("{\n\t"
      ".reg .b32 v0, v1, v2, v3, s1, s2, s3, lo, hi;\n\t"
      ".reg .b16 a, b;\n\t"
      "mov.b32 {a, b}, %5;\n\t"
      "mov.b32 lo, {a, a};\n\t"
      "mov.b32 hi, {b, b};\n\t"
      "shr.u32 s1, %4, 4;\n\t"
      "shr.u32 s2, %4, 8;\n\t"
      "shr.u32 s3, %4, 12;\n\t"
      "lop3.b32 v0, %4, 0x000F000F, 0x43004300, 0xEA;\n\t"
      "lop3.b32 v1, s1, 0x000F000F, 0x43004300, 0xEA;\n\t"
      "lop3.b32 v2, s2, 0x000F000F, 0x43004300, 0xEA;\n\t"
      "lop3.b32 v3, s3, 0x000F000F, 0x43004300, 0xEA;\n\t"
      "sub.rn.bf16x2 v0, v0, %6;\n\t"
      "sub.rn.bf16x2 v1, v1, %6;\n\t"
      "sub.rn.bf16x2 v2, v2, %6;\n\t"
      "sub.rn.bf16x2 v3, v3, %6;\n\t"
      "mul.rn.bf16x2 %0, v0, lo;\n\t"
      "mul.rn.bf16x2 %1, v2, hi;\n\t"
      "mul.rn.bf16x2 %2, v1, lo;\n\t"
      "mul.rn.bf16x2 %3, v3, hi;\n\t"
      "}\n"
      : "=&r"(d0), "=&r"(d1), "=&r"(d2), "=&r"(d3)
      : "r"(w), "r"(scales), "r"(0x43084308u));
}


// What two words with the same scales share, and one of them as a fragment.
template <bool kAnyScale, bool kAddExponents>
struct Dequant {
  ScaleFactors f;  // kAnyScale: f.lo is the scales
  __device__ __forceinline__ explicit Dequant(uint32_t scales) {
    if constexpr (kAnyScale) f.lo = scales;
    else f = scale_factors<kAddExponents>(scales);
  }
  __device__ __forceinline__ void operator()(uint32_t w, uint32_t& d0, uint32_t& d1, uint32_t& d2, uint32_t& d3) const {
    if constexpr (kAnyScale) dequant_fragment_any(w, f.lo, d0, d1, d2, d3);
    else dequant_fragment(w, f, d0, d1, d2, d3);
  }
};

// Whether all scales that the warp's lanes look at are below 2^-5 in magnitude; infinite and NaN
// ones are not.  Must be called by all 32 lanes.
__device__ __forceinline__ bool small_scales(uint2 scales) {
  constexpr uint32_t carry = (0x8000u - kSmallScaleEnd) * 0x10001u;  // reaches the sign bit from the end on
  const uint32_t over = (((scales.x & 0x7FFF7FFFu) + carry) | ((scales.y & 0x7FFF7FFFu) + carry)) & 0x80008000u;
  return __all_sync(0xffffffffu, over == 0);
}

// Activation ring cut into sub-slots of 128 token rows (both 64-wide K halves, 32 KB).
// A stage of a tile of at most 128 tokens takes one sub-slot, a 256-token stage an
// aligned pair (one sub-slot may be skipped to align), so that a launch mixing small and
// large tiles gives the small ones a ring twice as deep.  Every party keeps a cursor
// and one phase bit per sub-slot barrier of its own; all walk the same tile sequence.
// A pair is tracked by the barriers of its even sub-slot alone (the MMA issuer is the
// critical path of large tiles: no second wait or commit for it); the odd sub-slot's
// barriers keep the state of its last use on its own, which the loader checks without
// consuming it before it overwrites the memory.  That use is never outstanding when the
// odd sub-slot is next taken on its own, because the ring always passes through the even
// one (and so waits for the pair) first.
struct XSubRing {
  uint32_t next = 0;
  uint32_t phases = 0;
  __device__ __forceinline__ uint32_t take(bool pair, uint32_t count) {
    if (pair && (next & 1u)) next = next + 1u == count ? 0u : next + 1u;
    const uint32_t first = next;
    next += pair ? 2u : 1u;
    if (next >= count) next -= count;
    return first;
  }
  __device__ __forceinline__ uint32_t phase(uint32_t slot) const { return (phases >> slot) & 1u; }
  __device__ __forceinline__ void flip(uint32_t slot) { phases ^= 1u << slot; }
};

// Waits (bounded) for the latest use of every stage of a ring: nothing may stay in flight towards
// shared memory when a CTA retires, also when whoever reads the stages has given up.
__device__ __forceinline__ void drain_ring(const uint64_t* full, const StageCursor& issued, uint32_t stages) {
  for (uint32_t i = 0; i < stages; ++i) ptx::mbar_drain(ptx::smem_u32(full + i), issued.last_phase(i));
}

// kPair: clusters of two CTAs (p.pair).  kHold: two weight blocks per tile (on one CTA or on a
// pair), without SiLU*mul; whole tiles are held in registers while they are stored (see the
// epilogue).
template <int kDequantGroups, bool kPair, bool kHold>
__global__ void __launch_bounds__(32 * (12 + 4 * kDequantGroups), 1)
w4a16_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_s,
                  const __grid_constant__ CUtensorMap tm_x, const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  // Dynamic shared memory: [X ring | W ring | S ring | GemmShared], 1024-aligned.
  // One X stage holds two K halves, each mma_n rows of 128 bytes.
  const uint32_t raw_addr = ptx::smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
  uint8_t* smem = smem_raw + pad;
  // `pair`: this CTA is rank 0 (leader: issues the MMAs for both) or 1 of a cluster of two
  // and holds half of a tile's token rows.
  // (A kernel that contains cta_group::2 instructions can only be launched as clusters of
  // two, hence an instantiation of its own.)
  constexpr bool pair = kPair;
  uint32_t rank = 0;
  if constexpr (kPair) rank = ptx::cluster_ctarank();
  const uint32_t x_half_bytes = (static_cast<uint32_t>(p.mma_n) >> p.pair) * 128u;
  const uint32_t x_stage_bytes = 2u * x_half_bytes;
  const uint32_t w_stages = static_cast<uint32_t>(p.w_stages);
  const uint32_t x_stages = static_cast<uint32_t>(p.x_stages);
  uint8_t* smem_x = smem;
  uint8_t* smem_w = smem_x + x_stages * x_stage_bytes;
  uint8_t* smem_s = smem_w + w_stages * kWStageBytes;
  GemmShared& sh = *reinterpret_cast<GemmShared*>(smem_s + w_stages * kSStageBytes);

  // Read back through a shuffle so that the compiler knows the warp index (and what is
  // derived from it: roles, ring positions, barrier and tensor-memory addresses) to be
  // the same in all lanes and keeps them in uniform registers.
  const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const uint32_t lane = threadIdx.x & 31;
  constexpr uint32_t kFirstIssuerWarp = 4;
  constexpr uint32_t kFirstDequantWarp = 8;
  constexpr uint32_t kFirstEpilogueWarp = 8 + 4 * kDequantGroups;
  // Accumulators: `ni` issuers x `d_bufs` buffers of `d_cols` columns each in the
  // 256 TMEM columns after the A ring; buffer d of issuer i starts at column
  // 64 * a_stages + (d * ni + i) * d_cols.
  // With `ksplit` (layouts whose token tile exceeds 64) there are two issuers that do
  // not take turns: on tiles of at most 128 tokens issuer 0 takes the first 64-wide K
  // half of every stage and issuer 1 the second, each into its own 128-column
  // accumulator; on larger tiles issuer 0 does both halves into all 256 columns and
  // issuer 1 only keeps the barriers' phases moving.  One tcgen05.mma costs its issuing
  // thread ~100 cycles on a busy SM whatever its size, so a lone issuer caps small
  // tiles at ~900 cycles per stage.
  const bool ksplit = p.ksplit != 0;
  // `npair`: two issuers as well, but issuer i (with dequant group i) owns the weight block
  // n0 + 128 i of the tile: weight/scale stages alternate between the two blocks, one
  // activation stage serves both, and the two accumulators are two output blocks instead
  // of two partial sums.  An activation tile then crosses from L2 to the SM once per 256
  // weight rows instead of once per 128: with 128-row tiles the kernel was bound by that
  // traffic (about 10 TB/s between L2 and the SMs), not by the tensor pipe.
  static_assert(kHold || !kPair, "tiles on CTA pairs are always held");
  const bool npair = !kPair && (kHold || p.npair != 0);
  const int32_t w_per_kb = npair ? 2 : 1;  // weight/scale ring entries per K block
  // 256-token layouts with consecutive activation rows: sub-slot ring (see XSubRing).
  const bool subslots = ksplit && p.x_load == kXLoadTiled && p.mma_n == 256;
  constexpr uint32_t kSubBytes = 128u * 256u;
  const uint32_t ni = ksplit ? 2u : static_cast<uint32_t>(p.issuers);
  const uint32_t d_cols = ksplit ? 128u : static_cast<uint32_t>(p.mma_n);
  const uint32_t a_stages = static_cast<uint32_t>(p.a_stages);
  const uint32_t d_col0 = a_stages * kAColsPerStage;
  const uint32_t d_bufs = 2u * ni * d_cols <= kTmemCols - d_col0 ? 2u : 1u;
  const int32_t k_iters = (p.k + kBlockK - 1) / kBlockK;
  const bool k_tail_half = (p.k % kBlockK) != 0;  // last stage carries 64 K values only
  // Consecutive activation rows need one loading thread (warp 2) instead of two gathering
  // warps, and at most two issuers: warp 0 then feeds both the weight and the scale ring,
  // the issuers sit in warps 1 and 3, and warps 4-7 are a second group of epilogue warps
  // taking every other 16-column chunk.  Accumulators of 128 columns and more are
  // single-buffered, so the tensor core idles while a tile is drained: with K = 2048 the
  // four-warp drain was a quarter of the time of a two-block tile.
  const bool tiled_roles = kHold || (p.x_load == kXLoadTiled && ni <= 2u);
  const uint32_t epi_threads = tiled_roles ? 256u : 128u;

  // ------------------------------------------------------------------ setup --
  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tm_w);
    ptx::prefetch_tensormap(&tm_s);
    ptx::prefetch_tensormap(&tm_x);
    for (uint32_t s = 0; s < w_stages; ++s) {
      ptx::mbar_init(ptx::smem_u32(&sh.wfull[s]), 2);
      ptx::mbar_init(ptx::smem_u32(&sh.wempty[s]), 4);
    }
    // One arrival per gathering warp, or one transaction-count arrival.
    const uint32_t xfull_count = p.x_load == kXLoadCpAsync ? kHelperThreads / 32 : 1u;
    for (uint32_t s = 0; s < (subslots ? 2u * x_stages : x_stages); ++s) {
      ptx::mbar_init(ptx::smem_u32(&sh.xfull[s]), xfull_count);
      ptx::mbar_init(ptx::smem_u32(&sh.xempty[s]), (ksplit || npair) ? 2 : 1);
    }
    // `pair`: the leader's afull / dempty collect the arrivals of both CTAs' warps (four
    // dequant warps per stage, eight epilogue warps per CTA); the leader's commits reach
    // xempty / aempty / dfull of both CTAs.
    for (uint32_t a = 0; a < 2 * a_stages; ++a) {
      ptx::mbar_init(ptx::smem_u32(&sh.afull[a]), pair ? 8 : 4);
      ptx::mbar_init(ptx::smem_u32(&sh.aempty[a]), 1);
    }
    for (uint32_t d = 0; d < 2; ++d) {
      ptx::mbar_init(ptx::smem_u32(&sh.dfull[d]), ni);
      ptx::mbar_init(ptx::smem_u32(&sh.dempty[d]), (tiled_roles ? 8u : 4u) << p.pair);
    }
    ptx::mbar_init(ptx::smem_u32(&sh.mma_done), ni);
    sh.abort_flag = 0;
    sh.epilogue_failed = 0;
    ptx::fence_barrier_init();
  }
  if (warp == 2) {
    if constexpr (kPair) {
      ptx::tmem_alloc_pair(ptx::smem_u32(&sh.tmem_base), kTmemCols);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(ptx::smem_u32(&sh.tmem_base), kTmemCols);
      ptx::tmem_relinquish();
    }
  }
  // Token slots no load ever fills must not hold NaN patterns.
  for (uint32_t i = threadIdx.x; i < x_stages * x_stage_bytes / 16; i += blockDim.x) {
    reinterpret_cast<uint4*>(smem_x)[i] = make_uint4(0, 0, 0, 0);
  }
  // Up to here nothing an earlier kernel of the stream may still be writing has been
  // read: with programmatic dependent launch the set-up above overlaps that kernel's tail.
  ptx::grid_dependency_wait();
  // Number of M tiles.
  if (p.mode == kModeMasked) {
    if (threadIdx.x == 0) {
      int32_t acc = 0;
      for (int32_t g = 0; g < p.num_experts; ++g) {
        sh.group_prefix[g] = acc;
        int32_t mm = __ldg(p.masked_m + g);
        mm = mm < 0 ? 0 : (mm > p.max_m ? p.max_m : mm);
        acc += (mm + p.tile_tokens - 1) / p.tile_tokens;
      }
      sh.group_prefix[p.num_experts] = acc;
      sh.m_blocks = acc;
    }
  } else if (p.mode == kModeIndexed) {
    if (threadIdx.x == 0) {
      int32_t padded = __ldg(p.num_tokens_padded);
      padded = padded < 0 ? 0 : (padded > p.sorted_len ? p.sorted_len : padded);
      int32_t blocks = padded / p.tile_tokens;
      sh.m_blocks = blocks > p.expert_len ? p.expert_len : blocks;
      sh.have_tile_rows = sh.m_blocks <= kMaxMTiles ? 1 : 0;
    }
    __syncthreads();
    // One warp per routing block: one past the last slot whose id names a row.
    if (sh.have_tile_rows) {
      for (int32_t b = static_cast<int32_t>(warp); b < sh.m_blocks; b += static_cast<int32_t>(blockDim.x >> 5)) {
        int32_t last = 0;
        for (int32_t i = static_cast<int32_t>(lane); i < p.tile_tokens; i += 32) {
          const int32_t id = __ldg(p.sorted_ids + b * p.tile_tokens + i);
          if (id >= 0 && id < p.out_rows && id / p.top_k < p.x_rows) last = i + 1;
        }
        last = __reduce_max_sync(0xffffffffu, last);
        if (lane == 0) sh.tile_rows[b] = static_cast<uint16_t>(last);
      }
    }
  } else {
    // Expert of every 128-row block (its first row names it), then one warp drops padding
    // blocks and merges neighbouring blocks of one expert into 256-token tiles where the layout
    // takes those (the MMA runs at full rate only with N = 256).
    for (int32_t i = threadIdx.x; i < p.m_blocks; i += blockDim.x) {
      sh.mtile[i] = static_cast<uint32_t>(__ldg(p.m_indices + i * 128));
    }
    // One warp per block: one past its last row that belongs to an expert.
    for (int32_t b = static_cast<int32_t>(warp); b < p.m_blocks; b += static_cast<int32_t>(blockDim.x >> 5)) {
      int32_t last = 0;
#pragma unroll
      for (int32_t j = 0; j < 4; ++j) {
        const int32_t i = 32 * j + static_cast<int32_t>(lane);
        if (__ldg(p.m_indices + b * 128 + i) >= 0) last = i + 1;
      }
      last = __reduce_max_sync(0xffffffffu, last);
      if (lane == 0) sh.tile_rows[b] = static_cast<uint16_t>(last);
    }
    __syncthreads();
    // 32 blocks at a time, one per lane: a launch waits for this, and a single thread that walked
    // the blocks took 8 us for 48 of them and 12 for 96.  Within an expert's run of blocks a tile
    // starts at every even position (every position, where tiles are 128 tokens and all
    // blocks are taken).  In place: the write position never passes the read position.
    if (warp == 0) {
      int32_t count = 0, carry_expert = -1, carry_start = 0;
      for (int32_t i0 = 0; i0 < p.m_blocks; i0 += 32) {
        const int32_t i = i0 + static_cast<int32_t>(lane);
        const int32_t e = i < p.m_blocks ? static_cast<int32_t>(sh.mtile[i]) : -1;
        const int32_t next = i + 1 < p.m_blocks ? static_cast<int32_t>(sh.mtile[i + 1]) : -1;
        const int32_t rows = i < p.m_blocks ? sh.tile_rows[i] : 0;
        const int32_t next_rows = i + 1 < p.m_blocks ? sh.tile_rows[i + 1] : 0;
        int32_t prev = __shfl_up_sync(0xffffffffu, e, 1);
        if (lane == 0) prev = carry_expert;
        const uint32_t starts = __ballot_sync(0xffffffffu, e != prev) & (0xffffffffu >> (31u - lane));
        const int32_t run_start = starts != 0 ? i0 + 31 - __clz(static_cast<int32_t>(starts)) : carry_start;
        const bool valid = e >= 0 && e < p.num_experts;
        const bool even = ((i - run_start) & 1) == 0;
        const bool paired = next == e;  // (at an even position: with the next block)
        bool emit = valid && even;
        if (p.run_part == 1) emit = emit && !paired;
        else if (p.run_part == 2) emit = emit && paired;
        else if (p.tile_tokens != 256) emit = valid;
        const bool merged = p.tile_tokens == 256 && paired;
        const uint32_t mask = __ballot_sync(0xffffffffu, emit);
        carry_expert = __shfl_sync(0xffffffffu, e, 31);
        carry_start = __shfl_sync(0xffffffffu, run_start, 31);
        __syncwarp();  // all 32 blocks have been read
        if (emit) {
          const int32_t at = count + __popc(mask & ((1u << lane) - 1u));
          sh.tile_rows[at] = static_cast<uint16_t>(merged ? 128 + next_rows : rows);
          sh.mtile[at] = static_cast<uint32_t>(e) | (static_cast<uint32_t>(i) << 15) | (merged ? 0x80000000u : 0u);
        }
        count += __popc(mask);
        __syncwarp();
      }
      if (lane == 0) sh.m_blocks = count;
    }
  }
  ptx::fence_proxy_async();
  ptx::tc_fence_before();
  __syncthreads();
  // the peer's barriers must be initialised before anything arrives on them
  if constexpr (kPair) ptx::cluster_sync();
  ptx::tc_fence_after();
  ptx::grid_launch_dependents();

  const uint32_t tmem_base = __shfl_sync(0xffffffffu, sh.tmem_base, 0);  // uniform, see `warp`
  volatile uint32_t* abort_flag = &sh.abort_flag;
  // Offset that turns a shared-memory address of this CTA into the cluster address of the
  // same location in the leader (rank 0).
  const uint32_t sh_addr = ptx::smem_u32(&sh);
  uint32_t to_leader = 0;
  if constexpr (kPair) to_leader = ptx::map_to_cta(sh_addr, 0) - sh_addr;
  const int32_t tiles = __shfl_sync(0xffffffffu, sh.m_blocks, 0) *
                        (p.fuse_silu ? (p.n >> 1) / kBlockN : p.n / (kBlockN << (p.npair | p.pair)));
  // Both CTAs of a pair walk the same sequence of tiles.
  SegmentIterator iter;
  iter.init(tiles, k_iters, static_cast<int32_t>(gridDim.x >> p.pair),
            static_cast<int32_t>(blockIdx.x >> p.pair));
  Segment seg;

  if (warp == 0 && tiled_roles) {
    // ------------------------------ producer of both rings (packed weights, scales) --
    if (lane == 0) {
      StageCursor cur;
      bool ok = true;
      while (ok && iter.next(seg)) {
        const TileInfo t = decode_tile(p, sh, seg.tile, rank);
        if (!t.valid) continue;
        // to the tile's second weight block: the next 128 rows, or the up rows of a fused gate_up
        const int32_t block_step = p.fuse_silu ? (p.n >> 1) : kBlockN;
        int32_t w_row = t.expert * (p.k / 16) + seg.kb * (kBlockK / 16);
        int32_t s_row = t.expert * (p.k / 32) + seg.kb * (kBlockK / 32);
        for (int32_t kb = seg.kb; ok && kb < seg.ke; ++kb) {
          for (int32_t sub = 0; sub < w_per_kb; ++sub) {
            if (!ptx::mbar_wait(ptx::smem_u32(&sh.wempty[cur.s]), cur.ph ^ 1u, abort_flag)) {
              ok = false;
              break;
            }
            const uint32_t full = ptx::smem_u32(&sh.wfull[cur.s]);
            ptx::mbar_arrive_expect_tx(full, kWStageBytes);
            ptx::tma_load_2d(ptx::smem_u32(smem_w + cur.s * kWStageBytes), &tm_w, full,
                             2 * (t.n0 + sub * block_step), w_row);
            ptx::mbar_arrive_expect_tx(full, kSStageBytes);
            ptx::tma_load_2d(ptx::smem_u32(smem_s + cur.s * kSStageBytes), &tm_s, full,
                             t.n0 + sub * block_step, s_row);
            cur.advance(w_stages);
          }
          w_row += kBlockK / 16;
          s_row += kBlockK / 32;
        }
      }
      if (!ok) {
        sh.abort_flag = 1;
        if (p.status) atomicOr(p.status, kStatusProducerTimeout);
      }
      if constexpr (!kPair) drain_ring(sh.wfull, cur, w_stages);
    }
    __syncwarp();
  } else if (!tiled_roles && (warp == 0 || warp == 1)) {
    // ------------------------- producers: packed weights (warp 0), scales (warp 1) --
    if (lane == 0) {
      const bool weights = warp == 0;
      const CUtensorMap* map = weights ? &tm_w : &tm_s;
      uint8_t* ring = weights ? smem_w : smem_s;
      const uint32_t stage_bytes = weights ? kWStageBytes : kSStageBytes;
      const int32_t rows_per_stage = weights ? kBlockK / 16 : kBlockK / 32;
      const int32_t rows_per_expert = weights ? p.k / 16 : p.k / 32;
      StageCursor cur;
      bool ok = true;
      while (ok && iter.next(seg)) {
        const TileInfo t = decode_tile(p, sh, seg.tile, rank);
        if (!t.valid) continue;
        const int32_t col = weights ? 2 * t.n0 : t.n0;
        // to the tile's second weight block: the next 128 rows, or the up rows of a fused gate_up
        const int32_t block_step = p.fuse_silu ? (p.n >> 1) : kBlockN;
        const int32_t col_step = weights ? 2 * block_step : block_step;
        int32_t row = t.expert * rows_per_expert + seg.kb * rows_per_stage;
        for (int32_t kb = seg.kb; ok && kb < seg.ke; ++kb) {
          for (int32_t sub = 0; sub < w_per_kb; ++sub) {
            if (!ptx::mbar_wait(ptx::smem_u32(&sh.wempty[cur.s]), cur.ph ^ 1u, abort_flag)) {
              ok = false;
              break;
            }
            const uint32_t full = ptx::smem_u32(&sh.wfull[cur.s]);
            ptx::mbar_arrive_expect_tx(full, stage_bytes);
            ptx::tma_load_2d(ptx::smem_u32(ring + cur.s * stage_bytes), map, full, col + sub * col_step, row);
            cur.advance(w_stages);
          }
          row += rows_per_stage;
        }
      }
      if (!ok) {
        sh.abort_flag = 1;
        if (p.status) atomicOr(p.status, kStatusProducerTimeout);
      }
      if constexpr (!kPair) drain_ring(sh.wfull, cur, w_stages);
    }
    __syncwarp();
  } else if (warp == 2 || (warp == 3 && !tiled_roles)) {
    // ------------------------------------------------ warps 2-3: activations --
    StageCursor cur;
    XSubRing xring;
    bool ok = true;
    if (p.x_load == kXLoadTiled) {
      // Consecutive rows: one box per 64-wide K half, issued by one thread.
      while (ok && threadIdx.x == 64 && iter.next(seg)) {
        const TileInfo t = decode_tile(p, sh, seg.tile, rank);
        if (!t.valid) continue;
        int32_t k_col = seg.kb * kBlockK;
        // `pair`: this CTA's half of the tile's token rows
        const int32_t tile_rows_here = t.mma_n >> p.pair;
        const int32_t x_row0 = t.base + t.m0 + static_cast<int32_t>(rank) * tile_rows_here;
        const int32_t boxes = (tile_rows_here + p.x_box_rows - 1) / p.x_box_rows;
        const bool two_slots = t.mma_n > 128;
        for (int32_t kb = seg.kb; kb < seg.ke; ++kb) {
          if (subslots) {
            const uint32_t s0 = xring.take(two_slots, 2u * x_stages);
            if (!ptx::mbar_wait(ptx::smem_u32(&sh.xempty[s0]), xring.phase(s0) ^ 1u, abort_flag) ||
                (two_slots && !ptx::mbar_wait(ptx::smem_u32(&sh.xempty[s0 + 1]), xring.phase(s0 + 1) ^ 1u,
                                              abort_flag))) {  // odd half: checked, not consumed
              ok = false;
              break;
            }
            const uint32_t full = ptx::smem_u32(&sh.xfull[s0]);
            const uint32_t xs = ptx::smem_u32(smem_x + s0 * kSubBytes);
            const uint32_t half = two_slots ? kSubBytes : kSubBytes / 2;  // bytes of one K half
            ptx::mbar_arrive_expect_tx(full, static_cast<uint32_t>(boxes) * kSubBytes);
            for (int32_t b = 0; b < boxes; ++b) {
              const uint32_t off = static_cast<uint32_t>(b) * (kSubBytes / 2);
              ptx::tma_load_2d(xs + off, &tm_x, full, k_col, x_row0 + b * 128);
              ptx::tma_load_2d(xs + half + off, &tm_x, full, k_col + 64, x_row0 + b * 128);
            }
            xring.flip(s0);
            k_col += kBlockK;
            continue;
          }
          if (!ptx::mbar_wait(ptx::smem_u32(&sh.xempty[cur.s]), cur.ph ^ 1u, abort_flag)) {
            ok = false;
            break;
          }
          const uint32_t full = ptx::smem_u32(&sh.xfull[cur.s]);
          const uint32_t xs = ptx::smem_u32(smem_x + cur.s * x_stage_bytes);
          if constexpr (kPair) {
            // Both CTAs' boxes are counted on the leader's barrier, which expects the bytes
            // of both halves.  (A box of the peer that lands before the leader's arrival
            // only drives the transaction count negative for a moment: the phase cannot
            // complete before that arrival.)
            if (rank == 0) {
              ptx::mbar_arrive_expect_tx(full, 2u * static_cast<uint32_t>(boxes * p.x_box_rows) * 256u);
            }
            for (int32_t b = 0; b < boxes; ++b) {
              const uint32_t off = static_cast<uint32_t>(b * p.x_box_rows) * 128u;
              ptx::tma_load_2d_pair(xs + off, &tm_x, full + to_leader, k_col, x_row0 + b * p.x_box_rows);
              ptx::tma_load_2d_pair(xs + x_half_bytes + off, &tm_x, full + to_leader, k_col + 64,
                                    x_row0 + b * p.x_box_rows);
            }
            k_col += kBlockK;
            cur.advance(x_stages);
            continue;
          }
          ptx::mbar_arrive_expect_tx(full, static_cast<uint32_t>(boxes * p.x_box_rows) * 256u);
          for (int32_t b = 0; b < boxes; ++b) {
            const uint32_t off = static_cast<uint32_t>(b * p.x_box_rows) * 128u;
            ptx::tma_load_2d(xs + off, &tm_x, full, k_col, x_row0 + b * p.x_box_rows);
            ptx::tma_load_2d(xs + x_half_bytes + off, &tm_x, full, k_col + 64,
                             x_row0 + b * p.x_box_rows);
          }
          k_col += kBlockK;
          cur.advance(x_stages);
        }
      }
      if (!kPair && threadIdx.x == 64) {
        if (subslots) {
          for (uint32_t i = 0; i < 2u * x_stages; ++i) ptx::mbar_drain(ptx::smem_u32(&sh.xfull[i]), xring.phase(i) ^ 1u);
        } else {
          drain_ring(sh.xfull, cur, x_stages);
        }
      }
    } else if (p.x_load == kXLoadGather4) {
      // Routed rows by TMA: four rows per instruction, lanes of warp 2 own the row
      // groups lane and lane + 32.
      while (ok && warp == 2 && iter.next(seg)) {
        const TileInfo t = decode_tile(p, sh, seg.tile, rank);
        if (!t.valid) continue;
        int32_t rows[2][4];
        const int32_t load_groups = (t.ntok + 3) >> 2;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int32_t gi = static_cast<int32_t>(lane) + 32 * h;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int32_t slot = gi * 4 + j;
            rows[h][j] = (gi < load_groups && slot < t.ntok) ? x_row_of(p, t, slot) : p.x_rows;
          }
        }
        const uint32_t tx_bytes = static_cast<uint32_t>(load_groups) * 1024u;
        int32_t k_col = seg.kb * kBlockK;
        for (int32_t kb = seg.kb; kb < seg.ke; ++kb) {
          if (!ptx::mbar_wait_warp(ptx::smem_u32(&sh.xempty[cur.s]), cur.ph ^ 1u, abort_flag)) {
            ok = false;
            break;
          }
          const uint32_t full = ptx::smem_u32(&sh.xfull[cur.s]);
          const uint32_t xs = ptx::smem_u32(smem_x + cur.s * x_stage_bytes);
          if (lane == 0) ptx::mbar_arrive_expect_tx(full, tx_bytes);
          __syncwarp();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int32_t gi = static_cast<int32_t>(lane) + 32 * h;
            if (gi < load_groups) {
              ptx::tma_gather4(xs + gi * 512u, &tm_x, full, k_col, rows[h][0], rows[h][1],
                               rows[h][2], rows[h][3]);
              ptx::tma_gather4(xs + x_half_bytes + gi * 512u, &tm_x, full, k_col + 64, rows[h][0],
                               rows[h][1], rows[h][2], rows[h][3]);
            }
          }
          k_col += kBlockK;
          cur.advance(x_stages);
        }
      }
      if (warp == 2) drain_ring(sh.xfull, cur, x_stages);
    } else {
      // Routed rows by cp.async: thread = (16-byte chunk of the 256-byte stage row,
      // row modulo 4).
      const uint32_t ht = threadIdx.x - 64;
      const uint32_t ch = ht & 15;
      const uint32_t half = ch >> 3, ch8 = ch & 7;
      const uint32_t r0 = ht >> 4;
      // A stage is published (one arrival per warp: 32 lanes arriving on one mbarrier
      // would serialise) once its copies have landed, which is checked `depth` stages
      // later so that the copies of several stages stay in flight.
      const int32_t depth = x_stages >= 4 ? 2 : 1;
      StageCursor done;
      int32_t pending = 0;
      // A warp whose bounded wait ran out stops copying but keeps walking the tiles, so
      // that its sibling never waits alone at the three barriers below.
      while (iter.next(seg)) {
        const TileInfo t = decode_tile(p, sh, seg.tile, rank);
        if (!t.valid) continue;
        ptx::named_bar_sync(2, kHelperThreads);  // readers of the previous tile's rows are done
        // Element offset of each slot's activation row, or -1 for a slot without a token;
        // x_slots = one past the last slot that carries a token.  Slots beyond it keep
        // whatever an earlier tile left there: they only feed accumulator columns that
        // are never stored.
        if (ht == 0) sh.x_slots = 0;
        ptx::named_bar_sync(2, kHelperThreads);
        for (int32_t slot = ht; slot < t.ntok; slot += kHelperThreads) {
          const int32_t row = x_row_of(p, t, slot);
          sh.x_row[slot] = row < p.x_rows ? row * p.k : -1;
          if (row < p.x_rows) atomicMax(&sh.x_slots, slot + 1);
        }
        ptx::named_bar_sync(2, kHelperThreads);
        if (!ok) continue;
        const int32_t x_slots = sh.x_slots;
        int32_t k_col = seg.kb * kBlockK + static_cast<int32_t>(ch) * 8;
        // Decode-sized tiles (at most 16 rows with a token): each thread owns at most
        // four copies per stage, whose addresses live in registers for the whole tile.
        const bool few_rows = x_slots <= 16;
        const __nv_bfloat16* fsrc[4];
        uint32_t fdst[4];
        bool fact[4], fval[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const uint32_t rr = r0 + 4 * b;
          fact[b] = few_rows && static_cast<int32_t>(rr) < x_slots;
          const int32_t off = fact[b] ? sh.x_row[rr] : -1;
          fval[b] = off >= 0;
          fsrc[b] = p.x + (fval[b] ? off : 0) + k_col;
          fdst[b] = half * x_half_bytes + rr * 128u + ((ch8 ^ (rr & 7u)) << 4);
        }
        for (int32_t kb = seg.kb; kb < seg.ke; ++kb) {
          if (!ptx::mbar_wait_warp(ptx::smem_u32(&sh.xempty[cur.s]), cur.ph ^ 1u, abort_flag)) {
            ok = false;
            if (lane == 0) sh.abort_flag = 1;  // the sibling's waits end soon too
            break;
          }
          const uint32_t xs = ptx::smem_u32(smem_x + cur.s * x_stage_bytes);
          const bool col_ok = k_col + 8 <= p.k;
          if (few_rows) {
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              if (fact[b]) ptx::cp_async_16(xs + fdst[b], fsrc[b], fval[b] && col_ok);
              fsrc[b] += kBlockK;
            }
          } else {
            const __nv_bfloat16* xk = p.x + k_col;
            // Four rows per round: the offset loads go first so that the copies that
            // follow do not each wait on a shared-memory round trip.
            for (int32_t r = r0; r < x_slots; r += 16) {
              int32_t off[4];
#pragma unroll
              for (int b = 0; b < 4; ++b) off[b] = (r + 4 * b < x_slots) ? sh.x_row[r + 4 * b] : -1;
#pragma unroll
              for (int b = 0; b < 4; ++b) {
                const uint32_t rr = static_cast<uint32_t>(r + 4 * b);
                if (static_cast<int32_t>(rr) < x_slots) {
                  const bool valid = col_ok && off[b] >= 0;
                  ptx::cp_async_16(xs + half * x_half_bytes + rr * 128u + ((ch8 ^ (rr & 7u)) << 4),
                                   xk + (valid ? off[b] : 0), valid);
                }
              }
            }
          }
          ptx::cp_async_commit();
          if (++pending > depth) {
            // The MMA issuer adds the generic-to-async proxy fence after its wait.
            if (depth == 2) ptx::cp_async_wait_group<2>(); else ptx::cp_async_wait_group<1>();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&sh.xfull[done.s]));
            done.advance(x_stages);
            --pending;
          }
          k_col += kBlockK;
          cur.advance(x_stages);
        }
      }
      // Drain: publish what is still in flight (also when leaving on a timeout).
      ptx::cp_async_wait_all();
      __syncwarp();
      for (; pending > 0; --pending) {
        if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&sh.xfull[done.s]));
        done.advance(x_stages);
      }
    }
    __syncwarp();
    if (!ok && lane == 0) {
      sh.abort_flag = 1;
      if (p.status) atomicOr(p.status, kStatusProducerTimeout);
    }
  } else if (tiled_roles ? (warp == 1 || warp == 3) : (warp >= kFirstIssuerWarp && warp < kFirstDequantWarp)) {
    // ----------------------------------------------------------- MMA issuers --
    const uint32_t me = tiled_roles ? (warp >> 1) : warp - kFirstIssuerWarp;
    // The whole warp walks the stages and waits; one elected lane issues.  A loop inside
    // `if (lane == 0)` is divergent code to the compiler, which then moves every operand of
    // every MMA (addresses, descriptors: all the same in all lanes) into the uniform registers
    // the instruction reads, one by one, just before it: about 130 cycles per MMA.  (contiguous,
    // 8192 uneven rows, gate_up / down: 561 / 399 -> 534 / 381 us.)
    // A wait that gives up is recorded in `bad` and tested once per stage; until then the
    // issuer runs on, on whatever this CTA's operand buffers hold.
    if (me < ni && rank == 0) {
      const uint64_t xdesc0 = ptx::smem_desc_k_sw128(ptx::smem_u32(smem_x));
      const uint64_t xdesc_stage = x_stage_bytes >> 4;  // descriptor address units are 16 bytes
      const uint64_t xdesc_half = x_half_bytes >> 4;
      const uint32_t abort_addr = ptx::smem_u32(&sh.abort_flag);
      const uint32_t xfull0 = ptx::smem_u32(&sh.xfull[0]), xempty0 = ptx::smem_u32(&sh.xempty[0]);
      const uint32_t afull0 = ptx::smem_u32(&sh.afull[0]), aempty0 = ptx::smem_u32(&sh.aempty[0]);
      uint64_t xdesc = xdesc0;
      StageCursor cur, acur;
      XSubRing xring;
      uint32_t it = 0, segc = 0, bad = 0;
      while (iter.next(seg)) {
        const TileInfo t = decode_tile(p, sh, seg.tile, rank);
        if (!t.valid) continue;
        const uint32_t d = d_bufs == 2 ? (segc & 1u) : 0u;
        const uint32_t dph = d_bufs == 2 ? ((segc >> 1) & 1u) : (segc & 1u);
        ptx::mbar_wait_sticky(ptx::smem_u32(&sh.dempty[d]), dph ^ 1u, abort_addr, bad);
        if (__any_sync(0xffffffffu, bad != 0)) break;
        ptx::tc_fence_after();
        const uint32_t d_addr = tmem_base + d_col0 + (d * ni + me) * d_cols;
        // (through a shuffle: a value loaded from shared memory is not known to be uniform)
        const uint32_t mma_n = __shfl_sync(0xffffffffu, static_cast<uint32_t>(t.mma_n), 0);
        const uint32_t idesc = ptx::idesc_bf16_f32(kBlockN << p.pair, mma_n);
        uint32_t acc = 0;
        const bool split = ksplit && mma_n <= 128;
        for (int32_t kb = seg.kb; kb < seg.ke; ++kb, ++it) {
          const bool tail = k_tail_half && kb == k_iters - 1;  // no second K half
          if (kPair || npair) {
            // CTA pair: one MMA stream for both CTAs; every commit arrives on the barrier of
            // each.  `npair`: the K block's two operand-ring entries belong to the tile's two
            // weight blocks; this issuer takes the one of its block, with both K halves, into
            // its accumulator.
            uint32_t as = acur.s, aph = acur.ph;
            if (!kPair) {
              as += me;
              if (as >= a_stages) {
                as -= a_stages;
                aph ^= 1u;
              }
            }
            const uint32_t a_bar = as << 4;  // two 8-byte barriers per entry
            const uint32_t a_addr = tmem_base + as * kAColsPerStage;
            ptx::mbar_wait_sticky(xfull0 + cur.s * 8u, cur.ph, abort_addr, bad);
            ptx::mbar_wait_sticky(afull0 + a_bar, aph, abort_addr, bad);
            ptx::tc_fence_after();
            if (ptx::elect_one()) {
              if constexpr (kPair) {
                ptx::mma_ts_k64_pair(d_addr, a_addr, xdesc, idesc, acc);
                ptx::mma_commit_pair(aempty0 + a_bar);
              } else {
                ptx::mma_ts_k64(d_addr, a_addr, xdesc, idesc, acc);
                ptx::mma_commit(aempty0 + a_bar);
              }
            }
            __syncwarp();
            ptx::mbar_wait_sticky(afull0 + a_bar + 8u, aph, abort_addr, bad);
            ptx::tc_fence_after();
            if (ptx::elect_one()) {
              if constexpr (kPair) {
                if (!tail) ptx::mma_ts_k64_pair(d_addr, a_addr + 32, xdesc + xdesc_half, idesc, 1);
                ptx::mma_commit_pair(aempty0 + a_bar + 8u);
                ptx::mma_commit_pair(xempty0 + cur.s * 8u);
              } else {
                if (!tail) ptx::mma_ts_k64(d_addr, a_addr + 32, xdesc + xdesc_half, idesc, 1);
                ptx::mma_commit(aempty0 + a_bar + 8u);
                ptx::mma_commit(xempty0 + cur.s * 8u);
              }
            }
            __syncwarp();
            acc = 1;
            if (!kPair) acur.advance(a_stages);  // the other block's entry; the common advance below takes this one
          } else if (ksplit) {
            const uint32_t a_bar = acur.s << 4;
            const uint32_t aph = acur.ph;
            uint32_t xslot = cur.s;       // barrier (and, with sub-slots, buffer) of this stage
            uint64_t xd = xdesc, xd_half = xdesc_half;
            const bool two_slots = subslots && mma_n > 128;
            if (subslots) {
              xslot = xring.take(two_slots, 2u * x_stages);
              xd = xdesc0 + xslot * (kSubBytes >> 4);
              xd_half = two_slots ? (kSubBytes >> 4) : (kSubBytes >> 5);
              ptx::mbar_wait_sticky(xfull0 + xslot * 8u, xring.phase(xslot), abort_addr, bad);
              xring.flip(xslot);
            } else {
              ptx::mbar_wait_sticky(xfull0 + cur.s * 8u, cur.ph, abort_addr, bad);
            }
            if (p.x_load == kXLoadCpAsync) ptx::fence_proxy_async();
            const uint32_t a_addr = tmem_base + acur.s * kAColsPerStage;
            if (me == 0) {
              ptx::mbar_wait_sticky(afull0 + a_bar, aph, abort_addr, bad);
              ptx::tc_fence_after();
              if (ptx::elect_one()) {
                ptx::mma_ts_k64(d_addr, a_addr, xd, idesc, acc);
                ptx::mma_commit(aempty0 + a_bar);
              }
              __syncwarp();
              acc = 1;
            }
            if (me == 0 ? !split : split) {
              ptx::mbar_wait_sticky(afull0 + a_bar + 8u, aph, abort_addr, bad);
              ptx::tc_fence_after();
              if (ptx::elect_one()) {
                if (!tail) ptx::mma_ts_k64(d_addr, a_addr + 32, xd + xd_half, idesc, acc);
                ptx::mma_commit(aempty0 + a_bar + 8u);
              }
              __syncwarp();
              if (!tail) acc = 1;
            }
            // Both issuers account for the activation stage: a commit after MMAs of one's
            // own, a plain arrival otherwise.
            if (ptx::elect_one()) {
              if (me == 0 || split) ptx::mma_commit(xempty0 + xslot * 8u);
              else ptx::mbar_arrive(xempty0 + xslot * 8u);
            }
            __syncwarp();
          } else if ((it & (ni - 1)) == me) {
            const uint32_t a_bar = acur.s << 4;  // barrier of the first K half; the second follows it
            const uint32_t aph = acur.ph;
            ptx::mbar_wait_sticky(xfull0 + cur.s * 8u, cur.ph, abort_addr, bad);
            if (p.x_load == kXLoadCpAsync) ptx::fence_proxy_async();
            ptx::mbar_wait_sticky(afull0 + a_bar, aph, abort_addr, bad);
            ptx::tc_fence_after();
            const uint32_t a_addr = tmem_base + acur.s * kAColsPerStage;
            if (ptx::elect_one()) {
              ptx::mma_ts_k64(d_addr, a_addr, xdesc, idesc, acc);
              ptx::mma_commit(aempty0 + a_bar);
            }
            __syncwarp();
            ptx::mbar_wait_sticky(afull0 + a_bar + 8u, aph, abort_addr, bad);
            ptx::tc_fence_after();
            if (ptx::elect_one()) {
              if (!tail) ptx::mma_ts_k64(d_addr, a_addr + 32, xdesc + xdesc_half, idesc, 1);
              ptx::mma_commit(aempty0 + a_bar + 8u);
              ptx::mma_commit(xempty0 + cur.s * 8u);
            }
            __syncwarp();
            acc = 1;
          }
          xdesc += xdesc_stage;
          cur.advance(x_stages);
          acur.advance(a_stages);
          if (cur.s == 0) xdesc = xdesc0;
          if (__any_sync(0xffffffffu, bad != 0)) break;
        }
        if (__any_sync(0xffffffffu, bad != 0)) break;
        // One arrival per issuer and segment, also from an issuer that had no stage in it.
        if (ptx::elect_one()) {
          if constexpr (kPair) {
            ptx::mma_commit_pair(ptx::smem_u32(&sh.dfull[d]));
          } else if (acc != 0) {
            ptx::mma_commit(ptx::smem_u32(&sh.dfull[d]));
          } else {
            ptx::mbar_arrive(ptx::smem_u32(&sh.dfull[d]));
          }
        }
        __syncwarp();
        ++segc;
      }
      if (__any_sync(0xffffffffu, bad != 0) && lane == 0 && p.status) atomicOr(p.status, kStatusMmaTimeout);
      // Also when a role has given up, no MMA may run on into the release of tensor memory.
      if constexpr (!kPair) {
        if (ptx::elect_one()) ptx::mma_commit(ptx::smem_u32(&sh.mma_done));
        __syncwarp();
        ptx::mbar_drain(ptx::smem_u32(&sh.mma_done), 0);
      }
    }
    __syncwarp();
  } else if (warp >= kFirstDequantWarp && warp < kFirstEpilogueWarp) {
    // --------------------------------------------------------------- dequant --
    const uint32_t group = (warp - kFirstDequantWarp) >> 2;
    const uint32_t q = warp & 3;  // TMEM lane quarter == 32 weight rows
    // Byte offset of this thread's two packed words (slabs 2(q&1), 2(q&1)+1 of the
    // 64-row chunk q>>1) inside one K16 row of the stage, and of its four scales.
    const uint32_t w_off = (q >> 1) * 512u + lane * 16u + (q & 1) * 8u;
    const uint32_t s_off = (q >> 1) * 128u + (lane >> 2) * 16u + (q & 1) * 8u;
    // Which scales a loop over stages takes: those below 2^-5, others, or both by a branch.
    constexpr int kSmallOnly = 0, kAnyOnly = 1, kEither = 2;
    // Four lanes have the same scales, of the stage's four K32 groups; each looks at the range of one group's.
    const uint32_t probe_off = s_off + (lane & 3u) * 256u;
    StageCursor cur, acur;
    uint32_t it = 0;
    // Two such warps per scheduler: bound by the latency of their own chain (wait, load,
    // dequantise, store, publish), hence single-statement waits, running barrier offsets and
    // predicated arrivals (4096 routed tokens, down: 178 -> 174 us).
    uint32_t bad = 0;  // set by the first bounded wait that gives up; tested once per stage
    const uint32_t abort_addr = ptx::smem_u32(&sh.abort_flag);
    const uint32_t wfull0 = ptx::smem_u32(&sh.wfull[0]), wempty0 = ptx::smem_u32(&sh.wempty[0]);
    const uint32_t aempty0 = ptx::smem_u32(&sh.aempty[0]), afull0 = ptx::smem_u32(&sh.afull[0]);
    // A stored K half is published to the MMA issuer one compute step later (after
    // the next half has been dequantised), so that the latency of the tensor-memory
    // store and of the barrier round trip hides behind ALU work.  `pending` is the
    // slot whose store has been issued but not yet published.
    int32_t pending = -1;
    auto publish = [&]() {
      if (pending >= 0) {
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
        __syncwarp();
        const uint32_t full = afull0 + static_cast<uint32_t>(pending) * 8u;
        if constexpr (kPair) {
          // `pair`: the leader's barrier counts the warps of both CTAs
          if (lane == 0) ptx::mbar_arrive_cluster(full + to_leader);
        } else {
          ptx::mbar_arrive_lane0(full, lane);
        }
        pending = -1;
      }
    };
    auto load_half = [&](const uint8_t* wsrc, const uint8_t* ssrc, int h, uint2 (&words)[4],
                         uint2 (&scales)[2]) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        words[j] = *reinterpret_cast<const uint2*>(wsrc + (4 * h + j) * 1024);
      }
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        scales[g] = *reinterpret_cast<const uint2*>(ssrc + (2 * h + g) * 256);
      }
    };
    // scales[g].x = {slab A row r, slab A row r+8} of K32 group g; .y = the same for slab B.
    auto dequant_half = [&](auto any_scale, const uint2 (&words)[4], const uint2 (&scales)[2], uint32_t (&lo)[16],
                            uint32_t (&hi)[16]) {
      using Dq = Dequant<decltype(any_scale)::value, false>;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const Dq da(scales[g].x);
#pragma unroll
        for (int j = 2 * g; j < 2 * g + 2; ++j) da(words[j].x, lo[4 * j], lo[4 * j + 1], lo[4 * j + 2], lo[4 * j + 3]);
        const Dq db(scales[g].y);
#pragma unroll
        for (int j = 2 * g; j < 2 * g + 2; ++j) db(words[j].y, hi[4 * j], hi[4 * j + 1], hi[4 * j + 2], hi[4 * j + 3]);
      }
    };
    auto dequant_half_as = [&](auto way, bool small, const uint2 (&words)[4], const uint2 (&scales)[2], uint32_t (&lo)[16],
                               uint32_t (&hi)[16]) {
      constexpr int kWay = decltype(way)::value;
      if constexpr (kWay != kEither) dequant_half(std::bool_constant<kWay == kAnyOnly>{}, words, scales, lo, hi);
      else if (small) dequant_half(std::false_type{}, words, scales, lo, hi);
      else dequant_half(std::true_type{}, words, scales, lo, hi);
    };
    // Waits for the slot to be free, then stores one K half: lo to TMEM lanes 0-15 of
    // the quarter (first slab), hi to lanes 16-31 (second slab).
    auto store_half = [&](uint32_t slot, uint32_t aph, const uint32_t (&lo)[16],
                          const uint32_t (&hi)[16]) {
      ptx::mbar_wait_sticky(aempty0 + slot * 8u, aph ^ 1u, abort_addr, bad);
      ptx::tc_fence_after();
      const uint32_t a_addr = tmem_base + ((q * 32u) << 16) + slot * (kAColsPerStage / 2);
      ptx::tmem_st_16x128b_x8(a_addr, lo);
      ptx::tmem_st_16x128b_x8(a_addr + (16u << 16), hi);
      pending = static_cast<int32_t>(slot);
    };
    while (bad == 0 && iter.next(seg)) {
      const TileInfo t = decode_tile(p, sh, seg.tile, rank);
      if (!t.valid) continue;
      // This group owns the stages whose running index is `group` modulo the number
      // of groups: step over the others without visiting them.
      const uint32_t seg_len = static_cast<uint32_t>((seg.ke - seg.kb) * w_per_kb);  // ring entries
      const uint32_t first = (group - it) & (kDequantGroups - 1);
      const uint32_t it_end = it + seg_len;
      if (first >= seg_len) {
        it = it_end;
        cur.advance_by(seg_len, w_stages);
        acur.advance_by(seg_len, a_stages);
        continue;
      }
      it += first;
      cur.advance_by(first, w_stages);
      acur.advance_by(first, a_stages);
      // On single CTAs one loop per way to dequantise, each left at a stage that needs the other (which
      // waits for and loads that stage again): with a branch in one loop a half jumps to code beside the loop
      // and back, 48 experts of 60 rows, 4096 x 7168 / 7168 x 2048, us: 265 / 149, with two loops 256 / 138.  On
      // pairs, which the products bound, the branch is the better (24 of 250 rows 279 / 146.5, 280.4 / 148.5).
      auto run_stages = [&](auto way) {
        constexpr int kWay = decltype(way)::value;
        for (; it < it_end; it += kDequantGroups, cur.advance_by(kDequantGroups, w_stages),
                            acur.advance_by(kDequantGroups, a_stages)) {
          const uint32_t a = acur.s << 1;  // half-slots a (first K half) and a + 1 (second)
          const uint32_t aph = acur.ph;
          ptx::mbar_wait_sticky(wfull0 + cur.s * 8u, cur.ph, abort_addr, bad);
          const uint8_t* wsrc = smem_w + cur.s * kWStageBytes + w_off;
          const uint8_t* ssrc = smem_s + cur.s * kSStageBytes + s_off;
          uint2 words[4], scales[2];
          uint32_t lo[16], hi[16];
          load_half(wsrc, ssrc, 0, words, scales);
          const uint2 probe = *reinterpret_cast<const uint2*>(smem_s + cur.s * kSStageBytes + probe_off);
          const bool small = small_scales(probe);
          if (kWay != kEither && small == (kWay == kAnyOnly)) {
            bad = __any_sync(0xffffffffu, bad != 0) ? 1u : 0u;
            return;
          }
          dequant_half_as(way, small, words, scales, lo, hi);
          // Second half's words are fetched before the first half is stored, and the
          // stage goes back to the producers as soon as they are in registers.
          load_half(wsrc, ssrc, 1, words, scales);
          publish();  // previous stage's second half
          __syncwarp();
          ptx::mbar_arrive_lane0(wempty0 + cur.s * 8u, lane);
          store_half(a, aph, lo, hi);
          dequant_half_as(way, small, words, scales, lo, hi);
          publish();  // this stage's first half
          store_half(a + 1, aph, lo, hi);
          bad = __any_sync(0xffffffffu, bad != 0) ? 1u : 0u;
          if (bad != 0) return;
        }
      };
      while (bad == 0 && it < it_end) {
        if constexpr (kPair) {
          run_stages(std::integral_constant<int, kEither>{});
        } else {
          run_stages(std::integral_constant<int, kSmallOnly>{});
          if (bad == 0 && it < it_end) run_stages(std::integral_constant<int, kAnyOnly>{});
        }
      }
      // `it` overshoots the segment's end by less than one stride: bring the cursor back.
      if (bad == 0) {
        const uint32_t over = it - it_end;
        it = it_end;
        cur.advance_by(w_stages - over, w_stages);
        cur.ph ^= 1u;
        acur.advance_by(a_stages - over, a_stages);
        acur.ph ^= 1u;
      }
    }
    publish();
    if (bad != 0 && lane == 0 && p.status) atomicOr(p.status, kStatusDequantTimeout);
  } else {
    // -------------------------------------------------------------- epilogue --
    // Four warps, one per tensor-memory lane quarter; with `tiled_roles` a second group of
    // four (warps 4-7) takes every other 16-column chunk.
    const uint32_t q = warp & 3;
    const uint32_t kEpiThreads = epi_threads;
    const uint32_t egroup = warp < kFirstDequantWarp ? 1u : 0u;
    const uint32_t et = threadIdx.x - (egroup ? kFirstIssuerWarp : kFirstEpilogueWarp) * 32;  // 0..127 == TMEM lane
    const uint32_t efill = egroup * 128u + et;  // index among all epilogue threads
    uint32_t segc = 0, it0 = 0;
    bool ok = true;
    const size_t ws_block = static_cast<size_t>(kBlockN) * p.mma_n;  // partial sums of one weight block
    const size_t ws_slot = ws_block * w_per_kb;
    while (ok && iter.next(seg)) {
      const TileInfo t = decode_tile(p, sh, seg.tile, rank);
      if (!t.valid) continue;
      const uint32_t d = d_bufs == 2 ? (segc & 1u) : 0u;
      const uint32_t dph = d_bufs == 2 ? ((segc >> 1) & 1u) : (segc & 1u);
      ptx::named_bar_sync(1, kEpiThreads);  // previous segment's out_row readers are done
      const int32_t row_slots = (t.rows + 15) & ~15;  // >= t.mma_n; beyond it: rows written as zeros
      for (int32_t c = efill; c < row_slots; c += kEpiThreads) sh.out_row[c] = out_row_of(p, t, c);
      bool lock_ok = true;
      if (seg.type == kSegOwner && efill == 0) {
        // Wait (bounded) until every other slice of this tile has published its partial.
        const int* lock = p.locks + blockIdx.x;  // (`pair`: one word per CTA; the slices of its rows come from CTAs of its own rank)
        lock_ok = false;
        for (int32_t spin = 0; spin < p.lock_spins; ++spin) {
          if (ptx::ld_acquire(lock) >= seg.peer) {
            lock_ok = true;
            break;
          }
          __nanosleep(64);
        }
        if (!lock_ok && p.status) atomicOr(p.status, kStatusLockTimeout);
      }
      // The four warps must agree on the outcome before any of them leaves the loop,
      // or the named barriers below would wait for warps that are gone.
      if (!ptx::mbar_wait_warp(ptx::smem_u32(&sh.dfull[d]), dph, abort_flag) && lane == 0) {
        sh.epilogue_failed = 1;
      }
      ptx::tc_fence_after();
      ptx::named_bar_sync(1, kEpiThreads);  // out_row filled, lock observed, verdict published
      if (sh.epilogue_failed != 0) {
        ok = false;
        break;
      }
      const uint32_t d_addr = tmem_base + ((q * 32u) << 16) + d_col0 + d * ni * d_cols;
      // Issuer i accumulated the stages it0 + j with (it0 + j) % ni == i; it took part
      // in this segment only if one of them falls inside it.  (With `npair` accumulator
      // `sub` is the tile's weight block `sub` instead, and nothing is summed.)
      const uint32_t seg_len = static_cast<uint32_t>(seg.ke - seg.kb);
      // Fused SiLU*mul: one pass, which reads both accumulators (gate, up), combines them
      // and writes a [rows, N/2] tensor.
      const bool fuse = !kHold && p.fuse_silu != 0;
      const int32_t ldn = fuse ? (p.n >> 1) : p.n;
      __nv_bfloat16* stage = &sh.stage[egroup * 4u + q][0][0];
      // Transpose of 16 tokens through shared memory so that global stores are 16 bytes wide:
      // the warp holds 32 weight rows x 16 tokens, staged as [token][row]; each lane then
      // stores two 8-row pieces of a token's 64 bytes.
      auto store_staged = [&](int32_t c0, int32_t n_sub) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t idx = lane + 32 * i;
          const uint32_t tj = idx >> 2, piece = idx & 3;
          const int32_t row = sh.out_row[c0 + tj];
          const uint4 v = *reinterpret_cast<const uint4*>(stage + tj * 32 + piece * 8);
          if (row >= 0) {
            if (p.out_row_ptr != nullptr) {
              // the row lives wherever the caller's table says (possibly on another GPU)
              __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(
                  __ldg(reinterpret_cast<const unsigned long long*>(p.out_row_ptr) + row));
              if (dst != nullptr) *reinterpret_cast<uint4*>(dst + n_sub + piece * 8) = v;
            } else {
              *reinterpret_cast<uint4*>(p.out + static_cast<size_t>(row) * ldn + n_sub + piece * 8) = v;
            }
          }
        }
        __syncwarp();
      };
      if (kHold && seg.type == kSegFull) {
        // The warp's share of the accumulators (at most eight chunks of 16 columns) is read and
        // rounded first, the accumulators go back to the issuers, and only then are the rows
        // written.  Accumulators of this size are single-buffered: what is left between two
        // tiles is the reading alone.
        constexpr int kChunks = 8;
        uint32_t held[kChunks][8];
        const int32_t first = static_cast<int32_t>(egroup) * 16;
        constexpr bool two_blocks = !kPair;  // chunks 4-7 are the second weight block's
#pragma unroll
        for (int i = 0; i < kChunks; ++i) {
          const int32_t c0 = first + 32 * (two_blocks ? (i & 3) : i);
          if (c0 >= t.mma_n) {
#pragma unroll
            for (int j = 0; j < 8; ++j) held[i][j] = 0;  // padding rows of a contiguous block
            continue;
          }
          uint32_t v[16];
          ptx::tmem_ld_32x32b_x16(d_addr + (two_blocks ? (i >> 2) * d_cols : 0u) + c0, v);
          ptx::tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const __nv_bfloat162 pair2 = __floats2bfloat162_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
            held[i][j] = *reinterpret_cast<const uint32_t*>(&pair2);
          }
        }
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (kPair) ptx::mbar_arrive_cluster(ptx::smem_u32(&sh.dempty[d]) + to_leader);
          else ptx::mbar_arrive(ptx::smem_u32(&sh.dempty[d]));
        }
#pragma unroll
        for (int i = 0; i < kChunks; ++i) {
          const int32_t c0 = first + 32 * (two_blocks ? (i & 3) : i);
          if (c0 >= row_slots) continue;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const __nv_bfloat162 pair2 = *reinterpret_cast<const __nv_bfloat162*>(&held[i][j]);
            stage[2 * j * 32 + lane] = pair2.x;
            stage[(2 * j + 1) * 32 + lane] = pair2.y;
          }
          store_staged(c0, t.n0 + (two_blocks ? (i >> 2) * kBlockN : 0) + static_cast<int32_t>(q) * 32);
        }
        ++segc;
        it0 += seg_len;
        continue;
      }
      for (int32_t sub = 0; sub < (fuse ? 1 : w_per_kb); ++sub) {
      const int32_t n_sub = t.n0 + sub * kBlockN + static_cast<int32_t>(q) * 32;
      const size_t ws_sub = static_cast<size_t>(sub) * ws_block;
      for (int32_t c0 = static_cast<int32_t>(egroup) * 16; c0 < row_slots; c0 += tiled_roles ? 32 : 16) {
        float acc[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j] = 0.0f;
        // Slots past the tile's MMA N hold padding rows of a contiguous block: the product
        // of their all-zero activations is written without having been computed.
        const bool computed = c0 < t.mma_n;
        if (!computed && seg.type == kSegContrib) continue;
        for (uint32_t i = 0; computed && i < ni; ++i) {
          if (npair) {
            if (static_cast<int32_t>(i) != sub) continue;
          } else if (ksplit) {
            // issuer 1 holds the second K halves of tiles of at most 128 tokens, unless the
            // segment is nothing but the half-filled last stage
            if (i == 1 && (t.mma_n > 128 || seg_len == (k_tail_half && seg.ke == k_iters ? 1u : 0u))) continue;
          } else if (((i - it0) & (ni - 1)) >= seg_len) {
            continue;
          }
          uint32_t v[16];
          ptx::tmem_ld_32x32b_x16(d_addr + i * d_cols + c0, v);
          ptx::tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[j] += __uint_as_float(v[j]);
        }
        float up[16];
        if (fuse) {
#pragma unroll
          for (int j = 0; j < 16; ++j) up[j] = 0.0f;
          if (computed) {
            uint32_t v[16];
            ptx::tmem_ld_32x32b_x16(d_addr + d_cols + c0, v);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) up[j] = __uint_as_float(v[j]);
          }
        }
        if constexpr (kPair) {
          // On pairs (mma_n a multiple of 16 above 128) the partial sums lie as [four columns][weight
          // row][column]: 16-byte vectors, a warp's consecutive, two contributors' in flight.  Masked
          // launches of 4096 x 7168 / 7168 x 2048, words -> vectors, us, three runs of each in turn within
          // 0.4 of each other: 24 groups of 128 rows 191.6 -> 189.3 / 104.2 -> 103.7, 12 of 250 rows 138.7 ->
          // 136.9 / 81.6 -> 79.2, 7 of 250 rows 87.1 -> 85.0 / 57.3 -> 55.3, 48 of 200 rows the same; on single
          // CTAs vectors cost 1 %.
          if (seg.type != kSegFull) {
            float4* part = reinterpret_cast<float4*>(p.workspace + blockIdx.x * ws_slot + static_cast<size_t>(c0) * kBlockN) + et;
            if (seg.type == kSegContrib) {
#pragma unroll
              for (int j = 0; j < 4; ++j) __stcg(part + j * kBlockN, make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]));
              continue;
            }
            if (computed) {
#pragma unroll 2
              for (int32_t peer = 1; peer <= seg.peer; ++peer) {
                part += ws_slot / 2;  // the CTA of the same rank in the next pair
                float4 v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = __ldcg(part + j * kBlockN);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  acc[4 * j] += v[j].x;
                  acc[4 * j + 1] += v[j].y;
                  acc[4 * j + 2] += v[j].z;
                  acc[4 * j + 3] += v[j].w;
                }
              }
            }
          }
        } else if (seg.type == kSegContrib) {
          float* dst = p.workspace + blockIdx.x * ws_slot + ws_sub + static_cast<size_t>(c0) * kBlockN + et;
#pragma unroll
          for (int j = 0; j < 16; ++j) __stcg(dst + j * kBlockN, acc[j]);
          if (fuse) {
#pragma unroll
            for (int j = 0; j < 16; ++j) __stcg(dst + ws_block + j * kBlockN, up[j]);
          }
          continue;
        } else if (seg.type == kSegOwner && computed) {
          for (int32_t peer = 1; peer <= seg.peer; ++peer) {
            const float* src = p.workspace + (blockIdx.x + peer) * ws_slot + ws_sub +
                               static_cast<size_t>(c0) * kBlockN + et;
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[j] += __ldcg(src + j * kBlockN);
            if (fuse) {
#pragma unroll
              for (int j = 0; j < 16; ++j) up[j] += __ldcg(src + ws_block + j * kBlockN);
            }
          }
        }
        if (fuse) {
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[j] = acc[j] / (1.0f + __expf(-acc[j])) * up[j];
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) stage[j * 32 + lane] = __float2bfloat16_rn(acc[j]);
        store_staged(c0, n_sub);
      }
      }
      // Release the accumulator buffer to the MMA issuer.
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (kPair) ptx::mbar_arrive_cluster(ptx::smem_u32(&sh.dempty[d]) + to_leader);
        else ptx::mbar_arrive(ptx::smem_u32(&sh.dempty[d]));
      }
      if (seg.type == kSegContrib) {
        __threadfence();
        ptx::named_bar_sync(1, kEpiThreads);
        // the owner of this CTA's rows: the CTA of the same rank in the owning pair
        if (efill == 0) ptx::red_release_add(p.locks + ((seg.peer << p.pair) + static_cast<int32_t>(rank)), 1);
      } else if (seg.type == kSegOwner) {
        ptx::named_bar_sync(1, kEpiThreads);
        // After a timeout the word is left as it is: contributors that arrive late would
        // otherwise leave it non-zero behind a reset, and the caller has to clear the
        // buffer anyway once the status word reports the failure.
        if (efill == 0 && lock_ok) p.locks[blockIdx.x] = 0;
      }
      ++segc;
      it0 += seg_len;
    }
    if (!ok && lane == 0) {
      sh.abort_flag = 1;
      if (p.status) atomicOr(p.status, kStatusEpilogueTimeout);
    }
  }

  // --------------------------------------------------------------- teardown --
  ptx::tc_fence_before();
  __syncthreads();
  // `pair`: neither CTA may leave (or free tensor memory) while the other can still
  // signal its barriers or have MMAs reading its shared and tensor memory.  After a failure
  // boxes and MMAs of either may be under way that nobody waits for; a barrier of this CTA does
  // not tell about the other's, so they are left a millisecond, a thousand times what they
  // take.  (Waiting for them by role, as the other instantiation does, made every launch of
  // this one 2 % slower.)
  if constexpr (kPair) {
    if (sh.abort_flag != 0) {
      for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    ptx::cluster_sync();
  }
  if (warp == 2) {
    ptx::tc_fence_after();
    if constexpr (kPair) ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
    else ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace chord
