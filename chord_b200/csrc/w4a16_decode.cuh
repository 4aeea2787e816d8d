// Decode-sized variant of the W4A16 grouped GEMM (token tiles of at most 32 rows).
//
// Same data formats, scheduling and stream-K protocol as w4a16_gemm_kernel
// (w4a16_gemm.cuh) and the same dequantised BF16 weights; what changes is the matrix
// instruction.  A tile of a few tokens gives the tensor core next to nothing to do, and
// what bounds it is the stream of packed weights and the instructions spent on each of
// its words (the integer pipe that pulls the nibbles apart runs at half rate).  The packed
// format is the register fragment of the warp-level m16n8k16 instruction (one 32-bit word
// = the A fragment of 16 weight rows x 16 K values of one lane), so here the dequantised
// registers feed mma.sync directly: no store to tensor memory, no operand ring, no second
// warp that issues.  (tcgen05.mma takes its A operand from tensor or shared memory only;
// the version of this kernel built on it spent 219 issue slots per 2048 weights, with two
// barrier hand-overs per 64-wide K step, and read weights at 0.6 of the copy bandwidth.)
//
// A CTA is four independent workers.  A worker is a feeder warp and four computing warps:
//
//   * it has its own slice of the work (the grid of workers is 4 x the grid of CTAs), its
//     own shared-memory ring, lock word and scratch slot;
//   * a ring stage holds 128 K values of a tile: the activation rows (cp.async gather,
//     128-byte swizzle, so that ldmatrix reads them without bank conflicts), 8 KB of packed
//     weights and 1 KB of scales (two TMA boxes).  One barrier per stage counts all of it;
//   * a computing warp owns 32 of the tile's 128 weight rows over the whole K range: per
//     K16 it loads two words per lane and the token fragments, dequantises and multiplies.
//     The four warps share a stage but never wait for one another inside a tile;
//   * a tile runs with 8, 16, 24 or 32 token columns, by the rows it really has: at decode
//     sizes most routing blocks of 16 hold at most 8.
//
// Measured on a B200, gate_up [4096, 7168] / down [7168, 2048] of a layer's local experts, weights
// from HBM, replayed graph, us: tcgen05 version / with 15 instructions of dequantisation per word /
// now: 1 expert reached 19.2, 14.7 / 12.7, 10.2 / 12.2, 10.3; 11 experts of 1 row 53.7, 34.5 / 44.1, 27.4 /
// 40.1, 25.9; 48 of 5 rows 188, 111 / 153.6, 85.5 / 137.3, 77.1 (5.8 / 5.2 TB/s of packed weights and
// scales); 48 of 14 rows (Poisson) now 193, 110.  These are bursts at 1965 MHz, where the latency of the
// warps' work bounds it; in steady state the power cap does: 48 of 5 rows 181, 96 / 168, 89 at 1.6 to 1.7
// GHz.  About 10 us per launch do not depend on the experts: set-up, the first stages, and the
// stream-K slices at the end.
//
// Registers: 640 threads may have 96 each, of which the four feeder warps need 56 and the computing
// warps, with wide tiles or two blocks of a fused gate_up, more than 96: those take 104 (4 x 56 + 16 x 104
// <= 20 x 96), and only fused gate_up spills (8 bytes).
#pragma once

#include "register_split.h"
#include "w4a16_gemm.cuh"

namespace chord {

constexpr int kDecStageK = 128;                       // K elements per ring stage
constexpr int kDecWBytes = (kDecStageK / 16) * 1024;  // packed weights per stage
constexpr int kDecSBytes = (kDecStageK / 32) * 256;   // scales per stage
constexpr int kDecWSBytes = kDecWBytes + kDecSBytes;  // 9 KB: keeps stages 1024-aligned
constexpr int kDecMaxStages = 6;
constexpr int kDecMaxTokens = 32;
constexpr int kDecWorkers = 4;                        // workers per CTA
constexpr int kDecThreads = 32 * (kDecWorkers + 4 * kDecWorkers);  // feeders, computing warps
// Registers of a feeder's and of a computing warp's threads, once they have divided them
// (setmaxnreg: multiples of 8, by whole warpgroups of four warps).
constexpr int kDecFeederRegs = 56, kDecComputeRegs = 104;
static_assert(kDecWorkers == 4 && kDecFeederRegs % 8 == 0 && kDecComputeRegs % 8 == 0, "setmaxnreg");

// Whether the division is possible with what a kernel compiled to `num_regs` is launched with.
constexpr bool decode_registers_fit(int num_regs) {
  return register_split_fits(num_regs, kDecWorkers, kDecFeederRegs, 4 * kDecWorkers, kDecComputeRegs);
}
static_assert(decode_registers_fit(65536 / kDecThreads / 8 * 8), "the registers of an SM");

constexpr int kDecPitch = 40;  // BF16 per token row of the epilogue buffer: 32 rows, padded against bank conflicts

struct __align__(16) DecodeWorkerShared {
  uint64_t full[kDecMaxStages];   // stage landed (1 arrival + TMA bytes, 32 cp.async arrivals)
  uint64_t empty[kDecMaxStages];  // the four warps have read it (4 arrivals)
  __align__(16) __nv_bfloat16 stage[4][8][kDecPitch];  // epilogue transpose buffers, one per warp
};

struct __align__(16) DecodeShared {
  DecodeWorkerShared worker[kDecWorkers];
  uint32_t abort_flag;
  int32_t m_blocks;
  int32_t group_prefix[kMaxGroups + 1];  // masked: first M tile of each group
};

// Bytes of one ring stage: the activation rows of both 64-wide K halves first
// (1024-aligned for the swizzle), then packed weights and scales.
__host__ __device__ constexpr uint32_t decode_stage_bytes(int tokens) {
  return static_cast<uint32_t>(tokens) * 256u + kDecWSBytes;
}

// decode_tile() of the general kernel without its contiguous branch (not served here),
// with `ntok` = one past the last token slot that carries a row, which at decode sizes is
// commonly below 8 whatever block size the routing was aligned to.  A tile without any row
// is not valid (nothing to compute).  Must be called by all 32 lanes of a warp.
__device__ __forceinline__ TileInfo decode_tile_small(const GemmParams& p, const int32_t* group_prefix,
                                                      int32_t tile) {
  TileInfo t;
  const int32_t n_blocks = (p.n >> p.fuse_silu) / kBlockN;  // fused SiLU*mul: one tile per gate block
  const int32_t mb = tile / n_blocks;
  t.n0 = (tile - mb * n_blocks) * kBlockN;
  t.m0 = 0;
  t.limit = 0;
  t.mma_n = p.mma_n;
  if (p.mode == kModeIndexed) {
    // (through a shuffle: a loaded value is not known to be the same in all lanes)
    t.expert = __shfl_sync(0xffffffffu, __ldg(p.expert_ids + mb), 0);
    t.ntok = p.tile_tokens;
    t.base = mb * p.tile_tokens;
    const int32_t lane = static_cast<int32_t>(threadIdx.x & 31u);
    const int32_t id = lane < p.tile_tokens ? __ldg(p.sorted_ids + t.base + lane) : -1;
    const uint32_t rows = __ballot_sync(0xffffffffu, id >= 0 && id < p.out_rows && id / p.top_k < p.x_rows);
    t.ntok = 32 - __clz(static_cast<int32_t>(rows));  // one past the last slot that carries a row
  } else {
    int32_t lo = 0, hi = p.num_experts;
    while (hi - lo > 1) {
      const int32_t mid = (lo + hi) >> 1;
      if (group_prefix[mid] <= mb) lo = mid; else hi = mid;
    }
    lo = __shfl_sync(0xffffffffu, lo, 0);
    t.expert = lo;
    t.m0 = __shfl_sync(0xffffffffu, (mb - group_prefix[lo]) * p.tile_tokens, 0);
    int32_t mm = __shfl_sync(0xffffffffu, __ldg(p.masked_m + lo), 0);
    mm = mm < 0 ? 0 : (mm > p.max_m ? p.max_m : mm);
    t.limit = mm;
    const int32_t left = mm - t.m0;
    t.ntok = left < p.tile_tokens ? left : p.tile_tokens;
    t.base = lo * p.max_m;
  }
  t.rows = t.ntok;
  t.valid = t.expert >= 0 && t.expert < p.num_experts && t.ntok > 0;
  return t;
}

__device__ __forceinline__ float silu_f32(float v) { return v / (1.0f + __expf(-v)); }

// Where a computing warp finds its operands: shared-memory offsets into a ring stage.
struct DecodeLane {
  uint32_t w;      // packed words: slabs 2(q&1), 2(q&1)+1 of the 64-row chunk q>>1
  uint32_t s;      // scales of the same rows
  uint32_t probe;  // those of K32 group lane % 4
  uint32_t x[4];   // ldmatrix row addresses for the K16 steps of a 64-wide K half
};

// x[j] for NT = 1 (one ldmatrix covers two K16 steps; entries 0 and 1) or NT >= 2 (one
// ldmatrix covers 16 tokens of one K16 step).  Rows are 128 bytes, their 16-byte pieces
// stored at piece ^ (row % 8).
template <int NT>
__device__ __forceinline__ void decode_x_offsets(uint32_t lane, uint32_t (&x)[4]) {
  const uint32_t r = lane & 7u, mi = lane >> 3;
  if (NT == 1) {
    x[0] = r * 128u + ((mi ^ r) << 4);
    x[1] = x[0] ^ 64u;
    x[2] = x[3] = 0;
  } else {
    const uint32_t base = (r + 8u * (mi >> 1)) * 128u + (((mi & 1u) ^ r) << 4);
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) x[j] = base ^ (j * 32u);
  }
}

// Token fragments of one K16 step (NT >= 2).
template <int NT, int kX>
__device__ __forceinline__ void decode_tokens(uint32_t addr, uint32_t (&b)[2 * NT]) {
  uint32_t t[4];
  ptx::ldmatrix_x4<kX>(addr, t);
#pragma unroll
  for (int i = 0; i < 4; ++i) b[i] = t[i];
  if constexpr (NT == 3) {
    uint32_t u[2];
    ptx::ldmatrix_x2<kX + 2048>(addr, u);
    b[4] = u[0];
    b[5] = u[1];
  } else if constexpr (NT == 4) {
    ptx::ldmatrix_x4<kX + 2048>(addr, t);
#pragma unroll
    for (int i = 0; i < 4; ++i) b[4 + i] = t[i];
  }
}

// What a lane reads of one 64-wide K half: 32 weight rows, and the tokens where there are 8.
template <int NT>
struct DecodeHalf {
  uint2 words[4], scales[2];
  uint32_t tokens[NT == 1 ? 8 : 1];  // fragments of the four K16 steps (loaded as they are needed for NT > 1)
};

template <int kTokens, int NT, int kHalf>
__device__ __forceinline__ void decode_load(uint32_t st, const DecodeLane& at, DecodeHalf<NT>& h) {
  constexpr int kW = kTokens * 256 + 4096 * kHalf;
  constexpr int kS = kTokens * 256 + kDecWBytes + 512 * kHalf;
  constexpr int kX = kTokens * 128 * kHalf;
  h.words[0] = ptx::lds64<kW>(st + at.w);
  h.words[1] = ptx::lds64<kW + 1024>(st + at.w);
  h.words[2] = ptx::lds64<kW + 2048>(st + at.w);
  h.words[3] = ptx::lds64<kW + 3072>(st + at.w);
  h.scales[0] = ptx::lds64<kS>(st + at.s);
  h.scales[1] = ptx::lds64<kS + 256>(st + at.s);
  if constexpr (NT == 1) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      uint32_t t[4];
      ptx::ldmatrix_x4<kX>(st + at.x[j], t);
#pragma unroll
      for (int i = 0; i < 4; ++i) h.tokens[4 * j + i] = t[i];
    }
  }
}

// The products of one K half: 32 weight rows x 64 K x 8 NT tokens.
template <int kTokens, int NT, int kHalf, bool kAnyScale>
__device__ __forceinline__ void decode_half(uint32_t st, const DecodeLane& at, const DecodeHalf<NT>& h,
                                            float (&acc)[2][NT][4]) {
  constexpr int kX = kTokens * 128 * kHalf;
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    // scales[g].x = {slab A row r, slab A row r+8} of K32 group g; .y = the same for slab B.
    const Dequant<kAnyScale, true> da(h.scales[g].x), db(h.scales[g].y);
    uint32_t a[2][4], c[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) da(h.words[2 * g + i].x, a[i][0], a[i][1], a[i][2], a[i][3]);
#pragma unroll
    for (int i = 0; i < 2; ++i) db(h.words[2 * g + i].y, c[i][0], c[i][1], c[i][2], c[i][3]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j = 2 * g + i;
      uint32_t b[2 * NT];
      if constexpr (NT == 1) {
        b[0] = h.tokens[2 * j];
        b[1] = h.tokens[2 * j + 1];
      } else {
        decode_tokens<NT, kX>(st + at.x[j], b);
      }
#pragma unroll
      for (int n = 0; n < NT; ++n) ptx::mma_m16n8k16(acc[0][n], a[i], b[2 * n], b[2 * n + 1]);
#pragma unroll
      for (int n = 0; n < NT; ++n) ptx::mma_m16n8k16(acc[1][n], c[i], b[2 * n], b[2 * n + 1]);
    }
  }
}

// One stage whose first half has been loaded.
template <int kTokens, int NT, bool kAnyScale>
__device__ __forceinline__ void decode_stage_as(uint32_t st, const DecodeLane& at, bool second, DecodeHalf<NT>& h,
                                                float (&acc)[2][NT][4]) {
  decode_half<kTokens, NT, 0, kAnyScale>(st, at, h, acc);
  if (second) {
    decode_load<kTokens, NT, 1>(st, at, h);
    decode_half<kTokens, NT, 1, kAnyScale>(st, at, h, acc);
  }
}

// One stage.  Four lanes have the same scales, of its four K32 groups; each looks at the range of
// one group's, and one vote settles both halves.
template <int kTokens, int NT>
__device__ __forceinline__ void decode_stage(uint32_t st, const DecodeLane& at, bool second, float (&acc)[2][NT][4]) {
  DecodeHalf<NT> h;
  const uint2 probe = ptx::lds64<kTokens * 256 + kDecWBytes>(st + at.probe);
  decode_load<kTokens, NT, 0>(st, at, h);
  if (small_scales(probe)) decode_stage_as<kTokens, NT, false>(st, at, second, h, acc);
  else decode_stage_as<kTokens, NT, true>(st, at, second, h, acc);
}

// Ring position of a computing warp as running offsets (no multiplications in the loop).
struct DecodeRing {
  uint32_t base;              // shared address of stage 0
  uint32_t full0, empty0;     // barriers of stage 0
  uint32_t bytes;             // of the whole ring
  uint32_t abort_addr;
  uint32_t off = 0, bar = 0, ph = 0;
  uint32_t bad = 0;           // sticky: set by the first bounded wait that gives up
};

// One segment of a tile by one computing warp: K loop, stream-K fix-up, BF16 rows out.
// kBlocks = 2: gate_up with SiLU*mul; stages alternate between the gate and the up block of
// the tile (even / odd), each with accumulators of its own, and the warp stores
// bf16(silu(gate) * up).  A block no stage of the segment touched counts as zero.
template <int kTokens, int NT, int kBlocks>
__device__ __forceinline__ void decode_segment(const GemmParams& p, const Segment& seg, const TileInfo& t,
                                               DecodeRing& ring, bool tail, uint32_t q, uint32_t lane,
                                               uint32_t wt, uint32_t bar_id, int32_t worker_id,
                                               __nv_bfloat16* stage) {
  constexpr uint32_t kStageBytes = decode_stage_bytes(kTokens);
  DecodeLane at;
  at.w = (q >> 1) * 512u + lane * 16u + (q & 1) * 8u;
  at.s = (q >> 1) * 128u + (lane >> 2) * 16u + (q & 1) * 8u;
  at.probe = at.s + (lane & 3u) * 256u;
  decode_x_offsets<NT>(lane, at.x);
  // Output row of token slot `lane`: loaded now, used in the epilogue.
  const int32_t rows = out_row_of(p, t, static_cast<int32_t>(lane));
  float acc[kBlocks][2][NT][4];
#pragma unroll
  for (int b = 0; b < kBlocks; ++b)
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[b][m][n][i] = 0.0f;

  // The waits record a failure in `bad` and the code runs on (on stale data, within this
  // worker's own shared memory); `bad` is tested once per stage.  It is the same in all lanes
  // (the lanes vote inside the wait), so that a failure never splits the warp around the matrix
  // instructions and the barriers below.
  __syncwarp();
  if (ring.bad == 0) {
    for (int32_t kb = seg.kb; kb < seg.ke; ++kb) {
      const uint32_t st = ring.base + ring.off;
      ptx::mbar_wait_sticky<true>(ring.full0 + ring.bar, ring.ph, ring.abort_addr, ring.bad);
      // (the last stage holds one K half only when K is an odd multiple of 64, which no fused call has:
      // a branch less between its halves, 48 experts of 6 rows 150 -> 143 us)
      const bool second = kBlocks == 2 || !(tail && kb == seg.ke - 1);
      if (kBlocks == 1 || (kb & 1) == 0) decode_stage<kTokens, NT>(st, at, second, acc[0]);
      else decode_stage<kTokens, NT>(st, at, second, acc[kBlocks - 1]);
      __syncwarp();
      ptx::mbar_arrive_lane0(ring.empty0 + ring.bar, lane);
      ring.off += kStageBytes;
      ring.bar += 8u;
      if (ring.off == ring.bytes) {
        ring.off = 0;
        ring.bar = 0;
        ring.ph ^= 1u;
      }
      if (ring.bad != 0) break;
    }
  }

  // A whole tile needs nothing from the worker's other three warps; a stream-K slice does
  // (lock, partials), and only then do the four warps meet at named barriers.  A warp that
  // has given up skips the work but still meets its siblings there.
  const bool ok = ring.bad == 0;
  const bool shared_tile = seg.type != kSegFull;
  const size_t ws_slot = static_cast<size_t>(kBlockN) * kTokens * kBlocks;
  bool lock_ok = true;
  if (shared_tile) {
    if (ok && seg.type == kSegOwner && wt == 0) {
      const int* lock = p.locks + worker_id;
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
    ptx::named_bar_sync(bar_id, 128);  // lock observed
  }
  if (ok && seg.type == kSegContrib) {
    float4* dst = reinterpret_cast<float4*>(p.workspace + worker_id * ws_slot) + wt;
#pragma unroll
    for (int b = 0; b < kBlocks; ++b)
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const float* v = acc[b][m][n];
          __stcg(dst + ((b * 2 + m) * NT + n) * 128, make_float4(v[0], v[1], v[2], v[3]));
        }
    __threadfence();
  } else if (ok) {
    if (seg.type == kSegOwner) {
      // partials are added in worker order (deterministic)
      const float4* part = reinterpret_cast<const float4*>(p.workspace + (worker_id + 1) * ws_slot) + wt;
      for (int32_t peer = 1; peer <= seg.peer; ++peer, part += ws_slot / 4) {
        float4 v[kBlocks * 2 * NT];
#pragma unroll
        for (int i = 0; i < kBlocks * 2 * NT; ++i) v[i] = __ldcg(part + i * 128);
#pragma unroll
        for (int b = 0; b < kBlocks; ++b)
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n) {
              const float4& a = v[(b * 2 + m) * NT + n];
              acc[b][m][n][0] += a.x;
              acc[b][m][n][1] += a.y;
              acc[b][m][n][2] += a.z;
              acc[b][m][n][3] += a.w;
            }
      }
    }
    // Transpose through shared memory so that global stores are 16 bytes wide: eight
    // tokens at a time (32 weight rows x 8 tokens = one 16-byte piece per lane).  The lane's
    // accumulators are rows g, g+8 of each 16-row slab, tokens 2c, 2c+1.
    const uint32_t g = lane >> 2, c = lane & 3u;
    const int32_t col0 = t.n0 + static_cast<int32_t>(q) * 32;
    const int32_t ldn = kBlocks == 2 ? p.n >> 1 : p.n;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float v = acc[0][m][n][i];
          if (kBlocks == 2) v = silu_f32(v) * acc[kBlocks - 1][m][n][i];
          stage[(2 * c + (i & 1)) * kDecPitch + 16 * m + 8 * (i >> 1) + g] = __float2bfloat16_rn(v);
        }
      __syncwarp();
      const int32_t row = __shfl_sync(0xffffffffu, rows, 8 * n + static_cast<int32_t>(g));
      const uint4 val = *reinterpret_cast<const uint4*>(stage + g * kDecPitch + c * 8);
      if (row >= 0) {
        if (p.out_row_ptr != nullptr) {
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(
              __ldg(reinterpret_cast<const unsigned long long*>(p.out_row_ptr) + row));
          if (dst != nullptr) *reinterpret_cast<uint4*>(dst + col0 + c * 8) = val;
        } else {
          *reinterpret_cast<uint4*>(p.out + static_cast<size_t>(row) * ldn + col0 + c * 8) = val;
        }
      }
      __syncwarp();
    }
  }
  if (shared_tile) {
    ptx::named_bar_sync(bar_id, 128);  // all four warps' partials are written / read
    if (wt == 0) {
      // A contributor completes the handshake even after a failure, so that no owner
      // spins on a lock that would never move; the status word tells the host.  An owner
      // whose wait ran out leaves its word as it is (late contributors would make it
      // non-zero again behind a reset).
      if (seg.type == kSegContrib) ptx::red_release_add(p.locks + seg.peer, 1);
      else if (lock_ok) p.locks[worker_id] = 0;
    }
  }
}

// kTokens: token rows a ring stage has room for (16 or 32; p.mma_n).  kFuse: gate_up with
// SiLU*mul in the epilogue (16-token tiles and K % 128 == 0 only): a tile is a gate block
// and its up block (weight rows n0.. and N/2 + n0..), its ring stages alternate between the
// two (even stage = gate, odd = up, both of K block stage / 2).
template <int kTokens, bool kFuse>
__global__ void __launch_bounds__(kDecThreads, 1)
w4a16_decode_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_s,
                    const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  // Dynamic shared memory, 1024-aligned: one ring per worker, then DecodeShared.
  const uint32_t raw_addr = ptx::smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
  constexpr uint32_t kXBytes = kTokens * 256u;
  constexpr uint32_t kStageBytes = decode_stage_bytes(kTokens);
  const uint32_t stages = static_cast<uint32_t>(p.w_stages);
  const uint32_t worker_bytes = stages * kStageBytes;
  DecodeShared& sh = *reinterpret_cast<DecodeShared*>(smem + kDecWorkers * worker_bytes);

  // Read back through a shuffle so that the compiler knows the warp index (and every
  // ring position and barrier address derived from it) to be the same in all lanes and
  // keeps them in uniform registers.
  const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const uint32_t lane = threadIdx.x & 31;
  constexpr int32_t fuse = kFuse ? 1 : 0;
  const int32_t k_steps = ((p.k + kDecStageK - 1) / kDecStageK) << fuse;  // ring stages per tile
  const bool k_tail_half = (p.k % kDecStageK) != 0;             // last stage: first K half only

  // Set-up is on the critical path of a small launch: one thread per worker initialises
  // that worker's barriers.  (Activation rows that no gather fills keep whatever the shared
  // memory held: a token's column of the product depends on that token's row alone, and
  // columns without a row are not stored.)
  if (warp < kDecWorkers && lane == 0) {
    if (warp == 0) {
      ptx::prefetch_tensormap(&tm_w);
      ptx::prefetch_tensormap(&tm_s);
      sh.abort_flag = 0;
    }
    for (uint32_t s = 0; s < stages; ++s) {
      ptx::mbar_init(ptx::smem_u32(&sh.worker[warp].full[s]), 33);
      ptx::mbar_init(ptx::smem_u32(&sh.worker[warp].empty[s]), 4);
    }
    ptx::fence_barrier_init();
  }
  // Up to here nothing an earlier kernel of the stream may still be writing has been
  // read: with programmatic dependent launch the set-up above overlaps that kernel's tail.
  ptx::grid_dependency_wait();
  if (threadIdx.x == 0) {
    if (p.mode == kModeMasked) {
      int32_t acc = 0;
      for (int32_t g = 0; g < p.num_experts; ++g) {
        sh.group_prefix[g] = acc;
        int32_t mm = __ldg(p.masked_m + g);
        mm = mm < 0 ? 0 : (mm > p.max_m ? p.max_m : mm);
        acc += (mm + p.tile_tokens - 1) / p.tile_tokens;
      }
      sh.group_prefix[p.num_experts] = acc;
      sh.m_blocks = acc;
    } else {
      int32_t padded = __ldg(p.num_tokens_padded);
      padded = padded < 0 ? 0 : (padded > p.sorted_len ? p.sorted_len : padded);
      const int32_t blocks = padded / p.tile_tokens;
      sh.m_blocks = blocks > p.expert_len ? p.expert_len : blocks;
    }
  }
  __syncthreads();
  ptx::grid_launch_dependents();

  const uint32_t abort_addr = ptx::smem_u32(&sh.abort_flag);  // raised by any wait that gives up
  const int32_t tiles = __shfl_sync(0xffffffffu, sh.m_blocks, 0) * ((p.n >> fuse) / kBlockN);
  // warps 0-3 feed, warps 4-19 are the four workers' computing warps
  const uint32_t wk = warp < kDecWorkers ? warp : (warp - kDecWorkers) >> 2;
  // Worker ids interleave the CTAs (worker w of CTA c is c + w * grid), so that a launch
  // with fewer slices than workers spreads them over all SMs first.
  const int32_t worker_id = static_cast<int32_t>(wk * gridDim.x + blockIdx.x);
  const int32_t workers = static_cast<int32_t>(gridDim.x) * kDecWorkers;
  DecodeWorkerShared& ws = sh.worker[wk];
  const uint32_t ring0 = ptx::smem_u32(smem + wk * worker_bytes);  // shared address of stage 0
  const uint32_t full0 = ptx::smem_u32(&ws.full[0]);
  const uint32_t empty0 = ptx::smem_u32(&ws.empty[0]);

  if (warp < kDecWorkers) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kDecFeederRegs));
    // ------------------------- feeder of worker `warp`: weights, scales, activations --
    // Lane 0 issues the two TMA boxes of a stage; all lanes gather its activation rows with
    // cp.async (lane l fetches the 16-byte piece l % 8 of rows l / 8 + 4 b, b < kTokens / 4,
    // of both K halves) and leave an arrival on the stage's barrier behind their copies, so
    // that the feeder itself waits for nothing but free stages.
    constexpr int kRounds = kTokens / 4;
    const uint32_t piece = lane & 7u;
    const uint32_t r0 = lane >> 3;
    uint32_t dst_off[2];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const uint32_t r = r0 + 4u * b;
      dst_off[b] = r * 128u + ((piece ^ (r & 7u)) << 4);
    }
    SegmentIterator iter;
    iter.init(tiles, k_steps, workers, worker_id, true);
    Segment seg;
    StageCursor cur;
    uint32_t bad = 0;
    while (bad == 0 && iter.next(seg)) {
      const TileInfo t = decode_tile_small(p, sh.group_prefix, seg.tile);
      if (!t.valid) continue;
      // Once per segment: where the lane's rows are; a stage then only moves the pointers on.
      int32_t kb = seg.kb >> fuse;  // fused: both blocks of a pair of stages read the same K block
      const __nv_bfloat16* src[kRounds];
      uint32_t active = 0;  // bit b: the lane has a row to fetch in round b
#pragma unroll
      for (int b = 0; b < kRounds; ++b) {
        const int32_t slot = static_cast<int32_t>(r0) + 4 * b;
        const int32_t row = slot < t.ntok ? x_row_of(p, t, slot) : p.x_rows;
        const bool has = row < p.x_rows;
        src[b] = p.x + (has ? row * p.k : 0) + kb * kDecStageK + piece * 8;
        active |= has ? 1u << b : 0u;
      }
      const int32_t rounds = (t.ntok + 3) >> 2;
      int32_t w_row = t.expert * (p.k / 16) + kb * (kDecStageK / 16);
      int32_t s_row = t.expert * (p.k / 32) + kb * (kDecStageK / 32);
      for (int32_t step = seg.kb; step < seg.ke; ++step) {
        const int32_t w_col = t.n0 + (fuse ? (step & 1) * (p.n >> 1) : 0);
        ptx::mbar_wait_sticky(empty0 + cur.s * 8u, cur.ph ^ 1u, abort_addr, bad);
        bad = __any_sync(0xffffffffu, bad != 0) ? 1u : 0u;
        if (bad != 0) break;
        const uint32_t st = ring0 + cur.s * kStageBytes;
        const uint32_t full = full0 + cur.s * 8u;
        if (lane == 0) {
          ptx::mbar_arrive_expect_tx(full, kDecWSBytes);
          ptx::tma_load_2d(st + kXBytes, &tm_w, full, 2 * w_col, w_row);
          ptx::tma_load_2d(st + kXBytes + kDecWBytes, &tm_s, full, w_col, s_row);
        }
        __syncwarp();
        const bool second_half = !(k_tail_half && step == k_steps - 1);
#pragma unroll
        for (int b = 0; b < kRounds; ++b) {
          if (b >= rounds) break;
          if ((active >> b) & 1u) {
            const uint32_t dst = st + dst_off[b & 1] + (b >> 1) * 1024u;
            ptx::cp_async_16(dst, src[b], true);
            if (second_half) ptx::cp_async_16(dst + kTokens * 128u, src[b] + 64, true);
          }
        }
        ptx::cp_async_arrive_noinc(full);
        if (!kFuse || (step & 1)) {
#pragma unroll
          for (int b = 0; b < kRounds; ++b) src[b] += kDecStageK;
          w_row += kDecStageK / 16;
          s_row += kDecStageK / 32;
        }
        cur.advance(stages);
      }
    }
    // Nothing may stay in flight towards shared memory when the CTA retires, also when the
    // computing warps give up after this warp has issued its last stage: the gathers and the
    // boxes are waited for here (bounded), whoever else waits for them.
    ptx::cp_async_wait_all();
    for (uint32_t s = 0; s < stages; ++s) ptx::mbar_drain(full0 + s * 8u, cur.last_phase(s));
    if (bad != 0 && lane == 0 && p.status) atomicOr(p.status, kStatusProducerTimeout);
    __syncwarp();
  } else {
    // ---------------------------------------------------------- computing warps --
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kDecComputeRegs));  // (launch_decode has checked that they are there)
    const uint32_t q = (warp - kDecWorkers) & 3u;  // 32 weight rows of the tile
    const uint32_t wt = q * 32u + lane;            // 0..127 inside the worker
    const uint32_t bar_id = 1 + wk;
    DecodeRing ring;
    ring.base = ring0;
    ring.full0 = full0;
    ring.empty0 = empty0;
    ring.bytes = worker_bytes;
    ring.abort_addr = abort_addr;
    SegmentIterator iter;
    iter.init(tiles, k_steps, workers, worker_id, true);
    Segment seg;
    while (iter.next(seg)) {
      const TileInfo t = decode_tile_small(p, sh.group_prefix, seg.tile);
      if (!t.valid) continue;
      const bool tail = k_tail_half && seg.ke == k_steps;
      __nv_bfloat16* stage = &ws.stage[q][0][0];
      if (t.ntok <= 8) {
        decode_segment<kTokens, 1, 1 + fuse>(p, seg, t, ring, tail, q, lane, wt, bar_id, worker_id, stage);
      } else if (kTokens == 16 || t.ntok <= 16) {
        decode_segment<kTokens, 2, 1 + fuse>(p, seg, t, ring, tail, q, lane, wt, bar_id, worker_id, stage);
      } else if constexpr (kTokens > 16) {
        if (t.ntok <= 24) decode_segment<kTokens, 3, 1 + fuse>(p, seg, t, ring, tail, q, lane, wt, bar_id, worker_id, stage);
        else decode_segment<kTokens, 4, 1 + fuse>(p, seg, t, ring, tail, q, lane, wt, bar_id, worker_id, stage);
      }
    }
    if (ring.bad != 0 && lane == 0 && p.status) atomicOr(p.status, kStatusDequantTimeout);
  }
  __syncthreads();
}

}  // namespace chord
