// Routing alignment (moe_align_block_size) as a device routine.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "align_rules.h"
#include "ptx.cuh"

namespace chord {

// kCtas CTAs (one, or a cluster) of kWarps warps each (CUDA form of the reference's
// align_routing_blocks, tests/generators.py:192-230).  Pass 1 counts routes per (warp, expert);
// the per-expert totals give the padded block layout; pass 2 replays the same walk and places
// every id at expert offset + routes of lower CTAs and warps + routes seen so far by this warp, so
// ids inside an expert stay ascending and the result is deterministic.  `sentinel` pads the
// blocks (any value >= the number of routed rows the GEMM is told about).
//
// Bound by latency: few warps, every step waiting for L2 or shared memory.  A warp loads its ids
// kBatch rounds of 32 ahead (one L2 round trip per batch instead of one per round) and keeps
// them for pass 2 where it has no more than one batch; the offsets come from a warp scan.  The CTAs
// of a cluster read each other's totals from shared memory and compute the layout each for itself.
template <int kWarps, int kBatch, int kCtas>
__device__ __forceinline__ void moe_align_block(const int32_t* topk_ids, int32_t numel, int32_t sentinel,
                                                int32_t expert_base, int32_t num_experts,
                                                int32_t block_m, int32_t* sorted_ids,
                                                int32_t sorted_cap, int32_t* expert_ids,
                                                int32_t expert_cap, int32_t* num_tokens_padded) {
  extern __shared__ int32_t align_smem[];
  int32_t* counts = align_smem;                          // [kWarps][num_experts]
  int32_t* totals = align_smem + kWarps * num_experts;   // [num_experts]: of this CTA, read by its cluster
  int32_t* offsets = totals + num_experts;               // [num_experts + 1]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = kCtas > 1 ? static_cast<int>(ptx::cluster_ctarank()) : 0;
  for (int i = threadIdx.x; i < kWarps * num_experts; i += blockDim.x) counts[i] = 0;

  // Local expert of the ids i + 32 u + lane, or -1.
  const int32_t per_warp = ((numel + kWarps * kCtas - 1) / (kWarps * kCtas) + 31) / 32 * 32;
  const int32_t begin = (rank * kWarps + warp) * per_warp;
  const int32_t end = min(numel, begin + per_warp);
  int32_t e[kBatch];
  auto load = [&](int32_t i) {
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int32_t idx = i + 32 * u + lane;
      e[u] = idx < end ? __ldcg(topk_ids + idx) : -1;
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const uint32_t local = static_cast<uint32_t>(e[u]) - static_cast<uint32_t>(expert_base);
      e[u] = (i + 32 * u + lane < end && local < static_cast<uint32_t>(num_experts)) ? static_cast<int32_t>(local) : -1;
    }
  };
  constexpr int32_t kStep = 32 * kBatch;
  int32_t* mine = counts + warp * num_experts;
  if (begin < end) load(begin);
  __syncthreads();
  for (int32_t i = begin; i < end; i += kStep) {
    if (i != begin) load(i);
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      if (e[u] >= 0) atomicAdd(mine + e[u], 1);
    }
  }
  __syncthreads();

  // Per expert: totals, and per-warp counts turned into exclusive prefixes (with the routes of
  // lower CTAs in front).
  for (int x = threadIdx.x; x < num_experts; x += blockDim.x) {
    int32_t run = 0;
#pragma unroll 8
    for (int w = 0; w < kWarps; ++w) {
      const int32_t c = counts[w * num_experts + x];
      counts[w * num_experts + x] = run;
      run += c;
    }
    if constexpr (kCtas > 1) totals[x] = run;
    offsets[x] = (run + block_m - 1) / block_m * block_m;
  }
  if constexpr (kCtas > 1) {
    __syncwarp();
    ptx::cluster_sync();
    int32_t all[2] = {0, 0};  // (an expert per thread and round; both rounds of up to 2048 experts)
    int32_t below[2] = {0, 0};
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int x = threadIdx.x + t * kWarps * 32;
      if (x >= num_experts) continue;
      const uint32_t addr = ptx::smem_u32(totals + x);
#pragma unroll
      for (int r = 0; r < kCtas; ++r) {
        const int32_t c = ptx::ld_cluster(ptx::map_to_cta(addr, r));
        all[t] += c;
        below[t] += r < rank ? c : 0;
      }
    }
    __syncwarp();
    ptx::cluster_sync();  // every CTA has read the others' totals
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int x = threadIdx.x + t * kWarps * 32;
      if (x >= num_experts) continue;
      totals[x] = all[t];
      offsets[x] = (all[t] + block_m - 1) / block_m * block_m;
#pragma unroll 8
      for (int w = 0; w < kWarps; ++w) counts[w * num_experts + x] += below[t];
    }
  }
  __syncthreads();
  if (warp == 0) {
    int32_t acc = 0;
    for (int x0 = 0; x0 < num_experts; x0 += 32) {
      const int32_t padded = x0 + lane < num_experts ? offsets[x0 + lane] : 0;
      int32_t scan = padded;  // inclusive
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int32_t below = __shfl_up_sync(0xffffffffu, scan, d);
        if (lane >= d) scan += below;
      }
      if (x0 + lane < num_experts) offsets[x0 + lane] = acc + scan - padded;
      acc += __shfl_sync(0xffffffffu, scan, 31);
    }
    if (lane == 0) {
      offsets[num_experts] = acc;
      if (rank == 0) *num_tokens_padded = acc < sorted_cap ? acc : sorted_cap / block_m * block_m;
    }
  }
  __syncthreads();
  const int32_t total = min(offsets[num_experts], sorted_cap / block_m * block_m);
  if constexpr (kCtas > 1) {
    // Sentinels behind each expert's routes (no other CTA places an id there) and the experts of
    // its blocks; a warp per expert.
    for (int x = rank * kWarps + warp; x < num_experts; x += kWarps * kCtas) {
      const int32_t first = offsets[x], last = offsets[x + 1];
      for (int32_t i = first + totals[x] + lane; i < min(last, total); i += 32) sorted_ids[i] = sentinel;
      const int32_t blocks = (last - first) / block_m, block0 = first / block_m;
      for (int32_t b = lane; b < blocks; b += 32) {
        if (block0 + b < expert_cap) expert_ids[block0 + b] = x;
      }
    }
  } else {
    // Sentinels everywhere, then the ids over them: fewer dependent steps than a warp per expert
    // (512 ids over 48 experts: 4.1 against 5.0 us).
    for (int32_t i = threadIdx.x; i < total; i += blockDim.x) sorted_ids[i] = sentinel;
    for (int x = threadIdx.x; x < num_experts; x += blockDim.x) {
      for (int32_t b = offsets[x] / block_m; b < offsets[x + 1] / block_m; ++b) {
        if (b < expert_cap) expert_ids[b] = x;
      }
    }
    __syncthreads();
  }

  for (int32_t i = begin; i < end; i += kStep) {
    // (the ids of a single batch are still in the registers)
    if (end - begin > kStep) load(i);
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      if (i + 32 * u >= end) break;
      const uint32_t peers = __match_any_sync(0xffffffffu, e[u]);
      if (e[u] >= 0) {
        const int32_t rank_in_round = __popc(peers & ((1u << lane) - 1u));
        const int32_t pos = offsets[e[u]] + mine[e[u]] + rank_in_round;
        if (pos < total) sorted_ids[pos] = i + 32 * u + lane;
      }
      __syncwarp();
      if (e[u] >= 0 && lane == __ffs(peers) - 1) mine[e[u]] += __popc(peers);
      __syncwarp();
    }
  }
}

}  // namespace chord
