// Which kernel aligns a routing (routing.cuh): plain C++, so that a host without a GPU can check it too.
#pragma once

#include <cstddef>
#include <cstdint>

namespace chord {

constexpr int kAlignWarps = 32;
constexpr int kAlignWarpsFew = 16;
constexpr int kAlignCtas = 8;  // of the cluster that aligns many ids
constexpr size_t kAlignMaxSmem = 170 * 1024;

// Dynamic shared memory of a CTA of `warps` warps.
constexpr size_t moe_align_smem_bytes(int64_t num_experts, int warps) {
  return ((static_cast<size_t>(warps) + 2) * static_cast<size_t>(num_experts) + 1) * 4;
}

enum class AlignKernel { kShort = 0, kBatches = 1, kCluster = 2 };

// From 4096 ids on a cluster of eight CTAs of 32 warps (four rounds of loads ahead), where
// the counters fit 170 KB (up to 1279 experts) and the device can place such a cluster
// (`cluster_fits`: a part of a GPU may have too few SMs side by side).  Otherwise one CTA of 16 warps, with
// four rounds ahead from 513 ids on (more than the experts, where those are more); up to 512 a warp has
// one round, and the batch's unrolled code would only cost instruction fetches.
// One CTA / the cluster, us (replayed graph): 48 of 384 experts, 2048 ids 4.0 / 5.7, 4096 ids 5.7 / 5.8,
// 6144 ids 7.0 / 5.7, 32768 ids 24.7 / 6.7; 384 experts, 2048 ids 7.0 / 8.7, 4096 ids 10.0 / 8.6.
// One round / four rounds ahead: 48 of 384 experts, 1024 ids 4.2 / 3.6, 2048 ids 5.4 / 4.0; 640 experts, 640
// ids 6.8 / 6.8, 1024 ids 7.4 / 7.4, 1280 ids 8.4 / 7.7; 1024 experts, 1024 ids 8.7 / 9.0, 1280 ids 9.7 / 9.3; 2048
// experts, 1024 ids 12.5 / 13.7, 2048 ids 15.2 / 15.5.
constexpr AlignKernel align_kernel(int64_t numel, int64_t num_experts, bool cluster_fits) {
  if (numel >= 4096 && cluster_fits && moe_align_smem_bytes(num_experts, kAlignWarps) <= kAlignMaxSmem) return AlignKernel::kCluster;
  return numel > 32 * kAlignWarpsFew && numel > num_experts ? AlignKernel::kBatches : AlignKernel::kShort;
}

}  // namespace chord
