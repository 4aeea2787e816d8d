// The steps either side of the expert GEMMs: SiLU*mul between gate_up and
// down, and the routing alignment (moe_align_block_size) that produces the
// sorted_ids / expert_ids / num_tokens_padded contract `indexed` consumes.
#include <cuda_bf16.h>

#include "../../include/chord_b200.h"
#include "common.h"
#include "ptx.cuh"
#include "routing.cuh"

namespace chord {
namespace {

// The reciprocal instruction (1 ulp) instead of an IEEE division: at eight values per vector
// the divisions were as long as the memory traffic.  Subnormal reciprocals (v near -88) are kept.
__device__ __forceinline__ float silu(float v) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(1.0f + __expf(-v)));
  return v * r;
}

// Eight outputs per thread: out[r, c..c+7] = silu(in[r, c..]) * in[r, inter + c..].
__device__ __forceinline__ void silu_mul_vec8(const __nv_bfloat16* in_row, __nv_bfloat16* out_row,
                                              int64_t inter, int64_t c) {
  const uint4 g = __ldg(reinterpret_cast<const uint4*>(in_row + c));
  const uint4 u = __ldg(reinterpret_cast<const uint4*>(in_row + inter + c));
  const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
  const uint32_t uw[4] = {u.x, u.y, u.z, u.w};
  uint32_t ow[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 gf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gw[i]));
    const float2 uf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&uw[i]));
    const __nv_bfloat162 o = __floats2bfloat162_rn(silu(gf.x) * uf.x, silu(gf.y) * uf.y);
    ow[i] = *reinterpret_cast<const uint32_t*>(&o);
  }
  *reinterpret_cast<uint4*>(out_row + c) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
}

// Bound by HBM: two vectors in, one out.  A row of threads (x) per row of the tensor, so that
// no index is divided, and a block per few rows, so that many are in flight (30144 rows of
// 4096: 100 us with a flat 64-bit index and IEEE divisions, 94 us).
__global__ void __launch_bounds__(256)
silu_mul_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out,
                int64_t rows, int64_t inter) {
  ptx::grid_dependency_wait();
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.y + threadIdx.y; r < rows;
       r += static_cast<int64_t>(gridDim.x) * blockDim.y) {
    const __nv_bfloat16* in_row = in + r * 2 * inter;
    __nv_bfloat16* out_row = out + r * inter;
    for (int64_t c = threadIdx.x * 8; c < inter; c += blockDim.x * 8) silu_mul_vec8(in_row, out_row, inter, c);
  }
}

__global__ void __launch_bounds__(256)
silu_mul_routed_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out,
                       const int32_t* __restrict__ sorted_ids, int64_t sorted_len,
                       const int32_t* __restrict__ num_tokens_padded, int64_t row_limit,
                       int64_t inter) {
  ptx::grid_dependency_wait();
  int64_t count = __ldg(num_tokens_padded);
  count = count < 0 ? 0 : (count > sorted_len ? sorted_len : count);
  for (int64_t slot = blockIdx.x; slot < count; slot += gridDim.x) {
    const int64_t r = __ldg(sorted_ids + slot);
    if (r < 0 || r >= row_limit) continue;
    for (int64_t c = threadIdx.x * 8; c < inter; c += blockDim.x * 8) {
      silu_mul_vec8(in + r * 2 * inter, out + r * inter, inter, c);
    }
  }
}

template <int kWarps, int kBatch>
__global__ void __launch_bounds__(kWarps * 32)
moe_align_kernel(const int32_t* __restrict__ topk_ids, int32_t numel, int32_t expert_base,
                 int32_t num_experts, int32_t block_m, int32_t* __restrict__ sorted_ids,
                 int32_t sorted_cap, int32_t* __restrict__ expert_ids, int32_t expert_cap,
                 int32_t* __restrict__ num_tokens_padded) {
  moe_align_block<kWarps, kBatch>(topk_ids, numel, numel, expert_base, num_experts, block_m, sorted_ids,
                                  sorted_cap, expert_ids, expert_cap, num_tokens_padded);
}

}  // namespace
}  // namespace chord

extern "C" {

int chord_b200_silu_mul(const void* in, void* out, int64_t rows, int64_t inter, void* stream) {
  CHORD_REQUIRE(in != nullptr && out != nullptr, "null tensor pointer");
  CHORD_REQUIRE(rows >= 0 && inter > 0 && inter % 8 == 0,
                "need rows >= 0 and a positive intermediate size divisible by 8");
  CHORD_REQUIRE(((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0,
                "in and out must be 16-byte aligned");
  if (rows == 0) return chord::kOk;
  // As many threads along a row as it has vectors (a power of two, at most the block), the
  // rest of the block along the rows.
  unsigned tx = 1;
  while (tx < 256 && tx < inter / 8) tx *= 2;
  const dim3 block(tx, 256 / tx);
  int64_t blocks = (rows + block.y - 1) / block.y;
  if (blocks > 148 * 256) blocks = 148 * 256;
  CHORD_CUDA(chord::launch_kernel(chord::silu_mul_kernel, dim3(static_cast<unsigned>(blocks)), block, 0,
                                  static_cast<cudaStream_t>(stream), chord::options().pdl != 0,
                                  static_cast<const __nv_bfloat16*>(in), static_cast<__nv_bfloat16*>(out),
                                  rows, inter));
  return chord::kOk;
}

int chord_b200_silu_mul_routed(const void* in, void* out, const int32_t* sorted_ids,
                               int64_t sorted_len, const int32_t* num_tokens_padded,
                               int64_t row_limit, int64_t inter, void* stream) {
  CHORD_REQUIRE(in != nullptr && out != nullptr && sorted_ids != nullptr &&
                    num_tokens_padded != nullptr,
                "null tensor pointer");
  CHORD_REQUIRE(inter > 0 && inter % 8 == 0, "intermediate size must be a positive multiple of 8");
  CHORD_REQUIRE(((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0,
                "in and out must be 16-byte aligned");
  if (sorted_len <= 0) return chord::kOk;
  const int64_t blocks = sorted_len < 148 * 8 ? sorted_len : 148 * 8;
  CHORD_CUDA(chord::launch_kernel(chord::silu_mul_routed_kernel, dim3(static_cast<unsigned>(blocks)),
                                  dim3(256), 0, static_cast<cudaStream_t>(stream),
                                  chord::options().pdl != 0, static_cast<const __nv_bfloat16*>(in),
                                  static_cast<__nv_bfloat16*>(out), sorted_ids, sorted_len,
                                  num_tokens_padded, row_limit, inter));
  return chord::kOk;
}

int chord_b200_moe_align_block_size(const int32_t* topk_ids, int64_t numel, int64_t expert_base,
                                    int64_t num_experts, int64_t block_m, int32_t* sorted_ids,
                                    int64_t sorted_cap, int32_t* expert_ids, int64_t expert_cap,
                                    int32_t* num_tokens_padded, void* stream) {
  CHORD_REQUIRE(sorted_ids != nullptr && expert_ids != nullptr && num_tokens_padded != nullptr,
                "null routing pointer");
  CHORD_REQUIRE(numel >= 0 && numel < (1ll << 30), "numel out of range");
  CHORD_REQUIRE(numel == 0 || topk_ids != nullptr, "null topk_ids");
  CHORD_REQUIRE(num_experts > 0 && num_experts <= 2048, "num_experts must be in [1, 2048]");
  CHORD_REQUIRE(block_m > 0 && block_m % 8 == 0, "block_m must be a positive multiple of 8");
  const int64_t worst = numel + num_experts * (block_m - 1);
  const int64_t need = (worst < numel * block_m ? worst : numel * block_m);
  CHORD_REQUIRE(sorted_cap >= need / block_m * block_m,
                "sorted_ids capacity %lld is below the worst case %lld",
                static_cast<long long>(sorted_cap), static_cast<long long>(need / block_m * block_m));
  CHORD_REQUIRE(expert_cap >= need / block_m, "expert_ids capacity %lld is below the worst case %lld",
                static_cast<long long>(expert_cap), static_cast<long long>(need / block_m));
  // From 4096 ids on 32 warps, sixteen rounds of loads ahead, where the counters fit 160 KB (up
  // to 1240 experts).  Below that the short loop of 16 warps: a batch's unrolled code costs a
  // small call more (instruction fetches) than the loads it overlaps.
  // (32768 ids over 48 experts: 39.6 us with a load per round and 16 warps, 18.5 us now; 2048 ids:
  // 5.0 us with the short loop, 5.8 with the long one.)
  constexpr size_t kMaxSmem = 160 * 1024;
  const bool wide = numel >= 4096 && chord::moe_align_smem_bytes(num_experts, chord::kAlignWarps) <= kMaxSmem;
  const int warps = wide ? chord::kAlignWarps : chord::kAlignWarpsFew;
  const auto kernel = wide ? chord::moe_align_kernel<chord::kAlignWarps, 16>
                           : chord::moe_align_kernel<chord::kAlignWarpsFew, 1>;
  const size_t smem = chord::moe_align_smem_bytes(num_experts, warps);
  static bool attr_set[2][64] = {};
  int device = 0;
  CHORD_CUDA(cudaGetDevice(&device));
  if (smem > 48 * 1024 && !attr_set[wide][device & 63]) {
    CHORD_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
    attr_set[wide][device & 63] = true;
  }
  kernel<<<1, warps * 32, smem, static_cast<cudaStream_t>(stream)>>>(
      topk_ids, static_cast<int32_t>(numel), static_cast<int32_t>(expert_base),
      static_cast<int32_t>(num_experts), static_cast<int32_t>(block_m), sorted_ids,
      static_cast<int32_t>(sorted_cap < (1ll << 30) ? sorted_cap : (1ll << 30)), expert_ids,
      static_cast<int32_t>(expert_cap < (1ll << 30) ? expert_cap : (1ll << 30)),
      num_tokens_padded);
  CHORD_CUDA(cudaGetLastError());
  return chord::kOk;
}

}  // extern "C"
