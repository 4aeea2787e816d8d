// The steps either side of the expert GEMMs: SiLU*mul between gate_up and
// down, and the routing alignment (moe_align_block_size) that produces the
// sorted_ids / expert_ids / num_tokens_padded contract `indexed` consumes.
#include <cuda_bf16.h>

#include <mutex>

#include "../../include/chord_b200.h"
#include "common.h"
#include "ptx.cuh"
#include "routing.cuh"

namespace chord {
namespace {

__device__ __forceinline__ float silu(float v) { return v / (1.0f + __expf(-v)); }

// Eight outputs silu(g) * u.  A vector of zero gates (rows of a masked layout that hold no
// token) skips the divisions: their zero numerators take the slow branch of each, and silu(+-0)
// = +-0 leaves the same product.
__device__ __forceinline__ uint4 silu_mul_vec8(const uint4 g, const uint4 u) {
  const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
  const uint32_t uw[4] = {u.x, u.y, u.z, u.w};
  const bool zero = ((g.x | g.y | g.z | g.w) & 0x7FFF7FFFu) == 0;
  uint32_t ow[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 gf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gw[i]));
    const float2 uf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&uw[i]));
    if (!zero) gf = make_float2(silu(gf.x), silu(gf.y));
    const __nv_bfloat162 o = __floats2bfloat162_rn(gf.x * uf.x, gf.y * uf.y);
    ow[i] = *reinterpret_cast<const uint32_t*>(&o);
  }
  return make_uint4(ow[0], ow[1], ow[2], ow[3]);
}

// out[r, c..c+7] = silu(in[r, c..]) * in[r, inter + c..], a vector per thread and step; the
// tensor's vectors are numbered through, so that every thread has work whatever the number and
// the length of the rows.  Bound by the instructions of the divisions, some ten per element
// (with a reciprocal instruction in their place the copy rate is reached, at one more rounding
// of the quotient, which no caller asked for).  Index: 32 bits where they suffice, because a
// 64-bit division per vector shows.  30144 rows of 2 x 2048 in HBM, us: 64-bit index 69.0, this
// 66.4, a block per row 78.8; all but 8 of 256 rows zero: 125 without the branch for zeros, 58;
// 8 rows of 2 x 65536: 2.3, 2.2, 29.
template <typename Index>
__global__ void __launch_bounds__(256)
silu_mul_kernel(const uint4* __restrict__ in, uint4* __restrict__ out, Index total, Index row_vecs) {
  ptx::grid_dependency_wait();
  for (Index i = static_cast<Index>(blockIdx.x) * 256 + threadIdx.x; i < total; i += static_cast<Index>(gridDim.x) * 256) {
    const uint4* gate = in + static_cast<size_t>(i) + static_cast<size_t>(i / row_vecs) * row_vecs;
    out[i] = silu_mul_vec8(__ldg(gate), __ldg(gate + row_vecs));
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
    const uint4* gate = reinterpret_cast<const uint4*>(in + r * 2 * inter);
    uint4* row = reinterpret_cast<uint4*>(out + r * inter);
    for (int64_t c = threadIdx.x; c < inter / 8; c += blockDim.x) row[c] = silu_mul_vec8(__ldg(gate + c), __ldg(gate + inter / 8 + c));
  }
}

template <int kWarps, int kBatch, int kCtas>
__global__ void __launch_bounds__(kWarps * 32)
moe_align_kernel(const int32_t* __restrict__ topk_ids, int32_t numel, int32_t expert_base,
                 int32_t num_experts, int32_t block_m, int32_t* __restrict__ sorted_ids,
                 int32_t sorted_cap, int32_t* __restrict__ expert_ids, int32_t expert_cap,
                 int32_t* __restrict__ num_tokens_padded) {
  moe_align_block<kWarps, kBatch, kCtas>(topk_ids, numel, numel, expert_base, num_experts, block_m, sorted_ids,
                                  sorted_cap, expert_ids, expert_cap, num_tokens_padded);
}

using AlignFn = void (*)(const int32_t*, int32_t, int32_t, int32_t, int32_t, int32_t*, int32_t, int32_t*, int32_t, int32_t*);
const AlignFn kAlignKernels[3] = {moe_align_kernel<kAlignWarpsFew, 1, 1>, moe_align_kernel<kAlignWarpsFew, 4, 1>,
                                  moe_align_kernel<kAlignWarps, 4, kAlignCtas>};

// Whether the device can place the cluster at its largest, asked once per device.
bool align_cluster_fits(int device) {
  static std::mutex mutex;
  static int answer[64];  // 0 = not asked yet, 1 = no, 2 = yes
  std::lock_guard<std::mutex> guard(mutex);
  int& known = answer[device & 63];
  if (known == 0) {
    const AlignFn kernel = kAlignKernels[static_cast<int>(AlignKernel::kCluster)];
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = kAlignCtas;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(kAlignCtas);
    config.blockDim = dim3(kAlignWarps * 32);
    config.dynamicSmemBytes = kAlignMaxSmem;
    config.attrs = attribute;
    config.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kAlignMaxSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) != cudaSuccess) {
      cudaGetLastError();
      clusters = 0;
    }
    known = clusters >= 1 ? 2 : 1;
  }
  return known == 2;
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
  const int64_t total = rows * (inter / 8);
  int64_t blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  const dim3 grid(static_cast<unsigned>(blocks));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool pdl = chord::options().pdl != 0;
  const uint4* x = static_cast<const uint4*>(in);
  uint4* y = static_cast<uint4*>(out);
  if (total < (1ll << 31)) {
    CHORD_CUDA(chord::launch_kernel(chord::silu_mul_kernel<uint32_t>, grid, dim3(256), 0, s, pdl, x, y,
                                    static_cast<uint32_t>(total), static_cast<uint32_t>(inter / 8)));
  } else {
    CHORD_CUDA(chord::launch_kernel(chord::silu_mul_kernel<int64_t>, grid, dim3(256), 0, s, pdl, x, y, total, inter / 8));
  }
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
  int device = 0;
  CHORD_CUDA(cudaGetDevice(&device));
  const bool cluster_fits = numel >= 4096 && chord::align_cluster_fits(device);
  const chord::AlignKernel which = chord::align_kernel(numel, num_experts, cluster_fits);
  const int warps = which == chord::AlignKernel::kCluster ? chord::kAlignWarps : chord::kAlignWarpsFew;
  const chord::AlignFn kernel = chord::kAlignKernels[static_cast<int>(which)];
  const size_t smem = chord::moe_align_smem_bytes(num_experts, warps);
  static bool attr_set[3][64] = {};
  bool& attr = attr_set[static_cast<int>(which)][device & 63];
  if (smem > 48 * 1024 && !attr) {
    CHORD_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, chord::kAlignMaxSmem));
    attr = true;
  }
  const auto cap = [](int64_t v) { return static_cast<int32_t>(v < (1ll << 30) ? v : (1ll << 30)); };
  const int32_t n = static_cast<int32_t>(numel), base = static_cast<int32_t>(expert_base);
  const int32_t experts = static_cast<int32_t>(num_experts), block = static_cast<int32_t>(block_m);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (which == chord::AlignKernel::kCluster) {
    CHORD_CUDA(chord::launch_kernel_clusters(kernel, chord::kAlignCtas, dim3(chord::kAlignCtas), dim3(warps * 32), smem, s,
                                             false, topk_ids, n, base, experts, block, sorted_ids, cap(sorted_cap),
                                             expert_ids, cap(expert_cap), num_tokens_padded));
  } else {
    kernel<<<1, warps * 32, smem, s>>>(topk_ids, n, base, experts, block, sorted_ids, cap(sorted_cap), expert_ids,
                                       cap(expert_cap), num_tokens_padded);
    CHORD_CUDA(cudaGetLastError());
  }
  return chord::kOk;
}

}  // extern "C"
