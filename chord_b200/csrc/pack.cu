// Weight packer and scale permutation (load-time, integer / data-movement only).
//
// Output format, bit-exact with the reference's repack kernel
// (chord_kernels/operator/include/humming/kernel/repack.cuh:8-121 launched with
// interleave_mode 3, chord_kernels/operator/kernel/repack_weight.py:41-77):
//   packed int32 [E, K/16, 2N]; for word c of row kb let nb = c / 128,
//   t = (c % 128) / 4, s = c % 4; for rh, kh, kk in {0, 1} the 4-bit code of
//   weight (n, k) = (64 nb + 16 s + 8 rh + t / 4, 16 kb + 8 kh + 2 (t % 4) + kk)
//   sits at bit 4 (2 rh + kh) + 16 kk.
// The kernels below are organised around the output: one thread assembles 16-byte vectors
// (the four slabs s = 0..3 of one (kb, nb, t)), so stores are fully coalesced, and a CTA
// stages its 64-row x kTileK input tile in shared memory as nibbles with coalesced vector
// loads.  Both are bound by HBM (every byte is read and written once) as long as the
// shuffling of nibbles costs few instructions and enough bytes are in flight.
#include "../../include/chord_b200.h"
#include "common.h"
#include "ptx.cuh"

namespace chord {
namespace {

constexpr int kRows = 64;  // weight rows per CTA tile (one 64-row chunk)

// The four nibble pairs a packed word takes from the tile words b00, b01 (row r, K halves 0
// and 1) and b10, b11 (row r + 8): byte q of each word = codes of K offsets 2q, 2q + 1.  The
// bytes are collected in the order 2 rh + kh, then their low nibbles are moved to the lower
// and their high nibbles to the upper half of the word.
__device__ __forceinline__ uint32_t interleave_pairs(uint32_t b00, uint32_t b01, uint32_t b10, uint32_t b11,
                                                     uint32_t selector) {
  const uint32_t lo = __byte_perm(b00, b01, selector), hi = __byte_perm(b10, b11, selector);
  uint32_t x = __byte_perm(lo, hi, 0x5410);
  const uint32_t t = (x ^ (x >> 4)) & 0x00F000F0u;  // swap the middle nibbles of each half
  x ^= t ^ (t << 4);
  return __byte_perm(x, x, 0x3120);  // swap the middle bytes
}

// Shared tile: kRows rows of kTileK nibbles, eight nibbles per word (little-endian, i.e. the
// checkpoint form), four pad words per row so that the 16-byte reads of eight rows fall on
// different banks.  A thread reads 16 bytes (two K16 blocks) of each of its eight rows and
// assembles two output vectors from them; four lanes share every read.
// (4096 x 7168, 16 experts, checkpoint form, both kernels of a pack: 158 us = 3.3 TB/s with
// 32-bit copies into the tile and every output word put together nibble by nibble from
// 32-bit reads; 83 us = 6.4 TB/s with this layout.)
template <int kTileK, bool kPackedInput>
__global__ void __launch_bounds__(256)
repack_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int n, int k,
              int32_t* __restrict__ range_flag) {
  constexpr int kWordsPerRow = kTileK / 8;
  constexpr int kPitch = kWordsPerRow + 4;
  static_assert(kPitch % 32 == 4, "eight rows x 16 bytes must cover all banks");
  __shared__ __align__(16) uint32_t tile[kRows][kPitch];
  const int nb = blockIdx.x;
  const int k0 = blockIdx.y * kTileK;
  const int e = blockIdx.z;
  const int tid = threadIdx.x;
  const int k_here = min(kTileK, k - k0);  // multiple of 64

  if constexpr (kPackedInput) {
    constexpr int kVecs = kWordsPerRow / 4;
    const size_t row_words = static_cast<size_t>(k) / 8;
    const uint32_t* src = in + (static_cast<size_t>(e) * n + static_cast<size_t>(nb) * kRows) * row_words + k0 / 8;
    for (int i = tid; i < kRows * kVecs; i += blockDim.x) {
      const int r = i / kVecs, v = i % kVecs;
      if (v * 32 < k_here) ptx::cp_async_16(ptx::smem_u32(&tile[r][4 * v]), src + r * row_words + 4 * v, true);
    }
    ptx::cp_async_wait_all();
  } else {
    const uint32_t* src = in + (static_cast<size_t>(e) * n + static_cast<size_t>(nb) * kRows) * k + k0;
    uint32_t seen = 0;
#pragma unroll 4
    for (int i = tid; i < kRows * kWordsPerRow; i += 256) {
      const int r = i / kWordsPerRow, w = i % kWordsPerRow;
      if (w * 8 < k_here) {
        const uint4* p = reinterpret_cast<const uint4*>(src + static_cast<size_t>(r) * k + w * 8);
        const uint4 a = __ldg(p), b = __ldg(p + 1);
        const uint32_t c[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t word = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          seen |= c[j];
          word |= (c[j] & 15u) << (4 * j);
        }
        tile[r][w] = word;
      }
    }
    if (seen > 15u && range_flag != nullptr) atomicOr(range_flag, 1);
  }
  __syncthreads();

  // Two uint4 per (kb pair, t): words s = 0..3 of packed rows kb, kb + 1, columns 128 nb + 4 t + s.
  const int pairs = k_here / 32;
  const size_t out_pitch = 2 * static_cast<size_t>(n);
  uint32_t* dst0 = out + (static_cast<size_t>(e) * (k / 16) + k0 / 16) * out_pitch + 128 * nb;
  for (int i = tid; i < pairs * 32; i += blockDim.x) {
    const int kp = i >> 5, t = i & 31;
    const int r8 = t >> 2;
    const uint32_t q = t & 3u;
    const uint32_t selector = q | (4u + q) << 4;
    uint32_t words[2][4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const uint4 lo = *reinterpret_cast<const uint4*>(&tile[16 * s + r8][4 * kp]);
      const uint4 hi = *reinterpret_cast<const uint4*>(&tile[16 * s + 8 + r8][4 * kp]);
      words[0][s] = interleave_pairs(lo.x, lo.y, hi.x, hi.y, selector);
      words[1][s] = interleave_pairs(lo.z, lo.w, hi.z, hi.w, selector);
    }
    uint32_t* dst = dst0 + static_cast<size_t>(2 * kp) * out_pitch + 4 * t;
#pragma unroll
    for (int h = 0; h < 2; ++h, dst += out_pitch) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(words[h][0], words[h][1], words[h][2], words[h][3]);
    }
  }
}

// out[e, g, 64 c + j] = in[e, 64 c + 8 (j % 8) + j / 8, g]
// 64 rows (one chunk) x 64 groups per CTA, transposed through shared memory.  kVector: the
// tensors are aligned for 4-byte loads (two groups) and 16-byte stores (the eight rows
// 8 b + a of one group are consecutive in the output); otherwise element by element.
template <bool kVector>
__global__ void __launch_bounds__(256)
permute_scale_kernel(const uint16_t* __restrict__ in, uint16_t* __restrict__ out, int n, int groups) {
  __shared__ __align__(4) uint16_t tile[64][64 + 2];
  const int c = blockIdx.x, g0 = blockIdx.y * 64, e = blockIdx.z;
  const int tid = threadIdx.x;
  const uint16_t* src = in + (static_cast<size_t>(e) * n + static_cast<size_t>(c) * 64) * groups;
  uint16_t* dst = out + (static_cast<size_t>(e) * groups + g0) * n + static_cast<size_t>(c) * 64;
  if constexpr (kVector) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = (tid >> 5) + 8 * i, g = 2 * (tid & 31);
      if (g0 + g < groups) {  // (groups is even: K is a multiple of 64)
        *reinterpret_cast<uint32_t*>(&tile[r][g]) =
            __ldg(reinterpret_cast<const uint32_t*>(src + static_cast<size_t>(r) * groups + g0 + g));
      }
    }
  } else {
    for (int i = tid; i < 64 * 64; i += blockDim.x) {
      const int r = i >> 6, g = i & 63;
      if (g0 + g < groups) tile[r][g] = src[static_cast<size_t>(r) * groups + g0 + g];
    }
  }
  __syncthreads();
  if constexpr (kVector) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int g = (tid >> 3) + 32 * i, a = tid & 7;
      if (g0 + g < groups) {
        uint32_t v[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          v[b] = static_cast<uint32_t>(tile[16 * b + a][g]) | static_cast<uint32_t>(tile[16 * b + 8 + a][g]) << 16;
        }
        *reinterpret_cast<uint4*>(dst + static_cast<size_t>(g) * n + 8 * a) = make_uint4(v[0], v[1], v[2], v[3]);
      }
    }
  } else {
    for (int i = tid; i < 64 * 64; i += blockDim.x) {
      const int g = i >> 6, j = i & 63;
      if (g0 + g < groups) dst[static_cast<size_t>(g) * n + j] = tile[8 * (j & 7) + (j >> 3)][g];
    }
  }
}

}  // namespace
}  // namespace chord

extern "C" {

int chord_b200_repack_w4a16(const int32_t* in, int32_t* out, int64_t num_experts, int64_t n,
                            int64_t k, int packed_input, int32_t* range_flag, void* stream) {
  CHORD_REQUIRE(in != nullptr && out != nullptr, "null tensor pointer");
  CHORD_REQUIRE(num_experts > 0 && n > 0 && k > 0, "weight dimensions must be non-zero");
  CHORD_REQUIRE(n % 128 == 0, "shape_n must be divisible by 128, got %lld", static_cast<long long>(n));
  CHORD_REQUIRE(k % 64 == 0, "shape_k must be divisible by 64, got %lld", static_cast<long long>(k));
  CHORD_REQUIRE(num_experts <= 65535 && n * 2 < (1ll << 31) && k < (1ll << 31), "weight too large");
  CHORD_REQUIRE((reinterpret_cast<uintptr_t>(in) & 15u) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0,
                "weight tensors must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const uint32_t* src = reinterpret_cast<const uint32_t*>(in);
  uint32_t* dst = reinterpret_cast<uint32_t*>(out);
  if (packed_input) {
    constexpr int kTileK = 512;
    const dim3 grid(static_cast<unsigned>(n / 64), static_cast<unsigned>((k + kTileK - 1) / kTileK),
                    static_cast<unsigned>(num_experts));
    chord::repack_kernel<kTileK, true><<<grid, 256, 0, s>>>(src, dst, static_cast<int>(n),
                                                           static_cast<int>(k), nullptr);
  } else {
    constexpr int kTileK = 256;
    const dim3 grid(static_cast<unsigned>(n / 64), static_cast<unsigned>((k + kTileK - 1) / kTileK),
                    static_cast<unsigned>(num_experts));
    chord::repack_kernel<kTileK, false><<<grid, 256, 0, s>>>(src, dst, static_cast<int>(n),
                                                            static_cast<int>(k), range_flag);
  }
  CHORD_CUDA(cudaGetLastError());
  return chord::kOk;
}

int chord_b200_permute_scale(const void* in, void* out, int64_t num_experts, int64_t n, int64_t k,
                             void* stream) {
  CHORD_REQUIRE(in != nullptr && out != nullptr, "null tensor pointer");
  CHORD_REQUIRE(num_experts > 0 && n > 0 && k > 0, "scale dimensions must be non-zero");
  CHORD_REQUIRE(n % 64 == 0 && k % 32 == 0, "need N %% 64 == 0 and K %% 32 == 0");
  CHORD_REQUIRE(num_experts <= 65535, "too many experts");
  const int groups = static_cast<int>(k / 32);
  const dim3 grid(static_cast<unsigned>(n / 64), static_cast<unsigned>((groups + 63) / 64),
                  static_cast<unsigned>(num_experts));
  const bool vector = k % 64 == 0 && (reinterpret_cast<uintptr_t>(in) & 3u) == 0 &&
                      (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  const auto kernel = vector ? chord::permute_scale_kernel<true> : chord::permute_scale_kernel<false>;
  kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint16_t*>(in), static_cast<uint16_t*>(out), static_cast<int>(n), groups);
  CHORD_CUDA(cudaGetLastError());
  return chord::kOk;
}

}  // extern "C"
