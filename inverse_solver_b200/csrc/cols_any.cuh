// What the column passes of any length n = A R share (z_pass.cu, y_pass.cu):
// the split of a length, the tile layout, copies into shared memory and the
// tensor map of a [columns, n, batch] array.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include "cbs_kernels.cuh"
#include "fft_core.cuh"
#include "tma.cuh"

namespace odt {
namespace {

// columns per tile: 16; 32 for A <= 5, where step B would keep only 16 A of the
// threads busy (85 = 5 x 17 points behind an 88 x 88 plane, 8
// illuminations: 39.9 -> 33.3 us; 69 = 3 x 23, 125 x 108 plane: 53 -> 40 us)
__host__ __device__ constexpr int tile_w(int A) { return A <= 5 ? 32 : 16; }
constexpr int kThreads = 160;
constexpr int kMaxN = 256;      // rows of a TMA box
constexpr int kMaxR = 31;

// A of n = A R (0: none): 8 where it divides (kernels of their own, whose
// registers no other factor shares), else the largest A <= 10, else the
// smallest above
constexpr int z_split(int n) {
  if (n % 8 == 0 && n / 8 >= 8 && n / 8 <= kMaxR) return 8;
  for (int A = 10; A >= 2; --A)
    if (n % A == 0 && n / A >= A && n / A <= kMaxR) return A;
  for (int A = 11; A <= 16; ++A)
    if (n % A == 0 && n / A >= A && n / A <= kMaxR) return A;
  return 0;
}

template <int N>
struct ZSplit {   // z_split at compile time
  static constexpr int kA = z_split(N);
};

__host__ __device__ constexpr size_t a16(size_t b) { return (b + 15) & ~(size_t)15; }
__host__ __device__ constexpr size_t a1k(size_t b) { return (b + 1023) & ~(size_t)1023; }

// Shared memory: 2 mbarriers | twiddles | kq2 along z | kq2 x + y per column |
// two landing stages on 1024-byte boundaries (tiled copies need 128)
struct ZSmem {
  size_t tw, kz, gxy, s0, s1, total;
  __host__ __device__ ZSmem(int n, int w) {
    tw = 64;
    kz = tw + a16(sizeof(float2) * n);
    gxy = kz + a16(sizeof(float) * n);
    s0 = a1k(gxy + a16(sizeof(float) * w));
    s1 = s0 + sizeof(float2) * n * w;
    total = s1 + sizeof(float2) * n * w;
  }
};

// registers per thread: 5 CTAs of 160 threads allow 80
template <int R>
constexpr int min_ctas() {
  return R <= 20 ? 5 : R <= 25 ? 4 : 3;
}

#if defined(__CUDA_ARCH__)
__device__ __forceinline__ void tma_tile(void* dst, const CUtensorMap* map, int c0, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_addr(dst)),
      "l"(map), "r"(c0), "r"(0), "r"(c2), "r"(smem_addr(bar))
      : "memory");
}
__device__ __forceinline__ void copy8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
#endif

inline PFN_cuTensorMapEncodeTiled_v12000 encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    cudaDriverEntryPointQueryResult q;
    void* p = nullptr;
    const bool ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
                    q == cudaDriverEntryPointSuccess;
    return ok ? reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p) : nullptr;
  }();
  return fn;
}

// x [cols, n, nb] viewed as float32 pairs: dims (inner first) {2 cols, n, nb},
// box 2 W floats = W complex columns by all rows
inline bool make_map(float2* x, long long cols, int n, long long nb, int W, CUtensorMap* m) {
  auto enc = encoder();
  if (!enc) return false;
  const cuuint64_t plane = (cuuint64_t)cols;
  const cuuint64_t dims[3] = {2 * plane, (cuuint64_t)n, (cuuint64_t)nb};
  const cuuint64_t strides[2] = {plane * sizeof(float2), plane * sizeof(float2) * n};
  const cuuint32_t box[3] = {2 * (cuuint32_t)W, (cuuint32_t)n, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, x, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace
}  // namespace odt
