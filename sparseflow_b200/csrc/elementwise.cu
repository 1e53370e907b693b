// Standalone SiLU.mul: out = (g * 1/(1+exp(-g))) * u in fp32, stored in the 16-bit type.
// Same arithmetic as the reference's Triton kernel (sparseflow/kernels/fused_silu_mul.py:6-31);
// used on the dense branch of the shape gate and as the unfused A/B variant of the fused epilogue.
// HBM-bound: 3 x 2 bytes per element; 16-byte vector accesses.  Measured (B200): 4096 x 11008 55.6 -> 44.4 us (6.1 TB/s),
// 777 x 11008 14.4 -> 9.5 us, 24 x 14336 4.2 -> 2.0 us (before -> now; the small ones by the programmatic launch, launch.h).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"
#include "launch.h"
#include "sm100_ptx.cuh"

namespace sfb200 {
namespace {

template <bool BF16>
__device__ __forceinline__ float ld16(uint16_t b) {
  if (BF16) return __uint_as_float(static_cast<uint32_t>(b) << 16);
  return __half2float(__ushort_as_half(b));
}
template <bool BF16>
__device__ __forceinline__ uint16_t st16(float v) {
  if (BF16) return __bfloat16_as_ushort(__float2bfloat16_rn(v));
  return __half_as_ushort(__float2half_rn(v));
}
template <bool BF16>
__device__ __forceinline__ uint32_t silu_mul2(uint32_t g2, uint32_t u2) {
  uint32_t r = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float g = ld16<BF16>(static_cast<uint16_t>(g2 >> (16 * h)));
    const float u = ld16<BF16>(static_cast<uint16_t>(u2 >> (16 * h)));
    const float s = 1.0f / (1.0f + __expf(-g));
    r |= static_cast<uint32_t>(st16<BF16>((g * s) * u)) << (16 * h);
  }
  return r;
}

// vec path: cols % 8 == 0, all pitches % 8 == 0, 16-byte aligned bases.  One 16-byte piece per thread, numbered through the rows, so
// every thread of a block has work whatever the width.  The row is index / pieces per row, by multiplication (RowDivider):
// with a 64-bit division per piece the kernel ran at 4.8 TB/s, and with one block per 2048 columns of a row 64-wide pitched
// rows left 248 of 256 threads idle.  16384 x 64 / 262144 x 64 pitched: 2.8 / 21.9 us with the division, 17.4 / 77.7 us with blocks of
// columns, now 2.4 / 17.8 us; unpitched 262144 x 64 17.1 us.
struct RowDivider {
  uint64_t mul;
  int shift;
};
// For 1 <= d <= 2^28 and 0 <= i < 2^31: i / d == i * mul >> shift, with l = ceil(log2 d), shift = 31 + l and
// mul = floor(2^shift / d) + 1: 2^shift < mul * d <= 2^shift + 2^l, so the product is above i / d by less than
// i * 2^l / (d * 2^shift) < 1 / d.  mul <= 2^32: the product fits 64 bits.
RowDivider row_divider(uint32_t d) {
  int l = 0;
  while ((1ull << l) < d) ++l;
  return RowDivider{(1ull << (31 + l)) / d + 1, 31 + l};
}
template <bool BF16>
__global__ void __launch_bounds__(256) silu_mul_vec_kernel(const uint16_t* g, const uint16_t* u, uint16_t* o, uint32_t pieces,
                                                           uint32_t row_pieces, RowDivider div, int ldg, int ldu, int ldo) {
  dependency_wait();
  dependency_trigger();
  const uint32_t i = blockIdx.x * 256 + threadIdx.x;
  if (i >= pieces) return;
  const uint32_t r = static_cast<uint32_t>(i * div.mul >> div.shift), c = (i - r * row_pieces) * 8;
  const uint4 gv = *reinterpret_cast<const uint4*>(g + static_cast<size_t>(r) * ldg + c);
  const uint4 uv = *reinterpret_cast<const uint4*>(u + static_cast<size_t>(r) * ldu + c);
  uint4 ov;
  ov.x = silu_mul2<BF16>(gv.x, uv.x);
  ov.y = silu_mul2<BF16>(gv.y, uv.y);
  ov.z = silu_mul2<BF16>(gv.z, uv.z);
  ov.w = silu_mul2<BF16>(gv.w, uv.w);
  *reinterpret_cast<uint4*>(o + static_cast<size_t>(r) * ldo + c) = ov;
}

template <bool BF16>
__global__ void silu_mul_scalar_kernel(const uint16_t* g, const uint16_t* u, uint16_t* o, int rows,
                                       int cols, int ldg, int ldu, int ldo) {
  const size_t total = static_cast<size_t>(rows) * cols;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i / cols), c = static_cast<int>(i % cols);
    const float gv = ld16<BF16>(g[static_cast<size_t>(r) * ldg + c]);
    const float uv = ld16<BF16>(u[static_cast<size_t>(r) * ldu + c]);
    const float s = 1.0f / (1.0f + __expf(-gv));
    o[static_cast<size_t>(r) * ldo + c] = st16<BF16>((gv * s) * uv);
  }
}

}  // namespace

int launch_silu_mul(const void* gate, const void* up, void* out, int rows, int cols, int ld_g,
                    int ld_u, int ld_o, int fmt, cudaStream_t stream) {
  if (!gate || !up || !out || rows <= 0 || cols <= 0) return kErrInvalid;
  if (ld_g < cols || ld_u < cols || ld_o < cols) return kErrInvalid;
  if (fmt != kF16 && fmt != kBF16) return kErrInvalid;
  const uint16_t* g = static_cast<const uint16_t*>(gate);
  const uint16_t* u = static_cast<const uint16_t*>(up);
  uint16_t* o = static_cast<uint16_t*>(out);
  const bool vec = cols % 8 == 0 && ld_g % 8 == 0 && ld_u % 8 == 0 && ld_o % 8 == 0 &&
                   ((reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(up) |
                     reinterpret_cast<uintptr_t>(out)) % 16 == 0);
  if (vec) {
    const uint32_t row_pieces = static_cast<uint32_t>(cols) / 8;
    const RowDivider div = row_divider(row_pieces);
    const int most = static_cast<int>(((1ull << 31) - 1) / row_pieces);      // rows of a launch
    for (int r0 = 0, n; r0 < rows; r0 += n) {
      n = rows - r0 < most ? rows - r0 : most;
      const uint32_t pieces = static_cast<uint32_t>(n) * row_pieces;
      const int rc = launch_dependent(fmt == kBF16 ? silu_mul_vec_kernel<true> : silu_mul_vec_kernel<false>, (pieces + 255) / 256, 256, 0, 0,
                                      stream, g + static_cast<size_t>(r0) * ld_g, u + static_cast<size_t>(r0) * ld_u,
                                      o + static_cast<size_t>(r0) * ld_o, pieces, row_pieces, div, ld_g, ld_u, ld_o);
      if (rc != kOk) return rc;
    }
    return kOk;
  }
  const size_t work = static_cast<size_t>(rows) * cols;
  size_t blocks = (work + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (fmt == kBF16) silu_mul_scalar_kernel<true><<<blocks, 256, 0, stream>>>(g, u, o, rows, cols, ld_g, ld_u, ld_o);
  else silu_mul_scalar_kernel<false><<<blocks, 256, 0, stream>>>(g, u, o, rows, cols, ld_g, ld_u, ld_o);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrCuda;
}

}  // namespace sfb200
