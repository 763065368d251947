// fp32 operands as sums of three bf16 values (8 + 8 + 8 significant bits): a product of two such sums, kept to the six partial
// products (i, j), i + j <= 2, above 2^-24, gives up no operand bit of an fp32 product and has its range.
#pragma once
#include "px_rowpipe.cuh"

namespace px {

// x = b0 + b1 + b2 with bf16 terms.
__device__ __forceinline__ void split3(float x, bf16 (&b)[3]) {
  b[0] = __float2bfloat16_rn(x);
  const float r = x - __bfloat162float(b[0]);
  b[1] = __float2bfloat16_rn(r);
  b[2] = __float2bfloat16_rn(r - __bfloat162float(b[1]));
}
// Two values at a time, one conversion instruction a plane for both: w[p] = plane p of (x, y).
__device__ __forceinline__ void split3x2(float x, float y, uint32_t (&w)[3]) {
  w[0] = pack_bf16x2(x, y);
  const float2 a = unpack_bf16x2(w[0]);
  x -= a.x, y -= a.y;
  w[1] = pack_bf16x2(x, y);
  const float2 b = unpack_bf16x2(w[1]);
  w[2] = pack_bf16x2(x - b.x, y - b.y);
}

template <typename T>
__device__ __forceinline__ float4 ld4(const T* p);
template <>
__device__ __forceinline__ float4 ld4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <>
__device__ __forceinline__ float4 ld4<bf16>(const bf16* p) { return load4(p); }
template <>
__device__ __forceinline__ float4 ld4<__half>(const __half* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack_f16x2(u.x), b = unpack_f16x2(u.y);
  return make_float4(a.x, a.y, b.x, b.y);
}

// fp32 weight rows -> three bf16 planes; source row r goes to row (r / blk) * stride + off + r % blk.
static __global__ void split_weight_kernel(const float* __restrict__ w, bf16* __restrict__ out, int rows, int k, int out_rows,
                                    int blk, int stride, int off) {
  const int r = blockIdx.x, dst = (r / blk) * stride + off + r % blk;
  for (int c = threadIdx.x; c < k; c += blockDim.x) {
    bf16 b[3];
    split3(w[(size_t)r * k + c], b);
#pragma unroll
    for (int p = 0; p < 3; ++p) out[((size_t)p * out_rows + dst) * k + c] = b[p];
  }
}

// planes [3][rows][k] bf16, box [3][box_rows][64]
static bool make_plane_map(CUtensorMap* map, const bf16* base, int64_t rows, int64_t k, uint32_t box_rows) {
  return make_map_3d(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, (uint64_t)k, (uint64_t)rows, 3, (uint64_t)k * 2,
                     (uint64_t)rows * k * 2, 64, box_rows, CU_TENSOR_MAP_SWIZZLE_128B, 3);
}

}  // namespace px
