// fp32 numbers as sums of three bf16 numbers: what the kernels that multiply them on the tensor cores share.  Everything is
// in an unnamed namespace: each translation unit gets its own copy.
#pragma once
#include "wcn_common.cuh"

namespace {

// The six products that are kept (first part of the one factor, of the other; 0 = h, 1 = m, 2 = l), small ones first: the
// tensor core's accumulator drops what is below its last place.
__host__ __device__ constexpr int split_a(int q) { return (0x001102 >> (4 * q)) & 15; }
__host__ __device__ constexpr int split_b(int q) { return (0x010120 >> (4 * q)) & 15; }

// bf16 ends at 2^-133, the last bit of a small fp32 number lies at 2^-149.  So every number is multiplied by 2^24 before it is
// split, which brings all of them, the subnormal ones too, and the products of their parts into range; sums of products are
// taken back by 2^-48.  Both are exact.  (Split as they were, numbers lost bits from 2^-110 downwards: 6e-5 at 2^-120.)
constexpr float kSplitScale = 16777216.f, kSumScale = 1.f / (16777216.f * 16777216.f);

// x = h + m + l exactly (round to nearest twice; the rest has eight bits).
__device__ __forceinline__ void split3(float x, __nv_bfloat16& h, __nv_bfloat16& m, __nv_bfloat16& l) {
  h = __float2bfloat16_rn(x);
  const float r = __fsub_rn(x, __bfloat162float(h));
  m = __float2bfloat16_rn(r);
  l = __float2bfloat16_rn(__fsub_rn(r, __bfloat162float(m)));
}
// Infinities, NaN, and (scaled) numbers whose parts could have an infinite product where the numbers have none: their first
// part is NaN, which makes NaN of every sum that they are in, and such a sum is made again from the numbers themselves.
__device__ __forceinline__ bool unsplittable(float x) { return !(fabsf(x) < 9.223372e18f); }

// The parts of eight numbers times kSplitScale, 16 bytes each, `apart` bytes from one another.
__device__ __forceinline__ void store_parts(const float (&v)[8], char* dst, int64_t apart) {
  __align__(16) __nv_bfloat16 part[3][8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const float x = v[u] * kSplitScale;
    split3(x, part[0][u], part[1][u], part[2][u]);
    if (unsplittable(x)) part[0][u] = __ushort_as_bfloat16(0x7FC0);
  }
#pragma unroll
  for (int s = 0; s < 3; ++s) *reinterpret_cast<uint4*>(dst + s * apart) = *reinterpret_cast<const uint4*>(part[s]);
}
// Eight consecutive numbers of a row, zeros from `limit` on (a multiple of four; rows start on 16-byte boundaries).
__device__ __forceinline__ void load_eight(const float* row, int c, int limit, float (&v)[8]) {
  const float4 a = c < limit ? __ldg(reinterpret_cast<const float4*>(row + c)) : make_float4(0, 0, 0, 0);
  const float4 b = c + 4 < limit ? __ldg(reinterpret_cast<const float4*>(row + c + 4)) : make_float4(0, 0, 0, 0);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

}  // namespace
