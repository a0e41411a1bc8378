// Weights widened straight into tensor memory (qgemm_few.cu, qgemm_wide.cu): 64 k of a raw weight row in shared memory to 32 registers of fp16
// pairs, and the copies that bring the raw rows.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace cutb {
namespace {

constexpr uint32_t FT_ROWS = 128;  // weight rows of a tile
__host__ __device__ constexpr uint32_t ft_unit(int fmt) { return FT_ROWS * granule_bytes(fmt); }  // bytes of 256 k of them

// eight nibbles -> integers in fp16: 1024 + q from a low nibble, 64 + q from a high one, less the offset and OFF (both exact)
template <int OFF> __device__ __forceinline__ void ft_low(uint32_t x, uint32_t &p02, uint32_t &p13) {
  const __half2 k = __float2half2_rn(1024.f + OFF);
  p02 = h2_as_u32(__hsub2(u32_as_h2((x & 0x000F000Fu) | 0x64006400u), k));
  p13 = h2_as_u32(__hsub2(u32_as_h2(((x >> 8) & 0x000F000Fu) | 0x64006400u), k));
}
template <int OFF> __device__ __forceinline__ void ft_high(uint32_t x, uint32_t &p02, uint32_t &p13) {
  const __half2 k = __float2half2_rn(64.f + OFF);
  p02 = h2_as_u32(__hsub2(u32_as_h2((x & 0x00F000F0u) | 0x54005400u), k));
  p13 = h2_as_u32(__hsub2(u32_as_h2(((x >> 8) & 0x00F000F0u) | 0x54005400u), k));
}
__device__ __forceinline__ void ft_bytes(uint32_t x, uint32_t &p01, uint32_t &p23) {
  const uint32_t u = x ^ 0x80808080u;  // q + 128
  const __half2 k = __float2half2_rn(1152.f);
  p01 = h2_as_u32(__hsub2(u32_as_h2(__byte_perm(u, 0x64646464u, 0x4140)), k));
  p23 = h2_as_u32(__hsub2(u32_as_h2(__byte_perm(u, 0x64646464u, 0x4342)), k));
}

__device__ __forceinline__ uint4 ft_lds(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
// Chunk C (64 k) of the 256 k of a weight row at shared address `row`, rounded to fp16, in pairs.
template <int FMT, int C> __device__ __forceinline__ void ft_chunk(uint32_t row, uint32_t (&h)[32]) {
  constexpr int LINES = FMT == CUTB_Q8_0 ? 5 : 3;
  uint32_t w[LINES * 4];
#pragma unroll
  for (int i = 0; i < LINES; ++i) {
    const uint32_t at = FMT == CUTB_Q4_K ? (i ? 32u * C + 16u * i : 0u) : (((FMT == CUTB_Q8_0 ? 68u : 36u) * C) & ~15u) + 16u * i;
    const uint4 v = ft_lds(row + at);
    w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
  }
  if constexpr (FMT == CUTB_Q4_0) {  // two 18-byte blocks in nine words: {d0,u0} {u1,u2} {u3,u4} {u5,u6} {u7,d1} {v0,v1} ...
    const uint32_t *x = w + C;
    const __half2 d[2] = {u32_as_h2(__byte_perm(x[0], 0, 0x1010)), u32_as_h2(__byte_perm(x[4], 0, 0x3232))};
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t q = b ? __byte_perm(x[5 + i], 0, 0x3120) : __byte_perm(x[i], x[i + 1], 0x5342);  // bytes 0, 2, 1, 3 of the four
        uint32_t *lo = h + 16 * b + 2 * i, *hi = lo + 8;
        ft_low<8>(q, lo[0], lo[1]), ft_high<8>(q, hi[0], hi[1]);
#pragma unroll
        for (int e = 0; e < 2; ++e) lo[e] = h2_as_u32(__hmul2(u32_as_h2(lo[e]), d[b])), hi[e] = h2_as_u32(__hmul2(u32_as_h2(hi[e]), d[b]));
      }
  } else if constexpr (FMT == CUTB_Q8_0) {  // two 34-byte blocks in 17 words: {d0,u0} {u1,u2} ... {u13,u14} {u15,d1} then eight words
    const uint32_t *x = w + C;
    const __half2 d[2] = {u32_as_h2(__byte_perm(x[0], 0, 0x1010)), u32_as_h2(__byte_perm(x[8], 0, 0x3232))};
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      ft_bytes(i < 8 ? __funnelshift_r(x[i], x[i + 1], 16) : x[i + 1], h[2 * i], h[2 * i + 1]);
#pragma unroll
      for (int e = 0; e < 2; ++e) h[2 * i + e] = h2_as_u32(__hmul2(u32_as_h2(h[2 * i + e]), d[i >> 3]));
    }
  } else {
    const float d = h2f_bits(w[0] & 0xFFFFu), dmin = h2f_bits(w[0] >> 16);
    // 6-bit scales and minima of sub-blocks 2 C and 2 C + 1 (gguf_reader.cpp:668-676)
    constexpr uint32_t sh = (C & 1) * 16;
    uint32_t sc, mn;
    if (C < 2) sc = (w[1] >> sh) & 0x3F3Fu, mn = (w[2] >> sh) & 0x3F3Fu;
    else sc = ((w[3] >> sh) & 0x0F0Fu) | ((w[1] >> (sh + 2)) & 0x3030u), mn = ((w[3] >> (sh + 4)) & 0x0F0Fu) | ((w[2] >> (sh + 2)) & 0x3030u);
    const __half2 a0 = __float2half2_rn(d * (float)(sc & 0xFFu)), a1 = __float2half2_rn(d * (float)(sc >> 8));
    const __half2 b0 = __float2half2_rn(-(dmin * (float)(mn & 0xFFu))), b1 = __float2half2_rn(-(dmin * (float)(mn >> 8)));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t q = __byte_perm(w[4 + i], 0, 0x3120);
      uint32_t *lo = h + 2 * i, *hi = lo + 16;
      ft_low<0>(q, lo[0], lo[1]), ft_high<0>(q, hi[0], hi[1]);
#pragma unroll
      for (int e = 0; e < 2; ++e) lo[e] = h2_as_u32(__hfma2(u32_as_h2(lo[e]), a0, b0)), hi[e] = h2_as_u32(__hfma2(u32_as_h2(hi[e]), a1, b1));
    }
  }
}

// The weight as a 2-D tensor of 32-bit words, [N rows][row_bytes / 4]; a box is 256 k of 128 rows.
int ft_map(CUtensorMap *map, const cutb_qmatmul_desc &d) {
  EncodeTiledFn encode = nullptr;
  if (int rc = tc_encode_fn(&encode)) return rc;
  const uint64_t rb = row_bytes(d.format, d.K);
  const cuuint64_t dims[2] = {rb / 4, d.N}, strides[1] = {rb};
  const cuuint32_t box[2] = {granule_bytes(d.format) / 4, FT_ROWS}, estr[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void *>(d.W), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_error("qgemm: cuTensorMapEncodeTiled failed with %d for the weight (N=%u row bytes=%llu)", (int)r, d.N, (unsigned long long)rb);
    return CUTB_ERR_CUDA;
  }
  return CUTB_OK;
}

}  // namespace
}  // namespace cutb
