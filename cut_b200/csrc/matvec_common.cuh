// What the decode mat-vecs over GGUF blocks share (qgemv_row.cu: one or two virtual activation rows; qgemv_blocks.cu: up to 16).
#pragma once

#include "common.cuh"
#include "kernels.h"

namespace cutb {

// how the activations are read and staged: fp16; fp32 as two 16-bit levels; fp32 as one
constexpr int GV_A_HALF = 0, GV_A_F32_TWO = 1, GV_A_F32_ONE = 2;

struct GvParams {
  const uint8_t *W;
  uint64_t row_bytes;
  const void *A;
  uint32_t lda;
  float *C;
  uint32_t ldc;
  const float *D;
  uint32_t ldd;
  float *partial;  // [ksplit][M][N] when ksplit > 1
  uint32_t M, K, N;
  uint32_t gran_per_split;
  uint32_t ksplit;
  uint32_t stages;
  int fusion_type, fusion_op;
  int a_f32;
  int glu;              // rows in (gate, up) pairs: C[m, i] = unary(acc[2i]) * acc[2i + 1]
  const float *norm_w;  // fused RMSNorm of the activation rows (nullptr: none)
  float norm_eps;
  int *status;
  // Activations staged once for all CTAs by stage_acts_kernel (nullptr: every CTA stages its own; always so with one or two rows):
  // one blob per K split in the shared-memory layout [act | esc | sx], staged_bytes each.
  uint8_t *staged;
  uint32_t staged_bytes;
  // Row-sharded scatter epilogue (world > 1): instead of C, the output slice is stored into
  // every rank's full output at column n_off.  Peer-mapped pointers; plain stores, no
  // multicast, no fence here: the step's exchange kernel publishes them.
  uint32_t world, n_off, ldc_total;
  float *peer_C[CUTB_MAX_PEERS];
};

// Shared-memory loads by 32-bit shared address.  Plain loads through an
// address-space-qualified pointer rather than inline asm, so the compiler can
// schedule them freely between the (memory-clobbering) barrier waits.
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
  return *reinterpret_cast<const uint32_t *>(__cvta_shared_to_generic(addr));
}
__device__ __forceinline__ uint2 lds_u64(uint32_t addr) {
  return *reinterpret_cast<const uint2 *>(__cvta_shared_to_generic(addr));
}
__device__ __forceinline__ uint4 lds_u128(uint32_t addr) {
  return *reinterpret_cast<const uint4 *>(__cvta_shared_to_generic(addr));
}

// Low / high nibbles of four bytes -> four unsigned bytes 16 * q.  The Q4_0
// offset (q - 8) is applied after the MMA through the staged sum of the
// activations of the block: sum((q - 8) x) = sum(q x) - 8 sum(x).
__device__ __forceinline__ uint32_t nib_lo_s(uint32_t x) { return (x << 4) & 0xF0F0F0F0u; }
__device__ __forceinline__ uint32_t nib_hi_s(uint32_t x) { return x & 0xF0F0F0F0u; }

template <bool AF32> __device__ __forceinline__ float load_act(const void *A, uint64_t idx) {
  if constexpr (AF32) return __ldg(reinterpret_cast<const float *>(A) + idx);
  return __half2float(__ldg(reinterpret_cast<const __half *>(A) + idx));
}

// Balanced int8 digits of |v| <= 32639: v = 256 * hi + lo, both in [-128, 127].  Eight values
// packed four to a word: the low digit is the value's low byte as it stands (read as int8),
// the high digit is byte 1 of value + 128.
__device__ __forceinline__ void pack_digits(const int (&v)[8], uint32_t (&hi)[2], uint32_t (&lo)[2]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t a = (uint32_t)v[4 * h], b = (uint32_t)v[4 * h + 1], c = (uint32_t)v[4 * h + 2], d = (uint32_t)v[4 * h + 3];
    lo[h] = __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
    hi[h] = __byte_perm(__byte_perm(a + 128u, b + 128u, 0x0051), __byte_perm(c + 128u, d + 128u, 0x0051), 0x5410);
  }
}

constexpr float GV_QMAX = 32512.f;
constexpr float GV_MOST = 3e38f;  // of a scale's inverse: below 1e-34 the scale stays at what it can hold
// Steps of the second level (the residual of fp32 rows, at most half a step of the first) per step e of the first.  Two digits hold 32639, so the
// residual x - x^ e, up to e (1/2 + 32512 r) with r the error of e times its inverse (2^-23 where that is approximated) and of x times it
// (2^-24 where the product is rounded by itself), must not reach e * 32639 / GV_STEPS2.  With 2 * 32512 steps it did.
constexpr float GV_STEPS2 = 64000.f;
static_assert(GV_STEPS2 * (0.5f + 32512.f * (0x1p-23f + 0x1p-24f)) < 32639.f, "the second level wraps");

// One activation row at either precision, or two at one 16-bit level (qgemv_row.cu).
struct RowPlan {
  uint32_t grid_x, depth, groups;
  bool fixed;
  bool beside;  // the next launch's block is to fit beside this one's
  size_t smem;
};
// false: no shared-memory plan for this K split
bool row_matvec_plan(const cutb_qmatmul_desc &d, int amode, const DeviceInfo &di, uint32_t ksplit, uint32_t gran_per_split, RowPlan *pl);
int row_matvec_launch(const GvParams &p, int format, int amode, const RowPlan &pl, bool overlap, cudaStream_t stream);

// Three to eight fp16 rows (qgemv_few.cu).
bool few_matvec_plan(const cutb_qmatmul_desc &d, const DeviceInfo &di, uint32_t ksplit, uint32_t gran_per_split, RowPlan *pl);
int few_matvec_launch(const GvParams &p, int format, const RowPlan &pl, bool overlap, cudaStream_t stream);

}  // namespace cutb
