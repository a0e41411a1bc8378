// Decode mat-vec for three to eight fp16 activation rows over native Q4_0 and Q4_K blocks, as fp16 MMAs.
//
// C[m, n] = epilogue(sum_k A[m, k] * dequant(W)[n, k]), the reference's M = 1 variant (operators/impl/matmul/MatMulQ4GemvKPar8.cu:8-98)
// for a few rows at a time.
//
// Bound by latency (issue slots 37 % busy, shared memory 90 of the 100 cycles that HBM needs for 16 rows of 256 weights): the chain load ->
// MMA -> scale at four warps per scheduler, and, where a launch is short, the same hand-over and staging as in qgemv_row.cu.  What keeps them low:
//  * Quants enter m16n8k16 without a conversion: the bits of a nibble in the low mantissa bits of a half are the subnormal q * 2^-24,
//    exact, and one logic operation makes two of them (high nibbles: 16 q, in MMAs of their own).  Q4_0's offset times a block's sum of
//    activations is the accumulator's start, Q4_K's minima take the same sums; the sums are MMAs with a constant.  The activations
//    enter as they are.  The block scale is applied in fp32; all is in units of 2^-24 until the end.
//  * So there is nothing to quantise: a warp loads the granules (256 k) that fall to it, puts them into fragment order in shared memory,
//    and no launch goes before this one (the int8 digits of qgemv_blocks.cu take a launch of their own from three rows up).
//  * Weights come as in qgemv_row.cu: stages of 16 rows by eight granules by one tensor copy each.  The block keeps under half an SM where
//    that leaves four stages (up to four rows of 4096), else it takes a deep ring and the registers it likes (8 rows of 4096, Q4_0
//    11008 x 4096: 11.7 us a launch with eight stages alone on the SM, 12.1 with 56 registers, 15.1 with two stages beside the next block).
//  * Two groups of eight warps take a tile each, a granule per warp and stage; stages of both tiles come in turn.  A group meets in
//    barriers of its own, once to add up a tile and once before it writes the next tile's sums.
// us a launch, int8 digits -> here (graphs of 2 to 32): Q4_0 11008 x 4096 3 rows 14.6 -> 10.0, 8 rows 12.9 -> 11.7; 4096 x 4096 3 rows 8.6 ->
// 5.7, 8 rows 8.2 -> 7.2; 14336 x 2048 13.8 -> 8.9 and 12.5 -> 9.7; Q4_K 28672 x 1024 19.5 -> 12.2 and 23.7 -> 12.5.  Relative error against
// 64 bits 7e-7 (Q4_0) and 8e-6 (Q4_K) where the digits have 2.2e-5.  Q8_0 gained nothing (8 rows of 4096 x 4096 7.9 -> 9.4).
//
// Every wait on an mbarrier is bounded; on expiry the kernel stores CUTB_ERR_TIMEOUT in the caller's status word and leaves.
#include "matvec_common.cuh"
#include "tcgen05.cuh"

namespace cutb {

namespace {

constexpr uint32_t FW_ROWS = 16, FW_WARPS = 16, FW_CONSUMERS = FW_WARPS * 32, FW_THREADS = FW_CONSUMERS + 32;  // (one more warp issues the copies)
constexpr uint32_t FW_MAX_DEPTH = 8;
constexpr float FW_UNIT = 16777216.f;  // 2^24

constexpr uint32_t FW_GRANULES = 8, FW_GROUPS = FW_WARPS / FW_GRANULES;  // of a stage, one per warp of the group that takes it: 18 KB

struct FewParams : GvParams {
  uint32_t depth;  // stages of the ring
};

// D = A * B + C
__device__ __forceinline__ void mma_half(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, float c0, float c1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%10,%11};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1));
}
__device__ __forceinline__ void mma_half_add(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A stage that has not landed yet; true (and an error status) if it does not.  After the first time nobody waits long again.
__device__ __noinline__ bool few_wait_long(uint32_t bar, uint32_t phase, bool dead, int *status) {
  const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar, phase, dead ? 1u : 1u << 16));
  if (!ok && (threadIdx.x & 31) == 0 && status) atomicExch(status, (int)CUTB_ERR_TIMEOUT);
  return !ok;
}

// Loads of what the predecessor may have written: coherent ones that stay behind griddepcontrol.wait.
__device__ __forceinline__ uint4 load_halves(const __half *at) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(at) : "memory");
  return v;
}
// A granule (256 halves) of up to four rows that do not all start on sixteen bytes, into shared memory: [row][512 bytes], word by word as they
// lie.  Rows that start on a word are copied asynchronously (complete behind cp.async.wait_all); of one that starts between two words the
// last word is made of its last and first half.
__device__ __noinline__ void copy_rows(uint8_t *to, const __half *A, uint32_t lda, uint32_t rows, uint32_t lane) {
  uint32_t w[4][4];  // (all loads are in flight)
  auto between = [&](uint32_t m) { return (reinterpret_cast<uintptr_t>(A + (size_t)m * lda) & 2) != 0; };
#pragma unroll
  for (uint32_t m = 0; m < 4; ++m) {
    if (m >= rows) continue;
    const __half *row = A + (size_t)m * lda;
    if (!between(m)) {
      const uint32_t dst = smem_u32(to) + m * 512 + lane * 4;
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 128 * i), "l"(row + 2 * lane + 64 * i) : "memory");
      continue;
    }
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
      const uint32_t at = 1 + 2 * lane + 64 * i;
      if (at < 255) {
        asm volatile("ld.global.u32 %0, [%1];" : "=r"(w[m][i]) : "l"(row + at) : "memory");
      } else {
        uint16_t last, first;
        asm volatile("ld.global.u16 %0, [%1];" : "=h"(last) : "l"(row + 255) : "memory");
        asm volatile("ld.global.u16 %0, [%1];" : "=h"(first) : "l"(row) : "memory");
        w[m][i] = last | (uint32_t)first << 16;
      }
    }
  }
#pragma unroll
  for (uint32_t m = 0; m < 4; ++m) {
    if (m >= rows || !between(m)) continue;
    uint16_t *row = reinterpret_cast<uint16_t *>(to + m * 512);
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
      const uint32_t at = 1 + 2 * lane + 64 * i;
      row[at] = (uint16_t)w[m][i];
      row[(at + 1) & 255] = (uint16_t)(w[m][i] >> 16);
    }
  }
}

// Fragments: sixteen bytes per block, column (activation row, padded to CP) and lane t of a quad, the operands of the block's two MMAs
// (Q4_0: the low nibbles' and the high nibbles'; Q4_K: the lane's first and last four bytes).
template <int FMT, int CP, bool ALIGNED>
__device__ __forceinline__ void stage_granule(const FewParams &p, uint8_t *frag, float *off, uint32_t gs0, uint32_t gran, uint32_t lane) {
  const uint32_t kb = lane >> 2, q = lane & 3;
  const __half *A = reinterpret_cast<const __half *>(p.A) + (size_t)(gs0 + gran) * 256 + lane * 8;
  uint4 x[CP];
  if constexpr (ALIGNED) {
#pragma unroll
    for (int m = 0; m < CP; ++m)
      x[m] = (uint32_t)m < p.M ? load_halves(A + (size_t)m * p.lda) : make_uint4(0, 0, 0, 0);
  } else {
#pragma unroll
    for (int m = 0; m < CP; ++m)
      x[m] = (uint32_t)m < p.M ? *reinterpret_cast<const uint4 *>(frag + (size_t)gran * CP * 512 + m * 512 + lane * 16) : make_uint4(0, 0, 0, 0);
    __syncwarp();
  }
  uint8_t *to = frag + (size_t)(gran * 8 + kb) * CP * 64;
  const bool even = (kb & 1) == 0;
#pragma unroll
  for (int m = 0; m < CP; ++m) {
    uint32_t w0a = x[m].x, w0b = x[m].y, w1a = x[m].z, w1b = x[m].w;  // two words of four elements, as pairs
    if constexpr (FMT == CUTB_Q4_0) {
      // an aligned block's words start two elements late: the last pair is joined by a neighbour's first
      const uint32_t near = __shfl_xor_sync(0xffffffffu, w0a, 1);
      if (even) {
        const bool wraps = q & 1;  // elements {0, 1, 14, 15}
        const uint32_t last = w1b;
        w0a = w0b, w0b = w1a;
        w1a = wraps ? near : last, w1b = wraps ? last : near;
      }
    }
    const uint2 w0 = make_uint2(__byte_perm(w0a, w0b, 0x5410), __byte_perm(w0a, w0b, 0x7632));
    const uint2 w1 = make_uint2(__byte_perm(w1a, w1b, 0x5410), __byte_perm(w1a, w1b, 0x7632));
    uint8_t *at = to + m * 64;
    if constexpr (FMT == CUTB_Q4_K) {  // both MMAs of lane t = q
      *reinterpret_cast<uint4 *>(at + q * 16) = make_uint4(w0.x, w0.y, w1.x, w1.y);
    } else {  // words 2 (q % 2) and 2 (q % 2) + 1 of the first (q < 2) or the second MMA
      at += (q & 1) * 32 + (q >> 1) * 8;
      *reinterpret_cast<uint2 *>(at) = w0;
      *reinterpret_cast<uint2 *>(at + 16) = w1;
    }
  }
  __syncwarp();
  // the blocks' sums of activations, times the offset of their quants: products with a constant
  constexpr uint32_t K2 = FMT == CUTB_Q4_0 ? 0x80088008u : 0x00010001u;  // -8 or 1, times 2^-24
  const uint32_t g = lane >> 2, t = lane & 3, col = g % CP;
#pragma unroll
  for (uint32_t b = 0; b < 8; ++b) {
    const uint4 f = *reinterpret_cast<const uint4 *>(frag + (size_t)(gran * 8 + b) * CP * 64 + (col * 4 + t) * 16);
    float d[4];
    mma_half(d, K2, K2, K2, K2, f.x, f.y, 0.f, 0.f);
    mma_half_add(d, K2, K2, K2, K2, f.z, f.w);
    if (g == 0 && 2 * t < CP) *reinterpret_cast<float2 *>(off + (gran * 8 + b) * CP + 2 * t) = make_float2(d[0], d[1]);
  }
}

// One unit: 16 rows of 256 weights at shared address `unit` times the granule's fragments (x: this lane's sixteen bytes of its first
// block; o: the pair of sums of this lane's columns).  tot: rows g and g + 8 by columns 2t and 2t + 1, in units of 2^-24.
template <int FMT, int CP>
__device__ __forceinline__ void unit_few(uint32_t unit, uint32_t x, uint32_t o, uint32_t g, uint32_t t, float (&tot)[4]) {
  constexpr uint32_t GB = granule_bytes(FMT), XB = CP * 64, OB = CP * 4;
  const uint32_t ra = unit + g * GB, rb = ra + 8 * GB;
  auto sums_of = [&](uint32_t b) {
    const uint2 s = lds_u64(o + b * OB);
    return make_float2(__uint_as_float(s.x), __uint_as_float(s.y));
  };
  if constexpr (FMT == CUTB_Q4_0) {
    const uint32_t o1 = t == 3 ? 0u : 4u + 4u * t, selx = t == 3 ? 0x5432u : 0x3210u;
#pragma unroll
    for (uint32_t pr = 0; pr < 4; ++pr) {  // two blocks of 18 bytes in nine words
      const uint32_t pa = ra + pr * 36, pb = rb + pr * 36;
      const uint32_t a4 = lds_u32(pa + 16), b4 = lds_u32(pb + 16);
      const uint32_t wa[2] = {__byte_perm(lds_u32(pa + o1), a4, selx), lds_u32(pa + 20 + 4 * t)};
      const uint32_t wb[2] = {__byte_perm(lds_u32(pb + o1), b4, selx), lds_u32(pb + 20 + 4 * t)};
      const float da[2] = {h2f_bits(lds_u32(pa) & 0xFFFFu), h2f_bits(a4 >> 16)}, db[2] = {h2f_bits(lds_u32(pb) & 0xFFFFu), h2f_bits(b4 >> 16)};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint4 f = lds_u128(x + (2 * pr + i) * XB);
        const float2 s = sums_of(2 * pr + i);
        const uint32_t a8 = wa[i] >> 8, b8 = wb[i] >> 8;
        float lo[4], hi[4];
        mma_half(lo, wa[i] & 0x000F000Fu, wb[i] & 0x000F000Fu, a8 & 0x000F000Fu, b8 & 0x000F000Fu, f.x, f.y, s.x, s.y);
        mma_half(hi, wa[i] & 0x00F000F0u, wb[i] & 0x00F000F0u, a8 & 0x00F000F0u, b8 & 0x00F000F0u, f.z, f.w, 0.f, 0.f);
#pragma unroll
        for (int c = 0; c < 4; ++c) tot[c] = fmaf(c < 2 ? da[i] : db[i], fmaf(hi[c], 0.0625f, lo[c]), tot[c]);
      }
    }
  } else {
    const uint4 hA = lds_u128(ra), hB = lds_u128(rb);
    const float dA = h2f_bits(hA.x & 0xFFFFu), mA = h2f_bits(hA.x >> 16), dB = h2f_bits(hB.x & 0xFFFFu), mB = h2f_bits(hB.x >> 16);
    // 6-bit (scale, min) pairs, four sub-blocks per 32-bit word (gguf_reader.cpp:668-676)
    const uint32_t scA[2] = {hA.y & 0x3F3F3F3Fu, (hA.w & 0x0F0F0F0Fu) | ((hA.y >> 2) & 0x30303030u)};
    const uint32_t mnA[2] = {hA.z & 0x3F3F3F3Fu, ((hA.w >> 4) & 0x0F0F0F0Fu) | ((hA.z >> 2) & 0x30303030u)};
    const uint32_t scB[2] = {hB.y & 0x3F3F3F3Fu, (hB.w & 0x0F0F0F0Fu) | ((hB.y >> 2) & 0x30303030u)};
    const uint32_t mnB[2] = {hB.z & 0x3F3F3F3Fu, ((hB.w >> 4) & 0x0F0F0F0Fu) | ((hB.z >> 2) & 0x30303030u)};
    const float ndA = -dA * 8388608.f, nmA = -mA * 8388608.f, ndB = -dB * 8388608.f, nmB = -mB * 8388608.f;
#pragma unroll
    for (int gq = 0; gq < 4; ++gq) {
      const uint2 qa = lds_u64(ra + 16 + 32 * gq + 8 * t), qb = lds_u64(rb + 16 + 32 * gq + 8 * t);
#pragma unroll
      for (int hi = 0; hi < 2; ++hi) {
        const int j = 2 * gq + hi;  // sub-block 0..7; the odd ones are the high nibbles, which enter as 16 q
        const uint32_t sel = 0x7540u | (uint32_t)(j & 3), mask = hi ? 0x00F000F0u : 0x000F000Fu;
        const uint4 f = lds_u128(x + j * XB);
        const float2 s = sums_of(j);
        float c[4];
        mma_half(c, qa.x & mask, qb.x & mask, (qa.x >> 8) & mask, (qb.x >> 8) & mask, f.x, f.y, 0.f, 0.f);
        mma_half_add(c, qa.y & mask, qb.y & mask, (qa.y >> 8) & mask, (qb.y >> 8) & mask, f.z, f.w);
        // d * (2^23 + sc) - d * 2^23 == d * sc exactly
        const float one = hi ? 0.0625f : 1.f;
        const float dsA = one * fmaf(dA, __uint_as_float(__byte_perm(scA[j >> 2], 0x4B000000u, sel)), ndA);
        const float dmA = fmaf(mA, __uint_as_float(__byte_perm(mnA[j >> 2], 0x4B000000u, sel)), nmA);
        const float dsB = one * fmaf(dB, __uint_as_float(__byte_perm(scB[j >> 2], 0x4B000000u, sel)), ndB);
        const float dmB = fmaf(mB, __uint_as_float(__byte_perm(mnB[j >> 2], 0x4B000000u, sel)), nmB);
        tot[0] = fmaf(-dmA, s.x, fmaf(dsA, c[0], tot[0]));
        tot[1] = fmaf(-dmA, s.y, fmaf(dsA, c[1], tot[1]));
        tot[2] = fmaf(-dmB, s.x, fmaf(dsB, c[2], tot[2]));
        tot[3] = fmaf(-dmB, s.y, fmaf(dsB, c[3], tot[3]));
      }
    }
  }
}

// ALIGNED: all rows start on sixteen bytes.  MINB: blocks per SM that the registers are kept for.
template <int FMT, int CP, bool ALIGNED, int MINB>
__global__ void __launch_bounds__(FW_THREADS, MINB) qgemv_few_kernel(const __grid_constant__ CUtensorMap weights, const FewParams p) {
  constexpr uint32_t GB = granule_bytes(FMT), UNIT = FW_ROWS * GB, GPS = FW_GRANULES, STAGE = GPS * UNIT, GROUPS = FW_GROUPS;
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;

  // tiles of 16 rows of this block, granules [gs0, gs0 + ng) of this K split; a stage is GPS granules of a tile
  const uint32_t tiles = (p.N + FW_ROWS - 1) / FW_ROWS;
  const uint32_t t0 = (uint32_t)((uint64_t)blockIdx.x * tiles / gridDim.x), t1 = (uint32_t)((uint64_t)(blockIdx.x + 1) * tiles / gridDim.x);
  const uint32_t r0 = t0 * FW_ROWS, r1 = min(p.N, t1 * FW_ROWS), ntiles = t1 - t0;
  const uint32_t G = p.K >> 8, gs0 = blockIdx.y * p.gran_per_split, ng = min(G, gs0 + p.gran_per_split) - gs0;
  const uint32_t cpt = (ng + GPS - 1) / GPS, nstages = ntiles * cpt, D = p.depth;

  uint8_t *frag = smem + (size_t)D * STAGE;
  float *off = reinterpret_cast<float *>(frag + (size_t)p.gran_per_split * CP * 512);
  float *sums = off + (size_t)p.gran_per_split * CP * 8;  // [group][warp of it][column][row]
  uint64_t *bars = reinterpret_cast<uint64_t *>(sums + FW_WARPS * CP * FW_ROWS);
  // (a "full" barrier per slot and group, so that a group sees every phase of the barriers that it waits for)
  const uint32_t ring_u = smem_u32(smem), full_u = smem_u32(bars), empty_u = full_u + D * GROUPS * 8;

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == FW_WARPS) {
    // ---- copy warp: a stage is one box of the weights seen as [granule][row][bytes] ----
    if (lane == 0) {
      for (uint32_t s = 0; s < D; ++s) {
        mbar_init(empty_u + s * 8, GPS);
        for (uint32_t q = 0; q < GROUPS; ++q) mbar_init(full_u + (s * GROUPS + q) * 8, 1);
      }
      fence_mbar_init();
    }
    __syncwarp();
    // (tiles of all groups side by side, stage by stage)
    uint32_t slot = 0, par = 1, c = 0, set = 0, q = 0, issued = 0, seen[GROUPS] = {};
    auto fill = [&](uint32_t end) {
      for (; issued < end; ++issued) {
        if (issued >= D && !warp_wait(empty_u + slot * 8, par)) {
          if (lane == 0 && p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
          break;
        }
        if (lane == 0) {
          const uint32_t full = full_u + (slot * GROUPS + q) * 8;
          mbar_arrive_expect_tx(full, STAGE);
          tma_load_3d(ring_u + slot * STAGE, &weights, 0, r0 + (set + q) * FW_ROWS, gs0 + c * GPS, full);
        }
        __syncwarp();
#pragma unroll
        for (uint32_t i = 0; i < GROUPS; ++i)
          if (q == i) seen[i] ^= 1u << slot;  // copies into the slot for that group, modulo 2
        if (++slot == D) slot = 0, par ^= 1u;
        if (++q == min(GROUPS, ntiles - set)) {
          q = 0;
          if (++c == cpt) c = 0, set += GROUPS;
        }
      }
    };
    fill(min(D, nstages));
    __syncthreads();
    fill(nstages);
    // stay until every copy has landed (bounded): the last one of each slot and group
#pragma unroll
    for (uint32_t i = 0; i < GROUPS; ++i)
      for (uint32_t s = 0; s < D; ++s) mbar_drain(full_u + (s * GROUPS + i) * 8, ((seen[i] >> s) & 1u) ^ 1u);
    return;
  }
  __syncthreads();

  // What came before read only the (constant) weights; activations, D and C may be the predecessor's.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // Rows that start anywhere go to where the fragments will be first: one after the other, element by element, they took 0.3 us each.  us a
  // launch, rows K + 2 and (odd) K + 9 apart: Q4_0 4096 x 2048 with 8 rows 6.8 -> 5.6, Q4_K 14336 x 1792 with 5 rows 11.8 -> 10.1, Q4_0
  // 2368 x 4096 with 8 odd rows 8.7 -> 7.7 (the digits of qgemv_blocks.cu, at 16 bits: 6.2).
  if constexpr (!ALIGNED) {
    for (uint32_t gran = warp; gran < ng; gran += FW_WARPS)
      for (uint32_t h = 0; h < p.M; h += 4)
        copy_rows(frag + (size_t)gran * CP * 512 + h * 512, reinterpret_cast<const __half *>(p.A) + (size_t)(gs0 + gran) * 256 + (size_t)h * p.lda, p.lda, p.M - h, lane);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
  }
  for (uint32_t gran = warp; gran < ng; gran += FW_WARPS) stage_granule<FMT, CP, ALIGNED>(p, frag, off, gs0, gran, lane);
  asm volatile("bar.sync 1, %0;" ::"n"(FW_CONSUMERS) : "memory");

  const uint32_t group = warp / GPS, wg = warp % GPS, gtid = tid - group * GPS * 32;
  const uint32_t x_u = smem_u32(frag) + ((g % CP) * 4 + t) * 16, o_u = smem_u32(off) + (2 * t % CP) * 4;
  float *mine = sums + (size_t)warp * CP * FW_ROWS, *ours = sums + (size_t)group * GPS * CP * FW_ROWS;
  auto meet = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(2 + group), "n"(GPS * 32) : "memory"); };
  uint32_t seen = 0;  // seen: bit s: parity of the group's next visit to slot s
  bool dead = false;
  for (uint32_t tile = group; tile < ntiles; tile += GROUPS) {
    float tot[4] = {};
    const uint32_t set = tile - group, beside = min(GROUPS, ntiles - set);
    uint32_t slot = (set * cpt + group) % D;
    for (uint32_t c = 0; c < cpt; ++c) {
      const uint32_t full = full_u + (slot * GROUPS + group) * 8, phase = (seen >> slot) & 1u;
      if (!__all_sync(0xffffffffu, mbar_test(full, phase))) dead |= few_wait_long(full, phase, dead, p.status);
      const uint32_t gran = c * GPS + wg;
      if (gran < ng) unit_few<FMT, CP>(ring_u + slot * STAGE + wg * UNIT, x_u + gran * CP * 512, o_u + gran * CP * 32, g, t, tot);
      __syncwarp();
      if (lane == 0) mbar_arrive(empty_u + slot * 8);
      seen ^= 1u << slot;
      slot += beside;
      while (slot >= D) slot -= D;
    }
    // the sums of the group's warps meet; rows are turned by half a tile in every other lane pair's columns
    if (tile != group) meet();
    const uint32_t turn = (t & 1) * 8;
    if (2 * t < CP) {
      mine[(2 * t) * FW_ROWS + (g ^ turn)] = tot[0];
      mine[(2 * t + 1) * FW_ROWS + (g ^ turn)] = tot[1];
      mine[(2 * t) * FW_ROWS + ((g + 8) ^ turn)] = tot[2];
      mine[(2 * t + 1) * FW_ROWS + ((g + 8) ^ turn)] = tot[3];
    }
    meet();
    for (uint32_t o = gtid; o < FW_ROWS * p.M; o += GPS * 32) {
      const uint32_t row = o % FW_ROWS, m = o / FW_ROWS, n = r0 + tile * FW_ROWS + row;
      const float *at = ours + m * FW_ROWS + (row ^ ((m >> 1 & 1) * 8));
      float sum = 0.f;
#pragma unroll
      for (uint32_t w = 0; w < GPS; ++w) sum += at[w * CP * FW_ROWS];
      sum *= FW_UNIT;
      if (p.glu) {  // (gate, up) row pairs are neighbouring lanes: one output per pair
        // (an odd number of rows leaves half of the last warp)
        const float up = __shfl_down_sync((o & ~31u) + 32 <= FW_ROWS * p.M ? 0xffffffffu : 0x0000ffffu, sum, 1);
        if (!(row & 1) && n < r1) p.C[(size_t)m * p.ldc + (n >> 1)] = apply_epilogue(sum, CUTB_FUSION_UNARY, p.fusion_op, 0.f) * up;
        continue;
      }
      if (n >= r1) continue;
      if (p.ksplit > 1) {
        p.partial[((size_t)blockIdx.y * p.M + m) * p.N + n] = sum;
        continue;
      }
      const float dv = p.fusion_type == CUTB_FUSION_BINARY ? p.D[(size_t)m * p.ldd + n] : 0.f;
      const float out = apply_epilogue(sum, p.fusion_type, p.fusion_op, dv);
      if (p.world > 1) {
        const size_t to = (size_t)m * p.ldc_total + p.n_off + n;
        for (uint32_t q = 0; q < p.world; ++q) p.peer_C[q][to] = out;
      } else {
        p.C[(size_t)m * p.ldc + n] = out;
      }
    }
  }
}

template <int FMT, int CP, bool ALIGNED, int MINB>
int few_launch_inst(const CUtensorMap &map, const FewParams &p, const RowPlan &pl, bool overlap, cudaStream_t stream) {
  static bool configured[64] = {};  // per device: the attribute is set once on each
  int dev = 0;
  CUTB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    DeviceInfo di;
    if (int rc = get_device_info(&di)) return rc;
    CUTB_CUDA_TRY(cudaFuncSetAttribute(qgemv_few_kernel<FMT, CP, ALIGNED, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)di.smem_optin));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pl.grid_x, p.ksplit);
  cfg.blockDim = dim3(FW_THREADS);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  CUTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, qgemv_few_kernel<FMT, CP, ALIGNED, MINB>, map, p));
  return CUTB_OK;
}

template <int FMT, bool ALIGNED> int few_launch_rows(const CUtensorMap &map, const FewParams &p, const RowPlan &pl, bool overlap, cudaStream_t stream) {
  if (pl.beside) return p.M <= 4 ? few_launch_inst<FMT, 4, ALIGNED, 2>(map, p, pl, overlap, stream) : few_launch_inst<FMT, 8, ALIGNED, 2>(map, p, pl, overlap, stream);
  return p.M <= 4 ? few_launch_inst<FMT, 4, ALIGNED, 1>(map, p, pl, overlap, stream) : few_launch_inst<FMT, 8, ALIGNED, 1>(map, p, pl, overlap, stream);
}
template <int FMT> int few_launch_fmt(const CUtensorMap &map, const FewParams &p, const RowPlan &pl, bool overlap, cudaStream_t stream) {
  const bool aligned = reinterpret_cast<uintptr_t>(p.A) % 16 == 0 && p.lda % 8 == 0;
  return aligned ? few_launch_rows<FMT, true>(map, p, pl, overlap, stream) : few_launch_rows<FMT, false>(map, p, pl, overlap, stream);
}

}  // namespace

// Where it is the faster kernel, by 96 shapes of the two formats with 3, 4, 6 and 8 rows: up to 4096 weights of a row per block it takes 0.5
// to 0.96 of the digits' time (Q4_0 K = 512 to 4096), but for four rows, which are just one column tile there, of 3328 weights and more:
// these gain with two to five tiles to a block (N = 5000 8.3 -> 7.5 us) and lose with one (N = 2048 5.5 -> 6.2) or many (Q4_K N = 28672
// 23.2 -> 24.7).  Longer rows keep the digits (K = 8192, N = 5000: 13.7 / 14.4 for six rows) unless there are five rows and more and four
// tiles to a block (N = 28672 43.2 -> 40.7, K = 5120 33.6 -> 28.5).
bool few_matvec_plan(const cutb_qmatmul_desc &d, const DeviceInfo &di, uint32_t ksplit, uint32_t gran_per_split, RowPlan *pl) {
  if (d.a_dtype != CUTB_F16 || d.format == CUTB_Q8_0 || d.M < 3 || d.M > 8 || (d.flags & CUTB_FLAG_A_RMSNORM)) return false;
  const uint64_t all_tiles = (uint64_t)((d.N + FW_ROWS - 1) / FW_ROWS) * ksplit, sm = (uint64_t)di.sm_count;
  if (gran_per_split > 16 && (d.M < 5 || all_tiles < 4 * sm)) return false;
  if (d.M == 4 && gran_per_split > 12 && (all_tiles <= sm || all_tiles > 5 * sm)) return false;
  const uint32_t cp = d.M <= 4 ? 4 : 8;
  const uint32_t sms = (uint32_t)di.sm_count > ksplit ? (uint32_t)di.sm_count / ksplit : 1;
  const uint32_t tiles = (d.N + FW_ROWS - 1) / FW_ROWS;
  pl->grid_x = tiles < sms ? tiles : sms;
  pl->groups = 1;
  pl->fixed = false;
  const size_t stage = (size_t)FW_GRANULES * FW_ROWS * granule_bytes(d.format);
  const size_t fixed = (size_t)gran_per_split * cp * (512 + 32) + (size_t)FW_WARPS * cp * FW_ROWS * 4 + FW_MAX_DEPTH * (FW_GROUPS + 1) * 8;
  const size_t half = di.smem_per_sm > 2048 ? di.smem_per_sm / 2 - 1024 : di.smem_optin / 2;
  // Beside the next launch's block (56 registers, some spilled) where that leaves four stages, but for Q4_K's wide columns: us a launch, beside /
  // alone, Q4_K 8000 x 1024 with 8 rows 5.6 / 5.3, Q4_0 8000 x 1024 with 8 rows 4.9 / 5.1, 4096 x 2048 with 3 rows 3.8 / 4.1.
  pl->beside = (cp == 4 || d.format == CUTB_Q4_0) && fixed + 4 * stage <= half;
  const size_t room = pl->beside ? half : di.smem_optin;
  if (fixed + 2 * stage > room) return false;
  const size_t fit = (room - fixed) / stage;
  pl->depth = fit > FW_MAX_DEPTH ? FW_MAX_DEPTH : (uint32_t)fit;
  const uint32_t used = (tiles + pl->grid_x - 1) / pl->grid_x * ((gran_per_split + FW_GRANULES - 1) / FW_GRANULES);  // stages of a block
  if (!pl->beside && pl->depth > used) pl->depth = used > 2 ? used : 2;
  pl->smem = fixed + pl->depth * stage;
  return true;
}

int few_matvec_launch(const GvParams &gp, int format, const RowPlan &pl, bool overlap, cudaStream_t stream) {
  FewParams p;
  static_cast<GvParams &>(p) = gp;
  p.depth = pl.depth;
  CUtensorMap map;
  if (int rc = make_tmap_granules(&map, p.W, format, p.N, p.K, p.row_bytes, FW_ROWS, FW_GRANULES)) return rc;
  return format == CUTB_Q4_0 ? few_launch_fmt<CUTB_Q4_0>(map, p, pl, overlap, stream) : few_launch_fmt<CUTB_Q4_K>(map, p, pl, overlap, stream);
}

}  // namespace cutb
