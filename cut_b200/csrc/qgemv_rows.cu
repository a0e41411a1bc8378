// Matmul of a few activation rows (9 to 16, held as fp16) over native GGUF blocks: batched decode.
//
// C[m, n] = epilogue(sum_k A[m, k] * dequant(W)[n, k]).  The mat-vec of fewer rows (qgemv_blocks.cu) turns activations into
// int8 digits, two MMA columns per row; from nine rows up fp16 MMAs on the quants themselves cost less: a nibble becomes an fp16
// integer with one logic operation per two weights and one exact subtraction, the activations enter as they are, and a block's
// exact products (24-bit sums) are scaled in fp32.  From 17 rows up that scaling of every output costs more than scaling the weights,
// and qgemm_few.cu takes over.
//
//  * Work is dealt in units of 128 weight rows x 256 k, equal contiguous runs to one CTA per SM (stream-K).  A unit is one stage
//    of a ring: the raw block bytes (one 2-D TMA box) and the activations of these 256 k, already in MMA fragment order.
//  * 16 consumer warps: four groups of 32 rows x four groups of 64 k (two blocks).  A warp reads the bytes of its rows with
//    conflict-free 32-bit loads, widens them to A fragments of m16n8k16 MMAs in registers and meets every group of eight
//    activation rows with one 16-byte shared load per block; nothing goes through shared memory a second time.
//  * At the end of a tile's share the four k groups meet in shared memory.  A tile whose K one CTA covered is finished there;
//    otherwise the CTA stores its share, and the last of the tile's CTAs to arrive (a counter per tile) adds the shares in CTA
//    order -- a fixed summation order for a shape and a device -- and finishes the tile.
//  * A small kernel before it lays the activations out in fragment order (per 256 k: [block][8 rows][lane] 16 bytes; Q4_K: block
//    sums behind them) and clears the counters.  Weight stages are in flight while it runs (programmatic dependent launch).
//
// Bound by the latency of the chain shared load -> widen -> MMA -> scale at four warps per scheduler, and by about 5 us of start,
// staging and the meeting of the shares; 8192 x 8192 Q4_0, 12 rows: 22 us = 1.7 TB/s.
// Every wait is bounded; on expiry CUTB_ERR_TIMEOUT is recorded and the kernel runs to its end without waiting.
#include <cuda.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.h"
#include "tcgen05.cuh"

namespace cutb {
namespace {

constexpr int GR_NT = 2;  // groups of eight activation rows
constexpr uint32_t GR_ROWS = 128, GR_PITCH = 132, GR_WARPS = 16, GR_THREADS = (GR_WARPS + 1) * 32;
__host__ __device__ constexpr uint32_t gr_chunk(int fmt) { return fmt == CUTB_Q8_0 ? 272u : 144u; }  // bytes of 256 k of a row
__host__ __device__ constexpr bool gr_sums(int fmt) { return fmt == CUTB_Q4_K; }
__host__ __device__ constexpr uint32_t gr_act_bytes(int fmt, int nt) { return 4096u * nt + (gr_sums(fmt) ? 256u * nt : 0u); }
__host__ __device__ constexpr uint32_t gr_stage(int fmt, int nt) { return GR_ROWS * gr_chunk(fmt) + gr_act_bytes(fmt, nt); }
__host__ __device__ constexpr uint32_t gr_red(int nt) { return 8u * 1024u * nt + 8u * nt * GR_PITCH * 4u; }  // the k groups' sums, and a tile

struct GrParams {
  const void *A;
  uint32_t lda;
  float *C;
  uint32_t ldc;
  const float *D;
  uint32_t ldd;
  uint32_t M, K, N;
  uint32_t tiles, per, stages;
  int fusion_type, fusion_op;
  int quads;           // C (and D) rows allow 16-byte accesses
  int *status;
  uint8_t *acts;       // activations in fragment order, gr_act_bytes per 256 k
  uint32_t *arrived;   // a counter per tile
  float *shares;       // [2 * CTAs][8 nt][128]
};

// Element (0..31) of a block that half i (0..7) of lane t's fragment chunk holds: halves 0-3 feed the block's first MMA, 4-7 the
// second.  `even`: the block starts on a 4-byte boundary (Q4_0 and Q8_0 blocks alternate).
template <int FMT> __device__ __forceinline__ uint32_t gr_elem(bool even, uint32_t t, uint32_t i) {
  if constexpr (FMT == CUTB_Q8_0) {
    const uint32_t j = i & 3;
    if (!even) return (i < 4) ? 4 * t + j : 16 + 4 * t + j;
    if (i < 4) return 2 + 4 * t + j;
    if (t < 3) return 18 + 4 * t + j;
    return (j < 2) ? 30 + j : j - 2;  // {30, 31, 0, 1}
  } else {
    // nibbles: bytes 0 and 2 of a word make a pair, then bytes 1 and 3
    const uint32_t j = ((i & 1) << 1) | ((i >> 1) & 1), hi = i >> 2;
    if constexpr (FMT == CUTB_Q4_0) {
      uint32_t byte;
      if (!even) byte = 4 * t + j;
      else if (t < 3) byte = 2 + 4 * t + j;
      else byte = (j < 2) ? j : 12 + j;  // {0, 1, 14, 15}
      return byte + 16 * hi;
    } else {
      return 16 * hi + 4 * t + j;  // words t and t + 4 of the sub-block's 32 nibbles
    }
  }
}

template <int FMT, bool AF32, int NT> __global__ void __launch_bounds__(256) rows_stage_kernel(const GrParams p) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the activations may come from the kernel before; the scratch may be in use there
  const uint32_t id = blockIdx.x * 256 + threadIdx.x, lane = id & 31, g = lane >> 2, t = lane & 3;
  if (id < p.tiles) p.arrived[id] = 0;
  const uint32_t nt = (id >> 5) % NT, kb = (id >> 5) / NT;  // (a warp shares both)
  if (kb >= p.K / 32) return;
  const uint32_t m = nt * 8 + g;
  uint16_t v[8];
  float sum = 0.f;
  bool over = false;
#pragma unroll
  for (uint32_t i = 0; i < 8; ++i) {
    const uint32_t e = gr_elem<FMT>((kb & 1) == 0, t, i);
    __half x = __ushort_as_half(0);
    if (m < p.M) {
      const uint64_t at = (uint64_t)m * p.lda + kb * 32 + e;
      if constexpr (AF32) {
        const float f = __ldg(reinterpret_cast<const float *>(p.A) + at);
        over |= fabsf(f) > 65504.0f && fabsf(f) < __int_as_float(0x7f800000);
        x = __float2half_rn(f);
      } else {
        x = __ldg(reinterpret_cast<const __half *>(p.A) + at);
      }
    }
    v[i] = __half_as_ushort(x);
    if constexpr (gr_sums(FMT)) sum += __half2float(x);
  }
  uint8_t *unit = p.acts + (size_t)(kb / 8) * gr_act_bytes(FMT, NT);
  *reinterpret_cast<uint4 *>(unit + (((kb % 8) * NT + nt) * 32 + lane) * 16) =
      make_uint4(v[0] | (uint32_t)v[1] << 16, v[2] | (uint32_t)v[3] << 16, v[4] | (uint32_t)v[5] << 16, v[6] | (uint32_t)v[7] << 16);
  if constexpr (gr_sums(FMT)) {
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (t == 0) reinterpret_cast<float *>(unit + 4096 * NT)[((kb % 8) * NT + nt) * 8 + g] = sum;
  }
  if constexpr (AF32) {
    if (p.status && __any_sync(0xffffffffu, over) && lane == 0) atomicExch(p.status, (int)CUTB_ERR_RANGE);
  }
}

__device__ __forceinline__ uint32_t gr_lds(uint32_t a) { return *reinterpret_cast<const uint32_t *>(__cvta_shared_to_generic(a)); }
__device__ __forceinline__ uint4 gr_lds4(uint32_t a) { return *reinterpret_cast<const uint4 *>(__cvta_shared_to_generic(a)); }

__device__ __forceinline__ void gr_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// eight nibbles -> integers in fp16: 1024 + q from a low nibble, 64 + q from a high one, less the offset and OFF (both exact)
template <int OFF> __device__ __forceinline__ void gr_low(uint32_t x, uint32_t &p02, uint32_t &p13) {
  const __half2 k = __float2half2_rn(1024.f + OFF);
  p02 = h2_as_u32(__hsub2(u32_as_h2((x & 0x000F000Fu) | 0x64006400u), k));
  p13 = h2_as_u32(__hsub2(u32_as_h2(((x >> 8) & 0x000F000Fu) | 0x64006400u), k));
}
template <int OFF> __device__ __forceinline__ void gr_high(uint32_t x, uint32_t &p02, uint32_t &p13) {
  const __half2 k = __float2half2_rn(64.f + OFF);
  p02 = h2_as_u32(__hsub2(u32_as_h2((x & 0x00F000F0u) | 0x54005400u), k));
  p13 = h2_as_u32(__hsub2(u32_as_h2(((x >> 8) & 0x00F000F0u) | 0x54005400u), k));
}
__device__ __forceinline__ void gr_bytes(uint32_t x, uint32_t &p01, uint32_t &p23) {
  const uint32_t u = x ^ 0x80808080u;  // q + 128
  const __half2 k = __float2half2_rn(1152.f);
  p01 = h2_as_u32(__hsub2(u32_as_h2(__byte_perm(u, 0x64646464u, 0x4140)), k));
  p23 = h2_as_u32(__hsub2(u32_as_h2(__byte_perm(u, 0x64646464u, 0x4342)), k));
}

// One block (32 k) of a warp: its 32 rows (four per lane: f[row] = halves 0-1, 2-3 | 4-5, 6-7) and every group of eight
// activation rows.  sc / mn: the rows' scales and minima.
template <int FMT, int NT>
__device__ __forceinline__ void gr_block(float (&acc)[2][NT][4], const uint32_t (&f)[4][4], const float (&sc)[4], const float (&mn)[4], uint32_t act,
                                         uint32_t sums) {
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const uint4 b = gr_lds4(act + nt * 512);
    float2 sx = make_float2(0.f, 0.f);
    if constexpr (gr_sums(FMT)) sx = *reinterpret_cast<const float2 *>(__cvta_shared_to_generic(sums + nt * 32));
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      const uint32_t (&r0)[4] = f[2 * mt], (&r1)[4] = f[2 * mt + 1];
      float c[4] = {0.f, 0.f, 0.f, 0.f};
      gr_mma(c, r0[0], r1[0], r0[1], r1[1], b.x, b.y);
      gr_mma(c, r0[2], r1[2], r0[3], r1[3], b.z, b.w);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = 2 * mt + (e >> 1);
        acc[mt][nt][e] = fmaf(sc[r], c[e], acc[mt][nt][e]);
        if constexpr (gr_sums(FMT)) acc[mt][nt][e] = fmaf(-mn[r], (e & 1) ? sx.y : sx.x, acc[mt][nt][e]);
      }
    }
  }
}

template <int FMT, int NT>
__global__ void __launch_bounds__(GR_THREADS, 1) qgemv_rows_kernel(const __grid_constant__ CUtensorMap map_w, const GrParams p) {
  constexpr uint32_t CHUNK = gr_chunk(FMT), WB = GR_ROWS * CHUNK, AB = gr_act_bytes(FMT, NT), STAGE = WB + AB;
  extern __shared__ __align__(128) uint8_t gr_raw[];
  uint8_t *gr_smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gr_raw) + 127) & ~uintptr_t(127));  // (copied boxes)
  __shared__ uint32_t last_s;
  const uint32_t S = p.stages, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  float *red = reinterpret_cast<float *>(gr_smem + (size_t)S * STAGE);
  uint64_t *bars = reinterpret_cast<uint64_t *>(reinterpret_cast<uint8_t *>(red) + gr_red(NT));
  const uint32_t ring = smem_u32(gr_smem), full = smem_u32(bars), empty = full + S * 8;
  const uint32_t nk = p.K / 256, total = p.tiles * nk, u0 = blockIdx.x * p.per, n = min(p.per, total - u0);  // (the grid leaves no run empty)

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == 0) {
    for (uint32_t s = 0; s < S; ++s) mbar_init(full + s * 8, 1), mbar_init(empty + s * 8, GR_WARPS);
    fence_mbar_init();
  }
  __syncthreads();

  if (warp == GR_WARPS) {
    const bool leader = elect_one();
    auto weights = [&](uint32_t j, uint32_t slot) {
      const uint32_t u = u0 + j, bar = full + slot * 8;
      mbar_arrive_expect_tx(bar, STAGE);
      tma_load_2d(ring + slot * STAGE, &map_w, u % nk * (CHUNK / 4), u / nk * GR_ROWS, bar);
    };
    auto acts = [&](uint32_t j, uint32_t slot) {
      bulk_g2s(ring + slot * STAGE + WB, p.acts + (size_t)((u0 + j) % nk) * AB, AB, full + slot * 8);
    };
    const uint32_t first = min(S, n);
    if (leader)
      for (uint32_t j = 0; j < first; ++j) weights(j, j);  // constants: no wait for the kernel before
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (leader)
      for (uint32_t j = 0; j < first; ++j) acts(j, j);
    uint32_t slot = 0, ph = 0, issued = first;
    for (uint32_t j = S; j < n; ++j) {
      if (!__all_sync(0xffffffffu, mbar_wait_probe_first(empty + slot * 8, ph))) {
        if (leader && p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
        break;
      }
      if (leader) weights(j, slot), acts(j, slot);
      ++issued;
      if (++slot == S) slot = 0, ph ^= 1u;
    }
    // stay until every copy issued here has landed (bounded)
    for (uint32_t j = issued > S ? issued - S : 0; j < issued; ++j) (void)mbar_wait_bounded(full + (j % S) * 8, (j / S) & 1u);
    return;
  }

  const uint32_t rg = warp & 3, kg = warp >> 2;
  float acc[2][NT][4];
#pragma unroll
  for (int i = 0; i < 2 * NT * 4; ++i) (&acc[0][0][0])[i] = 0.f;
  uint32_t slot = 0, ph = 0, tile = u0 / nk, k = u0 % nk, k_begin = k, seg = 0;
  bool dead = false;
  // byte offset of row g of this warp's rows and of its 64 k in a stage
  const uint32_t row0 = (rg * 32 + g) * CHUNK + (FMT == CUTB_Q4_K ? 0u : kg * (FMT == CUTB_Q8_0 ? 68u : 36u));
  const uint32_t act0 = WB + kg * 2 * NT * 512 + lane * 16, sum0 = WB + 4096 * NT + kg * 2 * NT * 32 + t * 8;

  for (uint32_t j = 0; j < n; ++j) {
    if (!dead && !warp_wait(full + slot * 8, ph)) {
      dead = true;
      if (lane == 0 && p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
    }
    const uint32_t st = ring + slot * STAGE;
    if (!dead) {
      uint32_t f0[4][4], f1[4][4];  // the two blocks' fragments
      float s0[4], s1[4], m0[4], m1[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t pa = st + row0 + r * 8 * CHUNK;
        m0[r] = m1[r] = 0.f;
        if constexpr (FMT == CUTB_Q4_0) {
          // pairs of 18-byte blocks = 9 aligned words: {d0,u0} {u1,u2} {u3,u4} {u5,u6} {u7,d1} {v0,v1} ... {v6,v7}
          const uint32_t w0 = gr_lds(pa), w1 = gr_lds(pa + (t == 3 ? 0u : 4u + 4u * t)), w4 = gr_lds(pa + 16), w5 = gr_lds(pa + 20 + 4 * t);
          const uint32_t x = __byte_perm(w1, w4, t == 3 ? 0x5432u : 0x3210u);
          gr_low<8>(x, f0[r][0], f0[r][1]), gr_high<8>(x, f0[r][2], f0[r][3]);
          gr_low<8>(w5, f1[r][0], f1[r][1]), gr_high<8>(w5, f1[r][2], f1[r][3]);
          s0[r] = h2f_bits(w0 & 0xFFFFu), s1[r] = h2f_bits(w4 >> 16);
        } else if constexpr (FMT == CUTB_Q8_0) {
          // pairs of 34-byte blocks = 17 aligned words: {d0,u0} {u1,u2} ... {u13,u14} {u15,d1} then 8 words of block 1
          const uint32_t w0 = gr_lds(pa), w8 = gr_lds(pa + 32);
          gr_bytes(gr_lds(pa + 4 + 4 * t), f0[r][0], f0[r][1]);
          gr_bytes(__byte_perm(gr_lds(pa + 20 + 4 * t), w0, t == 3 ? 0x7610u : 0x3210u), f0[r][2], f0[r][3]);
          gr_bytes(gr_lds(pa + 36 + 4 * t), f1[r][0], f1[r][1]);
          gr_bytes(gr_lds(pa + 52 + 4 * t), f1[r][2], f1[r][3]);
          s0[r] = h2f_bits(w0 & 0xFFFFu), s1[r] = h2f_bits(w8 >> 16);
        } else {
          const uint4 h = gr_lds4(pa);
          const uint32_t x = gr_lds(pa + 16 + 32 * kg + 4 * t), y = gr_lds(pa + 32 + 32 * kg + 4 * t);
          const float d = h2f_bits(h.x & 0xFFFFu), dmin = h2f_bits(h.x >> 16);
          // 6-bit scales and minima of sub-blocks 2 kg and 2 kg + 1 (gguf_reader.cpp:668-676)
          const uint32_t sh = (kg & 1) * 16;
          uint32_t sc, mn;
          if (kg < 2) sc = (h.y >> sh) & 0x3F3Fu, mn = (h.z >> sh) & 0x3F3Fu;
          else sc = ((h.w >> sh) & 0x0F0Fu) | ((h.y >> (sh + 2)) & 0x3030u), mn = ((h.w >> (sh + 4)) & 0x0F0Fu) | ((h.z >> (sh + 2)) & 0x3030u);
          s0[r] = d * (float)(sc & 0xFFu), s1[r] = d * (float)(sc >> 8), m0[r] = dmin * (float)(mn & 0xFFu), m1[r] = dmin * (float)(mn >> 8);
          gr_low<0>(x, f0[r][0], f0[r][1]), gr_low<0>(y, f0[r][2], f0[r][3]);
          gr_high<0>(x, f1[r][0], f1[r][1]), gr_high<0>(y, f1[r][2], f1[r][3]);
        }
      }
      gr_block<FMT, NT>(acc, f0, s0, m0, st + act0, st + sum0);
      gr_block<FMT, NT>(acc, f1, s1, m1, st + act0 + NT * 512, st + sum0 + NT * 32);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + slot * 8);
    if (++slot == S) slot = 0, ph ^= 1u;
    if (++k < nk && j + 1 < n) continue;

    // ---- the tile, or this CTA's share of it, is complete: the k groups meet (fixed order) ----
    auto cell = [&](uint32_t upper) { return red + ((size_t)(upper * 4 + rg) * 8 * NT) * 32 + lane; };  // [2][4][8 NT][32]
    float *flat = &acc[0][0][0];
    if (kg >= 2) {
#pragma unroll
      for (int i = 0; i < 8 * NT; ++i) cell(kg - 2)[i * 32] = flat[i];
    }
    asm volatile("bar.sync 1, %0;" ::"n"(GR_WARPS * 32) : "memory");
    if (kg < 2) {
#pragma unroll
      for (int i = 0; i < 8 * NT; ++i) flat[i] += cell(kg)[i * 32];
      if (kg == 1) {
#pragma unroll
        for (int i = 0; i < 8 * NT; ++i) cell(1)[i * 32] = flat[i];
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(GR_WARPS * 32) : "memory");
    if (kg == 0) {
#pragma unroll
      for (int i = 0; i < 8 * NT; ++i) flat[i] += cell(1)[i * 32];
    }
    asm volatile("bar.sync 1, %0;" ::"n"(GR_WARPS * 32) : "memory");  // the buffer is free for the next tile
    if (kg == 0) {
      // The tile goes through shared memory, [activation row][128 weight rows], so that a thread stores four neighbouring
      // columns and the fused operation stands in the code once (unrolled over the accumulators it was several times the
      // instruction cache, and cost every launch with 32 rows 6 us).
      asm volatile("griddepcontrol.wait;" ::: "memory");
      const bool whole = k_begin == 0 && k == nk;
      float *cells = red + 8 * NT * 256;  // [8 NT][GR_PITCH]
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) cells[(nt * 8 + 2 * t + (e & 1)) * GR_PITCH + rg * 32 + mt * 16 + (e >> 1) * 8 + g] = acc[mt][nt][e];
      asm volatile("bar.sync 2, 128;" ::: "memory");
      bool finish = whole;
      if (!whole) {
        float *share = p.shares + (size_t)(2 * blockIdx.x + (seg ? 1u : 0u)) * 8 * NT * GR_ROWS + lane * 4;
#pragma unroll
        for (uint32_t i = 0; i < 2 * NT; ++i)
          *reinterpret_cast<float4 *>(share + (rg + 4 * i) * GR_ROWS) = *reinterpret_cast<const float4 *>(cells + (rg + 4 * i) * GR_PITCH + lane * 4);
        const uint32_t c_first = tile * nk / p.per, c_last = ((tile + 1) * nk - 1) / p.per;
        __threadfence();
        asm volatile("bar.sync 2, 128;" ::: "memory");
        if (tid == 0) last_s = atomicAdd(p.arrived + tile, 1u) == c_last - c_first;
        asm volatile("bar.sync 2, 128;" ::: "memory");
        finish = last_s != 0;
        if (finish) {  // every share of the tile is there: add them in CTA order
          __threadfence();
          // only the first of the tile's CTAs can have begun in an earlier tile
          const uint32_t tail = c_first * p.per / nk != tile ? 1u : 0u;
          float4 sum[2 * NT];
#pragma unroll
          for (uint32_t i = 0; i < 2 * NT; ++i) sum[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          for (uint32_t c = c_first; c <= c_last; ++c) {
            const float *src = p.shares + (size_t)(2 * c + (c == c_first ? tail : 0u)) * 8 * NT * GR_ROWS + rg * GR_ROWS + lane * 4;
            float4 v[2 * NT];  // a share's loads are all in flight
#pragma unroll
            for (uint32_t i = 0; i < 2 * NT; ++i) v[i] = __ldcg(reinterpret_cast<const float4 *>(src + i * 4 * GR_ROWS));
#pragma unroll
            for (uint32_t i = 0; i < 2 * NT; ++i) sum[i].x += v[i].x, sum[i].y += v[i].y, sum[i].z += v[i].z, sum[i].w += v[i].w;
          }
#pragma unroll
          for (uint32_t i = 0; i < 2 * NT; ++i) *reinterpret_cast<float4 *>(cells + (rg + 4 * i) * GR_PITCH + lane * 4) = sum[i];
        }
      }
      const uint32_t nn = tile * GR_ROWS + lane * 4;
      const bool quads = p.quads && nn + 4 <= p.N;
#pragma unroll 1
      for (uint32_t m = rg; finish && m < p.M; m += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(cells + m * GR_PITCH + lane * 4);
        float y[4] = {v.x, v.y, v.z, v.w}, dv[4] = {0.f, 0.f, 0.f, 0.f};
        float *dst = p.C + (size_t)m * p.ldc + nn;
        if (p.fusion_type != CUTB_FUSION_NONE) {
          const float *dsrc = p.D + (size_t)m * p.ldd + nn;
          if (p.fusion_type == CUTB_FUSION_BINARY) {
            if (quads) {
              const float4 f = *reinterpret_cast<const float4 *>(dsrc);
              dv[0] = f.x, dv[1] = f.y, dv[2] = f.z, dv[3] = f.w;
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (nn + e < p.N) dv[e] = dsrc[e];
            }
          }
          apply_epilogue_n<4>(y, dv, p.fusion_type, p.fusion_op);
        }
        if (quads) {
          *reinterpret_cast<float4 *>(dst) = make_float4(y[0], y[1], y[2], y[3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (nn + e < p.N) dst[e] = y[e];
        }
      }
      asm volatile("bar.sync 2, 128;" ::: "memory");  // last_s and the cells may be written again
    }
#pragma unroll
    for (int i = 0; i < 8 * NT; ++i) flat[i] = 0.f;
    if (k == nk) k = 0, ++tile;
    k_begin = k, ++seg;
  }
}

struct GrPlan {
  int nt;
  uint32_t tiles, per, grid, stages;
  uint64_t acts, arrived, shares;  // workspace bytes, each rounded up to 256
};

GrPlan gr_plan(const cutb_qmatmul_desc &d, uint32_t sms, size_t smem) {
  GrPlan pl{};
  pl.nt = GR_NT;
  pl.tiles = (d.N + GR_ROWS - 1) / GR_ROWS;
  const uint32_t total = pl.tiles * (d.K / 256);
  pl.grid = total < sms ? total : sms;
  pl.per = (total + pl.grid - 1) / pl.grid;
  pl.grid = (total + pl.per - 1) / pl.per;
  const size_t room = smem - gr_red(pl.nt) - 1024;
  pl.stages = (uint32_t)(room / (gr_stage(d.format, pl.nt) + 16));
  if (pl.stages > 8) pl.stages = 8;
  auto up = [](uint64_t b) { return (b + 255) / 256 * 256; };
  pl.acts = up((uint64_t)(d.K / 256) * gr_act_bytes(d.format, pl.nt));
  pl.arrived = up((uint64_t)pl.tiles * 4);
  pl.shares = (uint64_t)2 * pl.grid * 8 * pl.nt * GR_ROWS * 4;
  return pl;
}

// The weight as a 2-D tensor of 32-bit words, [N rows][row_bytes / 4]; a box is 256 k of 128 rows.
int gr_map(CUtensorMap *map, const cutb_qmatmul_desc &d) {
  EncodeTiledFn encode = nullptr;
  if (int rc = tc_encode_fn(&encode)) return rc;
  const uint64_t rb = row_bytes(d.format, d.K);
  const cuuint64_t dims[2] = {rb / 4, d.N}, strides[1] = {rb};
  const cuuint32_t box[2] = {gr_chunk(d.format) / 4, GR_ROWS}, estr[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void *>(d.W), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_error("qgemv: cuTensorMapEncodeTiled failed with %d for the weight (N=%u row bytes=%llu)", (int)r, d.N, (unsigned long long)rb);
    return CUTB_ERR_CUDA;
  }
  return CUTB_OK;
}

template <int FMT, int NT> int gr_launch(const cutb_qmatmul_desc &d, const GrParams &p, const GrPlan &pl, cudaStream_t stream) {
  static bool configured[64] = {};  // per device: the attribute is set once on each
  int dev = 0;
  CUTB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    DeviceInfo di;
    if (int rc = get_device_info(&di)) return rc;
    CUTB_CUDA_TRY(cudaFuncSetAttribute(qgemv_rows_kernel<FMT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)di.smem_optin - 512));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  CUtensorMap map;
  if (int rc = gr_map(&map, d)) return rc;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = d.flags & CUTB_FLAG_NO_OVERLAP ? 0 : 1;
  cfg.stream = stream;
  const uint32_t threads = d.K / 32 * NT * 32, least = pl.tiles;  // (a thread per tile clears its counter)
  cfg.gridDim = dim3(((threads > least ? threads : least) + 255) / 256);
  cfg.blockDim = dim3(256);
  if (d.a_dtype == CUTB_F32) CUTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, rows_stage_kernel<FMT, true, NT>, p));
  else CUTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, rows_stage_kernel<FMT, false, NT>, p));
  cfg.numAttrs = 1;  // its predecessor is this library's own kernel
  cfg.gridDim = dim3(pl.grid);
  cfg.blockDim = dim3(GR_THREADS);
  cfg.dynamicSmemBytes = (size_t)pl.stages * (gr_stage(FMT, NT) + 16) + gr_red(NT) + 128;
  CUTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, qgemv_rows_kernel<FMT, NT>, map, p));
  return CUTB_OK;
}

}  // namespace

bool qgemv_rows_supported(const cutb_qmatmul_desc &d) {
  if (d.layout != CUTB_LAYOUT_GGUF_BLOCKS || d.K == 0 || d.K % 256 != 0 || d.N == 0 || reinterpret_cast<uintptr_t>(d.W) % 16 != 0) return false;
  if (d.flags & (CUTB_FLAG_A_RMSNORM | CUTB_FLAG_GLU_PAIRS | CUTB_FLAG_STAGE_PER_CTA)) return false;
  return d.M >= 9 && d.M <= 32;
}

// Where this kernel is the faster one.  us per call in a chain, the kernel that runs otherwise (int8 mat-vec, or tcgen05 GEMM for few
// tokens) -> this one; tiles: 128 weight rows each, units: tiles x K / 256.
//   9 to 16 fp16 rows   From 20 tiles up always: 12 rows, 256 x 8192 10.5 -> 4.2, 2560 x 2560 Q4_0 x 0.79, 4096 x 4096 Q8_0 14.3 -> 10.3,
//                  8192 x 8192 Q4_0 26.3 -> 21.8.  Fewer tiles are shared by many CTAs, whose meeting costs more than it gives until the
//                  int8 kernel has to split K as well: 9 rows, 2048 x 2048 Q8_0 6.1 -> 7.7, 4608 x 2048 Q4_0 8.1 -> 10.3 and Q8_0 11.7 ->
//                  10.4, 8192 x 512 8.3 -> 12.2, so from 8 tiles of 192 (Q8_0: 3072 x 2048 x 0.75) or 384 units (Q4_0: 6144 x 2048 12.1 ->
//                  10.2; 16384 x 1024 alone loses 3 % up to 12 rows, and wins 25 % from 13); and where both are small, 1024 x 1000
//                  7.2 -> 6.2, 2048 x 768 8.1 -> 7.1.  Q4_K the same within 4 % either way (its minima cost a second product): stays.
//                  Eight rows, which fill the int8 kernel's columns: 12.8 -> 14.3: stays.
//   17 to 32 fp16 rows  The kernel is the tensor-core GEMM's for few rows (qgemm_few.cu) on either side; the line is where the variant that
//                  is reported for them changes.
//   fp32 rows      Rounded to fp16 by either kernel; here in the same pass that orders them.  All three formats gain on all of 35 weights
//                  from 512 x 512 to 28672 x 8192: x 0.44 to 0.94 (9 and 16 rows); 17 to 32 rows take qgemm_few.cu.
bool qgemv_rows_faster(const cutb_qmatmul_desc &d) {
  if (d.a_dtype == CUTB_F32) return true;
  if (d.format == CUTB_Q4_K) return false;
  const uint32_t tiles = (d.N + GR_ROWS - 1) / GR_ROWS;
  const uint64_t weights = (uint64_t)d.K * d.N, units = (uint64_t)tiles * (d.K / 256);
  const bool q8 = d.format == CUTB_Q8_0;
  if (d.M <= 16) return tiles >= 20 || (tiles >= 8 && units >= (q8 ? 192u : 384u)) || (tiles <= 8 && d.K <= 2048);
  if (q8) return weights >= (14ull << 20) || (weights >= (8ull << 20) && tiles >= 24);
  return weights >= (16ull << 20) && (tiles >= 48 || (tiles >= 32 && d.K <= 4096));
}

uint64_t qgemv_rows_workspace(const cutb_qmatmul_desc &d) {
  if (d.M > 8 * GR_NT) return qgemm_few_workspace(d, false);
  DeviceInfo di;
  uint32_t sms = 148;
  size_t smem = 232448;
  if (get_device_info(&di) == CUTB_OK) sms = (uint32_t)di.sm_count, smem = di.smem_optin;
  const GrPlan pl = gr_plan(d, sms, smem);
  return pl.acts + pl.arrived + pl.shares;
}

bool qgemv_rows_fits(const cutb_qmatmul_desc &d) {
  return d.workspace && reinterpret_cast<uintptr_t>(d.workspace) % 16 == 0 && d.workspace_bytes >= qgemv_rows_workspace(d);
}

int qgemv_rows_launch(const cutb_qmatmul_desc &d, cudaStream_t stream) {
  if (d.M > 8 * GR_NT) return qgemm_few_launch(d, stream);
  DeviceInfo di;
  if (int rc = get_device_info(&di)) return rc;
  const GrPlan pl = gr_plan(d, (uint32_t)di.sm_count, di.smem_optin);
  GrParams p{};
  p.A = d.A, p.lda = d.lda, p.C = d.C, p.ldc = d.ldc, p.D = d.D, p.ldd = d.ldd, p.M = d.M, p.K = d.K, p.N = d.N;
  p.tiles = pl.tiles, p.per = pl.per, p.stages = pl.stages, p.fusion_type = d.fusion_type, p.fusion_op = d.fusion_op, p.status = d.status;
  p.quads = reinterpret_cast<uintptr_t>(d.C) % 16 == 0 && d.ldc % 4 == 0 &&
            (d.fusion_type != CUTB_FUSION_BINARY || (reinterpret_cast<uintptr_t>(d.D) % 16 == 0 && d.ldd % 4 == 0));
  p.acts = reinterpret_cast<uint8_t *>(d.workspace);
  p.arrived = reinterpret_cast<uint32_t *>(p.acts + pl.acts);
  p.shares = reinterpret_cast<float *>(p.acts + pl.acts + pl.arrived);
  switch (d.format) {
    case CUTB_Q8_0: return gr_launch<CUTB_Q8_0, GR_NT>(d, p, pl, stream);
    case CUTB_Q4_0: return gr_launch<CUTB_Q4_0, GR_NT>(d, p, pl, stream);
    default: return gr_launch<CUTB_Q4_K, GR_NT>(d, p, pl, stream);
  }
}

}  // namespace cutb
