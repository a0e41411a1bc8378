// Tensor-core GEMM over native GGUF blocks for up to 64 activation rows: batched decode, short prompts.
//
// C[m, n] = epilogue(sum_k A[m, k] * dequant(W)[n, k]); fp16 operands, the dequantised weight rounded to fp16 as the reference's
// tensor-core variants round it (MatMulQ4CoopMatTiled.cu:84-87 / MatMulQ8CoopMatTiled.cu:71-74), fp32 accumulation.
//
//  * Weights are the MMA's A operand and go to it by tensor memory: a thread takes a weight row, widens 64 k of it in registers and
//    stores them to its lane (tcgen05.st), so that they pass through shared memory once, as raw blocks.  128 weight rows x 32 or 64
//    activation rows (shared memory, 128-byte swizzle) per instruction.
//  * Work is dealt in units of 128 weight rows x 256 k, equal contiguous runs to one CTA per SM.  Raw blocks come as one 2-D tensor box
//    a unit, activations as four, in rings of their own.
//  * 16 converter warps: four groups, the g-th 64 k of every unit each.  They ask for the next unit's blocks and for room in tensor memory
//    before they widen, so that the answers are there afterwards.  Two issuers, since an issuer's waits and eight MMAs take some 800
//    cycles a unit: each takes half a unit's k into accumulators of its own, which the epilogue adds.
//  * A tile whose K one CTA covered is finished there.  Shares of a tile go to the scratch; the kernel behind this one adds them in CTA
//    order (a fixed summation order for a shape and a device).  Activations that a tensor copy cannot read (fp32, odd strides) are laid
//    out by a kernel before it, which then also clears a counter per tile: the last of a tile's CTAs adds the shares, and the kernel
//    behind is not needed.
//
// Bound by the chain of the conversion (about 1000 cycles a unit, whose bytes HBM needs 770 for; issue slots are half busy), and by some 7 us of two dependent
// launches and the chain copy -> widen -> MMA -> share -> sum.  us a call in a chain, what ran before (MMAs of registers up
// to 32 rows, else qgemm_skinny.cu) -> here: Q4_0 4096 x 4096 32 rows 13.7 -> 8.5, 64 rows 17.7 -> 10.6; 8192 x 28672 32 rows 62.7 -> 48.7;
// Q8_0 8192 x 11008 64 rows 58.4 -> 27.0; Q4_K 4096 x 28672 64 rows 48.4 -> 34.0; Q4_0 4096 x 4096 with 50 fp32 rows 21.3 -> 11.9.  Over
// 36 weights from 512 x 500 to 14336 x 28672, each format, 17 to 64 rows: 1.4 to 1.8 times as fast on average, nowhere slower.  One issuer
// took 23.9 us where two take 21.4 (Q4_0 8192 x 8192, 32 rows), joining the shares in a launch behind instead of staging activations and
// counters before it 19.8, early questions to the barriers 18.3; two converter groups and two CTAs per SM 31.4.
//
// Every wait is bounded; on expiry CUTB_ERR_TIMEOUT is recorded, copies and MMAs under way are waited for (with a limit), tensor memory is
// given back and the kernel returns.
#include <cuda.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.h"
#include "tmem_weights.cuh"

namespace cutb {
namespace {

constexpr uint32_t FT_GROUPS = 4, FT_WARPS = 4 * FT_GROUPS, FT_THREADS = (FT_WARPS + 3) * 32;  // (copies, two issuers)
// Half units of widened weights in tensor memory per issuer, 64 columns each; beside them two accumulators per issuer.
__host__ __device__ constexpr uint32_t ft_slots(uint32_t T) { return T == 32 ? 3 : 2; }
__host__ __device__ constexpr uint32_t ft_act(uint32_t T) { return T * 512; }  // bytes of 256 k of the activation rows
__host__ __device__ constexpr uint32_t ft_act_stages(uint32_t T) { return T == 32 ? 4 : 3; }
__host__ __device__ constexpr uint32_t ft_stages(int fmt, uint32_t T) { return fmt == CUTB_Q8_0 ? (T == 32 ? 4 : 3) : 6; }
__host__ __device__ constexpr uint32_t ft_smem(int fmt, uint32_t T) {
  return 1024 + ft_stages(fmt, T) * (ft_unit(fmt) + 16) + ft_act_stages(T) * (ft_act(T) + 16) + ft_slots(T) * 32 + 40;
}

struct FtParams {
  const void *A;
  uint32_t lda;
  float *C;
  uint32_t ldc;
  const float *D;
  uint32_t ldd;
  uint32_t M, K, N;
  uint32_t tiles, per;  // tiles of 128 weight rows; units per CTA
  int fusion_type, fusion_op, glu;
  int *status;
  uint8_t *acts;      // fp16 rows of K (nullptr: the kernel reads A)
  uint32_t *arrived;  // a counter per tile (nullptr: the shares are joined by ft_join_kernel)
  float *shares;      // [2 * CTAs][share_rows][128]
  uint32_t share_rows;  // M rounded up to 8
};

// The shares of a tile, in CTA order: activation rows tok0 .. of its weight row `row`.
template <uint32_t TOK>
__device__ __forceinline__ void ft_add_shares(const FtParams &p, uint32_t tile, uint32_t nk, uint32_t c_first, uint32_t c_last, uint32_t tok0, uint32_t row,
                                              float (&sum)[TOK]) {
  // only the first of the tile's CTAs can have begun in an earlier tile
  const uint32_t tail = c_first * p.per / nk != tile ? 1u : 0u;
#pragma unroll
  for (uint32_t i = 0; i < TOK; ++i) sum[i] = 0.f;
#pragma unroll 1
  for (uint32_t c = c_first; c <= c_last; ++c) {
    const float *at = p.shares + (size_t)(2 * c + (c == c_first ? tail : 0u)) * p.share_rows * FT_ROWS + tok0 * FT_ROWS + row;
    float f[TOK];  // a share's loads are all in flight
#pragma unroll
    for (uint32_t i = 0; i < TOK; ++i) f[i] = tok0 + i / 8 * 8 < p.share_rows ? __ldcg(at + i * FT_ROWS) : 0.f;
#pragma unroll
    for (uint32_t i = 0; i < TOK; ++i) sum[i] += f[i];
  }
}
template <uint32_t TOK> __device__ __forceinline__ void ft_store(const FtParams &p, uint32_t tile, uint32_t tok0, uint32_t row, float (&v)[TOK]) {
  const uint32_t n = tile * FT_ROWS + row;
  float dv[TOK];
  if (p.glu) {  // gate and up rows are neighbouring lanes: the even one stores the pair's output
    float up[TOK];
#pragma unroll
    for (uint32_t i = 0; i < TOK; ++i) up[i] = __shfl_xor_sync(0xffffffffu, v[i], 1), dv[i] = 0.f;
    apply_epilogue_n<TOK>(v, dv, CUTB_FUSION_UNARY, p.fusion_op);
#pragma unroll
    for (uint32_t i = 0; i < TOK; ++i)
      if (n < p.N && !(row & 1) && tok0 + i < p.M) p.C[(size_t)(tok0 + i) * p.ldc + (n >> 1)] = v[i] * up[i];
    return;
  }
  if (n >= p.N) return;
#pragma unroll
  for (uint32_t i = 0; i < TOK; ++i) dv[i] = p.fusion_type == CUTB_FUSION_BINARY && tok0 + i < p.M ? p.D[(size_t)(tok0 + i) * p.ldd + n] : 0.f;
  if (p.fusion_type != CUTB_FUSION_NONE) apply_epilogue_n<TOK>(v, dv, p.fusion_type, p.fusion_op);
#pragma unroll
  for (uint32_t i = 0; i < TOK; ++i)
    if (tok0 + i < p.M) p.C[(size_t)(tok0 + i) * p.ldc + n] = v[i];
}

// The activations as fp16 rows of K, where the kernel below cannot read them as they are; clears the tiles' counters.
template <bool AF32> __global__ void __launch_bounds__(256) ft_stage_kernel(const FtParams p, int quads) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the activations may come from the kernel before; the scratch may be in use there
  const uint32_t id = blockIdx.x * 256 + threadIdx.x, m = id / (p.K / 8), k = id % (p.K / 8) * 8;
  if (id < p.tiles) p.arrived[id] = 0;
  if (m >= p.M) return;
  const uint64_t at = (uint64_t)m * p.lda + k;
  uint32_t h[4];
  bool over = false;
  if constexpr (AF32) {
    const volatile float *src = reinterpret_cast<const float *>(p.A) + at;
    float f[8];
    if (quads) {
      asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]) : "l"(src) : "memory");
      asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7]) : "l"(src + 4) : "memory");
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = src[i];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) over |= fabsf(f[i]) > 65504.0f && fabsf(f[i]) < __int_as_float(0x7f800000);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = h2_as_u32(__floats2half2_rn(f[2 * i], f[2 * i + 1]));
    if (over && p.status) atomicExch(p.status, (int)CUTB_ERR_RANGE);
  } else {
    const volatile uint16_t *src = reinterpret_cast<const uint16_t *>(p.A) + at;
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = src[2 * i] | (uint32_t)src[2 * i + 1] << 16;
  }
  *reinterpret_cast<uint4 *>(p.acts + ((size_t)m * p.K + k) * 2) = make_uint4(h[0], h[1], h[2], h[3]);
}

// The tiles that several CTAs share, where no counters tell the last of them: block x takes the tile that CTA x begins and another ends.
__global__ void __launch_bounds__(128) ft_join_kernel(const FtParams p, uint32_t nk) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t end = (blockIdx.x + 1) * p.per, tile = end / nk, c_first = tile * nk / p.per, c_last = ((tile + 1) * nk - 1) / p.per;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (end >= p.tiles * nk || end % nk == 0 || c_first != blockIdx.x) return;
  float v[8];
  ft_add_shares(p, tile, nk, c_first, c_last, blockIdx.y * 8, threadIdx.x, v);
  ft_store<8>(p, tile, blockIdx.y * 8, threadIdx.x, v);
}

template <int FMT, int T> __global__ void __launch_bounds__(FT_THREADS, 1)
    qgemm_few_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const FtParams p) {
  constexpr uint32_t CHUNK = granule_bytes(FMT), WB = ft_unit(FMT), CW = FT_WARPS, TOK = T / FT_GROUPS;  // (activation rows of a thread)
  constexpr uint32_t S = ft_stages(FMT, T), SA = ft_act_stages(T), SLOTS = ft_slots(T), ACT = ft_act(T), ACHUNK = T * 128;
  extern __shared__ __align__(128) uint8_t ft_raw[];
  uint8_t *ft_smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(ft_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint32_t last_s, tmem_s;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t acts_u = smem_u32(ft_smem), ring_u = acts_u + SA * ACT;
  const uint32_t wfull = ring_u + S * WB, wempty = wfull + S * 8, afull = wempty + S * 8, aempty = afull + SA * 8, xfull = aempty + SA * 8,
                 xempty = xfull + 2 * SLOTS * 8, dfull = xempty + 2 * SLOTS * 8, dempty = dfull + 16, idle = dempty + 16;
  const uint32_t nk = p.K / 256, total = p.tiles * nk, u0 = blockIdx.x * p.per, n = min(p.per, total - u0);  // (the grid leaves no run empty)

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (warp == CW) {
    if (lane == 0) {
      for (uint32_t s = 0; s < S; ++s) mbar_init(wfull + s * 8, 1), mbar_init(wempty + s * 8, CW);
      for (uint32_t s = 0; s < SA; ++s) mbar_init(afull + s * 8, 1), mbar_init(aempty + s * 8, 2);
      for (uint32_t s = 0; s < 2 * SLOTS; ++s) mbar_init(xfull + s * 8, 8), mbar_init(xempty + s * 8, 1);
      for (uint32_t s = 0; s < 2; ++s) mbar_init(dfull + s * 8, 2), mbar_init(dempty + s * 8, CW);
      mbar_init(idle, 2);
      fence_mbar_init();
    }
    __syncwarp();
  } else if (warp == CW + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_s, tmem_d = tmem + 2 * SLOTS * 64;  // two accumulators of 32 columns per issuer behind the chunks

  if (warp == CW) {
    // ---- copies ----
    const bool leader = elect_one();
    auto weights = [&](uint32_t j, uint32_t slot) {
      const uint32_t u = u0 + j, bar = wfull + slot * 8;
      mbar_arrive_expect_tx(bar, WB);
      tma_load_2d(ring_u + slot * WB, &map_w, u % nk * (CHUNK / 4), u / nk * FT_ROWS, bar);
    };
    auto acts = [&](uint32_t j, uint32_t slot) {
      mbar_arrive_expect_tx(afull + slot * 8, ACT);
      for (uint32_t c = 0; c < 4; ++c) tma_load_2d(acts_u + slot * ACT + c * ACHUNK, &map_a, (u0 + j) % nk * 256 + c * 64, 0, afull + slot * 8);
    };
    auto expired = [&]() {
      if (leader && p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
    };
    uint32_t wi = min(S, n), ai = min(SA, n);  // copies issued
    if (leader)
      for (uint32_t j = 0; j < wi; ++j) weights(j, j);  // constants: no wait for the kernel before
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (leader)
      for (uint32_t j = 0; j < ai; ++j) acts(j, j);
    uint32_t ws = 0, wp = 0, as = 0, ap = 0;
    while (wi < n || ai < n) {
      if (wi < n) {
        if (!warp_wait(wempty + ws * 8, wp)) {
          expired();
          break;
        }
        if (leader) weights(wi, ws);
        ++wi;
        if (++ws == S) ws = 0, wp ^= 1u;
      }
      if (ai < n && (ai + S <= wi + SA || wi == n)) {
        if (!warp_wait(aempty + as * 8, ap)) {
          expired();
          break;
        }
        if (leader) acts(ai, as);
        ++ai;
        if (++as == SA) as = 0, ap ^= 1u;
      }
    }
    // stay until every copy issued here has landed (bounded)
    for (uint32_t j = wi > S ? wi - S : 0; j < wi; ++j) mbar_drain(wfull + (j % S) * 8, (j / S) & 1u);
    for (uint32_t j = ai > SA ? ai - SA : 0; j < ai; ++j) mbar_drain(afull + (j % SA) * 8, (j / SA) & 1u);
  } else if (warp > CW) {
    // ---- MMAs: 128 weight rows (tensor memory) x 32 activation rows (shared memory), 16 k each; issuer h takes the h-th half of a unit ----
    const bool leader = elect_one();
    const uint32_t half = warp - CW - 1, xf = xfull + half * SLOTS * 8, xe = xempty + half * SLOTS * 8;
    const uint64_t proto = umma_desc_sw128(0);
    const uint32_t desc_hi = (uint32_t)(proto >> 32), b_lo0 = (uint32_t)proto + ((acts_u & 0x3FFFFu) >> 4) + half * (ACT / 32);
    const uint32_t idesc = umma_idesc_f16(128, T), a0 = tmem + half * SLOTS * 64, d0 = tmem_d + half * 2 * T;
    uint32_t as = 0, ap = 0, xs = 0, xp = 0, k = u0 % nk, seg = 0;
    bool first = true, ok = true;
    for (uint32_t j = 0; j < n; ++j) {
      if (first && seg >= 2) ok = mbar_spin_bounded(dempty + (seg & 1) * 8, ((seg >> 1) - 1) & 1u);
      if (ok) {
        const bool there = mbar_test(afull + as * 8, ap), widened = mbar_test(xf + xs * 8, xp);
        ok = (there || mbar_spin_bounded(afull + as * 8, ap)) && (widened || mbar_spin_bounded(xf + xs * 8, xp));
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t d = d0 + (seg & 1) * T, a = a0 + xs * 64, b = b_lo0 + as * (ACT / 16);
      if (leader) {
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) umma_ts(d, a + 8 * i, b + (i >> 2) * (ACHUNK / 16) + 2 * (i & 3), desc_hi, idesc, i ? 1u : (uint32_t)!first);
        umma_commit(xe + xs * 8);
        umma_commit(aempty + as * 8);
      }
      first = false;
      if (++xs == SLOTS) xs = 0, xp ^= 1u;
      if (++as == SA) as = 0, ap ^= 1u;
      if (++k < nk && j + 1 < n) continue;
      if (leader) umma_commit(dfull + (seg & 1) * 8);
      if (k == nk) k = 0;
      ++seg, first = true;
    }
    if (!ok && leader && p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
    if (leader) umma_commit(idle);
    __syncwarp();
    mbar_drain(idle, 0);  // no MMA is under way when the tensor memory goes back
    __syncwarp();
  } else {
    // ---- converters: one weight row per thread; group g widens the g-th chunk (64 k) of every unit ----
    const uint32_t quarter = (warp & 3) * 32, row = quarter + lane, group = warp >> 2, tok0 = group * TOK, half = group >> 1;
    const uint32_t xf = xfull + half * SLOTS * 8, xe = xempty + half * SLOTS * 8;
    const uint32_t to = tmem + (quarter << 16) + half * SLOTS * 64 + (group & 1) * 32;
    uint32_t ws = 0, wp = 0, xs = 0, xp = 0, tile = u0 / nk, k = u0 % nk, k_begin = k, seg = 0;
    bool dead = false;
    auto expect = [&](uint32_t bar, uint32_t parity) {
      if (!dead && !warp_wait(bar, parity)) {
        dead = true;
        if (lane == 0 && p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
      }
    };
    expect(wfull, 0);
    for (uint32_t j = 0; j < n; ++j) {
      // (barriers are asked early, so that an answer is there when it is needed)
      const bool room = mbar_test(xe + xs * 8, xp ^ 1u);
      const uint32_t src = ring_u + ws * WB + row * CHUNK;
      uint32_t h[32];
      switch (group) {
        case 0: ft_chunk<FMT, 0>(src, h); break;
        case 1: ft_chunk<FMT, 1>(src, h); break;
        case 2: ft_chunk<FMT, 2>(src, h); break;
        default: ft_chunk<FMT, 3>(src, h); break;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(wempty + ws * 8);
      if (++ws == S) ws = 0, wp ^= 1u;
      const bool more = j + 1 < n, landed = !more || mbar_test(wfull + ws * 8, wp);
      const bool ready = __all_sync(0xffffffffu, room && landed);
      if (!ready) expect(xe + xs * 8, xp ^ 1u);
      tc_fence_after();
      tmem_st16(to + xs * 64, *reinterpret_cast<const uint32_t (*)[16]>(&h[0]));
      tmem_st16(to + xs * 64 + 16, *reinterpret_cast<const uint32_t (*)[16]>(&h[16]));
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(xf + xs * 8);
      if (++xs == SLOTS) xs = 0, xp ^= 1u;
      if (more && !ready) expect(wfull + ws * 8, wp);
      if (++k < nk && more) continue;

      // ---- the tile, or this CTA's share of it, is complete ----
      expect(dfull + (seg & 1) * 8, (seg >> 1) & 1u);
      tc_fence_after();
      float v[TOK];
#pragma unroll
      for (uint32_t i = 0; i < TOK; i += 8) {  // the issuers' sums
        uint32_t a[8], b[8];
        tmem_ld8(tmem_d + (quarter << 16) + (seg & 1) * T + tok0 + i, a);
        tmem_ld8(tmem_d + (quarter << 16) + (2 + (seg & 1)) * T + tok0 + i, b);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[i + e] = __uint_as_float(a[e]) + __uint_as_float(b[e]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dempty + (seg & 1) * 8);
      asm volatile("griddepcontrol.wait;" ::: "memory");
      bool finish = k_begin == 0 && k == nk;
      if (!finish) {
        float *share = p.shares + (size_t)(2 * blockIdx.x + (seg ? 1u : 0u)) * p.share_rows * FT_ROWS + tok0 * FT_ROWS + row;
#pragma unroll
        for (uint32_t i = 0; i < TOK; ++i)
          if (tok0 + i / 8 * 8 < p.share_rows) share[i * FT_ROWS] = v[i];
      }
      if (!finish && p.arrived) {
        const uint32_t c_first = tile * nk / p.per, c_last = ((tile + 1) * nk - 1) / p.per;
        __threadfence();
        asm volatile("bar.sync 1, %0;" ::"n"(CW * 32) : "memory");
        if (tid == 0) last_s = atomicAdd(p.arrived + tile, 1u) == c_last - c_first;
        asm volatile("bar.sync 1, %0;" ::"n"(CW * 32) : "memory");
        finish = last_s != 0;
        if (finish) {  // every share of the tile is there: add them in CTA order
          __threadfence();
          ft_add_shares(p, tile, nk, c_first, c_last, tok0, row, v);
        }
      }
      if (finish) ft_store<TOK>(p, tile, tok0, row, v);
      if (k == nk) k = 0, ++tile;
      k_begin = k, ++seg;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == CW + 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

// Units that a CTA may have more than an equal share, if no tile is shared then: they take less than the launch that joins the shares.  us,
// tiles shared / whole: one unit more, Q8_0 512 x 20000 32 rows 9.2 / 7.3; three, 2048 x 11008 11.2 / 8.9; six, 4096 x 11776 Q8_0 15.8 / 14.3
// and Q4_0 15.2 / 14.5; seven and eight, 6144 x 12928 Q4_0 20.9 / 21.2, 6144 x 11800 19.4 / 20.6.
constexpr uint32_t FT_WHOLE = 6;

struct FtPlan {
  uint32_t T, tiles, per, grid, share_rows;
  uint64_t acts, arrived, shares;  // scratch bytes, each but the last rounded up to 256
};
FtPlan ft_plan(const cutb_qmatmul_desc &d, uint32_t sms) {
  FtPlan pl{};
  pl.T = d.M <= 32 ? 32 : 64;
  pl.tiles = (d.N + FT_ROWS - 1) / FT_ROWS;
  const uint32_t total = pl.tiles * (d.K / 256);
  pl.grid = total < sms ? total : sms;
  pl.per = (total + pl.grid - 1) / pl.grid;
  const uint32_t nk = d.K / 256, whole = (pl.per + nk - 1) / nk * nk;
  if (whole <= pl.per + FT_WHOLE) pl.per = whole;
  pl.grid = (total + pl.per - 1) / pl.per;
  pl.share_rows = (d.M + 7) / 8 * 8;
  auto up = [](uint64_t b) { return (b + 255) / 256 * 256; };
  pl.acts = up((uint64_t)d.M * d.K * 2);
  pl.arrived = up((uint64_t)pl.tiles * 4);
  pl.shares = pl.per % nk ? (uint64_t)2 * pl.grid * pl.share_rows * FT_ROWS * 4 : 0;
  return pl;
}
// A tensor copy can read the activations where they are.
bool ft_direct(const cutb_qmatmul_desc &d) { return d.a_dtype == CUTB_F16 && reinterpret_cast<uintptr_t>(d.A) % 16 == 0 && d.lda % 8 == 0; }

template <int FMT, int T> int ft_launch(const cutb_qmatmul_desc &d, const FtParams &p, const FtPlan &pl, cudaStream_t stream) {
  static bool configured[64] = {};  // per device: the attribute is set once on each
  int dev = 0;
  CUTB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    CUTB_CUDA_TRY(cudaFuncSetAttribute(qgemm_few_kernel<FMT, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ft_smem(FMT, T)));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  const bool staged = p.acts != nullptr;
  CUtensorMap map_w, map_a;
  if (int rc = ft_map(&map_w, d)) return rc;
  if (int rc = make_tmap_sw128(&map_a, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, staged ? p.acts : d.A, d.M, d.K, (uint64_t)(staged ? d.K : d.lda) * 2, T)) return rc;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = d.flags & CUTB_FLAG_NO_OVERLAP ? 0 : 1;
  cfg.stream = stream;
  if (staged) {
    const uint64_t threads = (uint64_t)d.M * (d.K / 8);
    cfg.gridDim = dim3((uint32_t)(((threads > pl.tiles ? threads : pl.tiles) + 255) / 256));
    cfg.blockDim = dim3(256);
    const int quads = reinterpret_cast<uintptr_t>(d.A) % 16 == 0 && d.lda % 4 == 0;
    if (d.a_dtype == CUTB_F32) CUTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, ft_stage_kernel<true>, p, quads));
    else CUTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, ft_stage_kernel<false>, p, quads));
    cfg.numAttrs = 1;  // its predecessor is this library's own kernel
  }
  cfg.gridDim = dim3(pl.grid);
  cfg.blockDim = dim3(FT_THREADS);
  cfg.dynamicSmemBytes = ft_smem(FMT, T);
  CUTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, qgemm_few_kernel<FMT, T>, map_w, map_a, p));
  const uint32_t nk = d.K / 256;
  if (!staged && p.per % nk != 0) {
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(pl.grid, p.share_rows / 8);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = 0;
    CUTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, ft_join_kernel, p, nk));
  }
  return CUTB_OK;
}
template <int FMT> int ft_dispatch(const cutb_qmatmul_desc &d, const FtParams &p, const FtPlan &pl, cudaStream_t stream) {
  return pl.T == 32 ? ft_launch<FMT, 32>(d, p, pl, stream) : ft_launch<FMT, 64>(d, p, pl, stream);
}

uint32_t ft_sms() {
  DeviceInfo di;
  return get_device_info(&di) == CUTB_OK ? (uint32_t)di.sm_count : 148u;
}

}  // namespace

bool qgemm_few_supported(const cutb_qmatmul_desc &d) {
  return d.layout == CUTB_LAYOUT_GGUF_BLOCKS && d.K != 0 && d.K % 256 == 0 && d.M != 0 && d.M <= 64 && d.N != 0 && reinterpret_cast<uintptr_t>(d.W) % 16 == 0;
}

uint64_t qgemm_few_workspace(const cutb_qmatmul_desc &d, bool direct) {
  const FtPlan pl = ft_plan(d, ft_sms());
  return direct ? pl.shares : pl.acts + pl.arrived + pl.shares;
}

bool qgemm_few_fits(const cutb_qmatmul_desc &d) {
  const uint64_t need = qgemm_few_workspace(d, ft_direct(d));
  return need == 0 || (d.workspace && reinterpret_cast<uintptr_t>(d.workspace) % 16 == 0 && d.workspace_bytes >= need);
}

int qgemm_few_launch(const cutb_qmatmul_desc &d, cudaStream_t stream) {
  const FtPlan pl = ft_plan(d, ft_sms());
  FtParams p{};
  p.A = d.A, p.lda = d.lda, p.C = d.C, p.ldc = d.ldc, p.D = d.D, p.ldd = d.ldd, p.M = d.M, p.K = d.K, p.N = d.N, p.tiles = pl.tiles, p.per = pl.per, p.share_rows = pl.share_rows;
  p.fusion_type = d.fusion_type, p.fusion_op = d.fusion_op, p.glu = d.flags & CUTB_FLAG_GLU_PAIRS ? 1 : 0, p.status = d.status;
  uint8_t *ws = reinterpret_cast<uint8_t *>(d.workspace);
  if (!ft_direct(d)) p.acts = ws, p.arrived = reinterpret_cast<uint32_t *>(ws + pl.acts), ws += pl.acts + pl.arrived;
  p.shares = reinterpret_cast<float *>(ws);
  switch (d.format) {
    case CUTB_Q8_0: return ft_dispatch<CUTB_Q8_0>(d, p, pl, stream);
    case CUTB_Q4_0: return ft_dispatch<CUTB_Q4_0>(d, p, pl, stream);
    default: return ft_dispatch<CUTB_Q4_K>(d, p, pl, stream);
  }
}

}  // namespace cutb
