// Attention of a prompt's tokens on the 5th-generation tensor cores, shared by the llama path (fp16 cache), windowed attention
// (bf16 ring caches) and latent attention over expanded keys and values (bf16).  Included by the translation units of the three.
//
// A block owns up to two tiles of 128 consecutive tokens of one query head; both meet the same tiles of 128 keys.
//   warps 0-3, 4-7  softmax of the first and of the second token tile, one token per thread (= tensor-memory lane).  Scores come
//                   by tcgen05.ld, the weights go back by tcgen05.st in the place of the scores: bf16 weights as the sum of two
//                   terms (16 significant bits), high parts in the first 64 columns and low parts in the other 64; fp16 weights as
//                   one term.  The running maximum is followed tile by tile, and the weighted values are rescaled in tensor memory
//                   when it rises: the largest weight is an exact 1 then.  Following it only past 2^8 was 2 to 9 % faster (32 heads,
//                   1500 tokens 46.9 against 47.7 us; 8 heads, 256 tokens behind 4000 82 against 91), but the error against 64 bits
//                   was up to 3.4 times (fp16) and 1.3 times (bf16) that of the kernels before; now 1.00 to 1.07 times.
//   warp 8          one lane copies the key and value tiles by TMA (boxes of 64 columns x 64 rows, 128-byte swizzle); columns past
//                   a head's elements and rows past the tensor read as zero.
//   warp 9          one lane issues the products: scores = Q K^T from shared memory, then weights (tensor memory, the A operand)
//                   times values (shared memory, read along the keys).  The two token tiles alternate, so that the tensor cores
//                   work for one while the other is in its softmax.
// Tensor memory: 2 x 128 columns of scores / weights, 2 x 128 of weighted values.
// Bound by the latency of a token tile's chain scores -> softmax -> weighted values (about 4500 cycles per 128 keys without rescaling,
// of which the tensor cores work 3000, in fp16 2000, and the exponentials 2000 for the two tiles together); the weights of 64 keys at a
// time are handed over, so that the products of the first half run beside the exponentials of the second.  32 heads of 128, window 1024,
// 2048 tokens: 207 us with warp MMAs -> 78 us (by ncu the tensor pipe is busy 30 % of a block's cycles).
// A row that comes out non-finite is computed again from the keys it sees alone (pa_row_again).
// Every wait is bounded; on expiry the block records CUTB_ERR_TIMEOUT, waits (bounded) for its copies, frees its tensor memory
// and returns.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "dense_common.cuh"
#include "tcgen05.cuh"

namespace cutb {
namespace {

constexpr int PA_BM = 128, PA_BN = 128, PA_THREADS = 320;
constexpr uint32_t PA_BOX = 64 * 128, PA_PLANE = 128 * 128;  // bytes of a copied box and of 64 columns of a 128-row tile
enum { PA_LLAMA = 0, PA_WINDOW = 1, PA_LATENT = 2 };

struct PaParams {
  const float *q;
  uint64_t ldq;
  uint32_t n_tokens, n_heads, rep, q_head;  // rep: query heads per KV head; q_head: elements of a query head
  uint32_t dim, rot;                        // PA_LATENT: elements that are not turned, and those that are, from column rot_col on
  uint32_t rot_col, pairing;
  const float *cos_t, *sin_t;
  const uint32_t *positions;  // PA_LLAMA: every token's cache row
  const uint32_t *pos_ptr;    // others: the first token's position
  uint32_t pos, max_pos, window, ring_rows;
  uint32_t step;              // tokens per block: 128 or 256
  uint32_t ksteps;            // 16-column steps of the score product
  uint32_t key_planes;        // 64-column planes that come from the heads' own keys (the others: the shared turned part)
  const uint16_t *k, *r, *v;  // what the tensor maps cover, for pa_row_again: keys, the shared turned part, values; strides in elements
  uint64_t ld_k, ld_r, ld_v;
  uint32_t k_head, v_head;
  int q_vec;                  // queries and tables allow eight pairs at a time (pa_set_vec)
  float scale, q_mul;         // |scale| log2(e), and the scale's sign: the maxima are taken of raw scores
  const float *sink;          // PA_LATENT: a logit per head
  int zero_sink;              // PA_WINDOW: a logit of zero
  void *out;
  uint64_t ldo;
  uint32_t vdim;
  int out_bf16;
  int *status;
};

template <int KP> struct PaRings {  // KP: 64-column planes of a key row
  static constexpr uint32_t K = 2, V = KP == 3 ? 1 : 2;
};
template <int KP, int VP> constexpr uint32_t pa_smem() {
  return 1024 + 2 * KP * PA_PLANE + PaRings<KP>::K * KP * PA_PLANE + PaRings<KP>::V * VP * PA_PLANE;
}

__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// waits for the loads before it; the registers pass through, so that nothing reads them earlier
__device__ __forceinline__ void tmem_wait32(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]),
                 "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
                 "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])::"memory");
}
// 2^x, subnormal results flushed (weights below 2^-126 of the largest)
__device__ __forceinline__ float pa_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Descriptor of a tile read along its rows (the MMA's N along the 64 columns of a plane, K along the rows): groups of eight rows
// 1024 bytes apart (stride byte offset), planes PA_PLANE apart (leading byte offset).
__device__ __forceinline__ uint64_t pa_value_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (uint64_t)(PA_PLANE >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

template <int MODE> __device__ __forceinline__ uint16_t pa_bits(float v) {
  if constexpr (MODE == PA_LLAMA) return __half_as_ushort(__float2half_rn(v));
  else return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// One token's output again, by one warp in fp32: a key that the token does not see has a weight of zero in its tile, and zero times an
// infinity or a NaN is not zero, so a row that came out non-finite may owe it to keys of other tokens.  `q`: the token tile's
// queries in shared memory, `r` the row; ms, inv: the token's followed maximum and 1 / sum.
template <int MODE>
__device__ __noinline__ void pa_row_again(const PaParams &p, const uint8_t *q, uint32_t r, uint32_t h, uint32_t tok, uint32_t pos, float ms, float inv) {
  const uint32_t lane = threadIdx.x & 31, kvh = h / p.rep, first = MODE == PA_WINDOW && pos + 1 > p.window ? pos + 1 - p.window : 0;
  auto number = [](uint32_t bits) {
    if constexpr (MODE == PA_LLAMA) return __half2float(__ushort_as_half((uint16_t)bits));
    else return __uint_as_float(bits << 16);
  };
  auto row_of = [&](uint32_t key) { return (uint64_t)(MODE == PA_WINDOW ? key % p.ring_rows : key); };
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (uint32_t k0 = first; k0 <= pos; k0 += 32) {
    const uint32_t key = k0 + lane;
    float w = 0.f;
    if (key <= pos) {
      const uint64_t row = row_of(key);
      float s = 0.f;
      for (uint32_t c = 0; c < p.ksteps * 16; ++c) {
        const bool turned = MODE == PA_LATENT && c >= p.rot_col;
        const uint32_t e = turned ? c - p.rot_col : c, n = MODE == PA_LATENT ? (turned ? p.rot : p.dim) : p.q_head;
        if (e >= n) continue;
        const uint32_t x = *reinterpret_cast<const uint16_t *>(q + (c >> 6) * PA_PLANE + r * 128u + ((((c & 63u) >> 3) ^ (r & 7u)) << 4) + (c & 7u) * 2u);
        s = fmaf(number(x), number(__ldg(turned ? p.r + row * p.ld_r + e : p.k + row * p.ld_k + (uint64_t)kvh * p.k_head + e)), s);
      }
      w = pa_exp2(fmaf(s, p.scale, -ms));
    }
    for (uint32_t j = 0; j < 32 && k0 + j <= pos; ++j) {
      const float wj = __shfl_sync(0xffffffffu, w, j);
      const uint16_t *src = p.v + row_of(k0 + j) * p.ld_v + (uint64_t)kvh * p.v_head;
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i)
        if (lane + 32 * i < p.vdim) acc[i] = fmaf(wj, number(__ldg(src + lane + 32 * i)), acc[i]);
    }
  }
#pragma unroll
  for (uint32_t i = 0; i < 4; ++i)
    if (lane + 32 * i < p.vdim) store_out(p.out, p.out_bf16, (uint64_t)tok * p.ldo + (uint64_t)h * p.vdim + lane + 32 * i, acc[i] * inv);
}

template <int MODE, int KP, int VP>
__global__ void __launch_bounds__(PA_THREADS, 1)
    prefill_attention_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_r,
                             const __grid_constant__ CUtensorMap map_v, const __grid_constant__ PaParams p) {
  constexpr bool BF16 = MODE != PA_LLAMA;
  constexpr uint32_t SK = PaRings<KP>::K, SV = PaRings<KP>::V, QT = KP * PA_PLANE, KT = KP * PA_PLANE, VT = VP * PA_PLANE;
  extern __shared__ __align__(1024) uint8_t pa_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(pa_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t bars[2 * SK + 2 * SV + 9];
  __shared__ uint32_t tmem_slot, abort_flag, hi_s[2];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t q_u = smem_u32(smem), k_u = q_u + 2 * QT, v_u = k_u + SK * KT;
  const uint32_t kfull = smem_u32(bars), kempty = kfull + SK * 8, vfull = kempty + SK * 8, vempty = vfull + SV * 8;
  const uint32_t sfull = vempty + SV * 8, pready = sfull + 16, odone = pready + 32, qready = odone + 16;  // pready: [token tile][half of the keys]

  if (tid == 0) {
    for (uint32_t i = 0; i < SK; ++i) mbar_init(kfull + i * 8, 1), mbar_init(kempty + i * 8, 1);
    for (uint32_t i = 0; i < SV; ++i) mbar_init(vfull + i * 8, 1), mbar_init(vempty + i * 8, 1);
    for (uint32_t x = 0; x < 2; ++x) mbar_init(sfull + x * 8, 1), mbar_init(odone + x * 8, 1);
    for (uint32_t x = 0; x < 4; ++x) mbar_init(pready + x * 8, 4);
    mbar_init(qready, 8);
    abort_flag = 0, hi_s[0] = hi_s[1] = 0;
    fence_mbar_init();
  }
  // the later tokens of every head (which see more keys) first: the short blocks fill what the long ones leave
  const uint32_t tok0 = (gridDim.y - 1 - blockIdx.y) * p.step, h = blockIdx.x, kvh = h / p.rep;
  uint32_t p0 = 0, ntok = min(p.step, p.n_tokens - tok0);
  pdl_enter();
  if constexpr (MODE != PA_LLAMA) {
    const uint64_t first = (uint64_t)(p.pos_ptr ? *p.pos_ptr : p.pos) + tok0;
    if (first + ntok > p.max_pos) {  // tokens without table rows are left out, as the cache write leaves them out
      if (p.status && tid == 0 && h == 0) atomicExch(p.status, (int)CUTB_ERR_INVALID);
      if (first >= p.max_pos) return;
      ntok = (uint32_t)(p.max_pos - first);
    }
    p0 = (uint32_t)first;
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  // this thread's token (softmax warps), its position, the first and last key each token tile sees
  const uint32_t grp = warp >> 2, row = tid & 127, tok = tok0 + grp * PA_BM + row;
  const bool live = warp < 8 && grp * PA_BM + row < ntok;
  uint32_t pos = p0 + grp * PA_BM + row;
  uint32_t lo[2], hi[2], first_pos[2];  // hi: one past the last key; 0: no tokens
  if constexpr (MODE == PA_LLAMA) {
    pos = 0;
    if (live) {
      pos = __ldg(p.positions + tok);
      if (pos >= p.max_pos) {  // never read outside the cache
        if (p.status && h == 0) atomicExch(p.status, (int)CUTB_ERR_INVALID);
        pos = p.max_pos - 1;
      }
      atomicMax(&hi_s[grp], pos + 1);
    }
    __syncthreads();
    lo[0] = lo[1] = 0, hi[0] = hi_s[0], hi[1] = hi_s[1];
    first_pos[0] = first_pos[1] = 0;  // (any order of positions: every tile is masked by key and position)
  } else {
#pragma unroll
    for (uint32_t x = 0; x < 2; ++x) {
      first_pos[x] = p0 + x * PA_BM;
      hi[x] = x * PA_BM < ntok ? p0 + min(ntok, (x + 1) * PA_BM) : 0;
      lo[x] = MODE == PA_WINDOW && first_pos[x] + 1 > p.window ? first_pos[x] + 1 - p.window : 0;
    }
  }
  const uint32_t key_lo = hi[0] ? lo[0] : lo[1], key_hi = max(hi[0], hi[1]);
  const uint32_t t_first = key_lo / PA_BN, t_end = (key_hi + PA_BN - 1) / PA_BN;
  auto sees = [&](uint32_t x, uint32_t t) { return t * PA_BN < hi[x] && (t + 1) * PA_BN > lo[x]; };
  auto give_up = [&]() {
    if (p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
    atomicExch(&abort_flag, 1u);
  };
  auto aborted = [&]() { return *reinterpret_cast<volatile uint32_t *>(&abort_flag) != 0; };

  if (warp == 8) {
    const bool leader = elect_one();
    uint32_t sk = 0, pk = 1, sv = 0, pv = 1;  // (a fresh barrier lets a wait on the phase before its first pass)
    for (uint32_t t = t_first; t < t_end; ++t) {
      uint32_t at[2];  // rows of the tile's halves
#pragma unroll
      for (uint32_t j = 0; j < 2; ++j) at[j] = MODE == PA_WINDOW ? (t * PA_BN + 64 * j) % p.ring_rows : t * PA_BN + 64 * j;
      if (!__all_sync(0xffffffffu, mbar_wait_probe_first(kempty + sk * 8, pk) && !aborted())) {
        if (leader) give_up();
        break;
      }
      if (leader) {
        mbar_arrive_expect_tx(kfull + sk * 8, KT);
#pragma unroll
        for (uint32_t c = 0; c < KP; ++c)
#pragma unroll
          for (uint32_t j = 0; j < 2; ++j) {
            const uint32_t dst = k_u + sk * KT + c * PA_PLANE + j * PA_BOX;
            if (MODE != PA_LATENT || c < p.key_planes) tma_load_3d(dst, &map_k, c * 64, kvh, at[j], kfull + sk * 8);
            else tma_load_3d(dst, &map_r, (c - p.key_planes) * 64, 0, at[j], kfull + sk * 8);
          }
      }
      if (++sk == SK) sk = 0, pk ^= 1u;
      if (!__all_sync(0xffffffffu, mbar_wait_probe_first(vempty + sv * 8, pv) && !aborted())) {
        if (leader) give_up();
        break;
      }
      if (leader) {
        mbar_arrive_expect_tx(vfull + sv * 8, VT);
#pragma unroll
        for (uint32_t c = 0; c < VP; ++c)
#pragma unroll
          for (uint32_t j = 0; j < 2; ++j)
            tma_load_3d(v_u + sv * VT + c * PA_PLANE + j * PA_BOX, &map_v, c * 64, kvh, at[j], vfull + sv * 8);
      }
      if (++sv == SV) sv = 0, pv ^= 1u;
    }
    // do not retire with copies still landing, whoever gives up and when: every slot's last fill (bounded; a slot that was never
    // filled answers at once)
    for (uint32_t i = 0; i < SK; ++i) {
      if (sk == 0) sk = SK, pk ^= 1u;
      --sk;
      mbar_drain(kfull + sk * 8, pk ^ 1u);
    }
    for (uint32_t i = 0; i < SV; ++i) {
      if (sv == 0) sv = SV, pv ^= 1u;
      --sv;
      mbar_drain(vfull + sv * 8, pv ^ 1u);
    }
    __syncwarp();
  } else if (warp == 9) {
    const bool leader = elect_one();
    const uint64_t kproto = umma_desc_sw128(0), vproto = pa_value_desc(0);
    const uint32_t k_hi = (uint32_t)(kproto >> 32), v_hi = (uint32_t)(vproto >> 32);
    const uint32_t q_lo = (uint32_t)kproto + ((q_u & 0x3FFFFu) >> 4), k_lo = (uint32_t)kproto + ((k_u & 0x3FFFFu) >> 4);
    const uint32_t v_lo = (uint32_t)vproto + ((v_u & 0x3FFFFu) >> 4);
    const uint32_t id_s = BF16 ? umma_idesc_bf16(128, 128) : umma_idesc_f16(128, 128);
    const uint32_t id_o = (BF16 ? umma_idesc_bf16(128, VP * 64) : umma_idesc_f16(128, VP * 64)) | (1u << 16);  // B along its rows
    uint32_t sk = 0, pk = 0, sv = 0, pv = 0, pp[2] = {0, 0}, acc[2] = {0, 0};
    bool ok = __all_sync(0xffffffffu, mbar_spin_bounded(qready, 0));
    tc_fence_after();
    auto scores = [&](uint32_t x) {
      if (leader) {
#pragma unroll
        for (uint32_t ks = 0; ks < KP * 4; ++ks) {
          if (ks >= p.ksteps) break;
          const uint32_t off = (ks >> 2) * (PA_PLANE >> 4) + (ks & 3) * 2;
          umma_f16(tmem + x * 128, q_lo + x * (QT >> 4) + off, k_lo + sk * (KT >> 4) + off, k_hi, id_s, ks != 0);
        }
        umma_commit(sfull + x * 8);
      }
    };
    // the value product of token tile x over the tile in value slot s; the last user of the slot gives it back
    auto values = [&](uint32_t x, bool last) {
      ok = ok && __all_sync(0xffffffffu, mbar_spin_bounded(vfull + sv * 8, pv));
#pragma unroll
      for (uint32_t half = 0; half < 2; ++half) {  // the weights of 64 keys at a time
        ok = ok && __all_sync(0xffffffffu, mbar_spin_bounded(pready + (2 * x + half) * 8, pp[x]));
        if (!ok) return;
        tc_fence_after();
        if (leader) {
#pragma unroll
          for (uint32_t term = 0; term < (BF16 ? 2u : 1u); ++term)
#pragma unroll
            for (uint32_t ks = 4 * half; ks < 4 * half + 4; ++ks)
              umma_ts(tmem + 256 + x * 128, tmem + x * 128 + term * 64 + ks * 8, v_lo + sv * (VT >> 4) + ks * (2048 >> 4), v_hi, id_o,
                            term | ks ? 1u : acc[x]);
        }
      }
      pp[x] ^= 1u;
      if (leader) {
        umma_commit(odone + x * 8);
        if (last) umma_commit(vempty + sv * 8);
      }
      acc[x] = 1;
      if (last && ++sv == SV) sv = 0, pv ^= 1u;
    };
    bool pending = false;  // the second token tile's value product over the tile before
    for (uint32_t t = t_first; t < t_end && ok; ++t) {
      const bool s0 = sees(0, t), s1 = sees(1, t);
      ok = __all_sync(0xffffffffu, mbar_spin_bounded(kfull + sk * 8, pk));
      if (!ok) break;
      tc_fence_after();
      if (s0) {
        scores(0);
        if (!s1 && leader) umma_commit(kempty + sk * 8);
      }
      if (pending) values(1, true);
      pending = s1;
      if (!ok) break;
      if (s1) {
        scores(1);
        if (leader) umma_commit(kempty + sk * 8);
      }
      if (s0) values(0, !s1);
      if (++sk == SK) sk = 0, pk ^= 1u;
    }
    if (ok && pending) values(1, true);
    if (!ok && leader) give_up();
    __syncwarp();
  } else {
    // queries: turned at their own positions, rounded
    {
      const uint32_t half = p.rot / 2, rows = p.step;
      const float *q0 = p.q + (uint64_t)tok0 * p.ldq + (uint64_t)h * p.q_head;
      auto turned = [](float x0, float x1, float c, float s, float &y0, float &y1) {
        if constexpr (MODE == PA_LLAMA) {  // products and sums rounded separately, as BatchedAttentionReadCache does
          y0 = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
          y1 = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
        } else {
          y0 = x0 * c - x1 * s, y1 = x1 * c + x0 * s;
        }
      };
      auto position = [&](uint32_t r) {
        if constexpr (MODE == PA_LLAMA) return min(__ldg(p.positions + tok0 + r), p.max_pos - 1);
        else return p0 + r;
      };
      auto at = [&](uint32_t r, uint32_t col) {
        return smem + (r >> 7) * QT + (col >> 6) * PA_PLANE + (r & 127u) * 128u + ((((col & 63u) >> 3) ^ (r & 7u)) << 4) + (col & 7u) * 2u;
      };
      if (p.q_vec) {
        // eight pairs per step: 16-byte loads and stores (pair by pair the 256 x 128 queries of a block took 22 us)
        constexpr uint32_t GP = KP * 4;
#pragma unroll 2
        for (uint32_t i = tid; i < rows * GP; i += 256) {
          const uint32_t r = i / GP, gi = i % GP, rc = min(r, ntok - 1);  // (rows past the last token repeat it)
          uint32_t e0 = 16 * gi, e1 = 16 * gi + 8, c0 = e0, c1 = e1, ti = 8 * gi;  // elements and columns of the two halves, table index
          bool turn, near = true, in = true;
          if constexpr (MODE == PA_LATENT) {  // columns: the unturned part padded to whole planes, then neighbours that turn
            turn = c0 >= p.rot_col;
            const uint32_t off = turn ? c0 - p.rot_col : c0;
            in = off < (turn ? p.rot : p.dim);
            e0 = turn ? p.dim + off : off, e1 = e0 + 8, ti = off / 2;
          } else {
            turn = ti < half;
            if (turn && !p.pairing) near = false, e0 = c0 = ti, e1 = c1 = ti + half;
            in = e1 < p.q_head;
          }
          float x[16], c[8], sn[8], y[16];
          const float *src = q0 + (uint64_t)rc * p.ldq;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float4 f = in ? __ldg(reinterpret_cast<const float4 *>(src + (u < 2 ? e0 : e1) + 4 * (u & 1))) : make_float4(0.f, 0.f, 0.f, 0.f);
            x[4 * u] = f.x * p.q_mul, x[4 * u + 1] = f.y * p.q_mul, x[4 * u + 2] = f.z * p.q_mul, x[4 * u + 3] = f.w * p.q_mul;
          }
          const uint64_t tb = turn && in ? (uint64_t)position(rc) * half + ti : 0;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float4 f = turn && in ? __ldg(reinterpret_cast<const float4 *>(p.cos_t + tb) + u) : make_float4(1.f, 1.f, 1.f, 1.f);
            const float4 g = turn && in ? __ldg(reinterpret_cast<const float4 *>(p.sin_t + tb) + u) : make_float4(0.f, 0.f, 0.f, 0.f);
            c[4 * u] = f.x, c[4 * u + 1] = f.y, c[4 * u + 2] = f.z, c[4 * u + 3] = f.w;
            sn[4 * u] = g.x, sn[4 * u + 1] = g.y, sn[4 * u + 2] = g.z, sn[4 * u + 3] = g.w;
          }
          if (near) {
#pragma unroll
            for (int u = 0; u < 8; ++u) turned(x[2 * u], x[2 * u + 1], c[u], sn[u], y[2 * u], y[2 * u + 1]);
          } else {
#pragma unroll
            for (int u = 0; u < 8; ++u) turned(x[u], x[8 + u], c[u], sn[u], y[u], y[8 + u]);
          }
          uint32_t w[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) w[u] = (uint32_t)pa_bits<MODE>(y[2 * u]) | (uint32_t)pa_bits<MODE>(y[2 * u + 1]) << 16;
          *reinterpret_cast<uint4 *>(at(r, c0)) = make_uint4(w[0], w[1], w[2], w[3]);
          *reinterpret_cast<uint4 *>(at(r, c1)) = make_uint4(w[4], w[5], w[6], w[7]);
        }
      } else {
        constexpr uint32_t PP = KP * 32;
#pragma unroll 4
        for (uint32_t i = tid; i < rows * PP; i += 256) {
          const uint32_t r = i / PP, pi = i % PP, rc = min(r, ntok - 1);
          uint32_t e0 = 2 * pi, e1 = 2 * pi + 1, c0 = e0, c1 = e1, ti = pi;
          bool turn;
          if constexpr (MODE == PA_LATENT) {
            turn = c0 >= p.rot_col;
            const uint32_t off = turn ? c0 - p.rot_col : c0;
            e0 = off < (turn ? p.rot : p.dim) ? (turn ? p.dim + off : off) : p.q_head, e1 = e0 + 1, ti = off / 2;
          } else {
            turn = pi < half;
            if (turn && !p.pairing) e0 = c0 = pi, e1 = c1 = pi + half;
          }
          const float *src = q0 + (uint64_t)rc * p.ldq;
          const float x0 = e0 < p.q_head ? __ldg(src + e0) * p.q_mul : 0.f, x1 = e1 < p.q_head ? __ldg(src + e1) * p.q_mul : 0.f;
          const bool in = turn && ti < half;
          const uint64_t tb = in ? (uint64_t)position(rc) * half + ti : 0;
          float y0, y1;
          turned(x0, x1, in ? __ldg(p.cos_t + tb) : 1.f, in ? __ldg(p.sin_t + tb) : 0.f, y0, y1);
          *reinterpret_cast<uint16_t *>(at(r, c0)) = pa_bits<MODE>(y0);
          *reinterpret_cast<uint16_t *>(at(r, c1)) = pa_bits<MODE>(y1);
        }
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(qready);
    }

    const uint32_t mine = tmem + ((warp & 3) << 21), s_t = mine + grp * 128, o_t = mine + 256 + grp * 128;
    const float scale = p.scale;
    const float sink = MODE == PA_LATENT ? (p.sink ? __ldg(p.sink + h) * 1.4426950408889634f : -INFINITY)
                                         : (MODE == PA_WINDOW && p.zero_sink ? 0.f : -INFINITY);
    float m = sink, l = 0.f;
    uint32_t ph = 0, pv = 0, sv = 0, done = 0;  // done: value products committed for this token tile
    bool dead = false;
    const uint32_t my_hi = hi[grp], my_lo = lo[grp];
    for (uint32_t t = t_first; t < t_end; ++t) {
      const uint32_t key0 = t * PA_BN;
      if (key0 < my_hi && key0 + PA_BN > my_lo) {
        if (!__all_sync(0xffffffffu, mbar_wait_probe_first(sfull + grp * 8, ph) && !aborted())) {
          dead = true;
          break;
        }
        ph ^= 1u;
        tc_fence_after();
        uint32_t s[4][32];
#pragma unroll
        for (int j = 0; j < 4; ++j) tmem_ld32_async(s_t + 32 * j, s[j]);
#pragma unroll
        for (int j = 0; j < 4; ++j) tmem_wait32(s[j]);
        // does every token of the tile see every key?
        const bool all = MODE != PA_LLAMA && key0 + PA_BN - 1 <= first_pos[grp] && (MODE != PA_WINDOW || key0 + p.window > my_hi - 1);
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // (independent chains)
        if (all) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) mx4[j] = fmaxf(mx4[j], __uint_as_float(s[j][i]));
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const uint32_t key = key0 + 32 * j + i;
              const bool in = key <= pos && (MODE != PA_WINDOW || pos - key < p.window);
              s[j][i] = in ? s[j][i] : 0xff800000u;
              mx4[j] = fmaxf(mx4[j], __uint_as_float(s[j][i]));
            }
        }
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale;
        if (done == 0) {  // nothing is summed yet
          m = fmaxf(m, mx);
        } else if (__any_sync(0xffffffffu, mx > m)) {
          const float mn = fmaxf(m, mx), f = mn == -INFINITY ? 1.f : pa_exp2(m - mn);
          m = mn, l *= f;
          if (!warp_wait(odone + grp * 8, (done - 1) & 1u)) {
            dead = true;
            break;
          }
          tc_fence_after();
#pragma unroll 1
          for (uint32_t c = 0; c < VP * 64; c += 32) {
            uint32_t o[32];
            tmem_ld32_async(o_t + c, o);
            tmem_wait32(o);
            uint32_t a[16], b[16];
#pragma unroll
            for (int i = 0; i < 16; ++i)
              a[i] = __float_as_uint(__uint_as_float(o[i]) * f), b[i] = __float_as_uint(__uint_as_float(o[16 + i]) * f);
            tmem_st16(o_t + c, a);
            tmem_st16(o_t + c + 16, b);
          }
        }
        const float ms = m == -INFINITY ? 0.f : m;  // nothing attended yet: keep exponents finite
        // Keys nobody in the block sees carry no weight, but a weight of zero times a stray NaN would not be zero.
        if (key0 < key_lo || key0 + PA_BN > key_hi) {
          if (!warp_wait(vfull + sv * 8, pv)) {
            dead = true;
            break;
          }
          for (uint32_t i = row; i < 128 * VP * 8; i += 128) {
            const uint32_t r = i / (VP * 8), c = i % (VP * 8), key = key0 + r;
            if (key < key_lo || key >= key_hi)
              *reinterpret_cast<uint4 *>(smem + (v_u - q_u) + sv * VT + (c >> 3) * PA_PLANE + r * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
          }
          fence_async_smem();  // (seen through the arrivals below: the first half's products wait for all four warps)
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t ph16[16], pl16[16];
          float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float a = pa_exp2(fmaf(__uint_as_float(s[j][2 * i]), scale, -ms)), b = pa_exp2(fmaf(__uint_as_float(s[j][2 * i + 1]), scale, -ms));
            sum0 += a, sum1 += b;
            if constexpr (BF16) {
              ph16[i] = pack_bf16(a, b);
              pl16[i] = pack_bf16(a - bf16_lo(ph16[i]), b - bf16_hi(ph16[i]));
            } else {
              ph16[i] = h2_as_u32(__floats2half2_rn(a, b));
            }
          }
          l += sum0 + sum1;
          tmem_st16(s_t + 16 * j, ph16);
          if constexpr (BF16) tmem_st16(s_t + 64 + 16 * j, pl16);
          if (j & 1) {
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(pready + (2 * grp + (j >> 1)) * 8);
          }
        }
        ++done;
      }
      if (++sv == SV) sv = 0, pv ^= 1u;
    }
    if (!dead && done && !warp_wait(odone + grp * 8, (done - 1) & 1u)) dead = true;
    if (dead) {
      if (lane == 0) give_up();
    } else if (done) {
      tc_fence_after();
      if (sink != -INFINITY) l += pa_exp2(sink - m);
      const float inv = MODE == PA_LLAMA ? (l > 0.f ? 1.0f / l : 0.f) : 1.0f / l;
      const uint64_t base = (uint64_t)tok * p.ldo + (uint64_t)h * p.vdim;
      const bool quads = p.vdim % 8 == 0 && p.ldo % 8 == 0 && reinterpret_cast<uintptr_t>(p.out) % 16 == 0;
      float stray = 0.f;  // becomes NaN with the first output that is not finite
#pragma unroll 1
      for (uint32_t c = 0; c < VP * 64; c += 32) {
        if (c >= p.vdim) break;
        uint32_t o[32];
        __syncwarp();  // (lanes without a token have gone ahead)
        tmem_ld32_async(o_t + c, o);
        tmem_wait32(o);
        if (!live) continue;
        float y[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) y[i] = __uint_as_float(o[i]) * inv, stray = fmaf(y[i], 0.f, stray);
        if (quads) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            if (c + i >= p.vdim) break;
            if (p.out_bf16) {
              *reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(p.out) + base + c + i) =
                  make_uint4(pack_bf16(y[i], y[i + 1]), pack_bf16(y[i + 2], y[i + 3]), pack_bf16(y[i + 4], y[i + 5]), pack_bf16(y[i + 6], y[i + 7]));
            } else {
              float4 *dst = reinterpret_cast<float4 *>(reinterpret_cast<float *>(p.out) + base + c + i);
              dst[0] = make_float4(y[i], y[i + 1], y[i + 2], y[i + 3]), dst[1] = make_float4(y[i + 4], y[i + 5], y[i + 6], y[i + 7]);
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c + i < p.vdim) store_out(p.out, p.out_bf16, base + c + i, y[i]);
        }
      }
      __syncwarp();  // (rows stored above are stored again below, by other lanes)
      for (uint32_t again = __ballot_sync(0xffffffffu, live && !(stray == 0.f)); again; again &= again - 1) {
        const int src = __ffs(again) - 1;
        pa_row_again<MODE>(p, smem + grp * QT, (warp & 3) * 32 + src, h, tok - lane + src, __shfl_sync(0xffffffffu, pos, src),
                           __shfl_sync(0xffffffffu, m == -INFINITY ? 0.f : m, src), __shfl_sync(0xffffffffu, inv, src));
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// Rows of `heads` heads of `cols` 16-bit elements (a head `head_step` elements after the one before); boxes of 64 elements x one
// head x 64 rows.
int pa_map(CUtensorMap *map, bool bf16, const void *base, uint32_t cols, uint32_t heads, uint64_t head_step, uint64_t rows, uint64_t ld) {
  EncodeTiledFn encode = nullptr;
  if (int rc = tc_encode_fn(&encode)) return rc;
  const cuuint64_t dims[3] = {cols, heads, rows}, strides[2] = {head_step * 2, ld * 2};
  const cuuint32_t box[3] = {64, 1, 64}, estr[3] = {1, 1, 1};
  const CUresult r = encode(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(base), dims, strides,
                            box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_error("attention: cuTensorMapEncodeTiled failed with %d (%u columns, %u heads, %llu rows)", (int)r, cols, heads, (unsigned long long)rows);
    return CUTB_ERR_CUDA;
  }
  return CUTB_OK;
}

// |scale| in log2 units, its sign with the queries (a scale of zero: queries of zero)
void pa_set_scale(PaParams *p, float scale) {
  p->scale = scale == 0.f ? 1.f : fabsf(scale) * 1.4426950408889634f;
  p->q_mul = scale == 0.f ? 0.f : (scale < 0.f ? -1.f : 1.f);
}

// Eight pairs at a time: groups of 16 columns that are turned whole or not at all, 16-byte aligned rows
void pa_set_vec(PaParams *p, int mode) {
  auto aligned = [](const void *a) { return reinterpret_cast<uintptr_t>(a) % 16 == 0; };
  p->q_vec = p->ldq % 4 == 0 && p->q_head % 16 == 0 && p->rot % 16 == 0 && (mode != PA_LATENT || p->dim % 16 == 0) && aligned(p->q) &&
             (!p->rot || (aligned(p->cos_t) && aligned(p->sin_t)));
}

template <int MODE, int KP, int VP>
int pa_launch_inst(const CUtensorMap &mk, const CUtensorMap &mr, const CUtensorMap &mv, const PaParams &params, cudaStream_t stream) {
  constexpr uint32_t smem = pa_smem<KP, VP>();
  PaParams p = params;
  pa_set_vec(&p, MODE);
  CUTB_CUDA_TRY(cudaFuncSetAttribute(prefill_attention_kernel<MODE, KP, VP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  CUTB_CUDA_TRY(launch_pdl(prefill_attention_kernel<MODE, KP, VP>, dim3(p.n_heads, (p.n_tokens + p.step - 1) / p.step), dim3(PA_THREADS), smem, stream,
                           mk, mr, mv, p));
  return CUTB_OK;
}

// Tokens per block: two tiles share the keys and hide one another's softmax; one tile where two would leave SMs without work.
uint32_t pa_step(uint32_t n_tokens, uint32_t n_heads, uint32_t sms) {
  return (uint64_t)((n_tokens + 255) / 256) * n_heads >= sms ? 256u : 128u;
}

}  // namespace
}  // namespace cutb
