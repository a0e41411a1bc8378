// Prefill GEMM over dense bf16 weights, C[M, N] = unary(A[M, K] W[N, K]^T + bias), and its 32-bit companion.
//
// dense_gemm_tc_kernel: persistent, warp-specialised tcgen05 kernel.  A CTA tile is 128 tokens x bn weight rows (up to 256);
// tokens are the MMA's M operand (one per tensor-memory lane), weight rows its N operand.  PAIR: two CTAs of a cluster share a
// tile of 256 tokens x bn rows (cta_group::2): each keeps its own 128 tokens' accumulators and copies its own tokens and half
// of the weight rows, a third fewer bytes per product; the first CTA's MMA warp issues for both.
//   warp 0      one lane copies the 64-k stages of both operands by TMA (128-byte swizzle; rows and k past the matrices read as
//               zero) into a ring that fills shared memory;
//   warp 1      allocates tensor memory (two accumulators of BN columns); one lane issues four K = 16 MMAs per stage and
//               commits them to the stage's "empty" barrier, and after the last stage to the accumulator's "full" barrier;
//   warps 2..5  epilogue of the previous tile meanwhile: tcgen05.ld (lane = token, 32 columns at a time), bias, elementwise
//               op, 16-byte stores along the row.
// GROUPED (experts): the rows of A are sorted by expert, expert e's are offsets[e] .. offsets[e + 1] - 1, and they meet its own N
// rows of the stacked weight.  Every CTA derives the list of tiles from the offsets on the device; a tile's copy may run into
// the next expert's rows, whose products are not stored.  Neighbouring outputs may pass through a gated unit (gate, up).
// Few tiles and a long K: the K stages of a tile are shared out over CTAs, partial sums go to the workspace and a second
// kernel adds them in a fixed order and applies the epilogue.
// Every wait is bounded; on expiry the CTA records CUTB_ERR_TIMEOUT in the caller's status word and tells the other CTA of its pair.
// Copies in flight are waited for (bounded; a pair's by its first CTA, before the two part), tensor memory is freed.
//
// dense_gemm_simt_kernel: fp32 fused multiply-adds (bf16 weights are exact in fp32), for the true 32-bit mode.
#include <algorithm>

#include <cuda.h>
#include <cuda_bf16.h>

#include "common.cuh"
#include "dense_common.cuh"
#include "kernels.h"
#include "tcgen05.cuh"

namespace cutb {
namespace {

constexpr int DG_BM = 128, DG_BK = 64, DG_THREADS = 192, DG_MAX_STAGES = 8;
constexpr uint32_t DG_A_BYTES = DG_BM * DG_BK * 2, DG_RING = 216 * 1024;
__host__ __device__ constexpr uint32_t dg_stage_bytes(uint32_t rows) { return DG_A_BYTES + (rows + 7) / 8 * 8 * DG_BK * 2; }  // rows: those a CTA copies

struct DgParams {
  const float *bias;
  void *C;
  float *partial;  // [ksplit][M][N] when K is split
  int *status;
  uint32_t M, K, N, ldc;
  uint32_t tiles_m, tiles_n, ksplit, nk, nk_per, a_box_rows;
  uint32_t bn, stages;  // weight rows of a tile (a multiple of 16, at most 256; pairs: of 32), 64-k stages in shared memory
  int c_bf16, unary;
  const uint32_t *offsets;  // grouped
  uint32_t experts;
  GluParams glu;
};
constexpr uint32_t DG_MAX_EXPERTS = 1024;

struct DgJob {
  uint32_t m0, m_end, n0, w0, k0, nk, z;  // rows m0 .. m_end - 1 are stored; w0 = row of the stacked weight
};

template <bool GROUPED, bool PAIR>
__global__ void __launch_bounds__(DG_THREADS, 1) dense_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a,
                                                                      const __grid_constant__ CUtensorMap map_w, const DgParams p) {
  const uint32_t S = p.stages, BN = p.bn, rows = PAIR ? BN / 2 : BN, STAGE = dg_stage_bytes(rows);
  constexpr uint32_t COLS = 512, TM = PAIR ? 2 * DG_BM : DG_BM;  // tokens of a tile
  const uint32_t rank = PAIR ? blockIdx.x & 1u : 0u, first_job = PAIR ? blockIdx.x / 2 : blockIdx.x, workers = PAIR ? gridDim.x / 2 : gridDim.x;
  extern __shared__ __align__(1024) uint8_t dg_raw[];
  uint8_t *ring = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(dg_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t bars[2 * DG_MAX_STAGES + 4];  // full[S], empty[S], accumulator full[2], accumulator empty[2]
  __shared__ uint32_t tmem_slot, abort_flag;
  __shared__ uint32_t offs[GROUPED ? DG_MAX_EXPERTS + 1 : 1], first_tile[GROUPED ? DG_MAX_EXPERTS + 1 : 1];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t full_u = smem_u32(bars), empty_u = full_u + S * 8, afull_u = empty_u + S * 8, aempty_u = afull_u + 16;
  const uint32_t ring_u = smem_u32(ring);

  if (tid == 0) {
    for (uint32_t s = 0; s < S; ++s) mbar_init(full_u + s * 8, 1), mbar_init(empty_u + s * 8, 1);
    for (int a = 0; a < 2; ++a) mbar_init(afull_u + a * 8, 1), mbar_init(aempty_u + a * 8, PAIR ? 8 : 4);
    abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  if (GROUPED && warp == 2) {  // row tiles before each expert
    uint32_t before = 0;
    for (uint32_t e0 = 0; e0 < p.experts; e0 += 32) {
      const uint32_t e = e0 + lane, lo = min(p.offsets[min(e, p.experts)], p.M), hi = min(p.offsets[min(e + 1, p.experts)], p.M);
      const uint32_t tiles = e < p.experts && hi > lo ? (hi - lo + TM - 1) / TM : 0;
      uint32_t sum = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= (uint32_t)o) sum += v;
      }
      if (e < p.experts) offs[e] = lo, first_tile[e] = before + sum - tiles;
      if (e + 1 == p.experts) offs[e + 1] = hi;
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) first_tile[p.experts] = before;
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) {  // the other CTA's barriers are there
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  }
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  auto give_up = [&]() {
    if (p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
    if constexpr (PAIR) {  // both CTAs of the pair (each stays until the other has come to its end)
#pragma unroll
      for (uint32_t r = 0; r < 2; ++r) {
        uint32_t at;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(&abort_flag)), "r"(r));
        asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(1u) : "memory");
      }
    } else {
      atomicExch(&abort_flag, 1u);
    }
  };
  auto aborted = [&]() { return *reinterpret_cast<volatile uint32_t *>(&abort_flag) != 0; };

  const uint32_t jobs = GROUPED ? first_tile[p.experts] * p.tiles_n : p.tiles_m * p.tiles_n * p.ksplit;
  // job -> token tile fastest (CTAs that run together share weight rows), then weight tile, then share of K; grouped: expert by
  // expert (a role's jobs ascend, so its cursor `e` only moves forward)
  uint32_t e = 0;
  auto job_of = [&](uint32_t j) {
    DgJob b;
    if constexpr (GROUPED) {
      while (j >= first_tile[e + 1] * p.tiles_n) ++e;
      const uint32_t rel = j - first_tile[e] * p.tiles_n, tm = first_tile[e + 1] - first_tile[e];
      b.m0 = offs[e] + rel % tm * TM, b.m_end = offs[e + 1];
      b.n0 = rel / tm * BN, b.w0 = e * p.N + b.n0;
      b.z = b.k0 = 0, b.nk = p.nk;
    } else {
      b.m0 = j % p.tiles_m * TM, b.m_end = p.M;
      b.n0 = b.w0 = j / p.tiles_m % p.tiles_n * BN;
      b.z = j / (p.tiles_m * p.tiles_n);
      b.k0 = b.z * p.nk_per;
      b.nk = min(p.nk_per, p.nk - b.k0);  // (the launcher leaves no share empty)
    }
    return b;
  };

  // The copy and MMA warps run converged, with one elected lane issuing: loop variables stay warp-uniform.  A wait that runs
  // out marks the warp dead; it then runs through its remaining steps without waiting, so that every loop ends.
  if (warp == 0) {
    const bool leader = elect_one();
    uint32_t s = 0, ph = 1;  // (a fresh barrier lets a wait on the phase before its first pass)
    const uint32_t bytes = (p.a_box_rows + rows) * DG_BK * 2 * (PAIR ? 2 : 1);
    bool dead = false;
    for (uint32_t j = first_job; j < jobs; j += workers) {
      const DgJob b = job_of(j);
      for (uint32_t ks = 0; ks < b.nk; ++ks) {
        if (!dead && !mbar_spin_bounded(empty_u + s * 8, ph)) {
          give_up();
          dead = true;
        }
        const uint32_t bar = full_u + s * 8, dst = ring_u + s * STAGE, x = (b.k0 + ks) * DG_BK;
        if (leader && !dead) {
          if constexpr (PAIR) {
            if (rank == 0) mbar_arrive_expect_tx(bar, bytes);  // both CTAs' copies
            const uint32_t to = first_cta(bar);
            tma_load_2d_pair(dst, &map_a, x, b.m0 + rank * DG_BM, to);
            tma_load_2d_pair(dst + DG_A_BYTES, &map_w, x, b.w0 + rank * rows, to);
          } else {
            mbar_arrive_expect_tx(bar, bytes);
            tma_load_2d(dst, &map_a, x, b.m0, bar);
            tma_load_2d(dst + DG_A_BYTES, &map_w, x, b.w0, bar);
          }
        }
        if (++s == S) s = 0, ph ^= 1u;
      }
    }
    // do not retire with copies still landing in shared memory, whoever gives up and when: every stage's last fill (bounded; a stage
    // that was never filled, or whose fill has landed, answers at once, a step that a dead warp left out runs into the small limit).
    // Both CTAs of a pair count on the first one's barriers, which waits for both; the second stays for the cluster barrier below.
    if (rank == 0) {
      for (uint32_t i = 0; i < S; ++i) {
        if (s == 0) s = S, ph ^= 1u;
        --s;
        mbar_drain(full_u + s * 8, ph ^ 1u);
      }
    }
    __syncwarp();
  } else if (warp == 1 && rank == 0) {
    const bool leader = elect_one();
    const uint64_t proto = umma_desc_sw128(0);
    const uint32_t desc_hi = (uint32_t)(proto >> 32), base = (uint32_t)proto + ((ring_u & 0x3FFFFu) >> 4);
    const uint32_t idesc = umma_idesc_bf16(TM, BN);
    uint32_t s = 0, ph = 0, turn = 0;
    bool dead = false;
    for (uint32_t j = first_job; j < jobs; j += workers, ++turn) {
      const uint32_t nk = job_of(j).nk, a = turn & 1, d = tmem + a * 256;
      if (turn >= 2 && !dead && !mbar_spin_bounded(aempty_u + a * 8, ((turn >> 1) - 1) & 1u)) {
        give_up();
        dead = true;
      }
      tc_fence_after();
      for (uint32_t ks = 0; ks < nk; ++ks) {
        if (!dead && !mbar_spin_bounded(full_u + s * 8, ph)) {
          give_up();
          dead = true;
        }
        tc_fence_after();
        const uint32_t at = base + s * (STAGE >> 4), wt = at + (DG_A_BYTES >> 4);
        if (leader) {
          if constexpr (PAIR) {
            umma_pair(d, at, wt, desc_hi, idesc, ks != 0);
            umma_pair(d, at + 2, wt + 2, desc_hi, idesc, 1);
            umma_pair(d, at + 4, wt + 4, desc_hi, idesc, 1);
            umma_pair(d, at + 6, wt + 6, desc_hi, idesc, 1);
            umma_commit_pair(empty_u + s * 8);
          } else {
            umma_f16(d, at, wt, desc_hi, idesc, ks != 0);
            umma_f16(d, at + 2, wt + 2, desc_hi, idesc, 1);
            umma_f16(d, at + 4, wt + 4, desc_hi, idesc, 1);
            umma_f16(d, at + 6, wt + 6, desc_hi, idesc, 1);
            umma_commit(empty_u + s * 8);
          }
        }
        if (++s == S) s = 0, ph ^= 1u;
      }
      if (leader) {
        if constexpr (PAIR) umma_commit_pair(afull_u + a * 8);
        else umma_commit(afull_u + a * 8);
      }
    }
    __syncwarp();
  } else if (warp >= 2) {
    const uint32_t quarter = warp & 3;  // tensor-memory lanes this warp may read
    uint32_t turn = 0;
    for (uint32_t j = first_job; j < jobs; j += workers, ++turn) {
      const DgJob b = job_of(j);
      const uint32_t a = turn & 1;
      uint32_t ok = 1;
      if (lane == 0) ok = !aborted() && mbar_wait_bounded(afull_u + a * 8, (turn >> 1) & 1u);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) {
        if (lane == 0) give_up();
        break;
      }
      tc_fence_after();
      const uint32_t m = b.m0 + rank * DG_BM + quarter * 32 + lane, n_end = min(p.N, b.n0 + BN);
#pragma unroll 1
      for (uint32_t c0 = 0; c0 < BN; c0 += 32) {
        const uint32_t n = b.n0 + c0;
        if (n >= p.N) break;
        uint32_t v[32];
        __syncwarp();  // (lanes without a row have gone ahead)
        tmem_ld32(tmem + ((quarter * 32) << 16) + a * 256 + c0, v);  // (the last piece of an odd number of 16s runs past the tile)
        if (m >= b.m_end) continue;
        const bool whole = n + 32 <= n_end;
        if constexpr (GROUPED) {
          if (p.glu.kind) {  // N is even: outputs 2 i and 2 i + 1 make one
            float y[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) y[i] = glu(p.glu, __uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
            const size_t base = (size_t)m * p.ldc + n / 2;
            if (whole && p.ldc % 8 == 0 && p.c_bf16) {
              uint4 *dst = reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(p.C) + base);
#pragma unroll
              for (int i = 0; i < 2; ++i)
                dst[i] = make_uint4(pack_bf16(y[8 * i], y[8 * i + 1]), pack_bf16(y[8 * i + 2], y[8 * i + 3]),
                                    pack_bf16(y[8 * i + 4], y[8 * i + 5]), pack_bf16(y[8 * i + 6], y[8 * i + 7]));
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (n + 2 * i < n_end) store_out(p.C, p.c_bf16, base + i, y[i]);
            }
            continue;
          }
        } else if (p.ksplit > 1) {
          float *dst = p.partial + ((size_t)b.z * p.M + m) * p.N + n;
          if (whole && p.N % 4 == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i) reinterpret_cast<uint4 *>(dst)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (n + i < n_end) dst[i] = __uint_as_float(v[i]);
          }
          continue;
        }
        float x[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = __uint_as_float(v[i]) + (p.bias && n + i < n_end ? __ldg(p.bias + n + i) : 0.f);
        if (p.unary == CUTB_UNARY_RELU_SQUARE) {
#pragma unroll
          for (int i = 0; i < 32; ++i) x[i] = fmaxf(x[i], 0.f) * fmaxf(x[i], 0.f);
        } else if (p.unary) {
          float (&x8)[32] = x;
          const float none[32] = {};
          apply_epilogue_n<32>(x8, none, CUTB_FUSION_UNARY, p.unary);
        }
        const size_t base = (size_t)m * p.ldc + n;
#pragma unroll
        for (int h = 0; h < 32; h += 16) {
          if (n + h + 16 <= n_end && p.ldc % 8 == 0) {
            if (p.c_bf16) {
              uint4 *dst = reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(p.C) + base + h);
#pragma unroll
              for (int i = 0; i < 2; ++i)
                dst[i] = make_uint4(pack_bf16(x[h + 8 * i], x[h + 8 * i + 1]), pack_bf16(x[h + 8 * i + 2], x[h + 8 * i + 3]),
                                    pack_bf16(x[h + 8 * i + 4], x[h + 8 * i + 5]), pack_bf16(x[h + 8 * i + 6], x[h + 8 * i + 7]));
            } else {
              float4 *dst = reinterpret_cast<float4 *>(reinterpret_cast<float *>(p.C) + base + h);
#pragma unroll
              for (int i = 0; i < 4; ++i) dst[i] = make_float4(x[h + 4 * i], x[h + 4 * i + 1], x[h + 4 * i + 2], x[h + 4 * i + 3]);
            }
          } else {
#pragma unroll
            for (int i = h; i < h + 16; ++i)
              if (n + i < n_end) store_out(p.C, p.c_bf16, base + i, x[i]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR)
          asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(first_cta(aempty_u + a * 8)) : "memory");
        else
          mbar_arrive(aempty_u + a * 8);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) {  // nobody leaves while the other may still signal it or use its shared memory
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  }
  if (warp == 1) {
    tc_fence_after();
    if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
  }
}

__global__ void __launch_bounds__(256) dense_splitk_reduce_kernel(const DgParams p) {
  const size_t idx = (size_t)blockIdx.x * 256 + threadIdx.x, total = (size_t)p.M * p.N;
  if (idx >= total) return;
  const uint32_t m = (uint32_t)(idx / p.N), n = (uint32_t)(idx % p.N);
  float sum = 0.f;
#pragma unroll 4
  for (uint32_t z = 0; z < p.ksplit; ++z) sum += p.partial[z * total + idx];
  store_out(p.C, p.c_bf16, (size_t)m * p.ldc + n, dense_unary(sum + (p.bias ? __ldg(p.bias + n) : 0.f), p.unary));
}

// 64 x 64 outputs per block of 256 threads, 4 x 4 per thread, k in steps of 16.  blockIdx.z = product of a batch; with `offsets`
// blockIdx.y = tile of an expert's rows.
struct DsParams {
  const void *A;
  const __nv_bfloat16 *W;
  const float *bias;
  void *C;
  uint32_t lda, ldw, ldc, M, N, K, a_batch, c_batch;
  int c_bf16, unary;
  const uint32_t *offsets;
  uint32_t experts;
  GluParams glu;
};

template <typename TA> __global__ void __launch_bounds__(256) dense_gemm_simt_kernel(const DsParams p) {
  __shared__ __align__(16) float as[16][64 + 4], ws[16][64 + 4];
  __shared__ uint32_t where[3];  // expert, first row, end of its rows
  pdl_enter();
  const uint32_t tid = threadIdx.x, tx = tid % 16, ty = tid / 16, n0 = blockIdx.x * 64, N = p.N, K = p.K, lda = p.lda, ldw = p.ldw;
  uint32_t m0 = blockIdx.y * 64, M = p.M;
  const TA *A = reinterpret_cast<const TA *>(p.A) + (size_t)blockIdx.z * p.a_batch;
  const __nv_bfloat16 *W = p.W + (size_t)blockIdx.z * N * ldw;
  if (p.offsets) {
    if (tid == 0) {
      uint32_t before = 0, e = 0, lo = 0, hi = 0;
      for (; e < p.experts; ++e) {
        lo = min(p.offsets[e], M), hi = min(p.offsets[e + 1], M);
        const uint32_t tiles = hi > lo ? (hi - lo + 63) / 64 : 0;
        if (blockIdx.y < before + tiles) break;
        before += tiles;
      }
      where[0] = e, where[1] = lo + (blockIdx.y - before) * 64, where[2] = hi;
    }
    __syncthreads();
    if (where[0] >= p.experts) return;  // (the grid is an upper bound)
    m0 = where[1], M = where[2];
    W += (size_t)where[0] * N * ldw;
  }
  float acc[4][4] = {};
  for (uint32_t k0 = 0; k0 < K; k0 += 16) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t r = tid / 16 + 16 * i, k = k0 + tid % 16;
      as[tid % 16][r] = m0 + r < M && k < K ? (float)A[(size_t)(m0 + r) * lda + k] : 0.f;
      ws[tid % 16][r] = n0 + r < N && k < K ? __bfloat162float(W[(size_t)(n0 + r) * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const float4 a = *reinterpret_cast<const float4 *>(&as[k][ty * 4]), w = *reinterpret_cast<const float4 *>(&ws[k][tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t m = m0 + ty * 4 + i, n = n0 + tx * 4;
    if (m >= M) continue;
    const size_t at = (size_t)m * p.ldc + (size_t)blockIdx.z * p.c_batch;
    if (p.glu.kind) {
#pragma unroll
      for (int j = 0; j < 4; j += 2)
        if (n + j < N) store_out(p.C, p.c_bf16, at + (n + j) / 2, glu(p.glu, acc[i][j], acc[i][j + 1]));
      continue;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < N) store_out(p.C, p.c_bf16, at + n + j, dense_unary(acc[i][j] + (p.bias ? __ldg(p.bias + n + j) : 0.f), p.unary));
  }
}

struct DgPlan {
  uint32_t bn, tiles_m, tiles_n, ksplit, nk, nk_per;
  bool pair;
};

// Pairs of CTAs that run at once (0: none, or no device)
uint32_t dg_pairs() {
  static uint32_t known[64] = {};  // per device: pairs + 1
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (!known[dev]) {
    const auto kernel = dense_gemm_tc_kernel<false, true>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2), cfg.blockDim = dim3(DG_THREADS), cfg.dynamicSmemBytes = 1024 + DG_RING;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(1024 + DG_RING)) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 0) {
      (void)cudaGetLastError();
      n = 0;
    }
    known[dev] = (uint32_t)n + 1;
  }
  return known[dev] - 1;
}

// The tile (width, one CTA's or a pair's) by the time of its waves.  Measured, relative: a 64-k stage of a wave of tiles; what a
// pair's start costs more.  A pair copies two thirds of the bytes per product, so it wins wherever its 256 tokens are filled; 256
// rows are slower than their share (six stages of copies in flight instead of seven, and a longer epilogue).  One CTA x 256 rows
// (all there was) -> now, us: 2048 x 4096 x 14336 181 -> 156 (pairs x 224), x 12288 177 -> 138 (224), x 6144 111 -> 80 (192),
// x 4096 65 -> 54 (256), 2048 x 14336 x 4096 186 -> 170 (256), 1501 x 4096 x 4096 59 -> 43 (192), 512 x 4096 x 14336 62 -> 50 (224);
// 2048 x 1024 x 2048 stays (16.9 against 19.0: the pair's start).  `row_tiles`: row tiles of a given height, as they are likely to fall.
// Grouped: 240 rows gain nothing over 256 (16 experts of 200 tokens x 4: 98 against 97 us).
template <class Tiles> void dg_width(uint32_t N, uint32_t nk, uint32_t sms, uint32_t pairs, bool grouped, Tiles row_tiles, DgPlan *pl) {
  static const struct { uint32_t bn, cost; } one[] = {{256, 140}, {240, 138}, {224, 125}, {208, 122}, {192, 112}, {128, 97}, {64, 90}},
                                             two[] = {{256, 115}, {224, 100}, {192, 92}, {160, 90}, {128, 86}};
  constexpr uint64_t PAIR_START = 570;
  uint64_t best = ~0ull;
  auto consider = [&](uint32_t bn, uint32_t cost, bool pair) {
    const uint32_t tm = row_tiles(pair ? 2 * DG_BM : DG_BM), tn = (N + bn - 1) / bn, workers = pair ? pairs : sms;
    const uint64_t t = (((uint64_t)tm * tn + workers - 1) / workers) * nk * cost + (pair ? PAIR_START : 0);
    if (t < best) best = t, pl->bn = bn, pl->tiles_m = tm, pl->tiles_n = tn, pl->pair = pair;
  };
  for (const auto &k : one)
    if (!grouped || k.bn != 240) consider(k.bn, k.cost, false);
  if (pairs)
    for (const auto &k : two) consider(k.bn, k.cost, true);
}
// K split when even narrow tiles leave most SMs idle.
DgPlan dg_plan(const cutb_dense_desc &d, uint32_t sms) {
  DgPlan b{};
  const uint32_t tm = (d.M + DG_BM - 1) / DG_BM;
  b.nk = (d.K + DG_BK - 1) / DG_BK;
  dg_width(d.N, b.nk, sms, d.M > DG_BM ? dg_pairs() : 0, false, [&](uint32_t rows) { return (d.M + rows - 1) / rows; }, &b);
  if (tm * ((d.N + 127) / 128) * 2 <= sms && b.nk >= 16) {
    b.bn = 128, b.pair = false, b.tiles_m = tm;
    b.tiles_n = (d.N + 127) / 128;
    uint32_t want = sms / (b.tiles_m * b.tiles_n);
    if (want > b.nk / 4) want = b.nk / 4;
    if (want > 16) want = 16;
    if (want < 1) want = 1;
    b.nk_per = (b.nk + want - 1) / want;
    b.ksplit = (b.nk + b.nk_per - 1) / b.nk_per;
  } else {
    b.ksplit = 1, b.nk_per = b.nk;
  }
  return b;
}

template <bool GROUPED, bool PAIR> int dg_launch_inst(const CUtensorMap &ma, const CUtensorMap &mw, const DgParams &p, uint32_t workers, cudaStream_t stream) {
  static bool configured[64] = {};
  int dev = 0;
  CUTB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    CUTB_CUDA_TRY(cudaFuncSetAttribute(dense_gemm_tc_kernel<GROUPED, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(1024 + DG_RING)));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  const uint32_t jobs = p.tiles_m * p.tiles_n * p.ksplit;  // (grouped: an upper bound)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((jobs < workers ? jobs : workers) * (PAIR ? 2 : 1));
  cfg.blockDim = dim3(DG_THREADS);
  // (what the ring takes and no more: the rest stays L1; 178 x 14336 x 4096 45.5 us with all of it, 44.3 so)
  cfg.dynamicSmemBytes = 1024 + p.stages * dg_stage_bytes(PAIR ? p.bn / 2 : p.bn);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr, cfg.numAttrs = PAIR ? 1 : 0;
  CUTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, dense_gemm_tc_kernel<GROUPED, PAIR>, ma, mw, p));
  return CUTB_OK;
}
template <bool GROUPED> int dg_launch(const CUtensorMap &ma, const CUtensorMap &mw, DgParams p, const DgPlan &pl, uint32_t sms, cudaStream_t stream) {
  p.bn = pl.bn, p.stages = DG_RING / dg_stage_bytes(pl.pair ? pl.bn / 2 : pl.bn);
  if (p.stages > DG_MAX_STAGES) p.stages = DG_MAX_STAGES;
  return pl.pair ? dg_launch_inst<GROUPED, true>(ma, mw, p, dg_pairs(), stream) : dg_launch_inst<GROUPED, false>(ma, mw, p, sms, stream);
}

}  // namespace

uint64_t dense_gemm_tc_workspace(const cutb_dense_desc &d) {
  DeviceInfo di;
  const uint32_t sms = get_device_info(&di) == CUTB_OK ? (uint32_t)di.sm_count : 148u;
  const DgPlan pl = dg_plan(d, sms);
  return pl.ksplit > 1 ? (uint64_t)pl.ksplit * d.M * d.N * sizeof(float) : 0;
}

bool dense_gemm_tc_supported(const cutb_dense_desc &d) {
  return d.a_dtype == CUTB_BF16 && d.lda % 8 == 0 && reinterpret_cast<uintptr_t>(d.A) % 16 == 0;
}

int dense_gemm_tc_launch(const cutb_dense_desc &d, cudaStream_t stream) {
  DeviceInfo di;
  if (int rc = get_device_info(&di)) return rc;
  DgPlan pl = dg_plan(d, (uint32_t)di.sm_count);
  if (pl.ksplit > 1 && (!d.workspace || d.workspace_bytes < (uint64_t)pl.ksplit * d.M * d.N * sizeof(float) ||
                        reinterpret_cast<uintptr_t>(d.workspace) % 16 != 0))
    pl.ksplit = 1, pl.nk_per = pl.nk;
  DgParams p{};
  p.bias = d.bias, p.C = d.C, p.status = d.status, p.M = d.M, p.K = d.K, p.N = d.N, p.ldc = d.ldc;
  p.partial = pl.ksplit > 1 ? reinterpret_cast<float *>(d.workspace) : nullptr;
  p.tiles_m = pl.tiles_m, p.tiles_n = pl.tiles_n, p.ksplit = pl.ksplit, p.nk = pl.nk, p.nk_per = pl.nk_per;
  p.a_box_rows = d.M >= DG_BM ? DG_BM : (d.M + 7) / 8 * 8;  // (rows of the tile that are not copied only feed outputs that are not stored)
  p.c_bf16 = d.c_dtype == CUTB_BF16, p.unary = d.unary_op;
  CUtensorMap ma, mw;
  if (int rc = make_tmap_sw128(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, d.A, d.M, d.K, (uint64_t)d.lda * 2, p.a_box_rows)) return rc;
  if (int rc = make_tmap_sw128(&mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, d.W, d.N, d.K, (uint64_t)d.ldw * 2, pl.pair ? pl.bn / 2 : pl.bn)) return rc;
  const int rc = dg_launch<false>(ma, mw, p, pl, (uint32_t)di.sm_count, stream);
  if (rc != CUTB_OK || pl.ksplit <= 1) return rc;
  dense_splitk_reduce_kernel<<<(unsigned)(((size_t)d.M * d.N + 255) / 256), 256, 0, stream>>>(p);
  CUTB_CUDA_TRY(cudaGetLastError());
  return CUTB_OK;
}

int moe_gemm_tc_launch(const cutb_moe_desc &d, cudaStream_t stream) {
  DeviceInfo di;
  if (int rc = get_device_info(&di)) return rc;
  const uint32_t sms = (uint32_t)di.sm_count, rows = d.n_tokens * d.top;
  DgParams p{};
  p.C = d.C, p.status = d.status, p.M = rows, p.K = d.K, p.N = d.N, p.ldc = (uint32_t)d.ldc;
  p.offsets = d.offsets, p.experts = d.experts, p.glu = GluParams{d.glu, d.alpha, d.beta, d.limit};
  p.c_bf16 = d.c_dtype == CUTB_BF16;
  p.nk = p.nk_per = (d.K + DG_BK - 1) / DG_BK, p.ksplit = 1;
  p.a_box_rows = rows >= DG_BM ? DG_BM : (rows + 7) / 8 * 8;
  // Row tiles: an expert in use has one at least; of two guesses, that experts are evenly used and that the last tile of each is half
  // full on average, the one with fewer tiles.  (Counted as rows / n + used / 2, pairs seemed to halve the tiles of experts with less than
  // a tile each, and the last wave went uncounted.)  us, counted so -> now, beside single CTAs x 256 rows: 16 experts, 200 tokens x 4,
  // 4096 -> 2 x 2048 gated 110 -> 97 (97), 1501 tokens x 4 215 -> 194 (189; its down projection 109 -> 102 (111)), 8 experts, 700 tokens x 2,
  // 1024 -> 2 x 1024 21.5 -> 14.8 (14.8), 2000 tokens x 4, 2560 -> 2 x 2048 130 -> 126 (138), 1500 tokens x 2, 4096 -> 2 x 2048 103 -> 94 (94).
  const uint32_t used = d.experts < rows ? d.experts : rows, each = (rows + used - 1) / used;
  DgPlan pl{};
  dg_width(d.N, p.nk, sms, rows > DG_BM ? dg_pairs() : 0, true, [&](uint32_t n) {
    return std::max(used, std::min(used * ((each + n - 1) / n), (2 * rows + used * n + 2 * n - 1) / (2 * n)));
  }, &pl);
  p.tiles_m = rows / (pl.pair ? 2 * DG_BM : DG_BM) + used, p.tiles_n = pl.tiles_n;
  CUtensorMap ma, mw;
  if (int rc = make_tmap_sw128(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, d.A, rows, d.K, d.lda * 2, p.a_box_rows)) return rc;
  if (int rc = make_tmap_sw128(&mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, d.W, d.experts * d.N, d.K, (uint64_t)d.ldw * 2, pl.pair ? pl.bn / 2 : pl.bn)) return rc;
  return dg_launch<true>(ma, mw, p, pl, sms, stream);
}

namespace {
int ds_launch(const DsParams &p, bool a_bf16, uint32_t tiles_m, uint32_t batch, cudaStream_t stream) {
  const dim3 grid((p.N + 63) / 64, tiles_m, batch);
  if (a_bf16) CUTB_CUDA_TRY(launch_pdl(dense_gemm_simt_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, p));
  else CUTB_CUDA_TRY(launch_pdl(dense_gemm_simt_kernel<float>, grid, dim3(256), 0, stream, p));
  return CUTB_OK;
}
}  // namespace

int dense_gemm_simt_launch(const cutb_dense_desc &d, cudaStream_t stream) {
  DsParams p{};
  p.A = d.A, p.W = reinterpret_cast<const __nv_bfloat16 *>(d.W), p.bias = d.bias, p.C = d.C;
  p.lda = d.lda, p.ldw = d.ldw, p.ldc = d.ldc, p.M = d.M, p.N = d.N, p.K = d.K, p.a_batch = d.a_batch, p.c_batch = d.c_batch;
  p.c_bf16 = d.c_dtype == CUTB_BF16, p.unary = d.unary_op;
  return ds_launch(p, d.a_dtype == CUTB_BF16, (d.M + 63) / 64, d.batch ? d.batch : 1, stream);
}

int moe_gemm_simt_launch(const cutb_moe_desc &d, cudaStream_t stream) {
  DsParams p{};
  const uint32_t rows = d.n_tokens * d.top, used = d.experts < rows ? d.experts : rows;
  p.A = d.A, p.W = reinterpret_cast<const __nv_bfloat16 *>(d.W), p.C = d.C;
  p.lda = (uint32_t)d.lda, p.ldw = d.ldw, p.ldc = (uint32_t)d.ldc, p.M = rows, p.N = d.N, p.K = d.K;
  p.c_bf16 = d.c_dtype == CUTB_BF16, p.offsets = d.offsets, p.experts = d.experts, p.glu = GluParams{d.glu, d.alpha, d.beta, d.limit};
  return ds_launch(p, d.a_dtype == CUTB_BF16, rows / 64 + used, 1, stream);
}

}  // namespace cutb
