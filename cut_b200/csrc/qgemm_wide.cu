// Tensor-core GEMM over native GGUF blocks for many activation rows (prompts): whole tiles, weights through tensor memory.
//
// C[m, n] = epilogue(sum_k A[m, k] * dequant(W)[n, k]); fp16 operands, the dequantised weight rounded to fp16 as in qgemm_tc.cu, fp32
// accumulation.
//
//  * A pair of CTAs (cta_group::2) takes tiles of 256 weight rows x T activation rows one after the other, K whole: nothing is shared and no
//    scratch is needed.  T (32 to 256) is chosen so that the tiles come out in full waves.
//  * Either CTA widens its 128 weight rows as in qgemm_few.cu: a thread takes a row, widens 64 k in registers and stores them to its lane of
//    tensor memory, the MMA's A operand.  (Widened into shared memory, as qgemm_tc.cu does, they are written there and read from there
//    once per 256 activation rows, beside the activations; its 512 rows a tile are bound by that, and two waves of 112 or 224 tiles leave
//    a quarter of the SMs idle.)
//  * Activations are the B operand, half of the rows in either CTA's shared memory, so that a byte of them leaves L2 once for 256 weight
//    rows: alone, a CTA's tiles ran into some 9 TB/s from L2 (Q4_K 512 x 4096 x 28672: 111 us with 128 x 256 tiles, 102 by pairs).
//  * One warp copies raw weights (256 k of 128 rows a box), one the activations, one of the first CTA issues the MMAs: 128 k a wait and a
//    commit, whose cost (some 600 cycles) bounded pieces of 64 k.  16 converter warps, four groups, the g-th 64 k of every unit each.
//  * Up to 128 rows there are two accumulators.  A tile is finished by the converters once a unit of the next one is on its way.
//
// Bound by the tensor cores (69 % busy at 512 rows) and, up to some 160 rows a tile, by the chain of the conversion: load, widen, store, hand over
// (a unit of 256 k takes 0.9 us with 64 rows, 1.4 us with 256, of which the MMAs need 1.1; issue slots are half busy).  us with the weights
// in L2, what ran before -> here: Q4_K 512 x 4096 x 14336 62 -> 54 (cycled weights 70 -> 64), x 28672 120 -> 103, x 6144 45 -> 28, x 4096
// 34 -> 25; Q8_0 512 x 4096 x 11008 64 -> 46; Q4_0 130 x 4096 x 11008 40 -> 24.  Two issuers, converters that take 128 k of every other unit, and an epilogue that holds the tile in registers
// (it spilled) gained nothing.
//
// Every wait is bounded; on expiry CUTB_ERR_TIMEOUT is recorded.  Both CTAs stay until copies, MMAs and signals between them are through.
#include "kernels.h"
#include "tmem_weights.cuh"

namespace cutb {
namespace {

constexpr uint32_t WG_GROUPS = 4, WG_WARPS = 4 * WG_GROUPS, WG_THREADS = (WG_WARPS + 3) * 32;  // (copies of weights, of activations, MMAs)
constexpr uint32_t WG_PIECES = 2, WG_SLOTS = 4;  // pieces (128 k) of a unit; of widened weights in tensor memory (64 columns each)
constexpr uint32_t WG_MAX_T = 256, WG_TWO_T = 128;  // activation rows of a tile; those that leave room for two accumulators
__host__ __device__ constexpr uint32_t wg_stages(int fmt) { return fmt == CUTB_Q8_0 ? 2u : 3u; }

struct WgParams {
  float *C;
  uint32_t ldc;
  const float *D;
  uint32_t ldd;
  uint32_t M, K, N;
  uint32_t T, blocks, tiles;  // activation rows of a tile, tiles side by side over M, all tiles
  uint32_t act_stages;        // pieces (128 k) of activations in shared memory, at most WG_SLOTS
  int fusion_type, fusion_op, glu;
  int *status;
};

template <int FMT> __global__ void __launch_bounds__(WG_THREADS, 1)
    qgemm_wide_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const WgParams p) {
  constexpr uint32_t CHUNK = granule_bytes(FMT), WB = ft_unit(FMT), CW = WG_WARPS, S = wg_stages(FMT), PP = WG_PIECES, SLOTS = WG_SLOTS;
  extern __shared__ __align__(128) uint8_t wg_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(wg_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint32_t tmem_s;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, T = p.T, SA = p.act_stages, ACT = T * 128;  // (of a piece: 128 k of half of the rows)
  const uint32_t ND = T <= WG_TWO_T ? 2 : 1;  // accumulators
  const uint32_t ring_u = smem_u32(smem), acts_u = ring_u + S * WB;
  const uint32_t wfull = acts_u + SA * ACT, wempty = wfull + S * 8, afull = wempty + S * 8, xfull = afull + SA * 8, used = xfull + SLOTS * 8,
                 dfull = used + SLOTS * 8, dempty = dfull + 16, idle = dempty + 16;
  const uint32_t worker = blockIdx.x >> 1, workers = gridDim.x >> 1, rank = blockIdx.x & 1u;
  const uint32_t nk = p.K / 256, mine = (p.tiles - worker + workers - 1) / workers, n = mine * nk;  // tiles and units of this pair

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (warp == CW) {
    if (lane == 0) {
      for (uint32_t s = 0; s < S; ++s) mbar_init(wfull + s * 8, 1), mbar_init(wempty + s * 8, CW);
      for (uint32_t s = 0; s < SA; ++s) mbar_init(afull + s * 8, 1);
      for (uint32_t s = 0; s < SLOTS; ++s) mbar_init(xfull + s * 8, 16), mbar_init(used + s * 8, 1);  // (a piece: 8 warps of each CTA)
      for (uint32_t s = 0; s < 2; ++s) mbar_init(dfull + s * 8, 1), mbar_init(dempty + s * 8, 2 * CW);
      mbar_init(idle, 1);
      fence_mbar_init();
    }
    __syncwarp();
  } else if (warp == CW + 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");  // the other CTA's barriers are there
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  tc_fence_after();
  const uint32_t tmem = tmem_s, tmem_d = tmem + SLOTS * 64;

  if (warp == CW) {
    // ---- copies of the raw weights, a unit (128 rows x 256 k) each; a caller of this many rows may have written them just before ----
    const bool leader = elect_one();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint32_t slot = 0, ph = 1, issued = 0;
    for (uint32_t tile = worker; tile < p.tiles; tile += workers)
      for (uint32_t k = 0; k < nk; ++k) {
        if (issued >= S && !warp_wait(wempty + slot * 8, ph)) {
          if (leader && p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
          tile = p.tiles;
          break;
        }
        if (leader) {
          mbar_arrive_expect_tx(wfull + slot * 8, WB);
          tma_load_2d(ring_u + slot * WB, &map_w, k * (CHUNK / 4), (tile / p.blocks * 2 + rank) * FT_ROWS, wfull + slot * 8);
        }
        ++issued;
        if (++slot == S) slot = 0, ph ^= 1u;
      }
    // stay until every copy issued here has landed (bounded)
    for (uint32_t j = issued > S ? issued - S : 0; j < issued; ++j) mbar_drain(wfull + (j % S) * 8, (j / S) & 1u);
  } else if (warp == CW + 1) {
    // ---- copies of the activations, a piece each: half of the tile's rows to either CTA, counted on the first one's barrier ----
    const bool leader = elect_one();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint32_t slot = 0, us = 0, up = 0, issued = 0;
    for (uint32_t tile = worker; tile < p.tiles; tile += workers)
      for (uint32_t c = 0; c < nk * PP; ++c) {
        if (issued >= SA) {  // piece `issued` - SA has been used
          if (!warp_wait(used + us * 8, up)) {
            if (leader && p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
            tile = p.tiles;
            break;
          }
          if (++us == SLOTS) us = 0, up ^= 1u;
        }
        if (leader) {
          if (rank == 0) mbar_arrive_expect_tx(afull + slot * 8, 2 * ACT);
          const uint32_t to = first_cta(afull + slot * 8), y = tile % p.blocks * T + rank * (T / 2);
          tma_load_2d_pair(acts_u + slot * ACT, &map_a, c * 128, y, to);
          tma_load_2d_pair(acts_u + slot * ACT + T * 64, &map_a, c * 128 + 64, y, to);
        }
        ++issued;
        if (++slot == SA) slot = 0;
      }
    // (the first CTA waits for both; the second stays for the barrier of the cluster)
    for (uint32_t j = issued > SA ? issued - SA : 0; j < issued && rank == 0; ++j) mbar_drain(afull + (j % SA) * 8, (j / SA) & 1u);
  } else if (warp == CW + 2) {
    // ---- MMAs: 256 weight rows (tensor memory of both CTAs) x T activation rows (shared memory), 16 k each ----
    if (rank == 0) {
      const bool leader = elect_one();
      const uint64_t proto = umma_desc_sw128(0);
      const uint32_t desc_hi = (uint32_t)(proto >> 32), b_lo0 = (uint32_t)proto + ((acts_u & 0x3FFFFu) >> 4), idesc = umma_idesc_f16(256, T);
      uint32_t as = 0, ap = 0, xs = 0, xp = 0;
      bool ok = true, early = false;  // early: the next piece's operands were there before this one's MMAs were issued
      for (uint32_t i = 0; i < mine && ok; ++i) {
        const uint32_t buf = ND == 2 ? i & 1 : 0, turn = ND == 2 ? i >> 1 : i, d = tmem_d + buf * WG_TWO_T;
        if (turn) ok = __all_sync(0xffffffffu, mbar_spin_bounded(dempty + buf * 8, (turn - 1) & 1u));
        for (uint32_t c = 0; c < nk * PP && ok; ++c) {
          if (!__all_sync(0xffffffffu, early)) {
            ok = mbar_spin_bounded(afull + as * 8, ap) && mbar_spin_bounded(xfull + xs * 8, xp);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
          }
          tc_fence_after();
          const uint32_t a = tmem + xs * 64, b = b_lo0 + as * (ACT / 16), bar = used + xs * 8;
          if (++as == SA) as = 0, ap ^= 1u;
          if (++xs == SLOTS) xs = 0, xp ^= 1u;
          const bool acts = mbar_test(afull + as * 8, ap), widened = mbar_test(xfull + xs * 8, xp);
          if (leader) {
#pragma unroll
            for (uint32_t e = 0; e < 8; ++e) umma_ts_pair(d, a + 8 * e, b + (e >> 2) * T * 4 + 2 * (e & 3), desc_hi, idesc, e ? 1u : (uint32_t)(c != 0));
            umma_commit_pair(bar);
          }
          early = acts && widened;
        }
        if (ok && leader) umma_commit_pair(dfull + buf * 8);
      }
      if (!ok && leader && p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
      if (leader) umma_commit_pair(idle);
      __syncwarp();
    }
  } else {
    // ---- converters: one weight row per thread; group g widens the g-th chunk (64 k) of every unit ----
    const uint32_t quarter = (warp & 3) * 32, row = quarter + lane, group = warp >> 2;
    const uint32_t to = tmem + (quarter << 16) + group * 32;
    uint32_t ws = 0, wp = 0, k = 0;
    bool dead = false;
    auto expect = [&](uint32_t bar, uint32_t parity) {
      if (!dead && !warp_wait(bar, parity)) {
        dead = true;
        if (lane == 0 && p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
      }
    };
    auto arrive_first = [&](uint32_t bar) { asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(first_cta(bar)) : "memory"); };
    // the pair's i-th tile: out of the accumulator, through the fused operation, to C
    auto finish = [&](uint32_t i) {
      const uint32_t at = worker + i * workers, buf = ND == 2 ? i & 1 : 0, turn = ND == 2 ? i >> 1 : i;
      expect(dfull + buf * 8, turn & 1u);
      tc_fence_after();
      if (i == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
      const uint32_t nn = (at / p.blocks * 2 + rank) * FT_ROWS + row, m0 = at % p.blocks * T;
      const bool n_ok = nn < p.N;
#pragma unroll 1
      for (uint32_t c = group * 8; c < T; c += WG_GROUPS * 8) {
        uint32_t v[8];
        __syncwarp();
        tmem_ld8(tmem_d + (quarter << 16) + buf * WG_TWO_T + c, v);
        const uint32_t m = m0 + c;
        if (m >= p.M) break;
        float x[8], dv[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(v[e]), dv[e] = 0.f;
        if (p.glu) {  // gate and up rows are neighbouring lanes: the even one stores the pair's output
          float up[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) up[e] = __shfl_xor_sync(0xffffffffu, x[e], 1);
          apply_epilogue_n<8>(x, dv, CUTB_FUSION_UNARY, p.fusion_op);
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (n_ok && !(lane & 1) && m + e < p.M) p.C[(size_t)(m + e) * p.ldc + (nn >> 1)] = x[e] * up[e];
          continue;
        }
        if (p.fusion_type != CUTB_FUSION_NONE) {
          if (p.fusion_type == CUTB_FUSION_BINARY) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (n_ok && m + e < p.M) dv[e] = p.D[(size_t)(m + e) * p.ldd + nn];
          }
          apply_epilogue_n<8>(x, dv, p.fusion_type, p.fusion_op);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (n_ok && m + e < p.M) p.C[(size_t)(m + e) * p.ldc + nn] = x[e];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_first(dempty + buf * 8);
    };
    uint32_t done = 0;
    expect(wfull, 0);
    for (uint32_t j = 0; j < n; ++j) {
      // (barriers are asked early, so that an answer is there when it is needed)
      const uint32_t xs = (group >> 1) + PP * (j & 1), xp = (j >> 1) & 1u;
      const bool room = mbar_test(used + xs * 8, xp ^ 1u);
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
      if (!ready) expect(used + xs * 8, xp ^ 1u);
      tc_fence_after();
      const uint32_t at = to + 128 * (j & 1);
      tmem_st16(at, *reinterpret_cast<const uint32_t (*)[16]>(&h[0]));
      tmem_st16(at + 16, *reinterpret_cast<const uint32_t (*)[16]>(&h[16]));
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_first(xfull + xs * 8);
      // a tile is finished when the next one's first unit is on its way
      if (k == 0 && j) finish(done++);
      if (++k == nk) k = 0;
      if (more && !ready) expect(wfull + ws * 8, wp);
    }
    finish(done);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == CW + 2) mbar_drain(idle, 0);  // no MMA is under way when the tensor memory goes back, and no signal when a CTA ends
  __syncthreads();
  asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if (warp == CW + 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

template <int FMT> constexpr size_t wg_fixed() { return 1024 + wg_stages(FMT) * (ft_unit(FMT) + 16) + WG_SLOTS * 16 + 40; }

// CTA pairs that the device runs at a time
uint32_t wg_pairs() {
  static uint32_t known[64] = {};  // per device: pairs + 1
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (!known[dev]) {
    const auto kernel = qgemm_wide_kernel<CUTB_Q8_0>;
    constexpr size_t smem = wg_fixed<CUTB_Q8_0>() + WG_SLOTS * (WG_MAX_T * 128 + 8);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2), cfg.blockDim = dim3(WG_THREADS), cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 0) {
      (void)cudaGetLastError();
      n = 0;
    }
    known[dev] = (uint32_t)n + 1;
  }
  return known[dev] - 1;
}

template <int FMT> int wg_launch(const cutb_qmatmul_desc &d, const void *a16, uint64_t stride, WgParams p, const DeviceInfo &di, cudaStream_t stream) {
  static bool configured[64] = {};  // per device: the attribute is set once on each
  const size_t room = di.smem_optin - 512;
  int dev = 0;
  CUTB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    CUTB_CUDA_TRY(cudaFuncSetAttribute(qgemm_wide_kernel<FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  const size_t fit = (room - wg_fixed<FMT>()) / (p.T * 128 + 8);
  p.act_stages = (uint32_t)(fit > WG_SLOTS ? WG_SLOTS : fit);
  CUtensorMap map_w, map_a;
  if (int rc = ft_map(&map_w, d)) return rc;
  if (int rc = make_tmap_sw128(&map_a, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a16, d.M, d.K, stride, p.T / 2)) return rc;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = d.flags & CUTB_FLAG_NO_OVERLAP ? 1 : 2;
  cfg.stream = stream;
  const uint32_t pairs = wg_pairs();
  cfg.gridDim = dim3(2 * (p.tiles < pairs ? p.tiles : pairs));
  cfg.blockDim = dim3(WG_THREADS);
  cfg.dynamicSmemBytes = wg_fixed<FMT>() + p.act_stages * (p.T * 128 + 8);
  CUTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, qgemm_wide_kernel<FMT>, map_w, map_a, p));
  return CUTB_OK;
}

}  // namespace

// The height of the tiles by the time of their waves (us): a unit, a tile's way out of the accumulator, and the launch.  Measured on the three
// formats at 64 to 2048 rows; units of up to 128 rows take what the conversion takes, larger ones the tensor cores and the activations
// through L2.
uint32_t qgemm_wide_plan(const cutb_qmatmul_desc &d, float *time) {
  static const float unit[8] = {0.89f, 0.89f, 0.93f, 0.95f, 0.98f, 1.12f, 1.17f, 1.36f};  // by rows / 32
  if (d.layout != CUTB_LAYOUT_GGUF_BLOCKS || d.K == 0 || d.K % 256 != 0) return 0;
  const uint32_t pairs = wg_pairs(), wide = (d.N + 2 * FT_ROWS - 1) / (2 * FT_ROWS), nk = d.K / 256;
  if (!pairs) return 0;
  uint32_t best = 0;
  for (uint32_t i = 8; i >= 1; --i) {
    const uint32_t T = 32 * i;
    const uint64_t tiles = (uint64_t)wide * ((d.M + T - 1) / T), waves = (tiles + pairs - 1) / pairs;
    if (tiles * nk > 0x7fffffffull) continue;
    const float t = 5.f + (float)waves * ((float)nk * unit[i - 1] + 0.009f * (float)T);
    if (!best || t < *time) best = T, *time = t;
  }
  return best;
}

int qgemm_wide_launch(const cutb_qmatmul_desc &d, const void *a16, uint64_t stride, uint32_t T, cudaStream_t stream) {
  DeviceInfo di;
  if (int rc = get_device_info(&di)) return rc;
  WgParams p{};
  p.C = d.C, p.ldc = d.ldc, p.D = d.D, p.ldd = d.ldd, p.M = d.M, p.K = d.K, p.N = d.N;
  p.T = T, p.blocks = (d.M + T - 1) / T, p.tiles = (d.N + 2 * FT_ROWS - 1) / (2 * FT_ROWS) * p.blocks;
  p.fusion_type = d.fusion_type, p.fusion_op = d.fusion_op, p.glu = d.flags & CUTB_FLAG_GLU_PAIRS ? 1 : 0, p.status = d.status;
  switch (d.format) {
    case CUTB_Q8_0: return wg_launch<CUTB_Q8_0>(d, a16, stride, p, di, stream);
    case CUTB_Q4_0: return wg_launch<CUTB_Q4_0>(d, a16, stride, p, di, stream);
    default: return wg_launch<CUTB_Q4_K>(d, a16, stride, p, di, stream);
  }
}

}  // namespace cutb
