// Decode mat-vec for one activation row (or two fp16 rows) over native GGUF blocks.
//
// C[m, n] = epilogue(sum_k A[m, k] * dequant(W)[n, k]), the reference's M = 1 variants MatMulQ4GemvKPar8 / MatMulQ8GemvKPar8
// (operators/impl/matmul/MatMulQ4GemvKPar8.cu:8-98, MatMulQ8GemvKPar8.cu:11-92) on the block layout its loader reads.
//
// What bounds it: each weight byte is read once, 25 MB in 3.9 us at the copy rate (11008 x 4096 of Q4_0), but a launch is as much a
// chain of latencies: 1.5 us from the predecessor's last block to the return of griddepcontrol.wait, 0.6 us until the activations
// have come from L2, 0.5 us until they are digits.  So the copies run ahead of that chain, and what follows it is short:
//  * The weights come through a ring of 18 KB stages, 16 rows of eight granules of 256 weights (four of Q8_0), one tensor copy each:
//    the weight seen as [granule][row][bytes] lands with rows 144 (272) bytes apart, on which the fragment loads meet no bank twice.
//    The ring is as deep as the SM allows (row_matvec_plan).  A chain that only copies takes 5.0 to 5.2 us a launch with five stages,
//    5.4 with sixteen padded row copies a stage, 7.7 with row copies of 576 bytes.
//  * Sixteen warps in two groups (Q8_0: four) take stages in turn, a granule per warp, and meet no other warp until the block's sums
//    are complete: a warp's partial sums go to shared memory per tile, and the epilogue runs once per eight tiles.  A barrier and an
//    epilogue per tile cost 0.35 us each.
//  * 4- and 8-bit quants feed the int8 MMA (m16n8k32) directly.  Lane t of a quad owns whole blocks (2t and 2t + 1 of a granule's
//    eight): its pair of activation columns is zero in the other lanes' k slots, so that column pair t ends as the dot product of the
//    lane's own block and the block scale is applied once, by the lane that loaded it.  Low nibbles enter as q and high ones as 16 q,
//    in MMAs of their own (one logic operation per four weights).  18- and 34-byte blocks are read in aligned pairs; the activations
//    are staged in the order that gives.
//  * A warp stages the activations of the granules that it multiplies, eight neighbouring elements to a lane (whole lines per load:
//    every block asks L2 for the same 8 KB at once; four-byte loads in block order took twice as long), and goes on without a barrier.
//    A fused RMSNorm stages x * weight; 1 / rms, a factor of the whole row, meets the sums in the epilogue.
// Measured, us a launch in a graph over cycled weights (before: 16 rows per tile through qgemv_blocks.cu's ring, a barrier per tile): Q4_0
// 11008 x 4096 (32 weights) 8.1 -> 6.4, Q4_0 28672 x 8192 (8) 33.4 -> 24.2, Q8_0 4096 x 4096 with fp32 rows (16) 5.95 -> 5.2.  Tried with
// five stages and slower for the first, in a run where this took 6.0: a lane to a row's blocks with dp4a (8.8), rings of cp.async per
// warp (7.5), the last warp of a group refilling the slot (6.4), eight warps with a unit each in registers before the wait (6.5),
// releasing the successor after the staging (7.7), stages of four granules (6.5).
//
// Activations are block floating point as in qgemv_blocks.cu: per 32-k block one fp32 scale e and 16-bit integers
// x^ = rint(x / e), |x^| <= 32512, as two balanced int8 digits; fp32 rows take a second such level for the residual.  The integer dot
// product of a block is exact; it is scaled in fp32 by (block scale) x e.
//
// Every wait on an mbarrier is bounded; on expiry the kernel stores CUTB_ERR_TIMEOUT in the caller's status word and leaves.
#include "matvec_common.cuh"
#include "tcgen05.cuh"

namespace cutb {

namespace {

constexpr uint32_t RW_ROWS = 16;
constexpr uint32_t RW_WARPS = 16, RW_CONSUMERS = RW_WARPS * 32, RW_THREADS = RW_CONSUMERS + 32;  // (one more warp issues the copies)
constexpr uint32_t RW_MAX_DEPTH = 8;
constexpr uint32_t RW_SUMS = RW_WARPS + 4;  // floats from one row's sums to the next: a thread reads them sixteen bytes at a time
constexpr uint32_t RW_GROUP = 8;                     // tiles whose sums a block keeps before it writes them out
constexpr float RW_LEVEL2 = 1.0f / GV_STEPS2;         // the second level's scale beside the first's
constexpr float RW_MAGIC = 12582912.f;               // 1.5 * 2^23: x + RW_MAGIC holds rint(x) in its low bits, |x| < 2^22


// Granules of a stage, one per warp of the group that takes it: 18 KB in each format
__host__ __device__ constexpr uint32_t rw_granules(int fmt) { return fmt == CUTB_Q8_0 ? 4u : 8u; }

struct RowParams : GvParams {
  uint32_t depth;   // stages of the ring
  uint32_t groups;  // tiles per group
  uint32_t box;     // granules of a copy
};

// int8 MMAs: D = A * B, and D += A * B
#define RW_MMA(AT, C)                                                                            \
  "mma.sync.aligned.m16n8k32.row.col.s32." AT ".s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {" C "};"
template <bool UA>
__device__ __forceinline__ void mma_bytes(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (UA)
    asm(RW_MMA("u8", "%10,%10,%10,%10") : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
  else
    asm(RW_MMA("s8", "%10,%10,%10,%10") : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
template <bool UA>
__device__ __forceinline__ void mma_bytes_add(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (UA)
    asm(RW_MMA("u8", "%0,%1,%2,%3") : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm(RW_MMA("s8", "%0,%1,%2,%3") : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
#undef RW_MMA
// A stage that has not landed yet; true (and an error status) if it does not.  After the first time nobody waits long again.
__device__ __noinline__ bool wait_long(uint32_t bar, uint32_t phase, bool dead, int *status) {
  const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar, phase, dead ? 1u : 1u << 16));
  if (!ok && (threadIdx.x & 31) == 0 && status) atomicExch(status, (int)CUTB_ERR_TIMEOUT);
  return !ok;
}
__device__ __forceinline__ float reciprocal(float a) {
  float d;
  asm("rcp.approx.f32 %0, %1;" : "=f"(d) : "f"(a));
  return d;
}
__device__ __forceinline__ float max_or_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}

// Layout of the staged activations, [granule][pass][v][half] rows of 128 bytes: sixteen bytes for each of the eight lanes that hold a
// column (column g: the block 2 (g / 2) + pass of the granule, digit g % 2), and {scale, sum} pairs at [granule][pass][row][block pair].
template <int FMT, int AMODE, int NR> struct RowShape {
  static constexpr bool TWO = AMODE == GV_A_F32_TWO;
  static constexpr bool AF32 = AMODE != GV_A_HALF;
  static constexpr int NV = TWO ? 2 : NR;  // digit pairs
  static constexpr uint32_t GB = granule_bytes(FMT), UNIT = RW_ROWS * GB;  // a warp's unit: 16 rows of 256 weights
  static constexpr uint32_t GPS = rw_granules(FMT), STAGE = GPS * UNIT;
};

// Loads of what the predecessor may have written: coherent ones that stay behind griddepcontrol.wait (the compiler may move loads of
// read-only data in front of it).
__device__ __forceinline__ uint4 load16(const void *at) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(at) : "memory");
  return v;
}
template <bool AF32> __device__ __forceinline__ uint32_t load1(const void *A, uint64_t idx) {
  if constexpr (AF32) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(reinterpret_cast<const uint32_t *>(A) + idx) : "memory");
    return v;
  } else {
    uint16_t v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(reinterpret_cast<const uint16_t *>(A) + idx) : "memory");
    return v;
  }
}

// Eight neighbouring elements, as they are loaded.
template <bool AF32> struct Octet {
  uint4 q[AF32 ? 2 : 1];
  __device__ __forceinline__ void load(const void *A, uint64_t idx, bool aligned) {
    if (aligned) {
      const uint8_t *at = reinterpret_cast<const uint8_t *>(A) + idx * (AF32 ? 4 : 2);
      q[0] = load16(at);
      if constexpr (AF32) q[1] = load16(at + 16);
      return;
    }
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = load1<AF32>(A, idx + i);
    if constexpr (AF32) q[0] = make_uint4(w[0], w[1], w[2], w[3]), q[1] = make_uint4(w[4], w[5], w[6], w[7]);
    else q[0] = make_uint4(w[0] | w[1] << 16, w[2] | w[3] << 16, w[4] | w[5] << 16, w[6] | w[7] << 16);
  }
  __device__ __forceinline__ void get(float (&x)[8]) const {
    if constexpr (AF32) {
      const uint32_t w[8] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w};
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = __uint_as_float(w[i]);
    } else {
      const uint32_t w[4] = {q[0].x, q[0].y, q[0].z, q[0].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(u32_as_h2(w[i]));
        x[2 * i] = f.x, x[2 * i + 1] = f.y;
      }
    }
  }
};

// Stages the blocks [0, nblk) from k0 on: four threads to a block, eight neighbouring elements each (read as they lie: a warp's loads
// are whole lines, which every block of the grid asks for at the same time).  With a fused RMSNorm the elements are staged times their
// norm weight alone: 1 / rms is a factor of the whole row and meets the sums in the epilogue; ss: this thread's share of the squares.
template <int FMT, int AMODE, int NR>
__device__ __forceinline__ void stage_row(const RowParams &p, uint8_t *act, float2 *scales, uint32_t k0, uint32_t nblk, float (&ss)[NR], uint32_t tid) {
  using S = RowShape<FMT, AMODE, NR>;
  const bool aligned = reinterpret_cast<uintptr_t>(p.A) % 16 == 0 && p.lda % (S::AF32 ? 4 : 8) == 0;
  const bool waligned = reinterpret_cast<uintptr_t>(p.norm_w) % 16 == 0, norm = p.norm_w != nullptr;
  constexpr float wscale = FMT == CUTB_Q4_0 ? 0.0625f : 1.0f, sxscale = FMT == CUTB_Q4_0 ? 8.0f : 1.0f;
  const uint32_t total = nblk * 4;  // (threads without a chunk read the last one and leave it)
  Octet<S::AF32> next;
  next.load(p.A, k0 + min(tid, total - 1) * 8, aligned);
#pragma unroll
  for (int m = 0; m < NR; ++m) {
    for (uint32_t base = 0; base < total; base += RW_CONSUMERS) {  // (as many rounds for every thread: shuffles inside)
      const bool live = base + tid < total;
      const uint32_t id = live ? base + tid : total - 1, kb = id >> 2, ct = id & 3;
      const Octet<S::AF32> now = next;
      Octet<true> wn;
      if (norm) wn.load(p.norm_w, k0 + id * 8, waligned);
      // the next round's elements, or the next row's first
      if (base + RW_CONSUMERS < total) next.load(p.A, (uint64_t)m * p.lda + k0 + min(base + RW_CONSUMERS + tid, total - 1) * 8, aligned);
      else if (m + 1 < NR) next.load(p.A, (uint64_t)(m + 1) * p.lda + k0 + min(tid, total - 1) * 8, aligned);
      float x[8];
      now.get(x);
      if (norm) {
        float w[8];
        wn.get(w);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (live) ss[m] = fmaf(x[i], x[i], ss[m]);
          x[i] *= w[i];
        }
      }
      float amax = 0.f;  // of the block; NaN if any of it is
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = max_or_nan(amax, fabsf(x[i]));
      amax = max_or_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
      amax = max_or_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
      const bool finite = amax < __int_as_float(0x7f800000);
      const float e = finite ? fmaxf(amax * (1.0f / GV_QMAX), 1.0f / GV_MOST) : __int_as_float(0x7fc00000);
      const float inv = finite ? fminf(reciprocal(e), GV_MOST) : 0.f;  // (of e itself: both roundings in one, see GV_STEPS2)
      const uint32_t pass = kb >> 3 << 1 | (kb & 1), pr = (kb & 7) >> 1;  // [granule][pass], the lane pair
      const bool even = (kb & 1) == 0;
      // v: floats whose low 16 bits are the integers.  A block's digits become eight words in the order in which the weights' aligned words
      // hold its elements: an unaligned block's as they are, an aligned block's (even: its scale takes half a word) from element 2 on, so
      // that a thread's last pair is joined by its neighbour's first and the last word is {0, 1, 14, 15} (Q8_0: {0, 1, 30, 31}).
      auto put = [&](const float (&v)[8], uint32_t vr) {
        int q[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) q[i] = __float_as_int(v[i]);
        uint32_t hi[2], lo[2];
        pack_digits(q, hi, lo);
        if constexpr (FMT != CUTB_Q4_K) {
          const uint32_t ends = __byte_perm(hi[0], lo[0], 0x5410);  // both digits' first pairs
          const uint32_t near = FMT == CUTB_Q4_0 ? __shfl_xor_sync(0xffffffffu, ends, 1) : __shfl_sync(0xffffffffu, ends, (ct + 1) & 3, 4);
          if (even) {
            const bool wraps = FMT == CUTB_Q4_0 ? (ct & 1) : ct == 3;
            const uint32_t h1 = __byte_perm(hi[1], near, wraps ? 0x3254 : 0x5432), l1 = __byte_perm(lo[1], near, wraps ? 0x3276 : 0x7632);
            hi[0] = __byte_perm(hi[0], hi[1], 0x5432), lo[0] = __byte_perm(lo[0], lo[1], 0x5432);
            hi[1] = h1, lo[1] = l1;
          }
        }
        if (!live) return;
        // word w of digit d lies at [half][lane 2 pr + d][..]: words 0 to 3 in the first half; Q4_0's are the low nibbles' words 0 and 1
        // and the high nibbles', then both nibbles' words 2 and 3: each pair of words is one MMA's operand
        uint8_t *to = act + ((size_t)pass * S::NV + vr) * 256 + pr * 32;
        to += FMT == CUTB_Q4_0 ? (ct & 1) * 128 + (ct >> 1) * 8 : (ct >> 1) * 128 + (ct & 1) * 8;
        *reinterpret_cast<uint2 *>(to) = make_uint2(hi[0], hi[1]);
        *reinterpret_cast<uint2 *>(to + 16) = make_uint2(lo[0], lo[1]);
      };
      auto sum_of = [&](const float (&v)[8]) {  // the block's integers
        int s = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) s += __float_as_int(v[i]);
        s -= 8 * __float_as_int(RW_MAGIC);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        return s + __shfl_xor_sync(0xffffffffu, s, 2);
      };
      float v[8], sum = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = fmaf(x[i], inv, RW_MAGIC);
      put(v, S::TWO ? 0 : m);
      if constexpr (FMT != CUTB_Q8_0) sum = e * (float)sum_of(v);
      if constexpr (S::TWO) {  // the residual x - x^ e in steps of e / GV_STEPS2
        float inv2 = inv * GV_STEPS2;
        if (inv2 > GV_MOST) inv2 = 0.f;  // (blocks below 1e-30: one level)
        float r[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = fmaf(fmaf(-(v[i] - RW_MAGIC), e, x[i]), inv2, RW_MAGIC);
        put(r, 1);
        if constexpr (FMT != CUTB_Q8_0) sum = fmaf(e * RW_LEVEL2, (float)sum_of(r), sum);
      }
      if (live && ct == 0) {
        // Q4_K's odd sub-blocks are the high nibbles and enter as 16 q, Q4_0's nibbles all do
        scales[((size_t)pass * NR + m) * 4 + pr] =
            make_float2(e * ((FMT == CUTB_Q4_K && (kb & 1)) ? 0.0625f : wscale), FMT != CUTB_Q8_0 ? sxscale * sum : 0.f);
      }
    }
  }
}

// One unit: 16 rows of 256 weights.  Lane t of a quad owns the blocks 2t and 2t + 1 of rows g and g + 8.
template <int FMT> struct Unit {
  static constexpr int N = FMT == CUTB_Q8_0 ? 17 : FMT == CUTB_Q4_0 ? 9 : 12;
  uint32_t a[N], b[N];  // the words of both blocks (Q4_K: the super-block's four, then the lane's eight) in rows g and g + 8

  __device__ __forceinline__ void load(uint32_t unit, uint32_t g, uint32_t t) {
    constexpr uint32_t GB = granule_bytes(FMT);
    const uint32_t ra = unit + g * GB, rb = ra + 8 * GB;
    if constexpr (FMT == CUTB_Q4_K) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const uint32_t at = i == 0 ? 0u : 32 * t + 16 * i;
        const uint4 wa = lds_u128(ra + at), wb = lds_u128(rb + at);
        a[4 * i] = wa.x, a[4 * i + 1] = wa.y, a[4 * i + 2] = wa.z, a[4 * i + 3] = wa.w;
        b[4 * i] = wb.x, b[4 * i + 1] = wb.y, b[4 * i + 2] = wb.z, b[4 * i + 3] = wb.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < N; ++k) {
        a[k] = lds_u32(ra + 4 * N * t + 4 * k);
        b[k] = lds_u32(rb + 4 * N * t + 4 * k);
      }
    }
  }
};

// A unit times its granule's staged activations: a lane's column pair (the digits) is zero in the other lanes' k slots, so that column
// pair t ends as the dot product of lane t's own block.  x: this lane's sixteen bytes of the granule's first row of columns (lanes
// without: of rows of zeros).
template <int FMT, int AMODE, int NR>
__device__ __forceinline__ void unit_dot(const Unit<FMT> &u, uint32_t x, uint32_t scales, uint32_t t, float (&tot)[NR][2]) {
  using S = RowShape<FMT, AMODE, NR>;
  constexpr int NV = S::NV;
  auto load_x = [&](int pass, int v, uint4 &x0, uint4 &x1) {
    x0 = lds_u128(x + ((pass * NV + v) * 2) * 128);
    x1 = lds_u128(x + ((pass * NV + v) * 2 + 1) * 128);
  };
  auto scale_of = [&](int pass, int m) {
    const uint2 s = lds_u64(scales + ((pass * NR + m) * 4 + t) * 8);
    return make_float2(__uint_as_float(s.x), __uint_as_float(s.y));
  };
  // integer dot products of rows g and g + 8 (two levels: in the first one's scale)
  auto join = [&](const int (&c)[NV][4], int m, float &fa, float &fb) {
    if constexpr (S::TWO) {
      fa = fmaf((float)(c[1][0] * 256 + c[1][1]), RW_LEVEL2, (float)(c[0][0] * 256 + c[0][1]));
      fb = fmaf((float)(c[1][2] * 256 + c[1][3]), RW_LEVEL2, (float)(c[0][2] * 256 + c[0][3]));
    } else {
      fa = (float)(c[m][0] * 256 + c[m][1]);
      fb = (float)(c[m][2] * 256 + c[m][3]);
    }
  };
  if constexpr (FMT == CUTB_Q4_0) {
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      uint32_t wa[4], wb[4];
      if (pass == 0) {
        wa[0] = u.a[1], wa[1] = u.a[2], wa[2] = u.a[3], wa[3] = __byte_perm(u.a[0], u.a[4], 0x5432);
        wb[0] = u.b[1], wb[1] = u.b[2], wb[2] = u.b[3], wb[3] = __byte_perm(u.b[0], u.b[4], 0x5432);
      } else {
        wa[0] = u.a[5], wa[1] = u.a[6], wa[2] = u.a[7], wa[3] = u.a[8];
        wb[0] = u.b[5], wb[1] = u.b[6], wb[2] = u.b[7], wb[3] = u.b[8];
      }
      const float dA = h2f_bits(pass == 0 ? u.a[0] & 0xFFFFu : u.a[4] >> 16), dB = h2f_bits(pass == 0 ? u.b[0] & 0xFFFFu : u.b[4] >> 16);
      int c[NV][4];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        uint4 x0, x1;
        load_x(pass, v, x0, x1);
        int lo[4], hi[4];  // low nibbles as q, high ones as 16 q
        mma_bytes<true>(lo, wa[0] & 0x0F0F0F0Fu, wb[0] & 0x0F0F0F0Fu, wa[1] & 0x0F0F0F0Fu, wb[1] & 0x0F0F0F0Fu, x0.x, x0.y);
        mma_bytes<true>(hi, wa[0] & 0xF0F0F0F0u, wb[0] & 0xF0F0F0F0u, wa[1] & 0xF0F0F0F0u, wb[1] & 0xF0F0F0F0u, x0.z, x0.w);
        mma_bytes_add<true>(lo, wa[2] & 0x0F0F0F0Fu, wb[2] & 0x0F0F0F0Fu, wa[3] & 0x0F0F0F0Fu, wb[3] & 0x0F0F0F0Fu, x1.x, x1.y);
        mma_bytes_add<true>(hi, wa[2] & 0xF0F0F0F0u, wb[2] & 0xF0F0F0F0u, wa[3] & 0xF0F0F0F0u, wb[3] & 0xF0F0F0F0u, x1.z, x1.w);
#pragma unroll
        for (int i = 0; i < 4; ++i) c[v][i] = lo[i] * 16 + hi[i];
      }
#pragma unroll
      for (int m = 0; m < NR; ++m) {
        const float2 s = scale_of(pass, m);
        float fa, fb;
        join(c, m, fa, fb);
        tot[m][0] = fmaf(dA, fmaf(s.x, fa, -s.y), tot[m][0]);  // d (e/16 sum 16 q x^ - 8 e sum x^)
        tot[m][1] = fmaf(dB, fmaf(s.x, fb, -s.y), tot[m][1]);
      }
    }
  } else if constexpr (FMT == CUTB_Q8_0) {
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      const int at = pass == 0 ? 1 : 9;  // two blocks of 34 bytes in seventeen words
      uint32_t wa[8], wb[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) wa[k] = u.a[at + k], wb[k] = u.b[at + k];
      if (pass == 0) wa[7] = __byte_perm(u.a[0], u.a[8], 0x5432), wb[7] = __byte_perm(u.b[0], u.b[8], 0x5432);
      const float dA = h2f_bits(pass == 0 ? u.a[0] & 0xFFFFu : u.a[8] >> 16), dB = h2f_bits(pass == 0 ? u.b[0] & 0xFFFFu : u.b[8] >> 16);
      int c[NV][4];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        uint4 x0, x1;
        load_x(pass, v, x0, x1);
        int c2[4];
        mma_bytes<false>(c[v], wa[0], wb[0], wa[1], wb[1], x0.x, x0.y);
        mma_bytes<false>(c2, wa[2], wb[2], wa[3], wb[3], x0.z, x0.w);
        mma_bytes_add<false>(c[v], wa[4], wb[4], wa[5], wb[5], x1.x, x1.y);
        mma_bytes_add<false>(c2, wa[6], wb[6], wa[7], wb[7], x1.z, x1.w);
#pragma unroll
        for (int i = 0; i < 4; ++i) c[v][i] += c2[i];
      }
#pragma unroll
      for (int m = 0; m < NR; ++m) {
        const float2 s = scale_of(pass, m);
        float fa, fb;
        join(c, m, fa, fb);
        tot[m][0] = fmaf(dA * s.x, fa, tot[m][0]);
        tot[m][1] = fmaf(dB * s.x, fb, tot[m][1]);
      }
    }
  } else {  // Q4_K: lane t owns the 64-weight group t = sub-blocks 2t (low nibbles) and 2t + 1 (high nibbles)
    const uint4 hA = make_uint4(u.a[0], u.a[1], u.a[2], u.a[3]), hB = make_uint4(u.b[0], u.b[1], u.b[2], u.b[3]);
    uint32_t wa[8], wb[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) wa[k] = u.a[4 + k], wb[k] = u.b[4 + k];
    const float dA = h2f_bits(hA.x & 0xFFFFu), mA = h2f_bits(hA.x >> 16);
    const float dB = h2f_bits(hB.x & 0xFFFFu), mB = h2f_bits(hB.x >> 16);
    // 6-bit (scale, min) fields of this lane's two sub-blocks (gguf_reader.cpp:668-676)
    const bool upper = t >= 2;  // sub-blocks 4..7 keep their high bits elsewhere
    const uint32_t scA = upper ? (hA.w & 0x0F0F0F0Fu) | ((hA.y >> 2) & 0x30303030u) : hA.y & 0x3F3F3F3Fu;
    const uint32_t mnA = upper ? ((hA.w >> 4) & 0x0F0F0F0Fu) | ((hA.z >> 2) & 0x30303030u) : hA.z & 0x3F3F3F3Fu;
    const uint32_t scB = upper ? (hB.w & 0x0F0F0F0Fu) | ((hB.y >> 2) & 0x30303030u) : hB.y & 0x3F3F3F3Fu;
    const uint32_t mnB = upper ? ((hB.w >> 4) & 0x0F0F0F0Fu) | ((hB.z >> 2) & 0x30303030u) : hB.z & 0x3F3F3F3Fu;
    const float ndA = -dA * 8388608.f, nmA = -mA * 8388608.f, ndB = -dB * 8388608.f, nmB = -mB * 8388608.f;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      const uint32_t sel = 0x7540u | (((2 * t) & 3) + pass), mask = pass ? 0xF0F0F0F0u : 0x0F0F0F0Fu;
      // d * (2^23 + sc) - d * 2^23 == d * sc exactly
      const float dsA = fmaf(dA, __uint_as_float(__byte_perm(scA, 0x4B000000u, sel)), ndA);
      const float dmA = fmaf(mA, __uint_as_float(__byte_perm(mnA, 0x4B000000u, sel)), nmA);
      const float dsB = fmaf(dB, __uint_as_float(__byte_perm(scB, 0x4B000000u, sel)), ndB);
      const float dmB = fmaf(mB, __uint_as_float(__byte_perm(mnB, 0x4B000000u, sel)), nmB);
      int c[NV][4];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        uint4 x0, x1;
        load_x(pass, v, x0, x1);
        int c2[4];
        mma_bytes<true>(c[v], wa[0] & mask, wb[0] & mask, wa[1] & mask, wb[1] & mask, x0.x, x0.y);
        mma_bytes<true>(c2, wa[2] & mask, wb[2] & mask, wa[3] & mask, wb[3] & mask, x0.z, x0.w);
        mma_bytes_add<true>(c[v], wa[4] & mask, wb[4] & mask, wa[5] & mask, wb[5] & mask, x1.x, x1.y);
        mma_bytes_add<true>(c2, wa[6] & mask, wb[6] & mask, wa[7] & mask, wb[7] & mask, x1.z, x1.w);
#pragma unroll
        for (int i = 0; i < 4; ++i) c[v][i] += c2[i];
      }
#pragma unroll
      for (int m = 0; m < NR; ++m) {
        const float2 s = scale_of(pass, m);
        float fa, fb;
        join(c, m, fa, fb);
        tot[m][0] = fmaf(-dmA, s.y, fmaf(dsA * s.x, fa, tot[m][0]));
        tot[m][1] = fmaf(-dmB, s.y, fmaf(dsB * s.x, fb, tot[m][1]));
      }
    }
  }
}

// FIXED: sixteen granules (K = 4096, or such a split): as many stages to a tile as there are groups, one granule per warp for good.
// MINB: blocks per SM that the registers are kept for: 2 (56 registers) only where the next launch's block is to copy beside this one, since
// all instantiations but the fixed ones of a single level spill there (up to 136 bytes a thread).
template <int FMT, int AMODE, int NR, bool FIXED, int MINB>
__global__ void __launch_bounds__(RW_THREADS, MINB) qgemv_row_kernel(const __grid_constant__ CUtensorMap weights, const RowParams p) {
  using S = RowShape<FMT, AMODE, NR>;
  constexpr int NV = S::NV;
  constexpr uint32_t NW = RW_WARPS, GPS = S::GPS, STAGE = S::STAGE, GROUPS = NW / GPS;
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;

  // tiles of 16 rows [t0, t1) of this block, granules [gs0, gs0 + ng) of this K split; a stage is GPS granules of a tile
  const uint32_t tiles = (p.N + RW_ROWS - 1) / RW_ROWS;
  const uint32_t t0 = (uint32_t)((uint64_t)blockIdx.x * tiles / gridDim.x), t1 = (uint32_t)((uint64_t)(blockIdx.x + 1) * tiles / gridDim.x);
  const uint32_t r0 = t0 * RW_ROWS, r1 = min(p.N, t1 * RW_ROWS), ntiles = t1 - t0;
  const uint32_t G = p.K >> 8, gs0 = blockIdx.y * p.gran_per_split, ng = min(G, gs0 + p.gran_per_split) - gs0;
  const uint32_t cpt = (ng + GPS - 1) / GPS, nstages = ntiles * cpt, D = p.depth;

  uint8_t *act = smem + (size_t)D * STAGE;
  uint8_t *zeros = act + (size_t)p.gran_per_split * NV * 512;  // a granule of them
  float2 *scales = reinterpret_cast<float2 *>(zeros + NV * 512);
  float *sums = reinterpret_cast<float *>(scales + (size_t)p.gran_per_split * NR * 8);  // [tile of the group][m][row][warp, padded]
  float *squares = sums + p.groups * NR * RW_ROWS * RW_SUMS;                           // [m][warp]
  uint64_t *bars = reinterpret_cast<uint64_t *>(squares + NR * NW);
  // A slot has a "full" barrier for each group: a group then sees every phase of the barriers that it waits for (with one barrier the
  // groups would pass each other's phases by, and a parity seen two phases late reads as done).
  const uint32_t ring_u = smem_u32(smem), full_u = smem_u32(bars), empty_u = full_u + D * GROUPS * 8;
  const uint32_t cycle = D % GROUPS == 0 ? D / GROUPS : D % 2 == 0 ? D / 2 : D;  // a group's stages from one use of a slot to its next

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == NW) {
    // ---- copy warp: a stage is one box of the weights seen as [granule][row][bytes] ----
    if (lane == 0) {
      for (uint32_t s = 0; s < D; ++s) {
        mbar_init(empty_u + s * 8, GPS);
        for (uint32_t q = 0; q < GROUPS; ++q) mbar_init(full_u + (s * GROUPS + q) * 8, 1);
      }
      fence_mbar_init();
    }
    __syncwarp();
    uint32_t slot = 0, par = 1, c = 0, row = r0, issued = 0;
    auto fill = [&](uint32_t end) {
      for (; issued < end; ++issued) {
        if (issued >= D && !warp_wait(empty_u + slot * 8, par)) {
          if (lane == 0 && p.status) atomicExch(p.status, (int)CUTB_ERR_TIMEOUT);
          break;
        }
        if (lane == 0) {
          const uint32_t full = full_u + (slot * GROUPS + issued % GROUPS) * 8;
          mbar_arrive_expect_tx(full, p.box * S::UNIT);
          tma_load_3d(ring_u + slot * STAGE, &weights, 0, row, gs0 + c * GPS, full);
        }
        __syncwarp();
        if (++slot == D) slot = 0, par ^= 1u;
        if (++c == cpt) c = 0, row += RW_ROWS;
      }
    };
    fill(min(D, nstages));
    __syncthreads();
    fill(nstages);
    // stay until every copy has landed (bounded)
    for (uint32_t j = issued > D ? issued - D : 0; j < issued; ++j)
      mbar_drain(full_u + (j % D * GROUPS + j % GROUPS) * 8, (j / GROUPS / cycle) & 1u);
    return;
  }

  // fields of the launch that the end needs: read now, while the copies are under way
  asm volatile("" ::"l"(p.C), "l"(p.D), "r"(p.ldc), "r"(p.fusion_type), "r"(p.fusion_op), "r"(p.world), "r"(p.ksplit), "l"(p.partial), "l"(p.norm_w));
  if (tid < NV * 32) reinterpret_cast<uint4 *>(zeros)[tid] = make_uint4(0, 0, 0, 0);
  __syncthreads();

  // The warp's group takes every GROUPS-th stage, the warp one granule of it.
  const uint32_t group = warp / GPS, wg = warp % GPS;
  uint32_t slot = group % D, visit = 0, phase = 0;
  bool dead = false;
  auto take = [&](Unit<FMT> &u) {
    const uint32_t full = full_u + (slot * GROUPS + group) * 8;
    if (!__all_sync(0xffffffffu, mbar_test(full, phase))) dead |= wait_long(full, phase, dead, p.status);
    u.load(ring_u + slot * STAGE + wg * S::UNIT, g, t);
    __syncwarp();
    if (lane == 0) mbar_arrive(empty_u + slot * 8);
    slot += GROUPS;
    if (slot >= D) slot -= D;
    if (++visit == cycle) visit = 0, phase ^= 1u;
  };
  // What came before read only the (constant) weights; activations, D and C may be the predecessor's.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  {
    float ss[NR] = {};
    stage_row<FMT, AMODE, NR>(p, act, scales, gs0 * 256, ng * 8, ss, tid);
    if (p.norm_w) {
#pragma unroll
      for (int m = 0; m < NR; ++m) {
        if (p.ksplit > 1)  // the rest of the row
          for (uint32_t k = tid; k < p.K; k += RW_CONSUMERS)
            if (k < gs0 * 256 || k >= (gs0 + ng) * 256) {
              const uint32_t bits = load1<S::AF32>(p.A, (uint64_t)m * p.lda + k);
              const float v = S::AF32 ? __uint_as_float(bits) : h2f_bits(bits);
              ss[m] = fmaf(v, v, ss[m]);
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss[m] += __shfl_xor_sync(0xffffffffu, ss[m], o);
        if (lane == 0) squares[m * NW + warp] = ss[m];
      }
    }
  }
  // A warp stages every sixteenth granule.  Where each group has as many stages of every tile, these are the ones it multiplies; else its
  // stages shift from tile to tile, and it reads what warps of other groups staged.
  if (FIXED || cpt % GROUPS == 0) __syncwarp();
  else asm volatile("bar.sync 1, %0;" ::"n"(RW_CONSUMERS) : "memory");

  // Where this lane reads its column: lanes without one read zeros, at a place in the row that the lanes beside them leave free.
  const bool mine = t == (g >> 1);
  const uint32_t x_u = mine ? smem_u32(act) + g * 16 : smem_u32(zeros) + (g ^ 4) * 16, x_step = mine ? NV * 512 : 0, scales_u = smem_u32(scales);
  uint32_t c = group;
  for (uint32_t first = 0; first < ntiles; first += p.groups) {
    const uint32_t end = min(ntiles, first + p.groups);
    float *to = sums + (g + 8 * (t & 1)) * RW_SUMS + warp;
    for (uint32_t tile = first; tile < end; ++tile) {
      float tot[NR][2] = {};
      do {
        if (!FIXED && c >= cpt) break;
        const uint32_t gran = FIXED ? warp : c * GPS + wg;
        Unit<FMT> u;
        take(u);
        if (FIXED || gran < ng) unit_dot<FMT, AMODE, NR>(u, x_u + gran * x_step, scales_u + gran * NR * 64, t, tot);
        c += GROUPS;
      } while (!FIXED);
      c -= cpt;
      // the four lanes of a quad hold parts of the same two rows: lane 0 ends with row g, lane 1 with row g + 8
#pragma unroll
      for (int m = 0; m < NR; ++m) {
        float v = (t & 1) ? tot[m][1] : tot[m][0];
        v += __shfl_xor_sync(0xffffffffu, (t & 1) ? tot[m][0] : tot[m][1], 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        if (t < 2) to[m * RW_ROWS * RW_SUMS] = v;
      }
      to += NR * RW_ROWS * RW_SUMS;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(RW_CONSUMERS) : "memory");

    // ---- epilogue of the group: a row's warps in a fixed order ----
    const uint32_t n0 = first * RW_ROWS, rows = min(r1 - r0, end * RW_ROWS) - n0;  // of the block's rows
    auto row_sum = [&](uint32_t row, uint32_t m) -> float {
      const float4 *at = reinterpret_cast<const float4 *>(sums + (((row / RW_ROWS) * NR + m) * RW_ROWS + row % RW_ROWS) * RW_SUMS);
      float s = 0.f;
#pragma unroll
      for (uint32_t w = 0; w < NW / 4; ++w) {
        const float4 v = at[w];
        s += (v.x + v.y) + (v.z + v.w);
      }
      return s;
    };
#pragma unroll
    for (uint32_t m = 0; m < NR; ++m) {
      float rs = 1.f;
      if (p.norm_w) {
        float ss = 0.f;
#pragma unroll
        for (uint32_t w = 0; w < NW; ++w) ss += squares[m * NW + w];
        rs = rsqrtf(ss / (float)p.K + p.norm_eps);
      }
      if (p.glu) {  // (gate, up) row pairs: one output per pair
        for (uint32_t i = tid; i < rows / 2; i += RW_CONSUMERS) {
          const float gate = rs * row_sum(2 * i, m), up = rs * row_sum(2 * i + 1, m);
          p.C[(size_t)m * p.ldc + (r0 + n0) / 2 + i] = apply_epilogue(gate, CUTB_FUSION_UNARY, p.fusion_op, 0.f) * up;
        }
        continue;
      }
      for (uint32_t i = tid; i < rows; i += RW_CONSUMERS) {
        const uint32_t n = r0 + n0 + i;
        const float sum = rs * row_sum(i, m);
        if (p.ksplit > 1) {
          p.partial[((size_t)blockIdx.y * p.M + m) * p.N + n] = sum;
          continue;
        }
        const float dv = p.fusion_type == CUTB_FUSION_BINARY ? p.D[(size_t)m * p.ldd + n] : 0.f;
        const float out = apply_epilogue(sum, p.fusion_type, p.fusion_op, dv);
        if (p.world > 1) {
          const size_t at = (size_t)m * p.ldc_total + p.n_off + n;
          for (uint32_t q = 0; q < p.world; ++q) p.peer_C[q][at] = out;
        } else {
          p.C[(size_t)m * p.ldc + n] = out;
        }
      }
    }
    if (end < ntiles) asm volatile("bar.sync 1, %0;" ::"n"(RW_CONSUMERS) : "memory");
  }
}

template <int FMT, int AMODE, int NR, bool FIXED, int MINB>
int row_launch_inst(const CUtensorMap &map, const RowParams &p, const RowPlan &pl, bool overlap, cudaStream_t stream) {
  static bool configured[64] = {};  // per device: the attribute is set once on each
  int dev = 0;
  CUTB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    DeviceInfo di;
    if (int rc = get_device_info(&di)) return rc;
    CUTB_CUDA_TRY(cudaFuncSetAttribute(qgemv_row_kernel<FMT, AMODE, NR, FIXED, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)di.smem_optin));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pl.grid_x, p.ksplit);
  cfg.blockDim = dim3(RW_THREADS);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  CUTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, qgemv_row_kernel<FMT, AMODE, NR, FIXED, MINB>, map, p));
  return CUTB_OK;
}

template <int FMT, int AMODE>
int row_launch_mode(const CUtensorMap &map, const RowParams &p, const RowPlan &pl, bool overlap, cudaStream_t stream) {
  if constexpr (AMODE != GV_A_F32_TWO) {
    if (p.M == 2) return row_launch_inst<FMT, AMODE, 2, false, 1>(map, p, pl, overlap, stream);
    if (pl.beside) return row_launch_inst<FMT, AMODE, 1, true, 2>(map, p, pl, overlap, stream);
  }
  return pl.fixed ? row_launch_inst<FMT, AMODE, 1, true, 1>(map, p, pl, overlap, stream) : row_launch_inst<FMT, AMODE, 1, false, 1>(map, p, pl, overlap, stream);
}

template <int FMT>
int row_launch_fmt(const CUtensorMap &map, const RowParams &p, int amode, const RowPlan &pl, bool overlap, cudaStream_t stream) {
  switch (amode) {
    case GV_A_F32_TWO: return row_launch_mode<FMT, GV_A_F32_TWO>(map, p, pl, overlap, stream);
    case GV_A_F32_ONE: return row_launch_mode<FMT, GV_A_F32_ONE>(map, p, pl, overlap, stream);
    default: return row_launch_mode<FMT, GV_A_HALF>(map, p, pl, overlap, stream);
  }
}

}  // namespace

bool row_matvec_plan(const cutb_qmatmul_desc &d, int amode, const DeviceInfo &di, uint32_t ksplit, uint32_t gran_per_split, RowPlan *pl) {
  const uint32_t nr = d.M, nv = amode == GV_A_F32_TWO ? 2 : nr;
  const uint32_t sms = (uint32_t)di.sm_count > ksplit ? (uint32_t)di.sm_count / ksplit : 1;
  const uint32_t tiles = (d.N + RW_ROWS - 1) / RW_ROWS;
  pl->grid_x = tiles < sms ? tiles : sms;
  const uint32_t per_block = (tiles + pl->grid_x - 1) / pl->grid_x;
  pl->groups = per_block < RW_GROUP ? per_block : RW_GROUP;
  const size_t stage = (size_t)rw_granules(d.format) * RW_ROWS * granule_bytes(d.format);
  const size_t fixed = (size_t)gran_per_split * (nv * 512 + nr * 64) + nv * 512 + (size_t)nr * (pl->groups * RW_ROWS * RW_SUMS + RW_WARPS) * 4 +
                       RW_MAX_DEPTH * (RW_WARPS / rw_granules(d.format) + 1) * 8;
  const uint32_t need = RW_WARPS / rw_granules(d.format);  // a slot for each group of warps at least
  const uint32_t used = per_block * ((gran_per_split + rw_granules(d.format) - 1) / rw_granules(d.format));  // stages of a block
  const uint32_t most = used > need ? used : need;
  pl->fixed = gran_per_split == RW_WARPS && d.K / 256 % RW_WARPS == 0;
  // The ring takes what the SM has, up to eight stages.  Four or five under half an SM, so that the next launch's block can start its copies
  // beside this one, were the slower plan almost everywhere, by 14 % on average of 346 one-row shapes.  us a launch, half an SM (56 registers) /
  // all of it: Q4_0 28672 x 8192 29.1 / 24.2, Q4_K 4096 x 14336 11.3 / 9.6, its fp32 rows at 32 bits 12000 x 14336 46.8 / 22.8, Q8_0 8000 x
  // 8192 16.0 / 13.7; a token of eight layers of a Q8_0 decoder (hidden 4096) 548 / 487, Q4_K 412 / 378, Q4_0 388 / 363, hidden 2048 270 / 233.
  // Only where a launch that starts early has all of a block's stages under half an SM at K = 4096 do neighbours gain: chains of Q4_0 4096 x
  // 4096 3.46 / 3.83, Q8_0 2368 x 4096 3.1 / 3.6.  (The same for any K gained 0.1 us in chains and lost 12 % of the hidden 2048 decoder.)
  const size_t half = di.smem_per_sm > 2048 ? di.smem_per_sm / 2 - 1024 : di.smem_optin / 2;
  pl->beside = pl->fixed && nv == 1 && !(d.flags & CUTB_FLAG_NO_OVERLAP) && fixed + most * stage <= half;
  const size_t room = di.smem_optin;
  if (fixed + need * stage > room) return false;
  const size_t fit = (room - fixed) / stage;
  pl->depth = fit > RW_MAX_DEPTH ? RW_MAX_DEPTH : (uint32_t)fit;
  if (pl->depth > most) pl->depth = most;
  pl->smem = fixed + pl->depth * stage;
  return true;
}

int row_matvec_launch(const GvParams &g, int format, int amode, const RowPlan &pl, bool overlap, cudaStream_t stream) {
  RowParams p;
  static_cast<GvParams &>(p) = g;
  p.depth = pl.depth;
  p.groups = pl.groups;
  p.box = p.gran_per_split < rw_granules(format) ? p.gran_per_split : rw_granules(format);
  CUtensorMap map;
  if (int rc = make_tmap_granules(&map, p.W, format, p.N, p.K, p.row_bytes, RW_ROWS, p.box)) return rc;
  switch (format) {
    case CUTB_Q8_0: return row_launch_fmt<CUTB_Q8_0>(map, p, amode, pl, overlap, stream);
    case CUTB_Q4_0: return row_launch_fmt<CUTB_Q4_0>(map, p, amode, pl, overlap, stream);
    default: return row_launch_fmt<CUTB_Q4_K>(map, p, amode, pl, overlap, stream);
  }
}

}  // namespace cutb
