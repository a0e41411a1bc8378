// Attention of a prompt's tokens over the fp16 KV cache of the llama path, on the tensor cores.
//
// Same contract as the batched mode of attention_decode_kernel (token i attends cache rows [0, positions[i]] with its query rotated
// here; BatchedAttentionReadCacheOpNode, operators/impl/attention/BatchedAttentionReadCache.cu), which serves a few tokens per
// block with SIMT dot products.  The kernel is prefill_attention_kernel (prefill_attention.cuh).  Arithmetic: q and the
// probabilities are rounded to fp16 (the cache already is), all sums are fp32 -- against the SIMT path the output differs by about
// 1e-3 of its magnitude.  32 heads of 128, us per call (warp MMAs of 64-token blocks before): 16 tokens 11.8 -> 9.0, 128 26.8 ->
// 11.1, 512 42.3 -> 18.1, 1501 160 -> 64.
//
// Used for an fp16 cache with head_dim 64 or 128, 16-byte aligned rows and at least 16 tokens; everything else stays on the SIMT
// kernel.
#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.h"
#include "prefill_attention.cuh"

namespace cutb {

bool batched_attention_tc_applies(int kv_dtype, const float *q_in, uint32_t q_stride, const void *kC, const void *vC, const float *out,
                                  uint32_t out_stride, uint32_t n_tokens, uint32_t nHeads, uint32_t nKvHeads, uint32_t headDim,
                                  uint64_t ld) {
  (void)q_in;
  (void)q_stride;
  if (kv_dtype != CUTB_F16 || (headDim != 64 && headDim != 128) || n_tokens < 16) return false;
  if (nKvHeads == 0 || nHeads % nKvHeads != 0) return false;
  // 16-byte cache rows for the copy engine
  if ((ld * 2) % 16 != 0 || reinterpret_cast<uintptr_t>(kC) % 16 != 0 || reinterpret_cast<uintptr_t>(vC) % 16 != 0) return false;
  if (reinterpret_cast<uintptr_t>(out) % 8 != 0 || out_stride % 2 != 0) return false;
  return true;
}

namespace {
template <int P> int ll_launch(const PaParams &p, const void *kC, const void *vC, uint32_t nKvHeads, uint64_t ld, cudaStream_t stream) {
  CUtensorMap mk, mv;
  if (int rc = pa_map(&mk, false, kC, P * 64, nKvHeads, P * 64, p.max_pos, ld)) return rc;
  if (int rc = pa_map(&mv, false, vC, P * 64, nKvHeads, P * 64, p.max_pos, ld)) return rc;
  return pa_launch_inst<PA_LLAMA, P, P>(mk, mk, mv, p, stream);
}
}  // namespace

int batched_attention_tc_launch(const float *q_in, uint32_t q_stride, const void *kC, const void *vC, const uint32_t *positions,
                                const float *cosT, const float *sinT, float *out, uint32_t out_stride, uint32_t n_tokens,
                                uint32_t nHeads, uint32_t nKvHeads, uint32_t headDim, uint64_t ld, uint32_t max_seq, float scale,
                                int *status, cudaStream_t stream) {
  DeviceInfo di;
  if (int rc = get_device_info(&di)) return rc;
  PaParams a{};
  a.q = q_in, a.ldq = q_stride, a.n_tokens = n_tokens, a.n_heads = nHeads, a.rep = nHeads / nKvHeads, a.q_head = headDim;
  a.rot = headDim, a.cos_t = cosT, a.sin_t = sinT, a.positions = positions, a.max_pos = max_seq;
  a.step = pa_step(n_tokens, nHeads, (uint32_t)di.sm_count), a.ksteps = headDim / 16, a.key_planes = headDim / 64;
  a.out = out, a.ldo = out_stride, a.vdim = headDim, a.status = status;
  a.k = reinterpret_cast<const uint16_t *>(kC), a.v = reinterpret_cast<const uint16_t *>(vC), a.ld_k = a.ld_v = ld, a.k_head = a.v_head = headDim;
  pa_set_scale(&a, scale);
  return headDim == 128 ? ll_launch<2>(a, kC, vC, nKvHeads, ld, stream) : ll_launch<1>(a, kC, vC, nKvHeads, ld, stream);
}

}  // namespace cutb
