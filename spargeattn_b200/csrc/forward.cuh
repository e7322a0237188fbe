// One call of the whole path, for the C entry point and the Python binding.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime_api.h>

#include "../../include/sparge_b200.h"

namespace sparge {

struct ForwardArgs {
  const void *q, *k, *v;            // [B,H,N,D] views, last dimension contiguous, 16-byte aligned rows
  void* o;                          // like q, in q's dtype
  long long q_st[3], k_st[3], v_st[3], o_st[3];   // strides of (batch, head, token) in elements
  const float *simthr, *cdf, *topk, *pvthr;       // [H]; pvthr NULL: no skip test
  const void* mask;                 // caller's block mask [B,H,nq,nk] instead of a selection rule
  int mask_elem_size;
  void* workspace;
  size_t workspace_bytes;
  int32_t* dev_status;
  const int32_t* q_ranges;          // see sparge_attn_fwd_rows
  int q_blocks_max;
  int B, H, N, D, dtype, v_dtype, is_causal, kernel_causal, sink, smooth_k;
  bool pv_fp16;                     // P and V in fp16 (sparge_attn_fwd_f16pv)
  float sm_scale;
};

enum { kWsKm, kWsScratch, kWsPq, kWsPk, kWsSimQ, kWsSimK, kWsQ8, kWsK8, kWsQs, kWsKs, kWsLut, kWsValid, kWsV8, kWsVs, kWsCount };

// fp16 V that the attention kernel can read where it is needs no copy of its own
inline bool forward_copies_v(bool pv_fp16, int v_dtype, const long long* v_st) {
  return pv_fp16 && (v_dtype != SPARGE_F16 || v_st[0] == 0 || v_st[1] == 0);
}
// offsets (may be NULL) of the workspace parts; v_bytes_per_value: 1 FP8 V, 2 fp16 copy, 0 none
size_t forward_layout(int B, int H, int N, int D, int v_bytes_per_value, size_t* off);
int forward(const ForwardArgs& a, cudaStream_t st);

}  // namespace sparge
