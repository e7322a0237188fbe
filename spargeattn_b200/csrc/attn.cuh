// Launch of the attention kernel (attn_sm100.cu) for the C entry points.
#pragma once
#include "common.cuh"

namespace sparge {

struct AttnArgs {
  const int8_t *q8, *k8;            // [B,H,N,D]
  const void* v;                    // e4m3 [B,H,N_pad,D], or fp16 [B,H,N,D] when v_f16 (any strides)
  long long v_st[3];                // fp16 V: strides of (batch, head, token) in elements
  void* o;
  long long o_st[3];
  const int32_t *lut, *valid;
  const float *pvthr, *q_scale, *k_scale, *v_scale;
  int32_t *dev_status, *pv_count;
  const int32_t* q_ranges;
  // Which row a CTA computes, without q_ranges: row_order [B*H*ceil(N/128)], or else late rows first in each of
  // order_groups groups of heads (0, or as many as there are heads: head by head)
  const int32_t* row_order;
  int order_groups;
  int q_blocks_max, B, H, N, D, out_dtype, causal, gran, pv_mode;
  bool v_f16, dependent;            // dependent: programmatic launch behind the kernel before it on the stream
  float sm_scale;
};

int attn_launch(const AttnArgs& a, cudaStream_t st);

}  // namespace sparge
