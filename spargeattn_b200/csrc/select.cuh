// Launches of the block selection (select.cu) for the C entry points.
#pragma once
#include "column_passes.cuh"

namespace sparge {

struct SelectArgs {
  const void *pq, *pk;              // pooled [B,H,nq,D], [B,H,nk,D]
  const uint8_t *sim_q, *sim_k;
  const float *topk, *cdf;          // [H], exactly one
  uint8_t* mask;                    // [B,H,nq,nk] or NULL
  int32_t *lut, *valid;
  int BH, H, nq, nk, D, dtype, causal, sink, best_first;
  bool dependent;                   // programmatic launch behind the kernel before it on the stream
  VQuantArgs vq;                    // V quantised beside the selection; v == NULL: none
};
int select_launch(const SelectArgs& a, cudaStream_t st);

// rows [heads * nq]: the row numbers, in `groups` even groups of heads, in a group the largest counts (of nk) first
int row_order_launch(const int32_t* valid, int32_t* rows, int heads, int nq, int groups, int nk, cudaStream_t st);

int mask_to_lut_launch(const void* mask, int elem_size, int32_t* lut, int32_t* valid, long long rows, int nk, bool dependent,
                       cudaStream_t st);

}  // namespace sparge
