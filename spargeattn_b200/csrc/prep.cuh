// What precedes the selection and the attention kernel of a call, in two launches (three for long sequences).
#pragma once
#include "column_passes.cuh"

namespace sparge {

enum { kVNone, kVFp8, kVHalf };   // V is used as it is / quantised to FP8 / copied as contiguous fp16

struct PrepArgs {
  const void *q, *k, *v;            // [B,H,N,D] views, last dimension contiguous
  long long q_st[3], k_st[3], v_st[3];   // strides of (batch, head, token) in elements
  const float* simthr;              // [H]; NULL: quantise only, no pooling
  void *pq, *pk;                    // pooled
  uint8_t *sim_q, *sim_k;
  int8_t *q8, *k8;
  float *qs, *ks;
  void* v_out;                      // v8 [B,H,N_pad,D] or fp16 [B,H,N,D]
  float* v_scale;                   // [B,H,D]
  void* km;                         // [B,H,D], written when smooth_k
  void* scratch;                    // prep_scratch_bytes()
  int BH, H, N, D, dtype, v_dtype, v_mode, smooth_k;
};

size_t prep_scratch_bytes(int BH, int N, int D);
// v_later: if not NULL, the FP8 quantisation of V is left to the caller, who gets what it needs (v stays NULL if V is not to
// be quantised).
int prep_launch(const PrepArgs& a, VQuantArgs* v_later, cudaStream_t st);

}  // namespace sparge
