// One call for the whole path of spas_sage2_attn_meansim_topk_cuda / spas_sage2_attn_meansim_cuda
// (spas_sage_attn/core.py:39-169), of their fp16-PV counterparts (:235-319) and of block_sparse_sage2_attn_cuda
// (:171-233): K mean, pooling + self-similarity + INT8 quantisation of Q and K, V quantiser, block selection + LUT,
// block-sparse attention, on one stream with every intermediate tensor carved out of one workspace. Four launches (five
// from 2 049 tokens on, six where the rows of a cdf selection are sorted by length), each a programmatic dependent of the
// one before it; issued entry by entry the path takes ten.
#include <algorithm>

#include "attn.cuh"
#include "forward.cuh"
#include "prep.cuh"
#include "select.cuh"

namespace sparge {

static size_t round_up_256(size_t x) { return (x + 255) / 256 * 256; }

size_t forward_layout(int B, int H, int N, int D, int v_bytes_per_value, size_t* off) {
  const size_t BH = (size_t)B * H, nq = ((size_t)N + 127) / 128, nk = ((size_t)N + 63) / 64, npad = nq * 128;
  const size_t bytes[kWsCount] = {
      BH * D * 2,                                  // km
      prep_scratch_bytes(B * H, N, D),             // partial sums and maxima
      BH * nq * D * 2, BH * nk * D * 2,            // pooled q, pooled k
      BH * nq, BH * nk,                            // self-similarity flags
      BH * (size_t)N * D, BH * (size_t)N * D,      // q_int8, k_int8
      BH * nq * 4, BH * nk * 4,                    // q_scale, k_scale
      BH * nq * nk * 4, BH * nq * 4,               // lut, valid
      BH * npad * D * v_bytes_per_value, BH * D * 4};   // v8 (or the fp16 copy of V), v_scale
  size_t total = 0;
  for (int i = 0; i < kWsCount; i++) {
    if (off) off[i] = total;
    total += round_up_256(bytes[i]);
  }
  return total;
}

int forward(const ForwardArgs& a, cudaStream_t st) {
  if (!a.q || !a.k || !a.v || !a.o || !a.workspace) return SPARGE_ERR_NULL;
  const bool select = a.mask == nullptr;
  if (select && !a.simthr) return SPARGE_ERR_NULL;
  if (select && (a.cdf == nullptr) == (a.topk == nullptr)) return SPARGE_ERR_INVALID_ARG;   // exactly one selection rule
  if (a.B <= 0 || a.H <= 0 || a.N < 128 || (a.D != 64 && a.D != 128)) return SPARGE_ERR_INVALID_ARG;
  if ((a.dtype != SPARGE_F16 && a.dtype != SPARGE_BF16) || (a.v_dtype != SPARGE_F16 && a.v_dtype != SPARGE_BF16))
    return SPARGE_ERR_INVALID_ARG;
  if (!select && a.mask_elem_size != 1 && a.mask_elem_size != 2 && a.mask_elem_size != 4 && a.mask_elem_size != 8)
    return SPARGE_ERR_INVALID_ARG;
  if (!(a.sm_scale > 0.f) || (a.q_ranges && a.q_blocks_max <= 0)) return SPARGE_ERR_INVALID_ARG;
  if ((long long)a.B * a.H > 65535) return SPARGE_ERR_TOO_LARGE;
  if (!strides_ok(a.q, a.q_st[0], a.q_st[1], a.q_st[2]) || !strides_ok(a.k, a.k_st[0], a.k_st[1], a.k_st[2]) ||
      !strides_ok(a.v, a.v_st[0], a.v_st[1], a.v_st[2]) || !strides_ok(a.o, a.o_st[0], a.o_st[1], a.o_st[2]))
    return SPARGE_ERR_INVALID_ARG;
  if (reinterpret_cast<uintptr_t>(a.workspace) & 255) return SPARGE_ERR_INVALID_ARG;
  const bool copy_v = forward_copies_v(a.pv_fp16, a.v_dtype, a.v_st);
  size_t off[kWsCount];
  if (a.workspace_bytes < forward_layout(a.B, a.H, a.N, a.D, copy_v ? 2 : a.pv_fp16 ? 0 : 1, off)) return SPARGE_ERR_INVALID_ARG;
  uint8_t* ws = static_cast<uint8_t*>(a.workspace);
  const int nq = (a.N + 127) / 128, nk = (a.N + 63) / 64;
  int32_t *lut = (int32_t*)(ws + off[kWsLut]), *valid = (int32_t*)(ws + off[kWsValid]);

  PrepArgs p = {};
  p.q = a.q, p.k = a.k, p.v = a.v;
  for (int i = 0; i < 3; i++) p.q_st[i] = a.q_st[i], p.k_st[i] = a.k_st[i], p.v_st[i] = a.v_st[i];
  p.simthr = select ? a.simthr : nullptr;
  p.pq = ws + off[kWsPq], p.pk = ws + off[kWsPk], p.sim_q = ws + off[kWsSimQ], p.sim_k = ws + off[kWsSimK];
  p.q8 = (int8_t*)(ws + off[kWsQ8]), p.k8 = (int8_t*)(ws + off[kWsK8]);
  p.qs = (float*)(ws + off[kWsQs]), p.ks = (float*)(ws + off[kWsKs]);
  p.v_out = ws + off[kWsV8], p.v_scale = (float*)(ws + off[kWsVs]), p.km = ws + off[kWsKm], p.scratch = ws + off[kWsScratch];
  p.BH = a.B * a.H, p.H = a.H, p.N = a.N, p.D = a.D, p.dtype = a.dtype, p.v_dtype = a.v_dtype, p.smooth_k = a.smooth_k;
  p.v_mode = copy_v ? kVHalf : a.pv_fp16 ? kVNone : kVFp8;
  // While the selection has at most eight rows per SM it is a chain of latencies that leaves the memory system idle: V is
  // quantised beside it. From there on it fills the chip, and V is cheaper beside K, where its rows are still in L2.
  // Whole call, topk 0.2, us, beside K / beside the selection, by rows of the selection:
  //   below   128 rows ([16 heads, 1000 tokens]) 39.6 / 37.1, 256 ([8,4096]) 49.8 / 48.1, 256 ([1,32760]) 386 / 380,
  //           576 ([16,4608]) 89.1 / 86.6, 864 ([24,4608]) 122.0 / 120.5, 931 ([1,119056]) 1 292 / 1 287,
  //           1 024 ([16,8191]) 250.8 / 251.5; two long heads lose: 1 024 ([2,65536]) 761 / 770
  //   above   1 440 ([40,4608]) 185.3 / 185.0, 1 668 ([12,17776]) 574 / 578, 2 304 ([12,24576]) 728 / 746 (cdf 750 / 771),
  //           3 072 ([12,32760]) 1 411 / 1 420; D = 64 still gains: 1 920 ([30,8192]) 244.2 / 240.8
  VQuantArgs v_later = {};
  const bool v_beside_selection = select && (long long)p.BH * nq <= 8 * 148;
  int rc = prep_launch(p, v_beside_selection ? &v_later : nullptr, st);
  if (rc != SPARGE_OK) return rc;

  if (select) {
    // the skip test exempts the last two live blocks of the visiting order: best-first order only without it
    const SelectArgs s = {p.pq, p.pk, p.sim_q, p.sim_k, a.topk, a.cdf, nullptr, lut, valid, p.BH, a.H, nq, nk, a.D, a.dtype,
                          a.is_causal, a.sink, a.pvthr == nullptr, true, v_later};
    rc = select_launch(s, st);
  } else {
    rc = mask_to_lut_launch(a.mask, a.mask_elem_size, lut, valid, (long long)p.BH * nq, nk, true, st);
  }
  if (rc != SPARGE_OK) return rc;

  // With cdf selection or a causal map the rows differ in length, and a long one that starts late keeps the chip waiting: they
  // are computed longest first, over even groups of as many heads as have their K and V in kOrderBytes. (Full groups and a rest
  // of one or two heads start the rest's longest rows last, which is slower than head by head: cdf [1,24,5632,128] 303 us head
  // by head, 312 as 22 + 2 heads, 295 as 12 + 12; causal top-k [1,17,8192,128] 267 / 271 / 244, [1,16,50000,64] 4 564 / 4 601 /
  // 4 411, fp16 P.V [1,16,16384,128] 944 / 991 / 876.) A causal row is the longer the later it is; other rows are sorted by
  // their counts.
  // kOrderBytes: with 16 MB the groups are short, above L2's 126 MB their K and V do not stay there; between, no size is the best.
  // Calls in us, head by head and with 16 / 32 / 64 / 96 MB, runs of one setting differ by 0.1-0.5 %, by up to 4 % where marked *:
  //   causal top-k  [1,40,15000,64] 1 400 and 1 306 / 1 301 / 1 298 / 1 298; * [1,32,32768,128] 5 408 and 5 270 / 5 160 / 5 137 /
  //                 5 147, [1,8,65536,128] 4 371 and 4 378 / 4 229 / 4 188 / 4 183; * fp16 P.V [1,9,32768,128] 1 900 and 1 900 /
  //                 1 830 / 1 766 / 1 780
  //   cdf           [1,24,5632,128] 303.0 and 295.4 / 292.8 / 295.3 / 295.4, [2,30,17776,64] 5 328 and 5 237 / 5 248 / 5 234 / 5 261;
  //                 * [1,12,32760,128] 3 457 and 3 305 / 3 245 / 3 297 / 3 233; fp16 P.V [1,24,16200,64] 1 919 and 1 838 / 1 820 /
  //                 1 836 / 1 827
  // Counts are sorted where there are more rows than the chip holds at a time; just above that the order gives 20 % or nothing,
  // by what the second wave happens to be (cdf [1,3,14400,64], 339 rows, three draws: 303 -> 252, 258, 251; 400 rows 299 -> 288,
  // 279 -> 285, 296 -> 264). Rows of one length, as when no query block is alike in itself, pay for the sort and gain nothing:
  // 239.5 -> 241.8 with 64 blocks ([1,24,4096,128]), 435.6 -> 437.1 with 94 ([1,24,6000,128]); kSortBlocks keeps that price
  // below 1 %. Rows that differ gain on both sides of it: 64 blocks 201.7 -> 197.1, [1,12,4096,64] 116.2 -> 105.2; 88 blocks
  // 303.0 -> 292.8; 48 blocks 201.5 -> 201.2 ([1,40,3072,128]).
  constexpr long long kOrderBytes = 32LL << 20;
  constexpr int kSortBlocks = 80;
  const long long head_bytes = (a.pv_fp16 ? 3LL : 2LL) * a.N * a.D;
  const int most_heads = (int)std::max(1LL, std::min((long long)p.BH, kOrderBytes / head_bytes));
  const int order_groups = (p.BH + most_heads - 1) / most_heads;
  int32_t* rows = nullptr;
  if (select && a.cdf && !a.q_ranges && nk > kSortBlocks && (long long)p.BH * nq > 2 * 148) {
    rows = static_cast<int32_t*>(p.scratch);   // free again: the preparation's partial sums
    rc = row_order_launch(valid, rows, p.BH, nq, order_groups, nk, st);
    if (rc != SPARGE_OK) return rc;
  }

  AttnArgs t = {};
  t.q8 = p.q8, t.k8 = p.k8, t.o = a.o, t.lut = lut, t.valid = valid, t.pvthr = a.pvthr;
  t.q_scale = p.qs, t.k_scale = p.ks, t.v_scale = p.v_scale, t.dev_status = a.dev_status;
  t.v_f16 = a.pv_fp16;
  t.v = a.pv_fp16 && !copy_v ? a.v : p.v_out;
  const long long packed[3] = {(long long)a.H * a.N * a.D, (long long)a.N * a.D, a.D};
  for (int i = 0; i < 3; i++) {
    t.o_st[i] = a.o_st[i];
    t.v_st[i] = copy_v ? packed[i] : a.v_st[i];
  }
  t.row_order = rows, t.order_groups = select && a.is_causal ? order_groups : 0;
  t.q_ranges = a.q_ranges, t.q_blocks_max = a.q_blocks_max, t.B = a.B, t.H = a.H, t.N = a.N, t.D = a.D;
  t.out_dtype = a.dtype, t.causal = a.kernel_causal, t.gran = 1, t.pv_mode = a.pvthr != nullptr, t.dependent = true;
  t.sm_scale = a.sm_scale;
  return attn_launch(t, st);
}

}  // namespace sparge

extern "C" size_t sparge_forward_workspace_bytes(int B, int H, int N, int D) {
  if (B <= 0 || H <= 0 || N <= 0 || (D != 64 && D != 128)) return 0;
  return sparge::forward_layout(B, H, N, D, 1, nullptr);
}

extern "C" int sparge_forward_workspace_layout(int B, int H, int N, int D, size_t* offsets, int n_offsets) {
  if (!offsets) return SPARGE_ERR_NULL;
  if (B <= 0 || H <= 0 || N <= 0 || (D != 64 && D != 128) || n_offsets != sparge::kWsCount) return SPARGE_ERR_INVALID_ARG;
  sparge::forward_layout(B, H, N, D, 1, offsets);
  return SPARGE_OK;
}

extern "C" int sparge_meansim_forward(const void* q, const void* k, const void* v, void* o, const float* simthreshd1,
                                      const float* cdfthreshd, const float* topk, const float* pvthreshd, void* workspace,
                                      size_t workspace_bytes, int32_t* dev_status, int B, int H, int N, int D, int dtype,
                                      int v_dtype, int is_causal, int kernel_causal, int attention_sink, int smooth_k,
                                      float sm_scale, const long long* q_strides, const long long* k_strides,
                                      const long long* v_strides, const long long* o_strides, sparge_stream_t stream) {
  if (!simthreshd1 || !q_strides || !k_strides || !v_strides || !o_strides) return SPARGE_ERR_NULL;
  sparge::ForwardArgs a = {};
  a.q = q, a.k = k, a.v = v, a.o = o, a.simthr = simthreshd1, a.cdf = cdfthreshd, a.topk = topk, a.pvthr = pvthreshd;
  for (int i = 0; i < 3; i++) a.q_st[i] = q_strides[i], a.k_st[i] = k_strides[i], a.v_st[i] = v_strides[i], a.o_st[i] = o_strides[i];
  a.workspace = workspace, a.workspace_bytes = workspace_bytes, a.dev_status = dev_status;
  a.B = B, a.H = H, a.N = N, a.D = D, a.dtype = dtype, a.v_dtype = v_dtype, a.is_causal = is_causal;
  a.kernel_causal = kernel_causal, a.sink = attention_sink, a.smooth_k = smooth_k, a.sm_scale = sm_scale;
  return sparge::forward(a, (cudaStream_t)stream);
}
