// LUT-driven block-sparse attention for sm_100a.
//   S = Q8 K8^T   : tcgen05.mma kind::i8, operands staged by TMA into 128B/64B-swizzled smem,
//                   s32 accumulator in tensor memory (TMEM). Two live 64-key blocks are paired into one
//                   N = 128 step: their K tiles sit next to each other in shared memory, so one
//                   instruction covers both (an odd last block runs as N = 64).
//   online softmax in registers, one thread per query row: one running-maximum update, one output rescale and
//                   one round of hand-offs per 128 keys; P rounded to e4m3 and stored to a 128B-swizzled
//                   shared-memory tile
//   O += P8 V8    : tcgen05.mma kind::f8f6f4, A = P tile (K-major), B = V tiles (token-major,
//                   MN-major descriptor), f32 accumulator in TMEM
// Replaces qk_int_sv_f8_block_sparse_attn_kernel (csrc/qattn/qk_int_sv_f8_cuda_sm89.cuh:42-755)
// and its host wrapper (csrc/qattn/qk_int_sv_f8_cuda_sm89.cu:392-585).
//
// One CTA per (q-block of 128 rows, head, batch); 6 warps:
//   warps 0-3  softmax / correction / epilogue (warp w owns query rows 32 w ... = TMEM lanes)
//   warp  4    TMA producer: walks the delta-encoded LUT and fetches only live K/V blocks
//   warp  5    MMA issuer (one elected lane) and TMEM owner
// TMEM columns: [0,128) S of the current step, [128,128+D) O  -> 256 columns, two CTAs per SM.
//
// What bounds it: the instruction stream of the softmax warps, two per scheduler (one of each CTA). Per score it takes
// the exponential unit 8 cycles of a warp and about four issue slots; everything else a step needs (hand-offs, TMEM
// reads, row maxima, stores) is latency that only the other CTA's warp can fill, so the step is arranged to have as few
// serial stages as possible: a thread reads its 128 scores at once and releases S (QK^T of the next step runs under this
// step's exponentials), and P has two buffers, so that nothing waits for P.V of the previous step except a rescale.
//
// Every wait is bounded; on expiry the kernel records a code in *dev_status and unwinds.
#include <cuda.h>

#include <atomic>

#include "attn.cuh"
#include "launch.cuh"
#include "row_groups.cuh"
#include "sm100_ptx.cuh"
#include "step_word.cuh"

namespace sparge {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kFp8Offset = 8.807f;     // csrc/qattn/attn_utils.cuh:28-30: 2^8.807 = 448 = e4m3 max
constexpr float kMaskValue = -5000000.0f;  // csrc/qattn/attn_utils.cuh:348-352

// PVF16: P and V in fp16 (tcgen05.mma kind::f16) instead of e4m3 -- the arithmetic of the reference's fp16-PV kernel
// (csrc/qattn/qk_int_sv_f16_cuda_sm80.cuh), which its Sage1-signature entry points run. V then is the caller's fp16
// tensor itself (no quantiser); a 64-key V tile is D/64 sub-tiles of [64 keys x 128 bytes] (64 channels each, 128B
// swizzle), P is two sub-tiles of [128 rows x 128 bytes], one per block of a pair. The tiles are twice as large,
// so the rings are shorter (see kKTiles), and at D = 128 P has one buffer, to keep two CTAs per SM.
template <int D, bool PVF16 = false>
struct AttnShape {
  // K ring of single tiles (fp16 variant at D = 128): three 64-key tile slots instead of two pair slots bring the CTA
  // down to 105 KB of shared memory so that two fit per SM; a step's two K tiles are then not
  // adjacent and QK^T is issued as two N = 64 instruction groups.
  static constexpr bool kKTiles = PVF16 && D == 128;
  static constexpr int kStagesK = kKTiles ? 3 : (D == 128 || PVF16) ? 2 : 4;   // ring slots: PAIRS of 64-key tiles (tiles if kKTiles)
  static constexpr int kSlotsV = PVF16 ? 2 : (D == 128 ? 3 : 8);   // single 64-key tiles
  static constexpr int kTileQ = 128 * D;
  static constexpr int kTileKV = 64 * D;
  static constexpr int kPairKV = 2 * kTileKV;
  static constexpr int kTileV = PVF16 ? 2 * kTileKV : kTileKV;
  static constexpr int kTileP = PVF16 ? 2 * 128 * 128 : 128 * 128;   // 128 rows x 128 keys of e4m3 / fp16
  static constexpr int kBuffersP = PVF16 && D == 128 ? 1 : 2;
  static constexpr int kRingK = kStagesK * (kKTiles ? kTileKV : kPairKV);
  static constexpr int kSmemBytes = 1024 + kTileQ + kBuffersP * kTileP + kRingK + kSlotsV * kTileV;
  static constexpr int kTmemCols = 256;
  static constexpr int kCtasPerSm = 2;
  static constexpr uint32_t kSwizzle = (D == 128) ? kSwizzle128B : kSwizzle64B;
};

__device__ __forceinline__ void report(int32_t* status, int code) {
  if (status) atomicCAS(status, 0, code);
}

template <typename OutT>
__device__ __forceinline__ uint32_t pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ void st_shared_v4(uint32_t addr, const uint32_t* w) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}

// Row maximum of a block's 64 scores, in log2 units.
__device__ __forceinline__ float block_rowmax(const uint32_t* sr, float c) {
  int m[4];   // four chains of 3-input maxima: short latency
#pragma unroll
  for (int g = 0; g < 4; g++) {
    m[g] = __vimax3_s32((int)sr[16 * g], (int)sr[16 * g + 1], (int)sr[16 * g + 2]);
#pragma unroll
    for (int k = 3; k < 15; k += 2) m[g] = __vimax3_s32(m[g], (int)sr[16 * g + k], (int)sr[16 * g + k + 1]);
  }
  m[0] = __vimax3_s32(m[0], m[1], (int)sr[15]);
  m[2] = __vimax3_s32(m[2], m[3], (int)sr[31]);
  m[0] = __vimax3_s32(m[0], m[2], (int)sr[47]);
  return __int2float_rn(max(m[0], (int)sr[63])) * c;   // c > 0: max commutes with the scaling
}

// The same with masks and per-column scales: keys with block-local index >= klim are masked. Per-thread granularity
// (QuantGranularity::kPerThread, qk_int_sv_f8_cuda_sm89.cuh:116-136): key column n of a
// block is scaled by entry (n % 8) / 2 of the block's four K scales, so a thread's 64 scores carry four different
// factors c4[0..3] and the integer maximum no longer commutes with the scaling: one maximum per factor.
__device__ __forceinline__ float block_rowmax_masked(const uint32_t* sr, const float* c4, int klim) {
  int mx[4] = {INT_MIN, INT_MIN, INT_MIN, INT_MIN};
#pragma unroll
  for (int k = 0; k < 64; k++) mx[(k & 7) >> 1] = (k < klim) ? max(mx[(k & 7) >> 1], (int)sr[k]) : mx[(k & 7) >> 1];
  float r = kMaskValue;
#pragma unroll
  for (int g = 0; g < 4; g++) r = (mx[g] != INT_MIN) ? fmaxf(r, __int2float_rn(mx[g]) * c4[g]) : r;
  return r;
}

// Probabilities of four neighbouring keys, packed for the P tile: four e4m3 bytes or four fp16.
template <bool PVF16>
__device__ __forceinline__ void pack_p(uint32_t* w, float a, float b, float c, float d) {
  if (PVF16) {
    w[0] = pack2<__half>(a, b);
    w[1] = pack2<__half>(c, d);
  } else {
    w[0] = cvt_e4m3x4(a, b, c, d);
  }
}

// P = 2^(S*c - m + offset) for a block's 64 scores (offset 8.807 for e4m3, 0 for fp16 whose values are at most 1): row
// sum in fp32 before the rounding (ComputeUnit::kCudaCore, qk_int_sv_f8_cuda_sm89.cuh:773); the packed values go to the
// row's 16-byte chunks chunk0 ... of the 128B-swizzled tile. `prow` = shared address of the row, rsw = row & 7.
// The scores are converted with the integer-to-float instruction: it is exact and runs at half rate beside the FMA
// pipe's packed f32x2 work (adding a float bias as an integer multiply-add instead cost 3 % of the kernel).
// EXACT: one factor per pair of key columns (c4, see block_rowmax_masked; all equal for the coarser granularities) and a key
// limit: keys >= klim get probability zero.
template <bool EXACT, bool PVF16>
__device__ __forceinline__ float block_exp(const uint32_t* sr, const float* c4, float m, int klim, uint32_t prow, int chunk0,
                                           int rsw) {
  constexpr int kKeysPerChunk = PVF16 ? 8 : 16;
  const float off = (PVF16 ? 0.f : kFp8Offset) - m;
  const float2 c2 = make_float2(c4[0], c4[0]), o2 = make_float2(off, off);
  float2 s0 = make_float2(0.f, 0.f), s1 = make_float2(0.f, 0.f);
#pragma unroll
  for (int ch = 0; ch < 64 / kKeysPerChunk; ch++) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < kKeysPerChunk; i += 4) {
      const int k = ch * kKeysPerChunk + i;
      float2 a = make_float2(__int2float_rn((int)sr[k]), __int2float_rn((int)sr[k + 1]));
      float2 b = make_float2(__int2float_rn((int)sr[k + 2]), __int2float_rn((int)sr[k + 3]));
      if (EXACT) {
        a = make_float2(fmaf(a.x, c4[(k & 7) >> 1], off), fmaf(a.y, c4[(k & 7) >> 1], off));
        b = make_float2(fmaf(b.x, c4[((k + 2) & 7) >> 1], off), fmaf(b.y, c4[((k + 2) & 7) >> 1], off));
      } else {
        a = __ffma2_rn(a, c2, o2);
        b = __ffma2_rn(b, c2, o2);
      }
      a = make_float2(ex2_approx(a.x), ex2_approx(a.y));
      b = make_float2(ex2_approx(b.x), ex2_approx(b.y));
      if (EXACT) {
        a = make_float2(k < klim ? a.x : 0.f, k + 1 < klim ? a.y : 0.f);
        b = make_float2(k + 2 < klim ? b.x : 0.f, k + 3 < klim ? b.y : 0.f);
      }
      s0 = __fadd2_rn(s0, a);
      s1 = __fadd2_rn(s1, b);
      pack_p<PVF16>(w + (PVF16 ? i / 2 : i / 4), a.x, a.y, b.x, b.y);
    }
    st_shared_v4(prow + (uint32_t)(((chunk0 + ch) ^ rsw) << 4), w);
  }
  s0 = __fadd2_rn(s0, s1);
  return s0.x + s0.y;
}

constexpr int kSoftmaxWarps = 4, kProducerWarp = 4, kMmaWarp = 5;
constexpr int kAttnThreads = 192;

// GRAN = qk_quant_gran: 1 one Q scale per 128-row block, 2 one per 32-row group (the K scale is per 64-key block in
// both), 3 per-thread Q/K scales. PV_MODE = PVThresholdMode: 0 no skip test, 1 the test decides per block, 2 per
// 32-row group. ORDERED: rows in the order of row_order or order_groups (AttnArgs), without row ranges and without counts of
// products. A variant of its own: it takes the row's place from shared memory in the epilogue, and the plain kernel, which has
// it from its block index, is slower like that (calls of [1,12,32760,128] 2 519 -> 2 549 us, [2,30,17776,64] 3 539 -> 3 595,
// with the skip test 2 737 -> 2 860 and 3 900 -> 4 117). With the same rows in the same order a call of the variant takes
// 2 502, 3 540, 2 709 and 3 853 us; in short CTAs the order's arithmetic shows ([1,24,4608,128] 170.7 -> 171.4).
template <int D, bool CAUSAL, int PV_MODE, typename OutT, int GRAN, bool PVF16 = false, bool ORDERED = false>
__global__ void __launch_bounds__(kAttnThreads, (AttnShape<D, PVF16>::kCtasPerSm))
attn_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
            const __grid_constant__ CUtensorMap tmap_v, OutT* __restrict__ o, const int32_t* lut, const int32_t* valid,
            const float* pvthr, const float* q_scale, const float* k_scale, const float* v_scale, int32_t* dev_status, int N,
            int H, int nq, int nk, float sm_scale_log2, long long osb, long long osh, long long osn,
            int32_t* __restrict__ pv_count, const int32_t* q_ranges, const int32_t* row_order, int order_groups) {
  using Shape = AttnShape<D, PVF16>;
  constexpr bool PV_SKIP = PV_MODE != 0, pv_per_warp = PV_MODE == 2, GRAN3 = GRAN == 3;
  constexpr int SK = Shape::kStagesK, NV = Shape::kSlotsV;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sP = smem + Shape::kTileQ;                                // buffer b: sP + b * kTileP
  uint8_t* sK = sP + Shape::kBuffersP * Shape::kTileP;               // slot s: sK + s * kPairKV
  uint8_t* sV = sK + Shape::kRingK;                                  // slot n: sV + n * kTileV
  constexpr bool KT = Shape::kKTiles;

  __shared__ uint64_t bar_q, bar_k_full[SK], bar_k_empty[SK], bar_v_full[NV], bar_v_empty[NV], bar_s_full, bar_s_free,
      bar_p_ready[2], bar_o_done[2], bar_vote[2];   // the pairs alternate by step
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_bh, s_qi;           // ORDERED: the CTA's head and query block
  __shared__ int s_skip[2][2], s_fail;   // [step parity][block of the pair]
  // PV-skip votes, one byte per softmax warp: [step parity][block of the pair]
  __shared__ uint32_t s_vote[2][2];
  __shared__ __align__(16) float s_vscale[PVF16 ? 4 : D];
  __shared__ int4 s_meta[8];           // per step (ring of 8): block indices of the pair and their K scales (as bits)

  // the shuffles let the compiler see that these are the same for the whole warp: branches on them need no convergence
  // bookkeeping and the operands of the MMA instructions can be kept in uniform registers
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  // Query blocks are issued last-first: under a causal mask the late rows hold the most live blocks, and the longest rows of
  // a head, or of a group of heads, start first. row_order names the rows of a map that is not known beforehand.
  // With q_ranges, (batch, head) bh computes only its query blocks [begin, begin + count): the unit of the
  // multi-GPU row sharding. The grid is sized for the largest count; the other CTAs leave at once.
  int at = 0;   // ORDERED: the CTA's row
  if (ORDERED) {
    if (row_order) {
      pdl_wait();
      at = __shfl_sync(0xffffffffu, row_order[blockIdx.y * nq + blockIdx.x], 0);
    } else {
      const HeadGroup group = head_group(group_of_head(blockIdx.y, gridDim.y, order_groups), gridDim.y, order_groups);
      const int j = (blockIdx.y - group.first) * nq + blockIdx.x;
      at = (group.first + j % group.heads) * nq + nq - 1 - j / group.heads;
    }
  }
  const int bh = ORDERED ? at / nq : blockIdx.y, h = bh % H;
  const int q_begin = !ORDERED && q_ranges ? q_ranges[2 * bh] : 0;
  const int q_count = !ORDERED && q_ranges ? min(q_ranges[2 * bh + 1], nq - q_begin) : (int)gridDim.x;
  if (!ORDERED && (int)blockIdx.x >= q_count) {
    pdl_wait();   // when every CTA leaves here, this kernel must still not end before the ones that it depends on
    return;
  }
  const int qi = ORDERED ? at - bh * nq : q_begin + q_count - 1 - (int)blockIdx.x;
  const size_t row_id = (size_t)bh * nq + qi;

  if (warp == kMmaWarp) {
    tmem_alloc(&s_tmem_base, Shape::kTmemCols);
    tmem_relinquish();
  }
  if (tid == kProducerWarp * 32) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    mbar_init(&bar_q, 1);
#pragma unroll
    for (int s = 0; s < SK; s++) {
      mbar_init(&bar_k_full[s], 1);
      mbar_init(&bar_k_empty[s], 1);
    }
#pragma unroll
    for (int s = 0; s < NV; s++) {
      mbar_init(&bar_v_full[s], 1);
      mbar_init(&bar_v_empty[s], 1);
    }
    mbar_init(&bar_s_full, 1);
    mbar_init(&bar_s_free, kSoftmaxWarps);
#pragma unroll
    for (int i = 0; i < 2; i++) {
      mbar_init(&bar_p_ready[i], kSoftmaxWarps);
      mbar_init(&bar_o_done[i], 1);
      mbar_init(&bar_vote[i], kSoftmaxWarps);
    }
    mbar_fence_init();
    s_fail = 0;
    // For the epilogue. A register that lives through the loop in their place costs 1-3 % of a call, and a division of the
    // row's number there 1 % without the skip test ([1,12,32760,128] 2 572 and 2 538 us against 2 500).
    if (ORDERED) {
      s_bh = bh;
      s_qi = qi;
    }
  }
  pdl_wait();   // everything below reads what the kernels before this one wrote
  // V's scales wait in shared memory for the epilogue, where 128 loads per thread from global memory were a fifth of a
  // short CTA's time: 15.2 -> 14.5 us at [1,4,2048,64], 122 -> 119 at [1,24,4608,128]
  if (!PVF16 && tid < D) s_vscale[tid] = v_scale[(size_t)bh * D + tid];
  const int cnt = __shfl_sync(0xffffffffu, min(valid[row_id], nk), 0);
  const int nsteps = (cnt + 1) >> 1;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = s_tmem_base;
  const uint32_t tO = tbase + 128;
  const int32_t* lrow = lut + row_id * nk;

  if (cnt <= 0) {   // no live block: defined output (zeros)
    const int rows = min(128, N - qi * 128);
    constexpr int kChunks = D * (int)sizeof(OutT) / 16;
    OutT* obase = o + (size_t)(bh / H) * osb + (size_t)(bh % H) * osh + (size_t)qi * 128 * osn;
    for (int i = tid; i < rows * kChunks; i += kAttnThreads)
      reinterpret_cast<uint4*>(obase + (size_t)(i / kChunks) * osn)[i % kChunks] = make_uint4(0, 0, 0, 0);
    if (!ORDERED && pv_count && tid < 4) pv_count[row_id * 4 + tid] = 0;
  } else if (warp == kProducerWarp) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      mbar_arrive_expect_tx(&bar_q, Shape::kTileQ);
      tma_load_3d(sQ, &tmap_q, &bar_q, 0, qi * 128, bh);
    }
    // absolute block index of live entry n (n must not decrease between calls): prefix sums of the delta LUT,
    // 32 entries at a time, so that no load depends on the previous one
    const float* ksc = k_scale + (size_t)bh * nk;
    int win = -32, jabs = 0, jcarry = 0;
    float ks_lane = 0.f, ks_out = 0.f;      // K scale of this lane's entry / of the entry last returned
    auto block_of = [&](int n) -> int {
      if (n >= win + 32) {
        win = n & ~31;
        int incl = (win + lane < cnt) ? lrow[win + lane] : 0;
#pragma unroll
        for (int ofs = 1; ofs < 32; ofs <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, ofs);
          if (lane >= ofs) incl += t;
        }
        jabs = jcarry + incl;
        jcarry = __shfl_sync(0xffffffffu, jabs, 31);
        jabs = max(0, min(jabs, nk - 1));
        ks_lane = ksc[jabs];
      }
      ks_out = __shfl_sync(0xffffffffu, ks_lane, n - win);
      return __shfl_sync(0xffffffffu, jabs, n - win);
    };
    int ok = 1, issued_k = 0, issued_v = 0;   // K slots (pairs, or tiles if KT) and V tiles requested
    // The step's block indices and K scales are published before its K tiles are requested: the softmax
    // warps read them once S of that step is complete, which is ordered after the tiles' arrival. The ring
    // slot was last used eight steps ago; the wait for a free K slot has just shown that step s - stages has retired.
    auto load_k = [&](int s, int ja, int jb, const int4& meta) {   // lane 0 only
      if (KT) {   // ring of single tiles: block n of the row's live list goes to slot n % SK
#pragma unroll
        for (int blk = 0; blk < 2; blk++) {
          if (blk == 1 && jb < 0) break;
          const int n = 2 * s + blk, ts = n % SK;
          if (n >= SK) ok = mbar_wait(&bar_k_empty[ts], ((n / SK) - 1) & 1) ? 1 : 0;
          if (!ok) return;
          if (blk == 0) s_meta[s & 7] = meta;
          mbar_arrive_expect_tx(&bar_k_full[ts], Shape::kTileKV);
          tma_load_3d(sK + ts * Shape::kTileKV, &tmap_k, &bar_k_full[ts], 0, (blk ? jb : ja) * 64, bh);
          issued_k = n + 1;
        }
      } else {
        const int slot = s % SK;
        if (s >= SK) ok = mbar_wait(&bar_k_empty[slot], ((s / SK) - 1) & 1) ? 1 : 0;
        if (!ok) return;
        s_meta[s & 7] = meta;
        uint8_t* dst = sK + slot * Shape::kPairKV;
        mbar_arrive_expect_tx(&bar_k_full[slot], (jb >= 0 ? 2 : 1) * Shape::kTileKV);
        tma_load_3d(dst, &tmap_k, &bar_k_full[slot], 0, ja * 64, bh);
        if (jb >= 0) tma_load_3d(dst + Shape::kTileKV, &tmap_k, &bar_k_full[slot], 0, jb * 64, bh);
        issued_k = s + 1;
      }
    };
    auto load_v = [&](int n, int j) {   // tile n of the row's live list; lane 0 only
      const int slot = n % NV;
      if (n >= NV) ok = mbar_wait(&bar_v_empty[slot], ((n / NV) - 1) & 1) ? 1 : 0;
      if (!ok) return;
      uint8_t* dst = sV + slot * Shape::kTileV;
      mbar_arrive_expect_tx(&bar_v_full[slot], Shape::kTileV);
      if (PVF16) {   // D/64 sub-tiles of 64 channels (128 bytes)
#pragma unroll
        for (int nh = 0; nh < D / 64; nh++)
          tma_load_4d(dst + nh * 8192, &tmap_v, &bar_v_full[slot], nh * 128, j * 64, bh % H, bh / H);
      } else {
        tma_load_3d(dst, &tmap_v, &bar_v_full[slot], 0, j * 64, bh);
      }
      issued_v = n + 1;
    };
    int ja = 0, jb = -1;
    for (int s = -1; s < nsteps && ok; s++) {   // K of step s + 1, then V of step s
      int na = -1, nb = -1;
      float ka = 0.f, kb = 0.f;
      if (s + 1 < nsteps) {
        na = block_of(2 * s + 2);
        ka = ks_out;
        if (2 * s + 3 < cnt) {
          nb = block_of(2 * s + 3);
          kb = ks_out;
        }
      }
      if (lane == 0) {
        if (s + 1 < nsteps) {
          // a second block that there is not counts as masked
          auto word = [&](int j) { return step_word(j, (j * 64 + 64 > N) || (CAUSAL && (j * 64 + 63 > qi * 128))); };
          load_k(s + 1, na, nb, make_int4(word(na), nb < 0 ? step_word(0, true) : word(nb), __float_as_int(ka), __float_as_int(kb)));
        }
        if (ok && s >= 0) load_v(2 * s, ja);
        if (ok && s >= 0 && jb >= 0) load_v(2 * s + 1, jb);
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      ja = na;
      jb = nb;
    }
    if (!ok && lane == 0) {
      report(dev_status, SPARGE_DEV_TIMEOUT_PRODUCER);
      // drain our own copies before the CTA's shared memory goes away
      for (int n = max(0, issued_k - SK); n < issued_k; n++) mbar_wait(&bar_k_full[n % SK], (n / SK) & 1);
      for (int n = max(0, issued_v - NV); n < issued_v; n++) mbar_wait(&bar_v_full[n % NV], (n / NV) & 1);
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp walks the loop and one elected lane issues: with warp-uniform control flow the operands of the
    // MMA instructions live in uniform registers. A single-lane loop has to move every descriptor word there by itself
    // first; issuing a step's four P.V instructions that way took about 580 cycles.
    constexpr uint32_t idesc_qk2 = make_idesc(2, 1, 1, 0, 0, 128, 128);  // s32 += s8 * s8, both K-major, two blocks
    constexpr uint32_t idesc_qk1 = make_idesc(2, 1, 1, 0, 0, 128, 64);   // odd last block
    constexpr uint32_t idesc_pv = make_idesc(1, 0, 0, 0, 1, 128, D);     // f32 += e4m3 * e4m3, B MN-major
    constexpr uint32_t idesc_pv16 = make_idesc(1, 0, 0, 0, 1, 128, D);   // f32 += f16 * f16, B MN-major
    constexpr uint32_t sbo = 8 * D;
    // a descriptor's low field is the address in 16-byte units: moving inside a tile or to another slot is one add
    const uint64_t qd = make_smem_desc(smem_u32(sQ), 16, sbo, Shape::kSwizzle);
    const uint64_t kd = make_smem_desc(smem_u32(sK), 16, sbo, Shape::kSwizzle);
    const uint64_t pd = make_smem_desc(smem_u32(sP), 16, 1024, kSwizzle128B);
    const uint64_t vd = PVF16 ? make_smem_desc(smem_u32(sV), 8192, 1024, kSwizzle128B)
                              : make_smem_desc(smem_u32(sV), 64 * D, sbo, Shape::kSwizzle);
    const bool leader = elect_one();
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) { ok = ok && __all_sync(0xffffffffu, mbar_wait(bar, parity)); };
    // waits for the K tiles of step s (one pair slot, or one or two tile slots of the tile ring)
    auto wait_k = [&](int s) {
      if (KT) {
        wait(&bar_k_full[(2 * s) % SK], ((2 * s) / SK) & 1);
        if (cnt - 2 * s >= 2) wait(&bar_k_full[(2 * s + 1) % SK], ((2 * s + 1) / SK) & 1);
      } else {
        wait(&bar_k_full[s % SK], (s / SK) & 1);
      }
    };
    auto issue_qk = [&](int s) {   // the K tiles of step s have arrived, S is free
      tc_fence_after();
      const bool two = cnt - 2 * s >= 2;
      if (KT) {   // the step's tiles are not adjacent in the ring: one N = 64 instruction group per block
        for (int blk = 0; blk < (two ? 2 : 1); blk++) {
          const int ts = (2 * s + blk) % SK;
          if (leader) {
#pragma unroll
            for (int ks = 0; ks < D / 32; ks++)
              mma_i8_ss(tbase + blk * 64, qd + 2 * ks, kd + ts * (Shape::kTileKV >> 4) + 2 * ks, idesc_qk1, ks > 0);
            tc_commit(&bar_k_empty[ts]);
          }
        }
        if (leader) tc_commit(&bar_s_full);
      } else {
        const int slot = s % SK;
        if (leader) {
#pragma unroll
          for (int ks = 0; ks < D / 32; ks++)
            mma_i8_ss(tbase, qd + 2 * ks, kd + slot * (Shape::kPairKV >> 4) + 2 * ks, two ? idesc_qk2 : idesc_qk1, ks > 0);
          tc_commit(&bar_k_empty[slot]);
          tc_commit(&bar_s_full);
        }
      }
    };
    wait(&bar_q, 0);
    wait_k(0);
    if (ok) issue_qk(0);
    bool started = false;          // the skip test may leave out the first products
    for (int s = 0; s < nsteps && ok; s++) {
      // Tiles arrive long before the softmax warps' hand-offs: their barriers are checked first, so that
      // only one wait stands between a hand-off and the MMAs it releases.
      if (s + 1 < nsteps) {
        wait_k(s + 1);
        wait(&bar_s_free, s & 1);      // every softmax warp has read S(s) into registers
        if (!ok) break;
        issue_qk(s + 1);
      }
      const bool two = cnt - 2 * s >= 2;
      wait(&bar_v_full[(2 * s) % NV], ((2 * s) / NV) & 1);
      if (two) wait(&bar_v_full[(2 * s + 1) % NV], ((2 * s + 1) / NV) & 1);
      wait(&bar_p_ready[s & 1], (s >> 1) & 1);
      if (!ok) break;
      tc_fence_after();
      const uint64_t pbuf = pd + (s % Shape::kBuffersP) * (Shape::kTileP >> 4);
#pragma unroll
      for (int blk = 0; blk < 2; blk++) {
        if (blk == 1 && !two) break;
        const int slot = (2 * s + blk) % NV;
        const uint64_t vtile = vd + slot * (Shape::kTileV >> 4);
        if (!(PV_SKIP && __any_sync(0xffffffffu, s_skip[s & 1][blk]))) {
          const uint32_t acc0 = PV_SKIP ? started : (s > 0 || blk > 0);
          if (leader) {
            // fp16: 16 keys by all channels at a time. The instruction is bound by its operands' way out of shared memory, and one
            // per 64 channels fetched every row of P twice at D = 128: 12 KB a step of 16 keys instead of 8 ([1,12,32760,128],
            // top-k 0.5: kernel 3 055 -> 2 963 us in turn under the power cap, 2 741 -> 2 658 before it sets in; whole call 3 167 ->
            // 3 099).
            if (PVF16) {
#pragma unroll
              for (int ks = 0; ks < 4; ks++)
                mma_f16_ss(tO, pbuf + blk * (16384 >> 4) + 2 * ks, vtile + ks * (2048 >> 4), idesc_pv16, ks > 0 ? 1u : acc0);
            } else {
#pragma unroll
              for (int ks = 0; ks < 2; ks++)
                mma_f8_ss(tO, pbuf + 2 * (2 * blk + ks), vtile + ks * (32 * D >> 4), idesc_pv, ks > 0 ? 1u : acc0);
            }
          }
          started = true;
        }
        if (leader) tc_commit(&bar_v_empty[slot]);
      }
      if (leader) tc_commit(&bar_o_done[s & 1]);
    }
    if (!ok && lane == 0) report(dev_status, SPARGE_DEV_TIMEOUT_MMA);
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax / correction / epilogue
    // One thread per query row (TMEM lane). Waits record a failure in s_fail and run on; it is looked at once, in the
    // epilogue.
    const int row = warp * 32 + lane;
    const uint32_t tlane = (uint32_t)(warp * 32) << 16;
    const uint32_t tS = tbase + tlane;
    const int qrow = qi * 128 + row;
    const float qs = (GRAN3 ? q_scale[row_id * 32 + warp * 8 + (lane & 7)]
                            : q_scale[GRAN == 1 ? row_id : row_id * 4 + warp]) * sm_scale_log2;
    const float* ks_row = k_scale + (size_t)bh * nk * 4;   // GRAN3 only: four K scales per block
    const float thr = PV_SKIP ? pvthr[h] : 0.f;
    const uint32_t prow = smem_u32(sP) + (uint32_t)row * 128u;
    const int rsw = row & 7;
    float m = kMaskValue, d = 0.f;
    int npv = 0;   // PV products issued for this query block (all of them unless the skip test fires)
    mbar_wait_or_flag(&bar_s_full, 0, &s_fail, SPARGE_DEV_TIMEOUT_SOFTMAX);
    for (int s = 0; s < nsteps; s++) {   // S of step s is complete
      tc_fence_after();
      uint32_t sr[128];
      tmem_ld32(tS, sr);
      tmem_ld32(tS + 32, sr + 32);
      tmem_ld32(tS + 64, sr + 64);
      tmem_ld32(tS + 96, sr + 96);
      const int4 mt = s_meta[s & 7];   // published by the producer warp before the step's K tiles were requested
      const bool two = cnt - 2 * s >= 2;                          // the last step of an odd count has one block
      // Key masks, or one block only: the general path for both blocks. One test, made while the scores travel, keeps the
      // ordinary step free of branches (with a test per block after the load: 2.44 instead of 2.33 ms at [1,12,32760,128]).
      const bool plain = !GRAN3 && __all_sync(0xffffffffu, !step_masked(mt.x | mt.y));
      float cc[2][4];   // scale of each block's scores (per-thread granularity: of each pair of key columns)
      int klim[2] = {64, 64};   // keys with block-local index >= klim are masked
#pragma unroll
      for (int b = 0; b < 2; b++) {
        cc[b][0] = cc[b][1] = cc[b][2] = cc[b][3] = qs * __int_as_float(b ? mt.w : mt.z);
        if (!plain) {
          const int word = b ? mt.y : mt.x, key0 = step_index(word) * 64;
          if (GRAN3) {
            const float4 k4 = *reinterpret_cast<const float4*>(ks_row + (size_t)step_block(word, nk) * 4);
            cc[b][0] = qs * k4.x; cc[b][1] = qs * k4.y; cc[b][2] = qs * k4.z; cc[b][3] = qs * k4.w;
          }
          klim[b] = min(64, N - key0);
          if (CAUSAL) klim[b] = min(klim[b], qrow - key0 + 1);
          klim[b] = max(klim[b], 0);
        }
      }
      tmem_wait_ld();
      // S is in registers: the MMA warp may overwrite it with the next step's scores
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_s_free);
      float r[2];
      if (plain) {
        r[0] = block_rowmax(sr, cc[0][0]);
        r[1] = block_rowmax(sr + 64, cc[1][0]);
      } else {
        r[0] = block_rowmax_masked(sr, cc[0], klim[0]);
        r[1] = two ? block_rowmax_masked(sr + 64, cc[1], klim[1]) : m;
      }
      const float m1 = fmaxf(m, r[0]);                            // maximum after block A
      const float m2 = fmaxf(m1, r[1]);
      // PV-skip test (qk_int_sv_f8_cuda_sm89.cuh:317-353), per 64-key block as in the reference: a block is dropped
      // when no row's maximum comes within `thr` of the running one -- block A against the maximum before it, block B
      // against the maximum after A. The warps publish their votes now and read the result only after the
      // exponentials, so the reduction latency is hidden; the last two live blocks are never skipped (so a candidate
      // step has two blocks).
      const bool candA = PV_SKIP && (2 * s < cnt - 2), candB = PV_SKIP && (2 * s + 1 < cnt - 2);
      bool own_skip[2] = {false, false};   // this warp's 32 rows vote to drop the block
      if (PV_SKIP && candA) {
        own_skip[0] = __all_sync(0xffffffffu, (r[0] - m) + thr <= 0.f);
        own_skip[1] = __all_sync(0xffffffffu, (r[1] - m1) + thr <= 0.f) && candB;
        if (lane == 0) {
          reinterpret_cast<volatile uint8_t*>(&s_vote[s & 1][0])[warp] = own_skip[0];
          reinterpret_cast<volatile uint8_t*>(&s_vote[s & 1][1])[warp] = own_skip[1];
          mbar_arrive(&bar_vote[s & 1]);
        }
      }
      const float alpha = (s > 0) ? ex2_approx(m - m2) : 0.f;
      const bool need_rescale = (s > 0) && __any_sync(0xffffffffu, m2 > m);
      m = m2;
      // P.V of the step that used this P buffer must have retired before the buffer is overwritten. With two buffers that
      // is step s - 2, whose products were issued before QK^T of this step, so S being complete shows it. With one buffer it
      // is the step before, block by block: its V tile is handed back when its product is done.
      auto wait_p = [&](int b) {
        if (Shape::kBuffersP == 1 && s > 0) {
          const int n = 2 * (s - 1) + b;
          mbar_wait_or_flag(&bar_v_empty[n % NV], (n / NV) & 1, &s_fail, SPARGE_DEV_TIMEOUT_SOFTMAX);
        }
      };
      const uint32_t pb = prow + (s % Shape::kBuffersP) * Shape::kTileP;
      float sum[2] = {0.f, 0.f};
      const uint32_t pb1 = pb + (PVF16 ? 16384u : 0u);
      constexpr int chunkB = PVF16 ? 0 : 4;
      if (plain && !(pv_per_warp && (own_skip[0] || own_skip[1]))) {
        wait_p(0);
        sum[0] = block_exp<false, PVF16>(sr, cc[0], m, 64, pb, 0, rsw);
        wait_p(1);
        sum[1] = block_exp<false, PVF16>(sr + 64, cc[1], m, 64, pb1, chunkB, rsw);
      } else {
        // A 32-row group that drops its block in per-warp mode still writes its rows of P (as zeros, no key being
        // visible): the other groups' rows of the same block may be multiplied.
        wait_p(0);
        wait_p(1);
        sum[0] = block_exp<true, PVF16>(sr, cc[0], m, pv_per_warp && own_skip[0] ? 0 : klim[0], pb, 0, rsw);
        if (two) sum[1] = block_exp<true, PVF16>(sr + 64, cc[1], m, pv_per_warp && own_skip[1] ? 0 : klim[1], pb1, chunkB, rsw);
      }
      // asked here, needed at the end of the step: the answer's latency is hidden
      const bool next_ready = s + 1 < nsteps && mbar_test(&bar_s_full, (s + 1) & 1);
      // A wait names a phase by its parity, so the waiter must know that the phase before it is complete: PV(s-3), the
      // previous user of this barrier, is (see above). With one barrier for all steps that would not hold.
      if (need_rescale) {   // some row of this warp raised its maximum: O must hold everything up to PV(s-1)
        mbar_wait_or_flag(&bar_o_done[(s - 1) & 1], ((s - 1) >> 1) & 1, &s_fail, SPARGE_DEV_TIMEOUT_SOFTMAX);
        tc_fence_after();
        const float2 al2 = make_float2(alpha, alpha);
#pragma unroll
        for (int c0 = 0; c0 < D; c0 += 16) {   // (64 at a time: 2 319 us against 2 307; D = 64: 3 308 against 3 262)
          uint32_t ov[16];
          tmem_ld16(tO + tlane + c0, ov);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const float2 r2 = __fmul2_rn(make_float2(__uint_as_float(ov[i]), __uint_as_float(ov[i + 1])), al2);
            ov[i] = __float_as_uint(r2.x);
            ov[i + 1] = __float_as_uint(r2.y);
          }
          tmem_st16(tO + tlane + c0, ov);
        }
        tmem_wait_st();
      }
      d *= alpha;
      bool skip[2] = {false, false};
      if (PV_SKIP && candA) {
        mbar_wait_or_flag(&bar_vote[s & 1], (s >> 1) & 1, &s_fail, SPARGE_DEV_TIMEOUT_SOFTMAX);
        // The product itself is left out only when all four groups drop the block, which is the per-block decision
        // in either mode.
        const bool skipA = s_vote[s & 1][0] == 0x01010101u, skipB = s_vote[s & 1][1] == 0x01010101u;
        skip[0] = pv_per_warp ? own_skip[0] : skipA;
        skip[1] = pv_per_warp ? own_skip[1] : skipB;
        if (tid == 0) {
          s_skip[s & 1][0] = skipA ? 1 : 0;
          s_skip[s & 1][1] = skipB ? 1 : 0;
        }
        npv += (skip[0] ? 0 : 1) + (skip[1] ? 0 : 1);
      } else {
        if (PV_SKIP && tid == 0) {
          s_skip[s & 1][0] = 0;
          s_skip[s & 1][1] = 0;
        }
        npv += two ? 2 : 1;
      }
      if (!skip[0]) d += sum[0];
      if (!skip[1]) d += sum[1];
      fence_proxy_async_smem();      // P bytes visible to the tensor core's operand fetch
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_p_ready[s & 1]);   // (two barriers: a warp may be a step ahead of another)
      if (s + 1 < nsteps && !__all_sync(0xffffffffu, next_ready))
        mbar_wait_or_flag(&bar_s_full, (s + 1) & 1, &s_fail, SPARGE_DEV_TIMEOUT_SOFTMAX);
    }
    mbar_wait_or_flag(&bar_o_done[(nsteps - 1) & 1], ((nsteps - 1) >> 1) & 1, &s_fail, SPARGE_DEV_TIMEOUT_SOFTMAX);
    tc_fence_after();
    const int fail = *(volatile int*)&s_fail;
    if (__all_sync(0xffffffffu, fail == 0)) {
      // One count per 32-row group, the layout of the reference's PV_Count (qk_int_sv_f8_cuda_sm89.cuh:650-656).
      // With the per-block decision the four entries of a block are equal; with the per-warp decision each group
      // has its own.
      const int bh_end = ORDERED ? *(volatile int*)&s_bh : bh;
      const int qrow_end = ORDERED ? *(volatile int*)&s_qi * 128 + row : qrow;
      if (!ORDERED && pv_count && lane == 0) pv_count[row_id * 4 + warp] = npv;
      // A row that saw no key at all (token-level causal mask over every live block of its row of blocks) has an
      // empty sum: it is written as zeros. (The reference gives such a row the plain average of V over the masked
      // keys, because its mask value is a large finite number and exp2(mask - mask) = 1.)
      const float inv = d > 0.f ? rcp_approx(d) : 0.f;
      OutT* orow = o + (size_t)(bh_end / H) * osb + (size_t)(bh_end % H) * osh + (size_t)qrow_end * osn;
#pragma unroll
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t ov[32];
        tmem_ld32(tO + tlane + c0, ov);
        tmem_wait_ld();
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          // fp16 V carries no scale
          const float4 vs = PVF16 ? make_float4(1.f, 1.f, 1.f, 1.f) : *reinterpret_cast<const float4*>(s_vscale + c0 + 2 * i);
          w[i] = pack2<OutT>(__uint_as_float(ov[2 * i]) * inv * vs.x, __uint_as_float(ov[2 * i + 1]) * inv * vs.y);
          w[i + 1] = pack2<OutT>(__uint_as_float(ov[2 * i + 2]) * inv * vs.z, __uint_as_float(ov[2 * i + 3]) * inv * vs.w);
        }
        if (qrow_end < N) {
          uint4* dst = reinterpret_cast<uint4*>(orow + c0);
#pragma unroll
          for (int i = 0; i < 4; i++) dst[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
        }
      }
    } else if (lane == 0) {
      report(dev_status, fail ? fail : SPARGE_DEV_TIMEOUT_SOFTMAX);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) tmem_dealloc(tbase, Shape::kTmemCols);
}

// ---------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) return nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// Byte tensor [planes, rows, inner] with a [1, box_rows, inner] box, swizzle span = inner bytes.
static bool make_map(CUtensorMap* m, const void* ptr, uint64_t inner, uint64_t rows, uint64_t planes, uint32_t box_rows) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  cuuint64_t dims[3] = {inner, rows, planes};
  cuuint64_t strides[2] = {inner, inner * rows};
  cuuint32_t box[3] = {(cuuint32_t)inner, box_rows, 1};
  cuuint32_t es[3] = {1, 1, 1};
  const CUtensorMapSwizzle sw = inner == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(ptr), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// fp16 V as bytes, any strides: [B, H, N, 2 D], copied as 64 rows of 128 bytes (64 channels; x is 0 or 128); rows past N
// read as zeros.
static bool make_map_v16(CUtensorMap* m, const AttnArgs& a) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  cuuint64_t dims[4] = {2 * (cuuint64_t)a.D, (cuuint64_t)a.N, (cuuint64_t)a.H, (cuuint64_t)a.B};
  cuuint64_t strides[3] = {2 * (cuuint64_t)a.v_st[2], 2 * (cuuint64_t)a.v_st[1], 2 * (cuuint64_t)a.v_st[0]};
  cuuint32_t box[4] = {128, 64, 1, 1};
  cuuint32_t es[4] = {1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void*>(a.v), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Function attributes are per device and outlive the call: set once for each (kernel, device).
static bool attn_attributes(const void* kern, int smem, std::atomic<uint64_t>& done) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  const uint64_t bit = 1ull << (dev & 63);
  if (dev < 64 && (done.load(std::memory_order_acquire) & bit)) return true;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return false;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess)
    return false;
  if (dev < 64) done.fetch_or(bit, std::memory_order_release);
  return true;
}

template <int D, bool CAUSAL, int PV_MODE, typename OutT, int GRAN, bool PVF16, bool ORDERED = false>
static int launch_attn(const AttnArgs& a, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, cudaStream_t st) {
  if (GRAN == 1 && PV_MODE != 2 && !ORDERED && !a.q_ranges && !a.pv_count && (a.row_order || (a.order_groups > 0 && a.order_groups < a.B * a.H)))
    return launch_attn<D, CAUSAL, PV_MODE, OutT, GRAN, PVF16, GRAN == 1 && PV_MODE != 2>(a, tq, tk, tv, st);
  auto kern = attn_kernel<D, CAUSAL, PV_MODE, OutT, GRAN, PVF16, ORDERED>;
  constexpr int smem = AttnShape<D, PVF16>::kSmemBytes;
  static std::atomic<uint64_t> done{0};
  if (!attn_attributes((const void*)kern, smem, done)) return SPARGE_ERR_CUDA;
  const int nq = (a.N + 127) / 128, nk = (a.N + 63) / 64;
  const int gx = a.q_ranges ? min(a.q_blocks_max, nq) : nq;
  const cudaError_t e = launch(kern, dim3(gx, a.B * a.H), kAttnThreads, smem, st, a.dependent, tq, tk, tv, (OutT*)a.o, a.lut,
                               a.valid, a.pvthr, a.q_scale, a.k_scale, a.v_scale, a.dev_status, a.N, a.H, nq, nk,
                               a.sm_scale * kLog2e, a.o_st[0], a.o_st[1], a.o_st[2], a.pv_count, a.q_ranges, a.row_order, a.order_groups);
  return e == cudaSuccess ? SPARGE_OK : SPARGE_ERR_CUDA;
}

// The checks are the callers'; fp16 V has per-block scales and the per-block skip test only.
int attn_launch(const AttnArgs& a, cudaStream_t st) {
  const int BH = a.B * a.H, n_pad = (a.N + 127) / 128 * 128;
  CUtensorMap tq, tk, tv;
  if (!make_map(&tq, a.q8, a.D, a.N, BH, 128) || !make_map(&tk, a.k8, a.D, a.N, BH, 64) ||
      !(a.v_f16 ? make_map_v16(&tv, a) : make_map(&tv, a.v, a.D, n_pad, BH, 64)))
    return SPARGE_ERR_CUDA;
  const bool bf = a.out_dtype == SPARGE_BF16;
#define SPARGE_ATTN_G(DD, C, S, G, F) \
  (bf ? launch_attn<DD, C, S, __nv_bfloat16, G, F>(a, tq, tk, tv, st) : launch_attn<DD, C, S, __half, G, F>(a, tq, tk, tv, st))
#define SPARGE_ATTN(DD, C, S) \
  (a.gran == 3 ? SPARGE_ATTN_G(DD, C, S, 3, false) : a.gran == 2 ? SPARGE_ATTN_G(DD, C, S, 2, false) : SPARGE_ATTN_G(DD, C, S, 1, false))
#define SPARGE_ATTN_S(DD, C) (a.pv_mode == 2 ? SPARGE_ATTN(DD, C, 2) : a.pv_mode == 1 ? SPARGE_ATTN(DD, C, 1) : SPARGE_ATTN(DD, C, 0))
#define SPARGE_F16PV_S(DD, C) (a.pv_mode != 0 ? SPARGE_ATTN_G(DD, C, 1, 1, true) : SPARGE_ATTN_G(DD, C, 0, 1, true))
  if (a.v_f16) {
    if (a.D == 64) return a.causal ? SPARGE_F16PV_S(64, true) : SPARGE_F16PV_S(64, false);
    return a.causal ? SPARGE_F16PV_S(128, true) : SPARGE_F16PV_S(128, false);
  }
  if (a.D == 64) return a.causal ? SPARGE_ATTN_S(64, true) : SPARGE_ATTN_S(64, false);
  return a.causal ? SPARGE_ATTN_S(128, true) : SPARGE_ATTN_S(128, false);
#undef SPARGE_F16PV_S
#undef SPARGE_ATTN_S
#undef SPARGE_ATTN
#undef SPARGE_ATTN_G
}

// One warp waits on an mbarrier that nobody arrives at, with a caller-chosen short limit, and reports
// the expiry through the same status word and code path as the attention kernel's bounded waits.
__global__ void wait_expiry_selftest_kernel(int32_t* dev_status, uint32_t slice_ns, uint32_t slices) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  const bool ok = mbar_wait(&bar, 0, slice_ns, slices);
  if (!ok && threadIdx.x == 0) report(dev_status, SPARGE_DEV_TIMEOUT_SOFTMAX);
}

}  // namespace sparge

extern "C" int sparge_selftest_wait_expiry(int32_t* dev_status, unsigned int slice_ns, unsigned int slices,
                                           sparge_stream_t stream) {
  if (!dev_status) return SPARGE_ERR_NULL;
  // a try lasts about 4 us even with a smaller hint: the test may not wait longer than 0.1 s either way
  if (slice_ns == 0 || slices == 0 || (unsigned long long)std::max(slice_ns, 4000u) * slices > 100000000ull)
    return SPARGE_ERR_INVALID_ARG;
  sparge::wait_expiry_selftest_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(dev_status, slice_ns, slices);
  return sparge::launch_status();
}

extern "C" int sparge_attn_fwd_gran(const int8_t* q_int8, const int8_t* k_int8, const uint8_t* v8, void* o,
                                    const int32_t* lut, const int32_t* valid, const float* pvthreshd,
                                    const float* q_scale, const float* k_scale, const float* v_scale,
                                    int32_t* dev_status, int B, int H, int N, int D, int out_dtype, int is_causal,
                                    float sm_scale, long long o_stride_b, long long o_stride_h, long long o_stride_n,
                                    int32_t* pv_count, const int32_t* q_block_ranges, int q_blocks_max,
                                    int qk_quant_gran, int pv_threshold_mode, sparge_stream_t stream) {
  using namespace sparge;
  if (q_block_ranges && q_blocks_max <= 0) return SPARGE_ERR_INVALID_ARG;
  if (qk_quant_gran < 1 || qk_quant_gran > 3 || pv_threshold_mode < 0 || pv_threshold_mode > 2) return SPARGE_ERR_INVALID_ARG;
  if (pv_threshold_mode == 0) pvthreshd = nullptr;
  else if (!pvthreshd) return SPARGE_ERR_NULL;
  // per-thread K scales are read four at a time
  if (qk_quant_gran == 3 && (reinterpret_cast<uintptr_t>(k_scale) & 15)) return SPARGE_ERR_INVALID_ARG;

  if (!q_int8 || !k_int8 || !v8 || !o || !lut || !valid || !q_scale || !k_scale || !v_scale) return SPARGE_ERR_NULL;
  if (B <= 0 || H <= 0 || N <= 0 || (D != 64 && D != 128) || (out_dtype != SPARGE_F16 && out_dtype != SPARGE_BF16))
    return SPARGE_ERR_INVALID_ARG;
  if (!(sm_scale > 0.f)) return SPARGE_ERR_INVALID_ARG;
  if ((long long)B * H > 65535) return SPARGE_ERR_TOO_LARGE;
  if (!strides_ok(o, o_stride_b, o_stride_h, o_stride_n)) return SPARGE_ERR_INVALID_ARG;
  AttnArgs a = {};
  a.q8 = q_int8, a.k8 = k_int8, a.v = v8, a.o = o;
  a.o_st[0] = o_stride_b, a.o_st[1] = o_stride_h, a.o_st[2] = o_stride_n;
  a.lut = lut, a.valid = valid, a.pvthr = pvthreshd, a.q_scale = q_scale, a.k_scale = k_scale, a.v_scale = v_scale;
  a.dev_status = dev_status, a.pv_count = pv_count, a.q_ranges = q_block_ranges, a.q_blocks_max = q_blocks_max;
  a.B = B, a.H = H, a.N = N, a.D = D, a.out_dtype = out_dtype, a.causal = is_causal, a.gran = qk_quant_gran;
  a.pv_mode = pv_threshold_mode, a.sm_scale = sm_scale;
  return attn_launch(a, (cudaStream_t)stream);
}

extern "C" int sparge_attn_fwd_f16pv(const int8_t* q_int8, const int8_t* k_int8, const void* v_f16, void* o,
                                     const int32_t* lut, const int32_t* valid, const float* pvthreshd,
                                     const float* q_scale, const float* k_scale, int32_t* dev_status, int B, int H, int N,
                                     int D, int out_dtype, int is_causal, float sm_scale, long long o_stride_b,
                                     long long o_stride_h, long long o_stride_n, int32_t* pv_count,
                                     const int32_t* q_block_ranges, int q_blocks_max, sparge_stream_t stream) {
  using namespace sparge;
  if (q_block_ranges && q_blocks_max <= 0) return SPARGE_ERR_INVALID_ARG;
  if (!q_int8 || !k_int8 || !v_f16 || !o || !lut || !valid || !q_scale || !k_scale) return SPARGE_ERR_NULL;
  if (B <= 0 || H <= 0 || N <= 0 || (D != 64 && D != 128) || (out_dtype != SPARGE_F16 && out_dtype != SPARGE_BF16))
    return SPARGE_ERR_INVALID_ARG;
  if (!(sm_scale > 0.f) || (reinterpret_cast<uintptr_t>(v_f16) & 15)) return SPARGE_ERR_INVALID_ARG;
  if ((long long)B * H > 65535) return SPARGE_ERR_TOO_LARGE;
  if (!strides_ok(o, o_stride_b, o_stride_h, o_stride_n)) return SPARGE_ERR_INVALID_ARG;
  AttnArgs a = {};
  a.q8 = q_int8, a.k8 = k_int8, a.v = v_f16, a.v_f16 = true, a.o = o;
  a.v_st[0] = (long long)H * N * D, a.v_st[1] = (long long)N * D, a.v_st[2] = D;
  a.o_st[0] = o_stride_b, a.o_st[1] = o_stride_h, a.o_st[2] = o_stride_n;
  a.lut = lut, a.valid = valid, a.pvthr = pvthreshd, a.q_scale = q_scale, a.k_scale = k_scale;
  a.dev_status = dev_status, a.pv_count = pv_count, a.q_ranges = q_block_ranges, a.q_blocks_max = q_blocks_max;
  a.B = B, a.H = H, a.N = N, a.D = D, a.out_dtype = out_dtype, a.causal = is_causal, a.gran = 1;
  a.pv_mode = pvthreshd != nullptr, a.sm_scale = sm_scale;
  return attn_launch(a, (cudaStream_t)stream);
}

extern "C" int sparge_attn_fwd_rows(const int8_t* q_int8, const int8_t* k_int8, const uint8_t* v8, void* o,
                                    const int32_t* lut, const int32_t* valid, const float* pvthreshd,
                                    const float* q_scale, const float* k_scale, const float* v_scale,
                                    int32_t* dev_status, int B, int H, int N, int D, int out_dtype, int is_causal,
                                    float sm_scale, long long o_stride_b, long long o_stride_h, long long o_stride_n,
                                    int32_t* pv_count, const int32_t* q_block_ranges, int q_blocks_max,
                                    sparge_stream_t stream) {
  return sparge_attn_fwd_gran(q_int8, k_int8, v8, o, lut, valid, pvthreshd, q_scale, k_scale, v_scale, dev_status, B, H, N, D,
                              out_dtype, is_causal, sm_scale, o_stride_b, o_stride_h, o_stride_n, pv_count, q_block_ranges,
                              q_blocks_max, 1, pvthreshd ? 1 : 0, stream);
}

extern "C" int sparge_attn_fwd_pv_count(const int8_t* q_int8, const int8_t* k_int8, const uint8_t* v8, void* o,
                                        const int32_t* lut, const int32_t* valid, const float* pvthreshd,
                                        const float* q_scale, const float* k_scale, const float* v_scale,
                                        int32_t* dev_status, int B, int H, int N, int D, int out_dtype, int is_causal,
                                        float sm_scale, long long o_stride_b, long long o_stride_h, long long o_stride_n,
                                        int32_t* pv_count, sparge_stream_t stream) {
  return sparge_attn_fwd_rows(q_int8, k_int8, v8, o, lut, valid, pvthreshd, q_scale, k_scale, v_scale, dev_status, B, H, N, D,
                              out_dtype, is_causal, sm_scale, o_stride_b, o_stride_h, o_stride_n, pv_count, nullptr, 0, stream);
}

extern "C" int sparge_attn_fwd_strided(const int8_t* q_int8, const int8_t* k_int8, const uint8_t* v8, void* o,
                                       const int32_t* lut, const int32_t* valid, const float* pvthreshd,
                                       const float* q_scale, const float* k_scale, const float* v_scale,
                                       int32_t* dev_status, int B, int H, int N, int D, int out_dtype, int is_causal,
                                       float sm_scale, long long o_stride_b, long long o_stride_h, long long o_stride_n,
                                       sparge_stream_t stream) {
  return sparge_attn_fwd_pv_count(q_int8, k_int8, v8, o, lut, valid, pvthreshd, q_scale, k_scale, v_scale, dev_status, B, H,
                                  N, D, out_dtype, is_causal, sm_scale, o_stride_b, o_stride_h, o_stride_n, nullptr, stream);
}

extern "C" int sparge_attn_fwd(const int8_t* q_int8, const int8_t* k_int8, const uint8_t* v8, void* o,
                               const int32_t* lut, const int32_t* valid, const float* pvthreshd, const float* q_scale,
                               const float* k_scale, const float* v_scale, int32_t* dev_status, int B, int H, int N,
                               int D, int out_dtype, int is_causal, float sm_scale, sparge_stream_t stream) {
  return sparge_attn_fwd_strided(q_int8, k_int8, v8, o, lut, valid, pvthreshd, q_scale, k_scale, v_scale, dev_status, B, H,
                                 N, D, out_dtype, is_causal, sm_scale, (long long)H * N * D, (long long)N * D, D, stream);
}
