// Mask predictor back end: pooled QK^T row -> softmax -> stable top-k (or cdf) selection ->
// forced blocks / causal / sink -> block mask + delta-encoded LUT, one warp per one or two (b, h, q-block) rows.
// Replaces spas_sage_attn/utils.py:386-420 (bmm, masked fills, softmax, sort, cumsum,
// triton_fill_block_map_kernel :282-292, triton_fill_causal_mask :304-311) and
// triton_block_map_to_lut_kernel (utils.py:54-74).
//
// Arithmetic contract (shared with the CPU oracle):
//   score  = T( fma-chain over ascending d, fp32 ) ; score = T( float(score) * float(D^-0.5) )
//   p      = T( float( exp(double(score) - max) / sum ) )           (fp64 softmax)
//   top-k  = first n_sel of a stable descending order of p (ties -> lower block index),
//            n_sel = clamp(int(topk[h] * nk), 1, nk)
//   cdf    = the reference runs torch.cumsum on the sorted probabilities in the 16-bit type and takes
//            torch.searchsorted(cdf, cdfthreshd[h], right=True) (utils.py:398-403). On the device that
//            cumsum is ATen's chunked Sklansky scan (ATen/native/cuda/ScanUtils.cuh,
//            tensor_kernel_scan_innermost_dim: chunks of 2 * num_threads_x values, every combine rounded to
//            the 16-bit type, num_threads_x derived from the row count and row length), and its rounding
//            decides the count on long rows (a bf16 running sum stops growing once the terms fall below
//            half an ulp). The kernel runs the same scan in the same order and the same binary search with
//            the fp32 comparison torch uses, so n_sel equals the reference's wherever the 16-bit
//            probabilities themselves agree; clamped to [1, nk].
//   a row with a score of +inf or NaN (a 16-bit score overflows from 65 520 in fp16) has NaN probabilities only, all equal
//            in the order: its first n_sel blocks, in cdf mode all of them.
#include <cfloat>

#include "launch.cuh"
#include "row_groups.cuh"
#include "select.cuh"

namespace sparge {

constexpr int kSelThreads = 256;

// The attribute is always set to what an SM gives a block, never to what one launch needs: it is the kernel's, and a thread
// with a shorter row would lower it between another thread's attribute and launch.
template <typename K>
static bool allow_dynamic_smem(K kernel, size_t smem) {
  return smem <= 48 * 1024 || cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) == cudaSuccess;
}

// Exclusive prefix count of `flag` over the CTA's threads in thread order, plus CTA total.
// s_warp must hold kSelThreads/32 ints. Contains two __syncthreads.
__device__ __forceinline__ int block_exclusive_count(bool flag, int* s_warp, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned b = __ballot_sync(0xffffffffu, flag);
  const int within = __popc(b & ((1u << lane) - 1u));
  if (lane == 0) s_warp[warp] = __popc(b);
  __syncthreads();
  int before = 0, tot = 0;
#pragma unroll
  for (int w = 0; w < kSelThreads / 32; w++) {
    const int c = s_warp[w];
    before += (w < warp) ? c : 0;
    tot += c;
  }
  __syncthreads();
  total = tot;
  return before + within;
}

// Writes one LUT row from the list of live block indices idx[0..count).
__device__ __forceinline__ void write_lut_row(const int* idx, int count, int nk, int32_t* lut_row, int32_t* valid_out) {
  for (int r = threadIdx.x; r < nk; r += kSelThreads) {
    int v = 0;
    if (r < count) v = idx[r] - (r > 0 ? idx[r - 1] : 0);
    lut_row[r] = v;
  }
  if (threadIdx.x == 0) *valid_out = count;
}

template <typename T>
__device__ __forceinline__ uint32_t key_bits(T v);
template <>
__device__ __forceinline__ uint32_t key_bits<__half>(__half v) { return (uint32_t)__half_as_ushort(v); }
template <>
__device__ __forceinline__ uint32_t key_bits<__nv_bfloat16>(__nv_bfloat16 v) { return (uint32_t)__bfloat16_as_ushort(v); }
template <typename T>
__device__ __forceinline__ float key_value(uint32_t k);
template <>
__device__ __forceinline__ float key_value<__half>(uint32_t k) { return __half2float(__ushort_as_half((unsigned short)k)); }
template <>
__device__ __forceinline__ float key_value<__nv_bfloat16>(uint32_t k) {
  return __bfloat162float(__ushort_as_bfloat16((unsigned short)k));
}

// ---- predictor -----------------------------------------------------------------------------------
// A warp owns RW rows (b, h, q-block) of one head, a CTA WARPS * RW consecutive ones.
//   1  scores: the CTA streams pooled K through shared memory in tiles of 64 rows; lane l of a warp runs the fp32 FMA
//      chains of keys j0 + l and j0 + 32 + l for each of its rows as one packed f32x2 chain (each half rounds on its own).
//      A score is a 16-bit value and is kept as one: two bytes per key and row are all that a row holds, and they become
//      in turn the softmax key, the sort buffer's source and the list of live blocks. (With 32-bit scores, an index list
//      and separate keys a row of 1 861 blocks took 12 KB, three warps fitted per scheduler, and the kernel waited:
//      2.26 ms for 24 heads of 931 x 1861 blocks, 1.14 ms now.)
//   2  per row, by its warp alone (shuffles and ballots): fp64 softmax, selection threshold by bisection over the 16 key
//      bits with eight keys per lane and load, final map and LUT.
// What bounds it: instruction issue of the score chains (1.3 per score and channel), then the fp64 pipe; a short row is a
// chain of dependent reductions. With one row per warp the first tile is asked for together with the query (kernel alone
// 6.64 -> 6.08 us for 64 rows of 32 blocks, 10.78 -> 10.14 for 864 of 72, cdf 16.05 -> 15.20 for 1 024 of 128; causal rows of
// 512 lose, 47.2 -> 48.0 for 3 072), and the three counts of a bisection round share one reduction: causal calls of
// [2,8,1000,128] 36.2 -> 35.6 us and [1,30,2500,128] 90.5 -> 90.0, [1,4,2048,64] 32.5 -> 32.2, cdf [1,16,8191,128] 379.6 ->
// 378.9, although the kernel alone, run again and again, takes 0.1-0.3 us longer.
constexpr int kSelTileKeys = 64;
// Marks of a block that is not self-similar: in place of its score, and in place of its probability (zero, with the sign
// bit telling that the block is live whatever the selection says).
constexpr uint16_t kNotSimilarScore = 0xffff, kNotSimilarKey = 0x8000;

__host__ __device__ inline int next_pow2(int n) {
  int p = 1;
  while (p < n) p <<= 1;
  return p;
}
// log2 of the x-extent of ATen's inner-dimension scan launch (get_log_num_threads_x_inner_scan, uint32 arithmetic)
__host__ __device__ inline int aten_scan_log_threads_x(uint32_t num_rows, uint32_t row_size) {
  uint32_t lx = 0, ly = 0;
  while ((1u << lx) < row_size) ++lx;
  while ((1u << ly) < num_rows) ++ly;
  const uint32_t diff = lx - ly;
  uint32_t v = (9u + diff) / 2u;
  v = v < 4u ? 4u : v;
  return (int)(v > 9u ? 9u : v);
}

// Shared memory of one row, in bytes: keys (16-bit, padded to whole 256-key groups of the bisection); the duplicated
// query (freed after the scores) or, in cdf mode, the sort buffer in the same place; the scanned probabilities.
struct SelectRow {
  int keys, work, cdf;
  __host__ __device__ int total() const { return keys + work + cdf; }
};
__host__ __device__ inline SelectRow select_row(int nk, int D, int cdf_len) {
  SelectRow r;
  r.keys = (nk + 255) / 256 * 512;
  const int sort = cdf_len ? next_pow2(nk) * 2 : 0;
  r.work = ((D * 8 > sort ? D * 8 : sort) + 15) / 16 * 16;
  r.cdf = (cdf_len * 2 + 15) / 16 * 16;
  return r;
}

// exp(x) for x <= 0: x = n ln 2 + r, Taylor polynomial of degree 11 in r (remainder below 7e-15), exponent added. Where
// exp(x) is below 1e-304 it is zero: no sum or 16-bit probability can tell.
__device__ __forceinline__ double exp_nonpositive(double x) {
  if (x < -700.0) return 0.0;
  constexpr double kLn2Hi = 0.6931471824645996, kLn2Lo = -1.90465429995776804525e-09;   // the nearest float (n * hi is exact) + the rest
  const float nf = rintf((float)x * 1.44269504f);
  double r = fma((double)nf, -kLn2Hi, x);
  r = fma((double)nf, -kLn2Lo, r);
  double p = 1.0 / 39916800.0;
  p = fma(p, r, 1.0 / 3628800.0);
  p = fma(p, r, 1.0 / 362880.0);
  p = fma(p, r, 1.0 / 40320.0);
  p = fma(p, r, 1.0 / 5040.0);
  p = fma(p, r, 1.0 / 720.0);
  p = fma(p, r, 1.0 / 120.0);
  p = fma(p, r, 1.0 / 24.0);
  p = fma(p, r, 1.0 / 6.0);
  p = fma(p, r, 0.5);
  p = fma(p, r, 1.0);
  p = fma(p, r, 1.0);
  return __hiloint2double(__double2hiint(p) + ((int)nf << 20), __double2loint(p));
}

// number of a lane's keys (8 in a 128-bit word) that are >= cand, both halves of cand2 holding cand: non-negative 16-bit
// floats order like their bit patterns
template <typename T>
__device__ __forceinline__ int count_ge(uint4 w, uint32_t cand2);
template <>
__device__ __forceinline__ int count_ge<__half>(uint4 w, uint32_t cand2) {
  const __half2 c = *reinterpret_cast<const __half2*>(&cand2);
  const __half2 s = __hadd2(__hadd2(__hge2(*reinterpret_cast<const __half2*>(&w.x), c), __hge2(*reinterpret_cast<const __half2*>(&w.y), c)),
                            __hadd2(__hge2(*reinterpret_cast<const __half2*>(&w.z), c), __hge2(*reinterpret_cast<const __half2*>(&w.w), c)));
  return (int)__low2float(s) + (int)__high2float(s);
}
template <>
__device__ __forceinline__ int count_ge<__nv_bfloat16>(uint4 w, uint32_t cand2) {
  const __nv_bfloat162 c = *reinterpret_cast<const __nv_bfloat162*>(&cand2);
  const __nv_bfloat162 s =
      __hadd2(__hadd2(__hge2(*reinterpret_cast<const __nv_bfloat162*>(&w.x), c), __hge2(*reinterpret_cast<const __nv_bfloat162*>(&w.y), c)),
              __hadd2(__hge2(*reinterpret_cast<const __nv_bfloat162*>(&w.z), c), __hge2(*reinterpret_cast<const __nv_bfloat162*>(&w.w), c)));
  return (int)__low2float(s) + (int)__high2float(s);
}

template <typename T>
__device__ __forceinline__ uint16_t add16(uint16_t a, uint16_t b) {
  return (uint16_t)key_bits<T>(Elem<T>::from_float(__fadd_rn(key_value<T>(a), key_value<T>(b))));
}

// Descending bitonic sort of P2 16-bit keys (two per word, unsigned order) by one warp in shared memory. The position of
// equal keys does not matter: only the sequence of values is used.
__device__ __forceinline__ void sort_descending(uint32_t* buf, int P2, int lane) {
  const int words = P2 / 2;
  for (int kk = 2; kk <= P2; kk <<= 1) {
    for (int jj = kk >> 1; jj > 1; jj >>= 1) {   // partners in different words
      const int jw = jj / 2;
      for (int t = lane; t < words / 2; t += 32) {
        const int i = ((t & ~(jw - 1)) << 1) | (t & (jw - 1)), ip = i | jw;
        const uint32_t a = buf[i], b = buf[ip];
        const uint32_t mx = __vmaxu2(a, b), mn = __vminu2(a, b);
        const bool down = ((2 * i) & kk) == 0;
        buf[i] = down ? mx : mn;
        buf[ip] = down ? mn : mx;
      }
      __syncwarp();
    }
    for (int i = lane; i < words; i += 32) {     // partners in one word
      const uint32_t a = buf[i], lo = min(a & 0xffffu, a >> 16), hi = max(a & 0xffffu, a >> 16);
      buf[i] = ((2 * i) & kk) == 0 ? (hi | (lo << 16)) : (lo | (hi << 16));
    }
    __syncwarp();
  }
}

// ATen's cumsum of nk sorted 16-bit values (see the contract above): chunks of W = 32 V values, the running total enters
// the first value of a chunk, Sklansky combine steps, each sum rounded to the 16-bit type. In registers: value i of a
// chunk is v[i / 32] of lane i % 32.
template <typename T, int V>
__device__ __forceinline__ void scan_chunks(const uint16_t* sorted, uint16_t* cdf, int nk, int lane) {
  uint16_t total = 0;
  for (int c0 = 0; c0 < nk; c0 += 32 * V) {
    uint16_t v[V];
#pragma unroll
    for (int i = 0; i < V; i++) v[i] = (c0 + 32 * i + lane < nk) ? sorted[c0 + 32 * i + lane] : (uint16_t)0;
    if (lane == 0) v[0] = add16<T>(v[0], total);
#pragma unroll
    for (int mm = 0; mm < 5; mm++) {
#pragma unroll
      for (int i = 0; i < V; i++) {
        const uint16_t o = (uint16_t)__shfl_sync(0xffffffffu, (int)v[i], (lane & ~((2 << mm) - 1)) + (1 << mm) - 1);
        if (lane & (1 << mm)) v[i] = add16<T>(v[i], o);
      }
    }
#pragma unroll
    for (int g = 1; g < V; g <<= 1) {
#pragma unroll
      for (int i = 0; i < V; i++)
        if (i & g) v[i] = add16<T>(v[i], (uint16_t)__shfl_sync(0xffffffffu, (int)v[(i & ~(2 * g - 1)) + g - 1], 31));
    }
#pragma unroll
    for (int i = 0; i < V; i++) cdf[c0 + 32 * i + lane] = v[i];
    total = (uint16_t)__shfl_sync(0xffffffffu, (int)v[V - 1], 31);
  }
  __syncwarp();
}
// the same for wider chunks, in shared memory
template <typename T>
__device__ __forceinline__ void scan_chunks_wide(const uint16_t* sorted, uint16_t* cdf, int nk, int log_nx, int lane) {
  const int nx = 1 << log_nx, W = 2 * nx;
  uint16_t total = 0;
  for (int c0 = 0; c0 < nk; c0 += W) {
    uint16_t* buf = cdf + c0;
    for (int i = lane; i < W; i += 32) buf[i] = (c0 + i < nk) ? sorted[c0 + i] : (uint16_t)0;
    __syncwarp();
    if (lane == 0) buf[0] = add16<T>(buf[0], total);
    __syncwarp();
    for (int mm = 0; mm <= log_nx; mm++) {
      const int sgm = 1 << mm;
      for (int t = lane; t < nx; t += 32) {
        const int a = ((t >> mm) << (mm + 1)) | sgm;
        const int ti = a + (t & (sgm - 1)), si = a - 1;
        buf[ti] = add16<T>(buf[ti], buf[si]);
      }
      __syncwarp();
    }
    total = buf[W - 1];
    __syncwarp();
  }
}

template <typename T, int D, int RW, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
select_kernel(const T* pq, const T* pk, const uint8_t* sim_q, const uint8_t* sim_k, const float* topk, const float* cdfthr,
              uint8_t* __restrict__ mask, int32_t* __restrict__ lut, int32_t* __restrict__ valid, int H, int nq, int nk,
              int is_causal, int sink, int best_first, int scan_log_nx, int cdf_len, const __grid_constant__ VQuantArgs vq, int row_ctas) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int kTileRowBytes = D * (int)sizeof(T) + 16;   // 16-byte pad: conflict-free 128-bit reads, one row per lane
  constexpr int kChunksPerRow = D * (int)sizeof(T) / 16;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int q0 = (blockIdx.x * WARPS + warp) * RW, bh = blockIdx.y, h = bh % H;   // this warp's first row
  const SelectRow layout = select_row(nk, D, cdf_len);
  unsigned char* base = smem_raw + kSelTileKeys * kTileRowBytes + (size_t)warp * RW * layout.total();
  auto keys_of = [&](int r) { return reinterpret_cast<uint16_t*>(base + r * layout.total()); };
  auto work_of = [&](int r) { return base + r * layout.total() + layout.keys; };
  // causal: a row sees the key blocks k < 2 (q + 1)
  auto limit_of = [&](int q) { return is_causal ? min(nk, (q + 1) * (kBlockQ / kBlockK)) : nk; };
  pdl_wait();
  // The grid's other blocks quantise V, which only the attention kernel waits for: a row is a chain of latencies or bound by
  // issue, V's pass is bound by memory.
  if ((int)blockIdx.x >= row_ctas) {
    // in the tile's place: the kernel has no static shared memory, which would count against the 48 KB of launch_select
    v_quant_span<D, WARPS * 32>(vq, *reinterpret_cast<float(*)[D]>(smem_raw), blockIdx.x - row_ctas, bh);
    pdl_trigger();
    return;
  }
  // asked for here, needed long after: a row is a chain of short steps, and a load in it would stall all of them
  const float n_or_thr = cdfthr ? cdfthr[h] : topk[h];
  uint8_t q_similar[RW];
#pragma unroll
  for (int r = 0; r < RW; r++) q_similar[r] = sim_q[(size_t)bh * nq + min(q0 + r, nq - 1)];

  // The query, each value twice (a packed FMA takes it as it is), and the first tile: asked for together, one latency less.
  const T* pkb = pk + (size_t)bh * nk * D;
  constexpr int kTileLoads = kSelTileKeys * kChunksPerRow / (WARPS * 32);   // 128-bit loads of a tile by a thread
  constexpr bool kFirstTile = RW == 1 && kTileLoads <= 8;
  auto tile_load = [&](int j0, int i) {
    const int row = i / kChunksPerRow, c = i % kChunksPerRow;
    return j0 + row < nk ? *reinterpret_cast<const uint4*>(pkb + (size_t)(j0 + row) * D + c * 8) : make_uint4(0, 0, 0, 0);
  };
  auto tile_store = [&](int i, const uint4& val) {
    *reinterpret_cast<uint4*>(smem_raw + i / kChunksPerRow * kTileRowBytes + i % kChunksPerRow * 16) = val;
  };
  {
    T qv[RW][D / 32];
#pragma unroll
    for (int r = 0; r < RW; r++)
#pragma unroll
      for (int d = 0; d < D / 32; d++) qv[r][d] = pq[((size_t)bh * nq + min(q0 + r, nq - 1)) * D + d * 32 + lane];
    uint4 first[kFirstTile ? kTileLoads : 1];
    if (kFirstTile) {
#pragma unroll
      for (int i = 0; i < kTileLoads; i++) first[i] = tile_load(0, threadIdx.x + i * WARPS * 32);
    }
#pragma unroll
    for (int r = 0; r < RW; r++)
#pragma unroll
      for (int d = 0; d < D / 32; d++) {
        const float v = Elem<T>::to_float(qv[r][d]);
        reinterpret_cast<float2*>(work_of(r))[d * 32 + lane] = make_float2(v, v);
      }
    if (kFirstTile) {
#pragma unroll
      for (int i = 0; i < kTileLoads; i++) tile_store(threadIdx.x + i * WARPS * 32, first[i]);
    }
  }

  // ---- 1: scores
  const float scale = (D == 64) ? 0.125f : 0.08838834764831845f;   // float(D ** -0.5)
  const uint8_t* simk = sim_k + (size_t)bh * nk;
  const int cta_limit = limit_of(min(nq, ((int)blockIdx.x + 1) * WARPS * RW) - 1);   // keys any row of the CTA sees
  const T minus_inf = Elem<T>::from_float(-INFINITY);
  float m[RW];
#pragma unroll
  for (int r = 0; r < RW; r++) m[r] = -INFINITY;
  for (int j0 = 0; j0 < nk; j0 += kSelTileKeys) {
    const bool seen = j0 < cta_limit;
    uint8_t similar[2];
#pragma unroll
    for (int hf = 0; hf < 2; hf++) similar[hf] = j0 + 32 * hf + lane < nk ? simk[j0 + 32 * hf + lane] : 0;
    if (seen) {
      if (!kFirstTile || j0 > 0) {
        __syncthreads();                                     // previous tile fully consumed
        for (int i = threadIdx.x; i < kSelTileKeys * kChunksPerRow; i += WARPS * 32) tile_store(i, tile_load(j0, i));
      }
      __syncthreads();
    }
    float2 acc[RW];
#pragma unroll
    for (int r = 0; r < RW; r++) acc[r] = make_float2(0.f, 0.f);
    if (seen) {
      const unsigned char* ka = smem_raw + lane * kTileRowBytes;
      const unsigned char* kb = ka + 32 * kTileRowBytes;
#pragma unroll 2
      for (int c = 0; c < kChunksPerRow; c++) {
        const Pack8<T> a = *reinterpret_cast<const Pack8<T>*>(ka + c * 16), b = *reinterpret_cast<const Pack8<T>*>(kb + c * 16);
        float2 k2[8];
#pragma unroll
        for (int i = 0; i < 8; i++) k2[i] = make_float2(Elem<T>::to_float(a.v[i]), Elem<T>::to_float(b.v[i]));
#pragma unroll
        for (int r = 0; r < RW; r++) {
          const float4* qv = reinterpret_cast<const float4*>(work_of(r)) + c * 4;
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float4 q2 = qv[i];
            acc[r] = __ffma2_rn(make_float2(q2.x, q2.y), k2[2 * i], acc[r]);
            acc[r] = __ffma2_rn(make_float2(q2.z, q2.w), k2[2 * i + 1], acc[r]);
          }
        }
      }
    }
#pragma unroll
    for (int hf = 0; hf < 2; hf++) {
      const int j = j0 + 32 * hf + lane;
      const bool in = j < nk;
#pragma unroll
      for (int r = 0; r < RW; r++) {
        T sc = minus_inf;
        if (similar[hf] && j < limit_of(q0 + r)) {
          sc = Elem<T>::from_float(hf ? acc[r].y : acc[r].x);
          sc = Elem<T>::from_float(__fmul_rn(Elem<T>::to_float(sc), scale));
          m[r] = fmaxf(m[r], Elem<T>::to_float(sc));
        }
        if (in) keys_of(r)[j] = similar[hf] ? (uint16_t)key_bits<T>(sc) : kNotSimilarScore;
      }
    }
  }
  __syncwarp();

  // ---- 2: row by row (no block-wide barrier below this line)
#pragma unroll 1
  for (int r = 0; r < RW; r++) {
    const int qi = q0 + r;
    if (qi >= nq) break;
    uint16_t* s_key = keys_of(r);
    const int k_limit = limit_of(qi);
    const float mx = warp_max(m[0]);
    const bool row_forced = q_similar[0] == 0;
#pragma unroll
    for (int i = 0; i + 1 < RW; i++) {                       // the next row's values, without indexing registers
      m[i] = m[i + 1];
      q_similar[i] = q_similar[i + 1];
    }

    // fp64 softmax -> 16-bit keys (p >= 0, so the bit pattern orders like the value). The exponentials are evaluated
    // twice, once for the sum and once for the probabilities, instead of being stored. (The first 256 kept in registers,
    // evaluated four at a time, made the kernel alone 0.1-2 us shorter and calls of short rows longer: a row of 40 blocks has
    // two per lane, and a call fetches the code anew. [1,30,2500,128] top-k 120.1 -> 121.2 us, cdf 162.3 -> 163.2, against cdf
    // [1,16,8191,128] 381.9 -> 380.6.)
    double Z = 0.0;
    for (int j = lane; j < nk; j += 32) {
      const uint16_t raw = s_key[j];
      const float sc = key_value<T>(raw);
      if (raw != kNotSimilarScore && sc != -INFINITY) Z += exp_nonpositive((double)sc - (double)mx);
    }
    Z = warp_sum(Z);
    const double rz = 1.0 / Z;
    // An infinite or NaN score makes all probabilities of its row NaN, which a descending order takes as equal: the first
    // n_sel blocks. Zeros are equal too, and the comparisons below can count them.
    const bool undefined = Z != Z;
    const int padded = (nk + 255) / 256 * 256;
    for (int j = lane; j < padded; j += 32) {
      uint16_t key = 0;
      if (j < nk) {
        const uint16_t raw = s_key[j];
        const float sc = key_value<T>(raw);
        if (raw == kNotSimilarScore) key = kNotSimilarKey;
        else if (sc != -INFINITY && !undefined) key = (uint16_t)key_bits<T>(Elem<T>::from_float((float)(exp_nonpositive((double)sc - (double)mx) * rz)));
      }
      s_key[j] = key;
    }
    __syncwarp();

    // how many blocks to select
    int n_sel;
    if (cdfthr == nullptr) {
      n_sel = (int)__fmul_rn(n_or_thr, (float)nk);           // top-k mode: same count for every row of a head
    } else {
      // cdf mode: the probabilities in descending order, ATen's cumsum of them, then torch.searchsorted(..., right=True):
      // upper-bound binary search, 16-bit cdf compared in fp32
      const float thr = n_or_thr;
      const int P2 = next_pow2(nk);
      uint16_t* sorted = reinterpret_cast<uint16_t*>(work_of(r));
      uint16_t* s_cdf = reinterpret_cast<uint16_t*>(work_of(r) + layout.work);
      for (int i = lane; i < P2; i += 32) sorted[i] = i < nk ? (uint16_t)(s_key[i] & 0x7fff) : (uint16_t)0;
      __syncwarp();
      sort_descending(reinterpret_cast<uint32_t*>(sorted), P2, lane);
      if (scan_log_nx == 4) scan_chunks<T, 1>(sorted, s_cdf, nk, lane);
      else if (scan_log_nx == 5) scan_chunks<T, 2>(sorted, s_cdf, nk, lane);
      else scan_chunks_wide<T>(sorted, s_cdf, nk, scan_log_nx, lane);
      int lo_i = 0, hi_i = nk;
      while (lo_i < hi_i) {
        const int mid = lo_i + ((hi_i - lo_i) >> 1);
        if (!(key_value<T>(s_cdf[mid]) > thr)) lo_i = mid + 1; else hi_i = mid;
      }
      n_sel = undefined ? nk : lo_i;                         // no sum of NaNs exceeds the threshold
    }
    n_sel = max(1, min(n_sel, nk));

    // n_sel-th largest key, two of its 15 value bits per round (three candidates counted at once: the rounds are a chain of
    // reductions); padding and not-similar keys count as zero
    const uint4* groups = reinterpret_cast<const uint4*>(s_key);
    const uint4 own = groups[lane];                          // all there is of a row of up to 256 blocks
    auto count_lane = [&](uint32_t cand) {
      const uint32_t cand2 = cand | (cand << 16);
      int c = count_ge<T>(own, cand2);
      for (int i = lane + 32; i < padded / 8; i += 32) c += count_ge<T>(groups[i], cand2);
      return (unsigned)c;
    };
    auto count = [&](uint32_t cand) { return (int)__reduce_add_sync(0xffffffffu, count_lane(cand)); };
    uint32_t thr_key = count(1u << 14) >= n_sel ? 1u << 14 : 0u;
#pragma unroll 1
    for (int bit = 12; bit >= 0; bit -= 2) {
      int c1, c2, c3;
      const unsigned l1 = count_lane(thr_key | (1u << bit)), l2 = count_lane(thr_key | (2u << bit)), l3 = count_lane(thr_key | (3u << bit));
      if (RW == 1 && padded < 1024) {                        // ten bits hold a count: one reduction for all three
        const unsigned c = __reduce_add_sync(0xffffffffu, l1 | (l2 << 10) | (l3 << 20));
        c1 = c & 1023, c2 = (c >> 10) & 1023, c3 = c >> 20;
      } else {
        c1 = (int)__reduce_add_sync(0xffffffffu, l1), c2 = (int)__reduce_add_sync(0xffffffffu, l2), c3 = (int)__reduce_add_sync(0xffffffffu, l3);
      }
      thr_key |= (uint32_t)((c1 >= n_sel) + (c2 >= n_sel) + (c3 >= n_sel)) << bit;
    }
    const int remaining = n_sel - count(thr_key + 1);

    // final map in index order (ties -> lower index), compacted in place into the list of live blocks: a lane takes eight
    // consecutive keys of a 256-key group, and a position of the list never lies past the keys already read. The best
    // block of the list (largest probability, lowest index) is found on the way.
    uint8_t* mrow = mask ? mask + ((size_t)bh * nq + qi) * nk : nullptr;
    int eq_seen = 0, live_seen = 0;
    uint32_t best = 0;                                       // (probability + 1) << 16 | 0xffff - position in the list
    for (int g0 = 0; g0 < nk; g0 += 256) {
      const int jb = g0 + lane * 8;
      const uint4 w = *reinterpret_cast<const uint4*>(s_key + jb);
      const uint32_t word[4] = {w.x, w.y, w.z, w.w};
      uint32_t eq = 0, live = 0;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t key = (word[i >> 1] >> (16 * (i & 1))) & 0xffffu;
        eq |= (jb + i < nk && (key & 0x7fff) == thr_key) ? 1u << i : 0u;
      }
      int eq_incl = __popc(eq);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, eq_incl, o);
        if (lane >= o) eq_incl += t;
      }
      int eq_rank = eq_seen + eq_incl - __popc(eq);
      eq_seen += __shfl_sync(0xffffffffu, eq_incl, 31);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int j = jb + i;
        const uint32_t key = (word[i >> 1] >> (16 * (i & 1))) & 0xffffu;
        bool on = false;
        if (j < nk) {
          const bool is_eq = (eq >> i) & 1;
          on = key > thr_key || (is_eq && eq_rank < remaining) || row_forced;   // (a not-similar key has the top bit)
          eq_rank += is_eq ? 1 : 0;
          if (is_causal) on = on && j < k_limit;
          if (sink && j == 0) on = true;
          if (mrow) mrow[j] = on ? 1 : 0;
        }
        live |= on ? 1u << i : 0u;
      }
      int incl = __popc(live);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      int pos = live_seen + incl - __popc(live);
      live_seen += __shfl_sync(0xffffffffu, incl, 31);
      __syncwarp();                                          // the whole group has been read
#pragma unroll
      for (int i = 0; i < 8; i++) {
        if ((live >> i) & 1) {
          const uint32_t key = (word[i >> 1] >> (16 * (i & 1))) & 0xffffu;
          best = max(best, (((key & 0x7fff) + 1) << 16) | (uint32_t)(0xffff - pos));
          s_key[pos++] = (uint16_t)(jb + i);
        }
      }
    }
    __syncwarp();
    // Visiting order. Reference order: ascending block index. Best-first: the live block with the largest
    // pooled probability (lowest index on ties) is moved to the front and the rest stay ascending; the
    // deltas may then be negative. Attention is order-independent, but starting at the block that most
    // likely holds the row maxima makes later rescales of the running output rare.
    const uint32_t top = __reduce_max_sync(0xffffffffu, best);
    const int rbest = (best_first && live_seen > 0) ? 0xffff - (int)(top & 0xffffu) : 0;
    const int jbest = live_seen > 0 ? s_key[rbest] : 0;
    int32_t* lrow = lut + ((size_t)bh * nq + qi) * nk;
    for (int i = lane; i < nk; i += 32) {
      int v = 0;
      if (i < live_seen) {
        // element at visiting position i: jbest first, then the ascending list without it
        const int cur = i == 0 ? jbest : s_key[i <= rbest ? i - 1 : i];
        const int prev = i == 0 ? 0 : i == 1 ? jbest : s_key[i - 1 <= rbest ? i - 2 : i - 1];
        v = cur - prev;
      }
      lrow[i] = v;
    }
    if (lane == 0) valid[(size_t)bh * nq + qi] = live_seen;
  }
  pdl_trigger();
}

// One CTA per mask row: compaction of a user block mask into the LUT.
// dynamic smem: int per warp, int idx[nk]
constexpr int kMaskWarps = kSelThreads / 32;
__global__ void __launch_bounds__(kSelThreads) mask_to_lut_kernel(const uint8_t* mask, int elem_size, int32_t* __restrict__ lut,
                                                                  int32_t* __restrict__ valid, int nk) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int* s_warp = reinterpret_cast<int*>(smem_raw);   // not static: that would count against the 48 KB of the launch too
  int* s_idx = s_warp + kMaskWarps;
  const size_t row = blockIdx.x;
  const uint8_t* mrow = mask + row * (size_t)nk * elem_size;
  int live_seen = 0;
  for (int j0 = 0; j0 < nk; j0 += kSelThreads) {
    const int j = j0 + threadIdx.x;
    bool live = false;
    if (j < nk) {
      const uint8_t* p = mrow + (size_t)j * elem_size;
      switch (elem_size) {
        case 1: live = *p != 0; break;
        case 2: live = *reinterpret_cast<const uint16_t*>(p) != 0; break;
        case 4: live = *reinterpret_cast<const uint32_t*>(p) != 0; break;
        default: live = *reinterpret_cast<const uint64_t*>(p) != 0; break;
      }
    }
    int tot;
    const int pos = live_seen + block_exclusive_count(live, s_warp, tot);
    live_seen += tot;
    if (live) s_idx[pos] = j;
  }
  __syncthreads();
  write_lut_row(s_idx, live_seen, nk, lut + row * (size_t)nk, valid + row);
  // nothing here depends on the kernels before this one, but the kernel after it relies on them too: it is released by
  // this one's end
  pdl_wait();
  pdl_trigger();
}

// Counting sort of a group of rows by their number of live blocks, longest first, by one CTA per group. Rows of one bucket
// come in any order: it decides when a row is computed, not what comes out.
constexpr int kOrderThreads = 1024, kOrderBuckets = 256;
__global__ void __launch_bounds__(kOrderThreads) row_order_kernel(const int32_t* valid, int32_t* __restrict__ rows, int heads,
                                                                  int nq, int nk) {
  __shared__ int s_place[kOrderBuckets], s_sum[kOrderBuckets / 32];
  const HeadGroup group = head_group(blockIdx.x, heads, gridDim.x);
  const int tid = threadIdx.x, first = group.first * nq, last = first + group.heads * nq;
  if (tid < kOrderBuckets) s_place[tid] = 0;
  pdl_wait();
  __syncthreads();
  auto bucket = [&](int i) { return kOrderBuckets - 1 - (int)((long long)min(max(valid[i], 0), nk) * (kOrderBuckets - 1) / nk); };
  for (int i = first + tid; i < last; i += kOrderThreads) atomicAdd(&s_place[bucket(i)], 1);
  __syncthreads();
  int mine = 0, incl = 0;
  if (tid < kOrderBuckets) {
    incl = mine = s_place[tid];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if ((tid & 31) >= o) incl += t;
    }
    if ((tid & 31) == 31) s_sum[tid >> 5] = incl;
  }
  __syncthreads();
  if (tid < kOrderBuckets) {
    for (int w = 0; w < tid >> 5; w++) incl += s_sum[w];
    s_place[tid] = first + incl - mine;
  }
  __syncthreads();
  for (int i = first + tid; i < last; i += kOrderThreads) rows[atomicAdd(&s_place[bucket(i)], 1)] = i;
  pdl_trigger();
}

int row_order_launch(const int32_t* valid, int32_t* rows, int heads, int nq, int groups, int nk, cudaStream_t st) {
  return launch(row_order_kernel, dim3(groups), kOrderThreads, 0, st, true, valid, rows, heads, nq, nk) == cudaSuccess ? SPARGE_OK
                                                                                                                      : SPARGE_ERR_CUDA;
}

template <typename T, int D, int RW, int WARPS>
static int launch_select(const SelectArgs& a, cudaStream_t st) {
  // cdf mode reproduces torch.cumsum over the [B*H*nq, nk] matrix of sorted probabilities: the scan's chunking
  // depends on both extents
  const int scan_log_nx = aten_scan_log_threads_x((uint32_t)a.BH * (uint32_t)a.nq, (uint32_t)a.nk);
  const int scan_w = 2 << scan_log_nx;
  const int cdf_len = a.cdf ? (a.nk + scan_w - 1) / scan_w * scan_w : 0;
  const size_t smem = kSelTileKeys * (D * sizeof(T) + 16) + (size_t)WARPS * RW * select_row(a.nk, D, cdf_len).total();
  if (smem > 200 * 1024) return SPARGE_ERR_TOO_LARGE;
  auto kern = select_kernel<T, D, RW, WARPS>;
  if (!allow_dynamic_smem(kern, smem)) return SPARGE_ERR_CUDA;
  const int row_ctas = (a.nq + WARPS * RW - 1) / (WARPS * RW);
  const cudaError_t e = launch(kern, dim3(row_ctas + (a.vq.v ? a.vq.spans : 0), a.BH), WARPS * 32, smem, st, a.dependent,
                               (const T*)a.pq, (const T*)a.pk, a.sim_q, a.sim_k, a.topk, a.cdf, a.mask, a.lut, a.valid, a.H, a.nq,
                               a.nk, a.causal, a.sink, a.best_first, scan_log_nx, cdf_len, a.vq, row_ctas);
  return e == cudaSuccess ? SPARGE_OK : SPARGE_ERR_CUDA;
}

// Two rows per warp share every K value and its conversion, but then a row's steps run behind the other's: worth it where
// the scores are most of the work and rows are plenty. One against two rows per warp, top-k mode, us, by rows per SM:
//   256 x 512 blocks:  59 / 71 at 21, 70 / 71 at 28, 78 / 71 at 31, 94 / 90 at 35, 101 / 90 at 42, 125 / 116 at 55
//   64 x 128:          23 / 26 at 26, 31 / 31 at 35, 34 / 31 at 42;   139 x 278, D = 64: 39 / 42 at 28, 51 / 51 at 34, 57 / 51 at 45
// Causal rows, whose pairs differ in length, gain nothing or lose: 256 x 512 68 / 80 at 35, 97 / 99 at 55. Long rows fill the
// SM's shared memory with fewer warps: 931 x 1861 blocks 324 / 397 at 38, 1 123 / 1 181 at 151. cdf mode, whose sort and scan
// are per row, is always one row per warp (84 / 108 at 21, 178 / 208 at 55).
constexpr long long kSelPairRows = 148 * 32;
template <typename T, int D>
static int dispatch_select(const SelectArgs& a, cudaStream_t st) {
  if (a.nk > 65535) return SPARGE_ERR_TOO_LARGE;             // block indices are kept in 16 bits
  int rc = SPARGE_ERR_TOO_LARGE;
  if (!a.cdf && (long long)a.BH * a.nq >= kSelPairRows) rc = launch_select<T, D, 2, 8>(a, st);
  if (rc == SPARGE_ERR_TOO_LARGE) rc = launch_select<T, D, 1, 4>(a, st);
  if (rc == SPARGE_ERR_TOO_LARGE) rc = launch_select<T, D, 1, 1>(a, st);   // very long rows: one fits an SM
  return rc;
}

int select_launch(const SelectArgs& a, cudaStream_t st) {
  if (a.dtype == SPARGE_F16) return a.D == 64 ? dispatch_select<__half, 64>(a, st) : dispatch_select<__half, 128>(a, st);
  return a.D == 64 ? dispatch_select<__nv_bfloat16, 64>(a, st) : dispatch_select<__nv_bfloat16, 128>(a, st);
}

int mask_to_lut_launch(const void* mask, int elem_size, int32_t* lut, int32_t* valid, long long rows, int nk, bool dependent,
                       cudaStream_t st) {
  if (nk > 50 * 1024 || rows > 2147483647LL) return SPARGE_ERR_TOO_LARGE;
  const size_t smem = ((size_t)kMaskWarps + nk) * sizeof(int);
  if (!allow_dynamic_smem(mask_to_lut_kernel, smem)) return SPARGE_ERR_CUDA;
  const cudaError_t e = launch(mask_to_lut_kernel, dim3((unsigned)rows), kSelThreads, smem, st, dependent, (const uint8_t*)mask,
                               elem_size, lut, valid, nk);
  return e == cudaSuccess ? SPARGE_OK : SPARGE_ERR_CUDA;
}

}  // namespace sparge

extern "C" int sparge_select(const void* pq, const void* pk, const uint8_t* sim_q, const uint8_t* sim_k,
                             const float* topk, const float* cdfthreshd, uint8_t* mask, int32_t* lut, int32_t* valid,
                             int B, int H, int nq, int nk, int D, int dtype, int is_causal, int attention_sink,
                             int lut_order, sparge_stream_t stream) {
  using namespace sparge;
  if (!pq || !pk || !sim_q || !sim_k || !lut || !valid) return SPARGE_ERR_NULL;
  if ((topk == nullptr) == (cdfthreshd == nullptr)) return SPARGE_ERR_INVALID_ARG;
  if (B <= 0 || H <= 0 || nq <= 0 || nk <= 0 || (D != 64 && D != 128) || (dtype != SPARGE_F16 && dtype != SPARGE_BF16))
    return SPARGE_ERR_INVALID_ARG;
  if ((long long)B * H > 65535) return SPARGE_ERR_TOO_LARGE;
  const SelectArgs a = {pq, pk, sim_q, sim_k, topk, cdfthreshd, mask, lut, valid, B * H, H, nq, nk, D, dtype, is_causal,
                        attention_sink, lut_order != 0, false, {}};
  return select_launch(a, (cudaStream_t)stream);
}

extern "C" int sparge_mask_to_lut(const void* mask, int elem_size, int32_t* lut, int32_t* valid, int B, int H, int nq,
                                  int nk, sparge_stream_t stream) {
  using namespace sparge;
  if (!mask || !lut || !valid) return SPARGE_ERR_NULL;
  if (B <= 0 || H <= 0 || nq <= 0 || nk <= 0 || (elem_size != 1 && elem_size != 2 && elem_size != 4 && elem_size != 8))
    return SPARGE_ERR_INVALID_ARG;
  return mask_to_lut_launch(mask, elem_size, lut, valid, (long long)B * H * nq, nk, false, (cudaStream_t)stream);
}
