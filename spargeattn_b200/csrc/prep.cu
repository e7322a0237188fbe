// Q, K and V of one call made ready for the selection and the attention kernel (see prep.cuh):
//   1  Q pooled and quantised | column sums of K | column maxima of V        (one read of each tensor)
//   1b partial sums and maxima combined, when there are many of them
//   2  K pooled and quantised with its mean taken out | V quantised to FP8   (a second read of K and V)
//      (beside a short selection V's part runs in the selection's grid instead: see forward.cu)
// The arithmetic is that of the standalone entries (kmean.cu, pool_quant.cu, quant_v.cu), so the bytes are the same.
//
// Why one launch for three tensors: pooling is bound by instruction issue and the column passes by memory, so their
// CTAs, interleaved in the grid, fill each other's gaps, and a call pays for two launches (three from
// 2 049 tokens on) instead of nine and a memset. The unit of the grid is a span of 256 tokens of one head: with 256 threads that is one or two 128-row
// blocks of Q, two or four 64-row blocks of K, or one column pass that is long enough to keep its loads in flight.
#include "column_passes.cuh"
#include "launch.cuh"
#include "pool_quant.cuh"
#include "prep.cuh"

namespace sparge {

// Up to this many partial results per head are combined by every CTA that needs them (8 KB from L2 at D = 128); from
// there on a kernel of its own does it once per head.
constexpr int kDirectParts = 8;

template <int D>
struct PrepShape {
  static constexpr int kQUnits = D == 128 ? 2 : 1, kQBlocks = D == 128 ? 1 : 2;   // units per span, 128-row blocks per unit
  static constexpr int kKUnits = D == 128 ? 2 : 1, kKBlocks = D == 128 ? 2 : 4;   // units per span, 64-row blocks per unit
};

struct PrepScratch {
  double *kpart, *ksum;   // [BH][spans][D], [BH][D]
  float *vpart, *vmax;
};

static size_t round_up(size_t x) { return (x + 255) / 256 * 256; }

static size_t prep_scratch(int BH, int N, int D, void* base, PrepScratch* s) {
  const size_t spans = ((size_t)N + kSpan - 1) / kSpan, row = (size_t)BH * D;
  const size_t bytes[4] = {row * spans * 8, row * 8, row * spans * 4, row * 4};
  uint8_t* p = static_cast<uint8_t*>(base);
  size_t total = 0;
  void* at[4];
  for (int i = 0; i < 4; i++) {
    at[i] = p + total;
    total += round_up(bytes[i]);
  }
  if (s) *s = PrepScratch{(double*)at[0], (double*)at[1], (float*)at[2], (float*)at[3]};
  return total;
}
size_t prep_scratch_bytes(int BH, int N, int D) { return prep_scratch(BH, N, D, nullptr, nullptr); }

template <typename T>
__device__ __forceinline__ const T* head_of(const void* x, const long long* st, int bh, int H) {
  return static_cast<const T*>(x) + (size_t)(bh / H) * st[0] + (size_t)(bh % H) * st[1];
}

// grid (spans * units, B*H), 256 threads, three CTAs per SM (the register limit of the pooling part).
template <typename T, int D, bool WANT_POOL>
__global__ void __launch_bounds__(kPassThreads, 3) prep_first_kernel(const __grid_constant__ PrepArgs a, PrepScratch s, int spans) {
  using Shape = PrepShape<D>;
  constexpr int QU = Shape::kQUnits, RPP = PassShape<D>::kRowsPerPass;
  __shared__ union {
    PoolQuantShared<D, 128, Shape::kQBlocks, WANT_POOL> pool;
    double sum[RPP][D];
    float amax[RPP][D];
  } sm;
  const int units = gridDim.x / spans, span = blockIdx.x / units, unit = blockIdx.x % units, bh = blockIdx.y;
  const int r0 = span * kSpan, r1 = min(a.N, r0 + kSpan);
  const size_t part = ((size_t)bh * spans + span) * D;
  if (unit < QU) {
    const int first = (span * QU + unit) * Shape::kQBlocks;
    if (first * 128 < a.N)
      pool_quant_blocks<T, D, 128, Shape::kQBlocks, false, WANT_POOL>(
          sm.pool, head_of<T>(a.q, a.q_st, bh, a.H), nullptr, WANT_POOL ? a.simthr[bh % a.H] : 0.f, (T*)a.pq, a.sim_q, a.q8, a.qs,
          a.N, (a.N + 127) / 128, bh, first, a.q_st[2], [] {});
  } else if (unit == QU && a.smooth_k) {
    const double v = column_sum<T, D>(sm.sum, head_of<T>(a.k, a.k_st, bh, a.H), r0, r1, a.k_st[2]);
    if (threadIdx.x < D) s.kpart[part + threadIdx.x] = v;
  } else if (a.v_mode == kVFp8) {
    const float m = a.v_dtype == SPARGE_F16
                        ? column_amax<__half, D>(sm.amax, head_of<__half>(a.v, a.v_st, bh, a.H), r0, r1, a.v_st[2])
                        : column_amax<__nv_bfloat16, D>(sm.amax, head_of<__nv_bfloat16>(a.v, a.v_st, bh, a.H), r0, r1, a.v_st[2]);
    if (threadIdx.x < D) s.vpart[part + threadIdx.x] = m;
  } else {
    __half* out = (__half*)a.v_out + (size_t)bh * a.N * D;
    if (a.v_dtype == SPARGE_F16) v_half_rows<__half, D>(head_of<__half>(a.v, a.v_st, bh, a.H), out, r0, r1, a.v_st[2]);
    else v_half_rows<__nv_bfloat16, D>(head_of<__nv_bfloat16>(a.v, a.v_st, bh, a.H), out, r0, r1, a.v_st[2]);
  }
  pdl_trigger();
}

// grid (B*H), 1024 threads: sums and maxima of a head's partial results.
template <int D>
__global__ void __launch_bounds__(1024) prep_combine_kernel(PrepScratch s, int spans, bool want_k, bool want_v) {
  constexpr int GROUPS = 1024 / D;
  __shared__ double rk[GROUPS][D];
  __shared__ float rv[GROUPS][D];
  pdl_wait();
  const int d = threadIdx.x % D, g = threadIdx.x / D;
  const size_t base = (size_t)blockIdx.x * spans * D + d;
  double k = 0.0;
  float v = 0.f;
#pragma unroll 8
  for (int c = g; c < spans; c += GROUPS) {
    if (want_k) k += s.kpart[base + (size_t)c * D];
    if (want_v) v = fmaxf(v, s.vpart[base + (size_t)c * D]);
  }
  rk[g][d] = k;
  rv[g][d] = v;
  __syncthreads();
  if (g == 0) {
    for (int i = 1; i < GROUPS; i++) {
      k += rk[i][d];
      v = fmaxf(v, rv[i][d]);
    }
    if (want_k) s.ksum[(size_t)blockIdx.x * D + d] = k;
    if (want_v) s.vmax[(size_t)blockIdx.x * D + d] = v;
  }
  pdl_trigger();
}

// grid (spans * units, B*H), 256 threads. kp: `parts` partial results per head. Walks the tensors back to front:
// what the first kernel read last is still in L2.
template <typename T, int D, bool SMOOTH_K, bool WANT_POOL>
__global__ void __launch_bounds__(kPassThreads, 3)
prep_second_kernel(const __grid_constant__ PrepArgs a, const __grid_constant__ VQuantArgs vq, const double* kp, int parts, int spans) {
  using Shape = PrepShape<D>;
  constexpr int KU = Shape::kKUnits;
  __shared__ PoolQuantShared<D, 64, Shape::kKBlocks, WANT_POOL> sm;
  __shared__ __align__(16) T s_km[D];
  __shared__ float s_mul[D];
  const int idx = gridDim.x - 1 - blockIdx.x, bh = gridDim.y - 1 - blockIdx.y, tid = threadIdx.x;
  const int units = gridDim.x / spans, span = idx / units, unit = idx % units;
  if (unit < KU) {
    const int first = (span * KU + unit) * Shape::kKBlocks;
    if (first * 64 < a.N) {
      pool_quant_blocks<T, D, 64, Shape::kKBlocks, SMOOTH_K, WANT_POOL>(
          sm, head_of<T>(a.k, a.k_st, bh, a.H), s_km, WANT_POOL ? a.simthr[bh % a.H] : 0.f, (T*)a.pk, a.sim_k, a.k8, a.ks, a.N,
          (a.N + 63) / 64, bh, first, a.k_st[2], [&] {
            pdl_wait();
            if (SMOOTH_K) {
              if (tid < D) {
                double m = 0.0;
                for (int c = 0; c < parts; c++) m += kp[((size_t)bh * parts + c) * D + tid];
                s_km[tid] = Elem<T>::from_float((float)(m / (double)a.N));
                if (first == 0) static_cast<T*>(a.km)[(size_t)bh * D + tid] = s_km[tid];
              }
              __syncthreads();
            }
          });
    }
  } else {
    pdl_wait();
    v_quant_span<D, kPassThreads>(vq, s_mul, span, bh);
  }
  pdl_trigger();
}

template <typename T, int D>
static int prep_launch_t(const PrepArgs& a, VQuantArgs* v_later, cudaStream_t st) {
  using Shape = PrepShape<D>;
  PrepScratch s;
  prep_scratch(a.BH, a.N, D, a.scratch, &s);
  const int spans = (a.N + kSpan - 1) / kSpan;
  const bool want = a.simthr != nullptr, smooth = a.smooth_k != 0, v8 = a.v_mode == kVFp8;
  const int units1 = Shape::kQUnits + (smooth ? 1 : 0) + (a.v_mode != kVNone ? 1 : 0);
  const int units2 = Shape::kKUnits + (v8 && !v_later ? 1 : 0);
  cudaError_t e = launch(want ? prep_first_kernel<T, D, true> : prep_first_kernel<T, D, false>, dim3(spans * units1, a.BH),
                         kPassThreads, 0, st, false, a, s, spans);
  const double* kp = s.kpart;
  const float* vp = s.vpart;
  int parts = spans;
  if (e == cudaSuccess && spans > kDirectParts && (smooth || v8)) {
    e = launch(prep_combine_kernel<D>, dim3(a.BH), 1024, 0, st, true, s, spans, smooth, v8);
    kp = s.ksum;
    vp = s.vmax;
    parts = 1;
  }
  auto second = smooth ? (want ? prep_second_kernel<T, D, true, true> : prep_second_kernel<T, D, true, false>)
                       : (want ? prep_second_kernel<T, D, false, true> : prep_second_kernel<T, D, false, false>);
  const VQuantArgs vq = {a.v, {a.v_st[0], a.v_st[1], a.v_st[2]}, a.v_out, a.v_scale, vp, parts, spans, a.N, a.H, a.v_dtype};
  if (v_later && v8) *v_later = vq;
  if (e == cudaSuccess) e = launch(second, dim3(spans * units2, a.BH), kPassThreads, 0, st, true, a, vq, kp, parts, spans);
  return e == cudaSuccess ? SPARGE_OK : SPARGE_ERR_CUDA;
}

int prep_launch(const PrepArgs& a, VQuantArgs* v_later, cudaStream_t st) {
  if (a.dtype == SPARGE_F16) return a.D == 64 ? prep_launch_t<__half, 64>(a, v_later, st) : prep_launch_t<__half, 128>(a, v_later, st);
  return a.D == 64 ? prep_launch_t<__nv_bfloat16, 64>(a, v_later, st) : prep_launch_t<__nv_bfloat16, 128>(a, v_later, st);
}

}  // namespace sparge
