// Passes of one 256-thread CTA over a range of rows of one [N, D] head: column sums (K mean), column maxima and FP8
// quantisation (V), fp16 conversion (V of the fp16-PV path). A thread owns 8 channels of every (256 / (D/8))-th row and
// keeps several 128-bit loads in flight: with one load per trip the column sum waited on memory with half of its issue
// slots idle (33.6 -> 27.5 us for a 100 MB tensor).
#pragma once
#include "common.cuh"
#include "sm100_ptx.cuh"

namespace sparge {

// What the FP8 quantisation of V needs once the column maxima are known.
struct VQuantArgs {
  const void* v;                    // [B,H,N,D] view; NULL: nothing to do
  long long st[3];                  // strides of (batch, head, token) in elements
  void* out;                        // [B,H,N_pad,D] e4m3
  float* v_scale;                   // [B,H,D]
  const float* vmax;                // [B*H, parts, D]
  int parts, spans, N, H, dtype;
};

constexpr int kPassThreads = 256;
constexpr int kSpan = 256;   // tokens of one head that a CTA takes
constexpr float kVScaleMax = 2.25f;   // spas_sage_attn/core.py:151

template <int D, int THREADS = kPassThreads>
struct PassShape {
  static constexpr int kThreadsPerRow = D / 8, kRowsPerPass = THREADS / kThreadsPerRow;
};

// fp16(v) of two neighbouring values: what the V quantiser sees whatever the input type. Pairs all through: converting,
// comparing and scaling one value at a time took a third more instructions.
template <typename T>
__device__ __forceinline__ __half2 to_half2(const T* v);
template <>
__device__ __forceinline__ __half2 to_half2<__half>(const __half* v) { return *reinterpret_cast<const __half2*>(v); }
template <>
__device__ __forceinline__ __half2 to_half2<__nv_bfloat16>(const __nv_bfloat16* v) {
  const uint32_t w = *reinterpret_cast<const uint32_t*>(v);
  return __float22half2_rn(make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)));
}

// a / b as fused.cu computes it under --use_fast_math
__device__ __forceinline__ float div_approx(float a, float b) {
  float q;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(q) : "f"(a), "f"(b));
  return q;
}
// multiplier of the V quantiser for a channel's maximum (an all-zero channel is emitted as zeros)
__device__ __forceinline__ float v_multiplier(float amax) { return amax > 0.f ? div_approx(kVScaleMax, amax) : 0.f; }

// f(row, values) for the rows of [row_begin, row_end) that this thread owns, UNROLL loads in flight
template <typename T, int D, int UNROLL, int THREADS = kPassThreads, typename F>
__device__ __forceinline__ void for_rows(const T* __restrict__ head, int row_begin, int row_end, long long sn, F f) {
  constexpr int TPR = PassShape<D, THREADS>::kThreadsPerRow, RPP = PassShape<D, THREADS>::kRowsPerPass;
  const int cg = threadIdx.x % TPR;
  int row = row_begin + threadIdx.x / TPR;
  for (; row + (UNROLL - 1) * RPP < row_end; row += UNROLL * RPP) {
    Pack8<T> p[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; u++) p[u] = *reinterpret_cast<const Pack8<T>*>(head + (size_t)(row + u * RPP) * sn + cg * 8);
#pragma unroll
    for (int u = 0; u < UNROLL; u++) f(row + u * RPP, p[u]);
  }
  for (; row < row_end; row += RPP) f(row, *reinterpret_cast<const Pack8<T>*>(head + (size_t)row * sn + cg * 8));
}

// Column sums in fp64 (independent of the order for all practical purposes): threads 0 .. D-1 return column tid's sum.
template <typename T, int D>
__device__ __forceinline__ double column_sum(double (*red)[D], const T* __restrict__ head, int row_begin, int row_end, long long sn) {
  constexpr int TPR = PassShape<D>::kThreadsPerRow, RPP = PassShape<D>::kRowsPerPass;
  const int tid = threadIdx.x, cg = tid % TPR, r0 = tid / TPR;
  double acc[8];
#pragma unroll
  for (int i = 0; i < 8; i++) acc[i] = 0.0;
  for_rows<T, D, 8>(head, row_begin, row_end, sn, [&](int, const Pack8<T>& p) {
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i] += (double)Elem<T>::to_float(p.v[i]);
  });
#pragma unroll
  for (int i = 0; i < 8; i++) red[r0][cg * 8 + i] = acc[i];
  __syncthreads();
  double s = 0.0;
  if (tid < D) {
#pragma unroll 4
    for (int r = 0; r < RPP; r++) s += red[r][tid];
  }
  return s;
}

// Column maxima of |fp16(v)|: threads 0 .. D-1 return column tid's maximum.
template <typename T, int D>
__device__ __forceinline__ float column_amax(float (*red)[D], const T* __restrict__ head, int row_begin, int row_end, long long sn) {
  constexpr int TPR = PassShape<D>::kThreadsPerRow, RPP = PassShape<D>::kRowsPerPass;
  const int tid = threadIdx.x, cg = tid % TPR, r0 = tid / TPR;
  __half2 mx[4];
#pragma unroll
  for (int i = 0; i < 4; i++) mx[i] = __floats2half2_rn(0.f, 0.f);
  for_rows<T, D, 8>(head, row_begin, row_end, sn, [&](int, const Pack8<T>& p) {
#pragma unroll
    for (int i = 0; i < 4; i++) mx[i] = __hmax2(mx[i], __habs2(to_half2<T>(p.v + 2 * i)));
  });
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float2 f = __half22float2(mx[i]);
    red[r0][cg * 8 + 2 * i] = f.x;
    red[r0][cg * 8 + 2 * i + 1] = f.y;
  }
  __syncthreads();
  float m = 0.f;
  if (tid < D) {
#pragma unroll 4
    for (int r = 0; r < RPP; r++) m = fmaxf(m, red[r][tid]);
  }
  return m;
}

// FP8 quantisation of rows [row_begin, row_end) of the padded output; r8: multipliers of this thread's 8 channels
template <typename T, int D, int THREADS = kPassThreads>
__device__ __forceinline__ void v_quant_rows(const T* __restrict__ head, uint8_t* __restrict__ out, const float* r8, int row_begin,
                                             int row_end, int N, long long sn) {
  constexpr int TPR = PassShape<D, THREADS>::kThreadsPerRow, RPP = PassShape<D, THREADS>::kRowsPerPass;
  const int cg = threadIdx.x % TPR, r0 = threadIdx.x / TPR;
  for_rows<T, D, 4, THREADS>(head, row_begin, min(row_end, N), sn, [&](int row, const Pack8<T>& p) {
    float2 f[4];
#pragma unroll
    for (int i = 0; i < 4; i++) f[i] = __fmul2_rn(__half22float2(to_half2<T>(p.v + 2 * i)), make_float2(r8[2 * i], r8[2 * i + 1]));
    *reinterpret_cast<uint2*>(out + (size_t)row * D + cg * 8) =
        make_uint2(cvt_e4m3x4(f[0].x, f[0].y, f[1].x, f[1].y), cvt_e4m3x4(f[2].x, f[2].y, f[3].x, f[3].y));
  });
  for (int row = max(row_begin, N) + r0; row < row_end; row += RPP)   // padding rows are zeros
    *reinterpret_cast<uint2*>(out + (size_t)row * D + cg * 8) = make_uint2(0u, 0u);
}

// FP8 quantisation of one span of one head by a CTA of THREADS threads, from the head's column maxima
template <int D, int THREADS>
__device__ __forceinline__ void v_quant_span(const VQuantArgs& a, float (&s_mul)[D], int span, int bh) {
  const int tid = threadIdx.x, n_pad = (a.N + 127) / 128 * 128, r0 = span * kSpan, r1 = min(n_pad, r0 + kSpan);
  for (int d = tid; d < D; d += THREADS) {
    float m = 0.f;
#pragma unroll 8
    for (int c = 0; c < a.parts; c++) m = fmaxf(m, a.vmax[((size_t)bh * a.parts + c) * D + d]);
    s_mul[d] = v_multiplier(m);
    if (span == 0) a.v_scale[(size_t)bh * D + d] = div_approx(m, kVScaleMax);
  }
  __syncthreads();
  float r8[8];
#pragma unroll
  for (int i = 0; i < 8; i++) r8[i] = s_mul[(tid % PassShape<D>::kThreadsPerRow) * 8 + i];
  uint8_t* out = (uint8_t*)a.out + (size_t)bh * n_pad * D;
  const size_t head = (size_t)(bh / a.H) * a.st[0] + (size_t)(bh % a.H) * a.st[1];
  if (a.dtype == SPARGE_F16) v_quant_rows<__half, D, THREADS>((const __half*)a.v + head, out, r8, r0, r1, a.N, a.st[2]);
  else v_quant_rows<__nv_bfloat16, D, THREADS>((const __nv_bfloat16*)a.v + head, out, r8, r0, r1, a.N, a.st[2]);
}

// fp16 copy of rows [row_begin, row_end)
template <typename T, int D>
__device__ __forceinline__ void v_half_rows(const T* __restrict__ head, __half* __restrict__ out, int row_begin, int row_end,
                                            long long sn) {
  const int cg = threadIdx.x % PassShape<D>::kThreadsPerRow;
  for_rows<T, D, 8>(head, row_begin, row_end, sn, [&](int row, const Pack8<T>& p) {
    alignas(16) __half2 h[4];
#pragma unroll
    for (int i = 0; i < 4; i++) h[i] = to_half2<T>(p.v + 2 * i);
    *reinterpret_cast<uint4*>(out + (size_t)row * D + cg * 8) = *reinterpret_cast<const uint4*>(h);
  });
}

}  // namespace sparge
