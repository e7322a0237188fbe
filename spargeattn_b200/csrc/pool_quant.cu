// Standalone entry of the pooling / INT8 quantiser of pool_quant.cuh: one block of rows per CTA.
#include "pool_quant.cuh"

namespace sparge {

// Registers are capped so that 768 threads stay resident per SM (three 128-row blocks of D = 128): measured
// 46 / 48 us for Q / K on a [1, 12, 32760, 128] tensor against 52 / 53 us with 512 resident threads and 63 / 50
// with 1024 (which spills).
constexpr int kPoolQuantResidentThreads = 768;

template <typename T, int D, int BS, bool HAS_KM, bool WANT_POOL>
__global__ void __launch_bounds__((BS / 8) * (D / 8), kPoolQuantResidentThreads / ((BS / 8) * (D / 8)))
pool_quant_kernel(const T* __restrict__ x, const T* __restrict__ km, const float* __restrict__ simthr,
                  T* __restrict__ pool, uint8_t* __restrict__ sim, int8_t* __restrict__ xq,
                  float* __restrict__ scale_out, int N, int H, int nb, long long sb, long long sh, long long sn) {
  __shared__ PoolQuantShared<D, BS, 1, WANT_POOL> sm;
  const int bh = blockIdx.y;
  pool_quant_blocks<T, D, BS, 1, HAS_KM, WANT_POOL>(sm, x + (size_t)(bh / H) * sb + (size_t)(bh % H) * sh,
                                                    HAS_KM ? km + (size_t)bh * D : nullptr, WANT_POOL ? simthr[bh % H] : 0.f,
                                                    pool, sim, xq, scale_out, N, nb, bh, blockIdx.x, sn, [] {});
}

template <typename T, int D, int BS>
static int launch_pq(const void* x, const void* km, const float* thr, void* pool, uint8_t* sim, int8_t* xq, float* sc,
                     int BH, int H, int N, long long sb, long long sh, long long sn, cudaStream_t st) {
  const int nb = BS == 32 ? (N + 127) / 128 * 4 : (N + BS - 1) / BS;
  dim3 grid(nb, BH);
  const bool has_km = km != nullptr, want = thr != nullptr;
#define SPARGE_PQ(KM, WP)                                                                                         \
  pool_quant_kernel<T, D, BS, KM, WP><<<grid, (BS / 8) * (D / 8), 0, st>>>((const T*)x, (const T*)km, thr, (T*)pool, sim, xq, sc, \
                                                            N, H, nb, sb, sh, sn)
  if (has_km && want) SPARGE_PQ(true, true);
  else if (has_km) SPARGE_PQ(true, false);
  else if (want) SPARGE_PQ(false, true);
  else SPARGE_PQ(false, false);
#undef SPARGE_PQ
  return launch_status();
}

template <typename T>
static int dispatch_pq(const void* x, const void* km, const float* thr, void* pool, uint8_t* sim, int8_t* xq, float* sc,
                       int BH, int H, int N, int D, int block, long long sb, long long sh, long long sn, cudaStream_t st) {
  if (D == 64 && block == 32) return launch_pq<T, 64, 32>(x, km, thr, pool, sim, xq, sc, BH, H, N, sb, sh, sn, st);
  if (D == 128 && block == 32) return launch_pq<T, 128, 32>(x, km, thr, pool, sim, xq, sc, BH, H, N, sb, sh, sn, st);
  if (D == 64 && block == 128) return launch_pq<T, 64, 128>(x, km, thr, pool, sim, xq, sc, BH, H, N, sb, sh, sn, st);
  if (D == 64 && block == 64) return launch_pq<T, 64, 64>(x, km, thr, pool, sim, xq, sc, BH, H, N, sb, sh, sn, st);
  if (D == 128 && block == 128) return launch_pq<T, 128, 128>(x, km, thr, pool, sim, xq, sc, BH, H, N, sb, sh, sn, st);
  return launch_pq<T, 128, 64>(x, km, thr, pool, sim, xq, sc, BH, H, N, sb, sh, sn, st);
}

}  // namespace sparge

extern "C" int sparge_pool_quant_strided(const void* x, const void* km, const float* simthreshd1, void* pool,
                                         uint8_t* sim, int8_t* x_int8, float* scale, int B, int H, int N, int D,
                                         int block, int dtype, long long stride_b, long long stride_h,
                                         long long stride_n, sparge_stream_t stream) {
  using namespace sparge;
  if (!x || !x_int8 || !scale) return SPARGE_ERR_NULL;
  if (simthreshd1 && (!pool || !sim)) return SPARGE_ERR_NULL;
  if (B <= 0 || H <= 0 || N <= 0 || (D != 64 && D != 128) || (block != 32 && block != 64 && block != 128) ||
      (dtype != SPARGE_F16 && dtype != SPARGE_BF16))
    return SPARGE_ERR_INVALID_ARG;
  if (block == 32 && simthreshd1) return SPARGE_ERR_UNSUPPORTED;   // 32-row groups are a quantiser granularity only
  if ((long long)B * H > 65535) return SPARGE_ERR_TOO_LARGE;
  if (!strides_ok(x, stride_b, stride_h, stride_n)) return SPARGE_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == SPARGE_F16)
    return dispatch_pq<__half>(x, km, simthreshd1, pool, sim, x_int8, scale, B * H, H, N, D, block, stride_b, stride_h,
                               stride_n, st);
  return dispatch_pq<__nv_bfloat16>(x, km, simthreshd1, pool, sim, x_int8, scale, B * H, H, N, D, block, stride_b,
                                    stride_h, stride_n, st);
}

extern "C" int sparge_pool_quant(const void* x, const void* km, const float* simthreshd1, void* pool, uint8_t* sim,
                                 int8_t* x_int8, float* scale, int B, int H, int N, int D, int block, int dtype,
                                 sparge_stream_t stream) {
  return sparge_pool_quant_strided(x, km, simthreshd1, pool, sim, x_int8, scale, B, H, N, D, block, dtype,
                                   (long long)H * N * D, (long long)N * D, D, stream);
}
