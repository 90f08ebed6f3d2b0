// Operand packing for the tensor-core Schur update.
//
// The reference converts the fp32 L and U panels into an fp16 copy with the
// same column-major layout as A (src/lu_nopiv.hxx:155-164, convert kernel
// src/convert.cu:324-360).  The tensor core wants both operands K-major, so
// here the L21 panel is transposed while it is converted (row-major copy)
// and the U12 panel keeps its column-major layout with a compact leading
// dimension.  e4m3 copies carry one power-of-two scale per 128-row /
// 128-column tile, the largest that keeps the tile's max |x| <= 448; split
// fp16 copies (hi + lo) the same with bound 32768, which keeps the lo parts
// of all but the tile's tiniest entries normal fp16 numbers.
#include "common.cuh"
#include "kernels.cuh"
#include "tc_gemm.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace lub {
namespace {

namespace cg = cooperative_groups;

template <typename T> __device__ __forceinline__ T to_low(float x);
template <> __device__ __forceinline__ __half to_low<__half>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ __nv_bfloat16 to_low<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ uint8_t to_low<uint8_t>(float x) {
  return (uint8_t)__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3);
}

__device__ __forceinline__ float to_f32(float x) { return x; }
__device__ __forceinline__ float to_f32(__half x) { return __half2float(x); }

constexpr int TA = 64;  // tile edge of the transposing pack

// Eight consecutive operand values: one 16-byte (fp8: 8-byte) store, or one by
// one where the destination is not aligned or fewer are inside.
template <typename T>
__device__ __forceinline__ void store8(T* dst, const float (&x)[8], int count) {
  T y[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) y[e] = to_low<T>(x[e]);
  if (count >= 8 && (reinterpret_cast<uintptr_t>(dst) & (8 * sizeof(T) - 1)) == 0) {
    if constexpr (sizeof(T) == 2) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<uint4*>(y);
    else *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<uint2*>(y);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (e < count) dst[e] = y[e];
  }
}

// Split fp16: x = hi + lo with hi = rn(x), lo = rn(x - hi) (x - hi exact).
__device__ __forceinline__ void split16(float x, float& hi, float& lo) {
  hi = __half2float(__float2half_rn(x));
  lo = __fsub_rn(x, hi);
}

// The value's eight copies: T itself, or (split, kp > 0) three fp16 segments of
// length kp, A [hi | hi | lo], B [hi ; lo ; hi], zeros in [K, kp).
template <typename T, bool SPLIT, bool IS_A>
__device__ __forceinline__ void put8(T* row, int64_t k, int64_t K, int64_t kp,
                                     const float (&x)[8]) {
  if constexpr (SPLIT) {
    float hi[8], lo[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) split16(x[e], hi[e], lo[e]);
    const int count = (int)((kp - k) < 8 ? (kp - k) : 8);
    store8(row + k, hi, count);
    store8(row + kp + k, IS_A ? hi : lo, count);
    store8(row + 2 * kp + k, IS_A ? lo : hi, count);
  } else {
    store8(row + k, x, (int)((K - k) < 8 ? (K - k) : 8));
  }
}

// R rows x 64 columns of A (from i0, k0) into the tile [k][i] by 256 threads:
// 16-byte loads of 4 (fp16: 8) rows where the source is aligned; m: the largest
// |x| seen.  Outside of A: zeros.
template <int R, typename S>
__device__ __forceinline__ void load_block(float* tile, int64_t M, int64_t K, const S* src,
                                           int64_t lds, int64_t i0, int64_t k0, float& m) {
  constexpr int V = 16 / sizeof(S);
  const bool vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0 && lds % V == 0 && i0 + R <= M;
  if (vec) {
    src += i0 + k0 * lds;
#pragma unroll
    for (int u = 0; u < R * TA / V / 256; ++u) {
      const int q = u * 256 + threadIdx.x;
      const int i = V * (q % (R / V)), k = q / (R / V);
      uint4 w = make_uint4(0, 0, 0, 0);
      if (k0 + k < K) w = *reinterpret_cast<const uint4*>(src + i + k * lds);
      const S* v = reinterpret_cast<const S*>(&w);
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const float x = to_f32(v[e]);
        m = fmaxf(m, fabsf(x));
        tile[k * (R + 1) + i + e] = x;
      }
    }
  } else {
#pragma unroll 8
    for (int q = threadIdx.x; q < R * TA; q += 256) {
      const int i = q % R, k = q / R;
      const float x = (i0 + i < M && k0 + k < K) ? to_f32(src[i0 + i + (k0 + k) * lds]) : 0.0f;
      m = fmaxf(m, fabsf(x));
      tile[k * (R + 1) + i] = x;
    }
  }
}

// The tile's rows out along K, eight values per thread and step, times 2^sc.
template <int R, typename T, bool SPLIT, bool SCALED>
__device__ __forceinline__ void store_block(const float* tile, int64_t M, int64_t K, int64_t kp,
                                            T* dst, int64_t ldd, int64_t i0, int64_t k0, int sc) {
  const int64_t kend = SPLIT ? kp : K;
#pragma unroll
  for (int u = 0; u < R * TA / 8 / 256; ++u) {
    const int q = u * 256 + threadIdx.x;
    const int k = 8 * (q & 7), i = q >> 3;
    if (i0 + i < M && k0 + k < kend) {
      float x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        x[e] = tile[(k + e) * (R + 1) + i];
        if (SCALED) x[e] = ldexpf(x[e], sc);
      }
      put8<T, SPLIT, true>(dst + (i0 + i) * ldd, k0 + k, K, kp, x);
    }
  }
}

// Values [k, k + 8) of a column of B; zeros past K.
template <typename S>
__device__ __forceinline__ void load8(const S* col, int64_t k, int64_t K, bool vec, float (&x)[8]) {
  if (vec && k + 8 <= K) {
    uint4 u[sizeof(S) / 2];
#pragma unroll
    for (int e = 0; e < (int)sizeof(S) / 2; ++e) u[e] = reinterpret_cast<const uint4*>(col + k)[e];
    const S* v = reinterpret_cast<const S*>(u);
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = to_f32(v[e]);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = k + e < K ? to_f32(col[k + e]) : 0.0f;
  }
}

template <typename S>
__device__ __forceinline__ bool cols_aligned(const S* src, int64_t lds) {
  return (reinterpret_cast<uintptr_t>(src) & 15) == 0 && lds % (16 / sizeof(S)) == 0;
}

// S: source element type (fp32, or fp16 for the fp16-operand gemm entry,
// whose values pass through unchanged).  16-byte loads and stores through the
// transposing tile: 6000 x 500 fp16 11.5 -> 6.0 us.  err (optional) is cleared: the error
// word of the update that reads the copy.
template <typename T, typename S = float>
__global__ void __launch_bounds__(256)
pack_a_kernel(int64_t M, int64_t K, const S* __restrict__ src, int64_t lds,
              T* __restrict__ dst, int64_t ldd, int* err) {
  __shared__ float tile[TA * (TA + 1)];  // [k][i]
  dependency_wait();
  const int64_t i0 = (int64_t)blockIdx.x * TA, k0 = (int64_t)blockIdx.y * TA;
  if (err && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *err = 0;
  float m = 0.0f;
  load_block<TA>(tile, M, K, src, lds, i0, k0, m);
  __syncthreads();
  store_block<TA, T, false, false>(tile, M, K, 0, dst, ldd, i0, k0, 0);
}

constexpr int kBCols = 8;   // columns per block of the B copy: one per warp

template <typename T, typename S = float>
__global__ void __launch_bounds__(256)
pack_b_kernel(int64_t K, int64_t N, const S* __restrict__ src, int64_t lds,
              T* __restrict__ dst, int64_t ldd) {
  dependency_wait();
  const int64_t j = (int64_t)blockIdx.x * kBCols + (threadIdx.x >> 5);
  if (j >= N) return;
  const bool vec = cols_aligned(src, lds);
  for (int64_t k = 8 * (threadIdx.x & 31); k < K; k += 256) {
    float x[8];
    load8(src + j * lds, k, K, vec, x);
    put8<T, false, false>(dst + j * ldd, k, K, 0, x);
  }
}

// s = largest integer with amax * 2^s <= bound (0 for an all-zero or
// non-finite tile).
__device__ __forceinline__ int scale_of(float a, float bound) {
  int s = 0;
  if (a > 0.0f && isfinite(a)) {
    int e, eb;
    frexpf(a, &e);      // a in [2^(e-1), 2^e)
    frexpf(bound, &eb); // bound in [2^(eb-1), 2^eb)
    s = eb - 1 - e;     // a * 2^s < 2^(eb-1) <= bound
    while (ldexpf(a, s + 1) <= bound) ++s;
    while (ldexpf(a, s) > bound) --s;
  }
  return s;
}

// Scaled kinds: a cluster of four CTAs per 128-row tile of A (the first nA) or
// 128-column tile of B.  Each CTA holds 64 of the K values of the tile's rows
// (columns) in shared memory (registers), the four find the largest |x| and so
// the scale over distributed shared memory, and write the copy: the source is
// read once for K <= 256, the outer step, twice beyond.  Eight launches before
// (two clears, two maxima, two scales, two copies), on the panel's critical
// path: 39 us per outer step at 8192 rows and columns, K = 256; now 10 (bound
// by one round trip to memory, the cluster's exchange and the stores; the whole
// e4m3 factorization at n = 8192 5.39 -> 4.46 ms).
constexpr int kScaledCtas = 4;
constexpr int kScaledK = kScaledCtas * TA;

template <typename T, bool SPLIT>
__global__ void __cluster_dims__(kScaledCtas, 1, 1) __launch_bounds__(256)
pack_scaled_kernel(int nA, int64_t M, int64_t N, int64_t K, int64_t kp,
                   const float* __restrict__ a, int64_t lda, T* __restrict__ da,
                   int* __restrict__ sa, const float* __restrict__ b, int64_t ldb,
                   T* __restrict__ db, int* __restrict__ sb, int64_t ldd, float bound) {
  __shared__ float tile[TA * (128 + 1)];  // [k][i]
  __shared__ float red[8];
  __shared__ float part[kScaledCtas];     // each CTA's maximum, from all four
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  cg::cluster_group cl = cg::this_cluster();
  dependency_wait();
  cl.barrier_arrive();   // waited for before the first remote store
  const int rank = (int)cl.block_rank();
  const int t = (int)(blockIdx.x / kScaledCtas);
  const bool is_a = t < nA;
  const int64_t t0 = (int64_t)(is_a ? t : t - nA) * 128;
  const int64_t kend = SPLIT ? kp : K;
  const bool vec = cols_aligned(b, ldb);
  const int64_t kfirst = (int64_t)rank * TA;
  float x[4][8];   // B: thread's column t0 + tid / 8 + 32 u, values k + 8 (tid % 8) ..
  float m = 0.0f;
  for (int64_t k0 = kfirst; k0 < K; k0 += kScaledK) {
    if (is_a) {
      load_block<128>(tile, M, K, a, lda, t0, k0, m);
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t j = t0 + (tid >> 3) + 32 * u;
        load8(b + j * ldb, k0 + 8 * (tid & 7), j < N ? K : 0, vec, x[u]);
#pragma unroll
        for (int e = 0; e < 8; ++e) m = fmaxf(m, fabsf(x[u][e]));
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) red[warp] = m;
  __syncthreads();
  cl.barrier_wait();
  if (tid < kScaledCtas) {
    float y = red[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) y = fmaxf(y, red[w]);
    *cl.map_shared_rank(&part[rank], tid) = y;
  }
  cl.sync();
  m = fmaxf(fmaxf(part[0], part[1]), fmaxf(part[2], part[3]));
  const int sc = scale_of(m, bound);
  if (rank == 0 && tid == 0) (is_a ? sa : sb)[t0 / 128] = sc;
  const bool again = K > kScaledK;  // the tile was overwritten
  for (int64_t k0 = kfirst; k0 < kend; k0 += kScaledK) {
    if (is_a) {
      if (again || k0 >= K) {
        __syncthreads();
        load_block<128>(tile, M, K, a, lda, t0, k0, m);
        __syncthreads();
      }
      store_block<128, T, SPLIT, true>(tile, M, K, kp, da, ldd, t0, k0, sc);
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t j = t0 + (tid >> 3) + 32 * u, k = k0 + 8 * (tid & 7);
        if (j >= N || k >= kend) continue;
        if (again || k0 >= K) load8(b + j * ldb, k, K, vec, x[u]);
        float y[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = ldexpf(x[u][e], sc);
        put8<T, SPLIT, false>(db + j * ldd, k, K, kp, y);
      }
    }
  }
}

template <typename T, typename S>
lu_status pack_a_typed(cudaStream_t st, int64_t M, int64_t K, const S* src,
                       int64_t lds, void* dst, int64_t ldd, int* err = nullptr) {
  dim3 grid((unsigned)ceil_div(M, TA), (unsigned)ceil_div(K, TA));
  LUB_CUDA_TRY(launch_dependent(pack_a_kernel<T, S>, grid, 256, 0, st, M, K, src, lds, (T*)dst,
                                ldd, err));
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

template <typename T, typename S>
lu_status pack_b_typed(cudaStream_t st, int64_t K, int64_t N, const S* src,
                       int64_t lds, void* dst, int64_t ldd) {
  LUB_CUDA_TRY(launch_dependent(pack_b_kernel<T, S>, (unsigned)ceil_div(N, kBCols), 256, 0, st, K,
                                N, src, lds, (T*)dst, ldd));
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

}  // namespace

lu_status launch_pack_a(cudaStream_t st, TcOperand kind, int64_t M, int64_t K,
                        const float* src, int64_t lds, void* dst, int64_t ldd) {
  if (M <= 0 || K <= 0) return LU_SUCCESS;
  switch (kind) {
    case TcOperand::F16: return pack_a_typed<__half>(st, M, K, src, lds, dst, ldd);
    case TcOperand::BF16: return pack_a_typed<__nv_bfloat16>(st, M, K, src, lds, dst, ldd);
    default: return LU_ERR_INVALID_ARG;
  }
}

lu_status launch_pack_b(cudaStream_t st, TcOperand kind, int64_t K, int64_t N,
                        const float* src, int64_t lds, void* dst, int64_t ldd) {
  if (N <= 0 || K <= 0) return LU_SUCCESS;
  switch (kind) {
    case TcOperand::F16: return pack_b_typed<__half>(st, K, N, src, lds, dst, ldd);
    case TcOperand::BF16: return pack_b_typed<__nv_bfloat16>(st, K, N, src, lds, dst, ldd);
    default: return LU_ERR_INVALID_ARG;
  }
}

lu_status launch_pack_a_f16(cudaStream_t st, int64_t M, int64_t K, const __half* src,
                            int64_t lds, __half* dst, int64_t ldd, int* err) {
  if (M <= 0 || K <= 0) return LU_SUCCESS;
  return pack_a_typed<__half>(st, M, K, src, lds, dst, ldd, err);
}

lu_status launch_pack_b_f16(cudaStream_t st, int64_t K, int64_t N, const __half* src,
                            int64_t lds, __half* dst, int64_t ldd) {
  if (N <= 0 || K <= 0) return LU_SUCCESS;
  return pack_b_typed<__half>(st, K, N, src, lds, dst, ldd);
}

lu_status launch_pack_scaled(cudaStream_t st, TcOperand kind, int64_t M, int64_t N, int64_t K,
                             const float* a, int64_t lda, void* da, int* sa, const float* b,
                             int64_t ldb, void* db, int* sb, int64_t ldd) {
  M = std::max<int64_t>(M, 0);
  N = std::max<int64_t>(N, 0);
  const int64_t nA = ceil_div(M, 128), nB = ceil_div(N, 128);
  if (nA + nB == 0 || K <= 0) return LU_SUCCESS;
  const int64_t kp = (K + 15) / 16 * 16;
  const float bound = tc_scale_bound(kind);
  const unsigned grid = (unsigned)(kScaledCtas * (nA + nB));
  if (kind == TcOperand::E4M3) {
    LUB_CUDA_TRY(launch_dependent(pack_scaled_kernel<uint8_t, false>, grid, 256, 0, st, (int)nA,
                                  M, N, K, kp, a, lda, (uint8_t*)da, sa, b, ldb, (uint8_t*)db, sb,
                                  ldd, bound));
  } else if (kind == TcOperand::SPLIT16) {
    if (ldd < 3 * kp) return LU_ERR_INVALID_ARG;
    LUB_CUDA_TRY(launch_dependent(pack_scaled_kernel<__half, true>, grid, 256, 0, st, (int)nA, M,
                                  N, K, kp, a, lda, (__half*)da, sa, b, ldb, (__half*)db, sb, ldd,
                                  bound));
  } else {
    return LU_ERR_INVALID_ARG;
  }
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

}  // namespace lub
