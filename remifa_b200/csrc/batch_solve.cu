// Batched solves and adjoint for the factors a batch plan produced (new; the
// reference has neither a batch nor a derivative).
//
// Two kernels share a batch, by size (launch_batch_solve): batch_solve_kernel
// takes the larger matrices, batch_solve_warp_kernel small ones in great number.
// Both keep b, x and the residual in shared memory (fp64) and read the fp32
// factors and matrices from global memory / L2.
//
// batch_solve_kernel: one CTA of eight warps per (matrix, group of up to NR
// right-hand sides).
//   * The 32 x 32 diagonal blocks of L and U are inverted once per item, in
//     fp64, by substitution (one warp per block, lane j column j), and kept
//     packed L^-1 \ U^-1 in shared memory; all 1 + refine_iters solves use
//     them.
//   * A triangle is then one step per block of 32 unknowns: x_t = Dinv_t (b_t -
//     sum over the solved blocks), the sum split over the eight warps.  Not
//     transposed: lanes are the block's rows, warp w sums the columns w, w +
//     8, ...; transposed: warp w owns four of the block's columns, lanes run
//     down the rows, one shuffle tree per column.  Both read the factor's
//     columns coalesced.  While one warp multiplies by Dinv_t the others
//     already sum block t+1's row over the blocks before t.
// batch_solve_warp_kernel: one warp per (matrix, right-hand side), down the
// triangles column by column with no barrier; it fills the chip with matrices
// where a CTA per matrix would mostly wait (4,000 of n = 40, one right-hand side:
// 38 us, 129 with the CTA kernel).
// With the original fp32 matrices given, refine_iters rounds of FP64
// refinement follow: r = b - op(A) x in fp64, x += op(LU)^-1 r.  Every sum has
// a fixed order, so results do not depend on scheduling.
//
// What bounds the CTA kernel: the chain of dependent block steps (2 (1 + iters) n / 32 of
// them, each an L2 latency and the inverse's product), hidden by three CTAs
// per SM at n <= 256; there the factors of the resident matrices outgrow L2,
// so every round reads them from DRAM again (2 TB/s).  The fp32 -> fp64
// conversions (one warp instruction per 8 cycles and scheduler) take a
// seventh of the time, the arithmetic less.  1,024 matrices of 64..256, one
// right-hand side, 4 refinement rounds on B200: 0.42 ms (transposed 0.44),
// 6.3 ms as one warp per (matrix, right-hand side) walking single columns.
//
// The adjoint of X = A^-1 B: dB = A^-T G (the transposed solve above, in
// place in G) and dA = -dB X^T (fp64 dot products, stored fp32).
#include "common.cuh"
#include "kernels.cuh"

#include <algorithm>

struct lu_batch_plan_t;

namespace lub {

// plan accessors (batch.cu)
int64_t batch_plan_size(const lu_batch_plan_t* p);
const int32_t* batch_plan_dev_n(const lu_batch_plan_t* p);
const int32_t* batch_plan_dev_order(const lu_batch_plan_t* p);  // by decreasing size
const int32_t* batch_plan_upto(const lu_batch_plan_t* p);  // [n]: matrices of size <= n
int batch_plan_nmax(const lu_batch_plan_t* p);

namespace {

constexpr int kWarps = 8;
constexpr int kT = 32 * kWarps;
constexpr int BS = 32;                 // unknowns per step
constexpr int kDS = BS + 1;            // row stride of an inverted block (doubles)

// Shared memory of one item, in doubles: inverted diagonal blocks, x, b and r of
// the group, the warps' partial sums.
__host__ __device__ inline size_t smem_doubles(int nmax, int nr) {
  const size_t nb = (size_t)(nmax + BS - 1) / BS;
  return nb * BS * kDS + 3 * nb * BS * nr + (size_t)kWarps * nr * BS;
}

// Inverses of the unit lower and the upper triangle of every diagonal block,
// packed in place of the block at S + t BS kDS (row-major, stride kDS), one
// warp per block.  The 16 x 16 diagonal halves by substitution (half-warp h
// half h, lane j column j), then the off-diagonal quarters as products:
// -L22^-1 L21 L11^-1 by the lower half-warp, -U11^-1 U12 U22^-1 by the upper
// one (half the registers of a 32-row substitution).  This sets the kernel's
// register need: at the 80 that three CTAs per SM leave, its instances spill 120 to
// 570 bytes a thread, most of them here; two CTAs at 128 registers took 465 us
// where three take 430, a rolled form of this code 25 us more (1,024 matrices of
// 64..256).
__device__ __forceinline__ void invert_blocks(const float* __restrict__ F, int64_t ld, int n,
                                              int nb, double* S) {
  constexpr int H = BS / 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int h = lane >> 4, j = lane & (H - 1);
#pragma unroll 1
  for (int t = warp; t < nb; t += kWarps) {
    double* D = S + (size_t)t * BS * kDS;
    const int r0 = t * BS;
    const bool rowok = r0 + lane < n;
    const float* src = F + (r0 + lane) + (int64_t)r0 * ld;
#pragma unroll 16
    for (int c = 0; c < BS; ++c) {
      const bool ok = rowok && r0 + c < n;
      D[lane * kDS + c] = ok ? (double)src[(int64_t)c * ld] : (c == lane ? 1.0 : 0.0);
    }
    __syncwarp();
    double* Dh = D + h * H * (kDS + 1);
    const double rd = 1.0 / D[lane * kDS + lane];
    {
      double z[H];
#pragma unroll
      for (int i = 0; i < H; ++i) z[i] = i == j ? 1.0 : 0.0;
#pragma unroll
      for (int k = 0; k < H; ++k)
#pragma unroll
        for (int i = k + 1; i < H; ++i) z[i] = fma(-Dh[i * kDS + k], z[k], z[i]);
      __syncwarp();  // every read of L is done
#pragma unroll
      for (int i = 1; i < H; ++i)
        if (i > j) Dh[i * kDS + j] = z[i];
#pragma unroll
      for (int i = 0; i < H; ++i) z[i] = i == j ? rd : 0.0;
#pragma unroll
      for (int k = H - 1; k >= 0; --k) {
        // row k takes its reciprocal in the columns right of k; the columns
        // left of k have nothing there
        const double rk = __shfl_sync(0xffffffffu, rd, h * H + k);
        if (k < j) z[k] *= rk;
#pragma unroll
        for (int i = 0; i < k; ++i) z[i] = fma(-Dh[i * kDS + k], z[k], z[i]);
      }
      __syncwarp();  // every read of U is done
#pragma unroll
      for (int i = 0; i < H; ++i)
        if (i <= j) Dh[i * kDS + j] = z[i];
    }
    __syncwarp();
    double* P = h ? D + H : D + H * kDS;              // U12 or L21
    const double* Q = h ? D : D + H * (kDS + 1);      // U11^-1 or L22^-1
    double a[H], w[H];
#pragma unroll
    for (int k = 0; k < H; ++k)
      a[k] = (h ? k <= j : k > j) ? Dh[k * kDS + j] : (k == j ? 1.0 : 0.0);
#pragma unroll
    for (int i = 0; i < H; ++i) {
      w[i] = 0.0;
#pragma unroll
      for (int k = 0; k < H; ++k) w[i] = fma(P[i * kDS + k], a[k], w[i]);
    }
    __syncwarp();  // every read of the quarters is done
#pragma unroll
    for (int i = 0; i < H; ++i) {
      double v = h ? Q[i * kDS + i] * w[i] : w[i];
#pragma unroll
      for (int k = 0; k < H; ++k)
        if (h ? k > i : k < i) v = fma(Q[i * kDS + k], w[k], v);
      P[i * kDS + j] = -v;
    }
  }
}

// Row lane of the packed inverse (transposed: column lane) times y (16-byte
// aligned).  lower: L^-1 (unit diagonal) else U^-1.  Entries of the other
// triangle are skipped.
__device__ __forceinline__ double dinv_mul(const double* D, bool trans, bool lower,
                                           const double* y) {
  const int lane = threadIdx.x & 31;
  const bool below = lower != trans;  // op(triangle) is lower
  const double own = lower ? 1.0 : D[lane * kDS + lane];
  const double* d = trans ? D + lane : D + lane * kDS;
  const int st = trans ? kDS : 1;
  double s[4] = {own * y[lane], 0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < BS; k += 2) {
    const double2 y2 = *reinterpret_cast<const double2*>(y + k);
    if (below ? k < lane : k > lane) s[k & 3] = fma(d[k * st], y2.x, s[k & 3]);
    if (below ? k + 1 < lane : k + 1 > lane)
      s[(k + 1) & 3] = fma(d[(k + 1) * st], y2.y, s[(k + 1) & 3]);
  }
  return (s[0] + s[1]) + (s[2] + s[3]);
}

// Sums of four per-lane partials over the 32 lanes: two halving exchanges,
// then three full steps.  Lanes 8 q .. 8 q + 7 end with sum q.
__device__ __forceinline__ double reduce4(const double (&a)[4]) {
  const int lane = threadIdx.x & 31;
  const bool b4 = lane & 16, b3 = lane & 8;
  double v0 = (b4 ? a[2] : a[0]) + __shfl_xor_sync(0xffffffffu, b4 ? a[0] : a[2], 16);
  double v1 = (b4 ? a[3] : a[1]) + __shfl_xor_sync(0xffffffffu, b4 ? a[1] : a[3], 16);
  double v = (b3 ? v1 : v0) + __shfl_xor_sync(0xffffffffu, b3 ? v0 : v1, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The warp's share of rows [r0, r0 + 32) of op(F) times x over whole blocks of
// 32 columns: not transposed, lane = row, columns 4 warp .. 4 warp + 3 of each
// block; transposed, rows 4 warp .. 4 warp + 3 of the row block (columns of
// F), lanes over the block's 32.  Rows past n read the last valid one instead
// (their sums are dropped); columns past n are zero, as x is there.
template <bool TRANS, int NR>
struct Partial {
  static constexpr int NA = TRANS ? 4 : 1;
  double acc[NA][NR];
  const float* p[4];  // column 4 warp + q of F (transposed: r0 + 4 warp + q, from row lane)
  int row;            // lane's row (not transposed)

  __device__ __forceinline__ void init(const float* __restrict__ F, int64_t ld) {
    const int warp = threadIdx.x >> 5;
    if (!TRANS) {
#pragma unroll
      for (int q = 0; q < 4; ++q) p[q] = F + (4 * warp + q) * ld;
    }
  }
  // the row block of the next sums
  __device__ __forceinline__ void start(const float* __restrict__ F, int64_t ld, int n, int r0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (!TRANS) {
      row = min(r0 + lane, n - 1);
    } else {
      const float* c = F + lane + (r0 + 4 * warp) * ld;
      if (r0 + BS <= n) {
#pragma unroll
        for (int q = 0; q < 4; ++q) p[q] = c + q * ld;
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          p[q] = F + lane + (int64_t)min(r0 + 4 * warp + q, n - 1) * ld;
      }
    }
#pragma unroll
    for (int q = 0; q < NA; ++q)
#pragma unroll
      for (int c = 0; c < NR; ++c) acc[q][c] = 0.0;
  }
  // The warp's entries of block q0: of a whole block, of any.
  __device__ __forceinline__ void fetch_whole(float (&v)[4], int64_t ld, int q0) const {
    const int64_t at = TRANS ? (int64_t)(q0 * BS) : row + q0 * (BS * ld);
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = p[q][at];
  }
  __device__ __forceinline__ void fetch(float (&v)[4], int64_t ld, int n, int q0) const {
    if ((q0 + 1) * BS <= n) return fetch_whole(v, ld, q0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t at = TRANS ? (int64_t)(q0 * BS) : row + q0 * (BS * ld);
    if (TRANS && NR == 1) {
      // loaded and dropped: 442 us, 460 with the load left out (1,024 matrices of
      // 64..256; the other instances are the faster ones without it)
      const int over = max(0, q0 * BS + lane - (n - 1));
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = p[q][at - over];
      if (over > 0) v[0] = v[1] = v[2] = v[3] = 0.0f;
    } else {
      const int left = n - q0 * BS - (TRANS ? lane : 4 * warp);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        v[q] = 0.0f;
        if (left > (TRANS ? 0 : q)) v[q] = p[q][at];
      }
    }
  }
  // block q0's entries v times x
  __device__ __forceinline__ void add(const float (&v)[4], int q0, const double* x, int np) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < NR; ++c) {
      const double* xc = x + c * np + q0 * BS;
      if (TRANS) {
        const double xv = xc[lane];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q][c] = fma((double)v[q], xv, acc[q][c]);
      } else {
        const double2 x0 = *reinterpret_cast<const double2*>(xc + 4 * warp);
        const double2 x1 = *reinterpret_cast<const double2*>(xc + 4 * warp + 2);
        acc[0][c] = fma((double)v[0], x0.x, acc[0][c]);
        acc[0][c] = fma((double)v[1], x0.y, acc[0][c]);
        acc[0][c] = fma((double)v[2], x1.x, acc[0][c]);
        acc[0][c] = fma((double)v[3], x1.y, acc[0][c]);
      }
    }
  }
  // M whole blocks from q0, their loads all in flight before the first use
  template <int M>
  __device__ __forceinline__ void add_whole(int64_t ld, int q0, const double* x, int np) {
    float v[M][4];
#pragma unroll
    for (int u = 0; u < M; ++u) fetch_whole(v[u], ld, q0 + u);
#pragma unroll
    for (int u = 0; u < M; ++u) add(v[u], q0 + u, x, np);
  }
  // blocks q0 .. q1 - 1
  __device__ __forceinline__ void add_range(int64_t ld, int n, int q0, int q1, const double* x,
                                            int np) {
    const int full = min(q1, n / BS);
    float vt[4];
    if (full < q1) fetch(vt, ld, n, full);
#pragma unroll 1
    for (; q0 + 4 <= full; q0 += 4) add_whole<4>(ld, q0, x, np);
    if (full - q0 == 3) add_whole<3>(ld, q0, x, np);
    else if (full - q0 == 2) add_whole<2>(ld, q0, x, np);
    else if (full - q0 == 1) add_whole<1>(ld, q0, x, np);
    if (full < q1) add(vt, full, x, np);
  }

  // Partial sums to part: [warp][c][row] not transposed, [c][row] transposed
  __device__ __forceinline__ void publish(double* part) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < NR; ++c) {
      if (!TRANS) {
        part[(warp * NR + c) * BS + lane] = acc[0][c];
      } else {
        const double a[4] = {acc[0][c], acc[NA > 1 ? 1 : 0][c], acc[NA > 2 ? 2 : 0][c],
                             acc[NA > 3 ? 3 : 0][c]};
        const double v = reduce4(a);
        if ((lane & 7) == 0) part[c * BS + 4 * warp + (lane >> 3)] = v;
      }
    }
  }
  // Sum of row lane of column c (after a CTA barrier)
  static __device__ __forceinline__ double total(const double* part, int c) {
    const int lane = threadIdx.x & 31;
    if (TRANS) return part[c * BS + lane];
    double s = part[c * BS + lane];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) s += part[(w * NR + c) * BS + lane];
    return s;
  }
};

// x <- op(T)^-1 x for the lower (unit) or upper triangle of F; all threads.
// Ends with a CTA barrier.
template <bool TRANS, int NR>
__device__ __forceinline__ void tri_solve(const float* __restrict__ F, int64_t ld, int n, int nb,
                                          bool lower, const double* S, double* x, int np,
                                          double* part) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool fwd = lower != TRANS;
  Partial<TRANS, NR> p;
  float pv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  p.init(F, ld);
  p.start(F, ld, n, (fwd ? 0 : nb - 1) * BS);
#pragma unroll 1
  for (int s = 0; s < nb; ++s) {
    const int t = fwd ? s : nb - 1 - s;
    if (s > 0) p.add(pv, fwd ? t - 1 : t + 1, x, np);
    p.publish(part);
    __syncthreads();
    if (s + 1 < nb) {
      p.start(F, ld, n, (fwd ? t + 1 : t - 1) * BS);
      p.fetch(pv, ld, n, t);
    }
    if (warp < NR) {
      double* xc = x + warp * np + t * BS;
      // rows past n stay zero whatever the sums hold
      const bool ok = t * BS + lane < n;
      const double y = xc[lane] - Partial<TRANS, NR>::total(part, warp);
      xc[lane] = ok ? y : 0.0;
      __syncwarp();
      const double v = dinv_mul(S + (size_t)t * BS * kDS, TRANS, lower, xc);
      __syncwarp();
      xc[lane] = ok ? v : 0.0;
    }
    // the blocks solved before t
    if (s > 0 && s + 1 < nb) p.add_range(ld, n, fwd ? 0 : t + 1, fwd ? t : nb, x, np);
    __syncthreads();
  }
}

template <bool TRANS, int NR>
__device__ __forceinline__ void solve(const float* F, int64_t ld, int n, int nb, const double* S,
                                      double* x, int np, double* part) {
  tri_solve<TRANS, NR>(F, ld, n, nb, !TRANS, S, x, np, part);
  tri_solve<TRANS, NR>(F, ld, n, nb, TRANS, S, x, np, part);
}

// r = b - op(A) x (A fp32, fp64 arithmetic), one row block per barrier pair.
template <bool TRANS, int NR>
__device__ __forceinline__ void residual(const float* __restrict__ A, int64_t ld, int n, int nb,
                                         const double* b, const double* x, double* r, int np,
                                         double* part) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Partial<TRANS, NR> p;
  p.init(A, ld);
#pragma unroll 1
  for (int t = 0; t < nb; ++t) {
    p.start(A, ld, n, t * BS);
    p.add_range(ld, n, 0, nb, x, np);
    __syncthreads();  // the previous block's sums are read
    p.publish(part);
    __syncthreads();
    if (warp < NR) {
      const int i = warp * np + t * BS + lane;
      r[i] = t * BS + lane < n ? b[i] - Partial<TRANS, NR>::total(part, warp) : 0.0;
    }
  }
  __syncthreads();
}

struct SolveArgs {
  const float* const* lu;
  const int32_t* ldlu;
  const float* const* a;    // original matrices (refinement), or null
  const int32_t* lda;
  double* const* x;         // n_i x nrhs, ld n_i: b on entry, x on exit
  const int32_t* n;
  int64_t batch;
  int nrhs;
  int iters;
  const int32_t* order;     // this launch's matrices (batch of them)
};

// The launches of one call share a stream and take disjoint matrices: each lets
// the next one start beside it, and completes only after the one in front.
__device__ __forceinline__ void launch_begin() { dependents_launch(); }
__device__ __forceinline__ void launch_end() {
  if (blockIdx.x == 0) dependency_wait();
}

template <bool TRANS, int NR>
__global__ void __launch_bounds__(kT, 3)
batch_solve_kernel(SolveArgs s) {
  extern __shared__ __align__(16) double sh[];
  launch_begin();
  const int groups = (s.nrhs + NR - 1) / NR;
  const int64_t item = blockIdx.x;
  const int64_t m = s.order[item / groups];
  const int c0 = (int)(item % groups) * NR;
  const int nc = min(NR, s.nrhs - c0);
  const int n = s.n[m];
  const int nb = (n + BS - 1) / BS, np = nb * BS;
  double* S = sh;
  double* xb = S + (size_t)nb * BS * kDS;
  double* bb = xb + (size_t)NR * np;
  double* rb = bb + (size_t)NR * np;
  double* part = rb + (size_t)NR * np;
  const float* F = s.lu[m];
  const int64_t ldf = s.ldlu ? s.ldlu[m] : n;
  double* xg = s.x[m] + (int64_t)c0 * n;
  for (int e = threadIdx.x; e < NR * np; e += kT) {
    const int c = e / np, i = e - c * np;
    const double v = (c < nc && i < n) ? xg[i + (int64_t)c * n] : 0.0;
    xb[e] = v;
    bb[e] = v;
  }
  invert_blocks(F, ldf, n, nb, S);
  __syncthreads();
  solve<TRANS, NR>(F, ldf, n, nb, S, xb, np, part);
  if (s.a) {
    const float* A = s.a[m];
    const int64_t lda = s.lda ? s.lda[m] : n;
    for (int k = 0; k < s.iters; ++k) {
      residual<TRANS, NR>(A, lda, n, nb, bb, xb, rb, np, part);
      solve<TRANS, NR>(F, ldf, n, nb, S, rb, np, part);
      for (int e = threadIdx.x; e < NR * np; e += kT) xb[e] += rb[e];
      __syncthreads();
    }
  }
  for (int e = threadIdx.x; e < nc * np; e += kT) {
    const int c = e / np, i = e - c * np;
    if (i < n) xg[i + (int64_t)c * n] = xb[e];
  }
  launch_end();
}

// ---- one warp per (matrix, right-hand side) --------------------------------
namespace warp {

constexpr int kWarpsPerCta = 4;

// x (shared, fp64, length n) <- L^-1 x, L unit lower (fp32, column-major).
__device__ __forceinline__ void lower_solve(const float* __restrict__ F, int64_t ld,
                                            int n, double* x) {
  const int lane = threadIdx.x & 31;
  for (int j = 0; j < n - 1; ++j) {
    __syncwarp();
    const double xj = x[j];
    const float* col = F + (int64_t)j * ld;
    for (int i = j + 1 + lane; i < n; i += 32) x[i] = fma(-(double)col[i], xj, x[i]);
  }
  __syncwarp();
}

// x <- U^-1 x, U upper with its diagonal (column form, bottom up).
__device__ __forceinline__ void upper_solve(const float* __restrict__ F, int64_t ld,
                                            int n, double* x) {
  const int lane = threadIdx.x & 31;
  for (int j = n - 1; j >= 0; --j) {
    __syncwarp();
    const float* col = F + (int64_t)j * ld;
    const double xj = x[j] / (double)col[j];
    __syncwarp();
    if (lane == 0) x[j] = xj;
    for (int i = lane; i < j; i += 32) x[i] = fma(-(double)col[i], xj, x[i]);
  }
  __syncwarp();
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// x <- U^-T x (dot form, top down: x_j = (x_j - U[0:j, j] . x[0:j]) / U_jj).
__device__ __forceinline__ void upper_t_solve(const float* __restrict__ F, int64_t ld,
                                              int n, double* x) {
  const int lane = threadIdx.x & 31;
  for (int j = 0; j < n; ++j) {
    const float* col = F + (int64_t)j * ld;
    double p = 0.0;
    for (int i = lane; i < j; i += 32) p = fma((double)col[i], x[i], p);
    p = warp_sum(p);
    if (lane == 0) x[j] = (x[j] - p) / (double)col[j];
    __syncwarp();
  }
}

// x <- L^-T x (dot form, bottom up: x_j = x_j - L[j+1:n, j] . x[j+1:n]).
__device__ __forceinline__ void lower_t_solve(const float* __restrict__ F, int64_t ld,
                                              int n, double* x) {
  const int lane = threadIdx.x & 31;
  for (int j = n - 2; j >= 0; --j) {
    const float* col = F + (int64_t)j * ld;
    double p = 0.0;
    for (int i = j + 1 + lane; i < n; i += 32) p = fma((double)col[i], x[i], p);
    p = warp_sum(p);
    if (lane == 0) x[j] = x[j] - p;
    __syncwarp();
  }
}

template <bool TRANS>
__device__ __forceinline__ void solve(const float* F, int64_t ld, int n, double* x) {
  if (!TRANS) {
    lower_solve(F, ld, n, x);
    upper_solve(F, ld, n, x);
  } else {
    upper_t_solve(F, ld, n, x);
    lower_t_solve(F, ld, n, x);
  }
}

// r = b - op(A) x (A fp32, fp64 arithmetic).
template <bool TRANS>
__device__ __forceinline__ void residual(const float* __restrict__ A, int64_t ld, int n,
                                         const double* b, const double* x, double* r) {
  const int lane = threadIdx.x & 31;
  if (!TRANS) {
    for (int i = lane; i < n; i += 32) r[i] = b[i];
    for (int j = 0; j < n; ++j) {
      __syncwarp();
      const double xj = x[j];
      const float* col = A + (int64_t)j * ld;
      for (int i = lane; i < n; i += 32) r[i] = fma(-(double)col[i], xj, r[i]);
    }
  } else {
    for (int j = 0; j < n; ++j) {
      const float* col = A + (int64_t)j * ld;
      double p = 0.0;
      for (int i = lane; i < n; i += 32) p = fma((double)col[i], x[i], p);
      p = warp_sum(p);
      if (lane == 0) r[j] = b[j] - p;
    }
  }
  __syncwarp();
}

}  // namespace warp

// nmax: the largest of this launch's matrices.
template <bool TRANS>
__global__ void __launch_bounds__(32 * warp::kWarpsPerCta)
batch_solve_warp_kernel(SolveArgs s, int nmax) {
  extern __shared__ __align__(16) double sh[];
  launch_begin();
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* xb = sh + (size_t)wid * 3 * nmax;
  double* bb = xb + nmax;
  double* rb = bb + nmax;
  const int64_t items = s.batch * s.nrhs;
  for (int64_t it = (int64_t)blockIdx.x * warp::kWarpsPerCta + wid; it < items;
       it += (int64_t)gridDim.x * warp::kWarpsPerCta) {
    const int64_t q = it / s.nrhs;
    const int c = (int)(it - q * s.nrhs);
    const int64_t m = s.order[q];
    const int n = s.n[m];
    const float* F = s.lu[m];
    const int64_t ldf = s.ldlu ? s.ldlu[m] : n;
    double* xg = s.x[m] + (int64_t)c * n;
    for (int i = lane; i < n; i += 32) {
      xb[i] = xg[i];
      bb[i] = xg[i];
    }
    __syncwarp();
    warp::solve<TRANS>(F, ldf, n, xb);
    if (s.a) {
      const float* A = s.a[m];
      const int64_t lda = s.lda ? s.lda[m] : n;
      for (int k = 0; k < s.iters; ++k) {
        warp::residual<TRANS>(A, lda, n, bb, xb, rb);
        warp::solve<TRANS>(F, ldf, n, rb);
        for (int i = lane; i < n; i += 32) xb[i] += rb[i];
        __syncwarp();
      }
    }
    for (int i = lane; i < n; i += 32) xg[i] = xb[i];
    __syncwarp();
  }
  launch_end();
}

// dA_m[i, j] = -sum_r dB_m[i, r] X_m[j, r], one CTA per matrix (largest
// first): warps take columns j, lanes rows i, dB and X through L1; the writes
// of dA bound it (1,024 matrices of 64..256: 38 us = 3.0 TB/s; 147 us with a
// thread and an index division per element, which is the faster one below 64
// rows, where it keeps all threads busy: 16000 of n = 16 20 us, 35 by columns; n
// = 48 112 and 119, n = 64 190 and 138).
__global__ void __launch_bounds__(kT)
batch_outer_kernel(const double* const* __restrict__ db, const double* const* __restrict__ x,
                   float* const* __restrict__ da, const int32_t* __restrict__ ldda,
                   const int32_t* __restrict__ ns, const int32_t* __restrict__ order, int nrhs) {
  const int m = order[blockIdx.x];
  const int n = ns[m];
  const int64_t ld = ldda ? (int64_t)ldda[m] : n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double* __restrict__ G = db[m];
  const double* __restrict__ X = x[m];
  float* __restrict__ D = da[m];
  if (n < 64) {
    for (int e = threadIdx.x; e < n * n; e += kT) {
      const int j = e / n, i = e - j * n;
      double acc = 0.0;
      for (int r = 0; r < nrhs; ++r)
        acc = fma(G[i + (int64_t)r * n], X[j + (int64_t)r * n], acc);
      D[i + j * ld] = (float)(-acc);
    }
    return;
  }
  constexpr int CW = 4;  // columns of a warp per pass over the rows
  for (int j0 = CW * warp; j0 < n; j0 += CW * kWarps) {
    for (int i = lane; i < n; i += 32) {
      double acc[CW] = {0.0, 0.0, 0.0, 0.0};
      for (int r = 0; r < nrhs; ++r) {
        const double g = G[i + (int64_t)r * n];
#pragma unroll
        for (int q = 0; q < CW; ++q)
          if (j0 + q < n) acc[q] = fma(g, X[j0 + q + (int64_t)r * n], acc[q]);
      }
#pragma unroll
      for (int q = 0; q < CW; ++q)
        if (j0 + q < n) D[i + (j0 + q) * ld] = (float)(-acc[q]);
    }
  }
}

// One launch of a call; `behind`: another launch of the call is in front of it.
template <typename... P, typename... A>
lu_status launch_part(bool behind, void (*kernel)(P...), int64_t grid, int threads, size_t smem,
                      cudaStream_t st, A... args) {
  LUB_CUDA_TRY(set_smem_limit((const void*)kernel, smem));
  if (behind) {
    LUB_CUDA_TRY(launch_dependent(kernel, (unsigned)grid, threads, smem, st, args...));
  } else {
    kernel<<<(unsigned)grid, threads, smem, st>>>(args...);
  }
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

// CTAs of batch_solve_kernel an SM holds: its shared memory, at most three.
int ctas_per_sm(int n, int nr) {
  return (int)std::min<size_t>(3, 233472 / (smem_doubles(n, nr) * sizeof(double) + 1024));
}

// The size up to which matrices go to the warp kernel: where the time it needs --
// the longer of one warp's chain and the sum over all -- stays below what the same
// matrices cost as CTAs, three to an SM (a fifth less while they stay in L2).  In
// us, fitted on B200 to uniform batches of 64 .. 16000 matrices of 16 .. 192 rows, 1
// .. 8 right-hand sides and 0 .. 4 rounds, where 98 % of the cases come within 5 % of the
// better kernel (the CTA kernel alone takes up to 7 times the warp kernel's time,
// 16000 of n = 16; the warp kernel alone up to 25 times the other's, 64 of n =
// 192).
int warp_limit(const int32_t* upto, int nmax, int nrhs, int nr, int iters, bool trans) {
  const double block = nr < 4 ? 7.7 : 8.7;
  const double round = trans ? (nr < 4 ? 3.0 : 8.5) : (nr < 4 ? 2.5 : 4.1);
  const double slots = 3.0 * sm_count() / ((nrhs + nr - 1) / nr);
  const double passes = 1.0 + (trans ? 1.45 : 1.27) * iters;
  double cta = 0.0, sum = 0.0, bytes = 0.0, best = 0.0;
  int limit = 0;
  for (int n = 1; n <= std::min(nmax, 160); ++n) {
    const double c = upto[n] - upto[n - 1], n2 = (double)n * n;
    if (c == 0.0) continue;
    const int nb = (n + BS - 1) / BS;
    cta += c / slots * (12.6 + nb * (block + round * iters));
    bytes += c * n2 * (iters > 0 ? 8.0 : 4.0);
    sum += c * nrhs * passes * 1e-3 * (trans ? 0.19 * n + 0.0027 * n2 : 0.052 * n + 0.0045 * n2);
    const double chain = passes * (trans ? 0.84 * n + 0.0045 * n2 : 0.37 * n + 0.0105 * n2);
    const double gain = (bytes < 64e6 ? 0.8 : 1.0) * cta - std::max(chain, sum);
    if (gain > best) {
      best = gain;
      limit = n;
    }
  }
  return limit;
}

template <bool TRANS, int NR>
lu_status launch_sizes(cudaStream_t st, SolveArgs s, const int32_t* upto, int nmax) {
  const int32_t* order = s.order;
  const int64_t batch = s.batch, groups = (s.nrhs + NR - 1) / NR;
  const int limit = warp_limit(upto, nmax, s.nrhs, NR, s.iters, TRANS);
  const int64_t big = batch - upto[limit];   // the first ones of `order`
  if (big * groups > 0x7fffffffll) return LU_ERR_INVALID_ARG;
  int64_t at = 0;
  int top = nmax;                            // the largest size from `at` on
  while (at < big) {
    // matrices that fit more CTAs on an SM get a launch of their own once they
    // fill it (1,000 of 64 .. 200 rows and one of 300, five right-hand sides:
    // 504 us in one launch)
    const int fit = ctas_per_sm(top, NR);
    int64_t to = big;
    int n = top;
    while (n > limit && ctas_per_sm(n, NR) == fit) --n;
    if (n > limit && (upto[n] - upto[limit]) * groups > (int64_t)sm_count() * (fit + 1))
      to = batch - upto[n];
    s.order = order + at;
    s.batch = to - at;
    LUB_TRY(launch_part(at > 0, batch_solve_kernel<TRANS, NR>, s.batch * groups, kT,
                        smem_doubles(top, NR) * sizeof(double), st, s));
    at = to;
    for (top = n; top > limit && upto[top] == upto[top - 1]; --top) {}
  }
  if (big == batch) return LU_SUCCESS;
  s.order = order + big;
  s.batch = batch - big;
  const int64_t ctas = std::min<int64_t>(
      (s.batch * s.nrhs + warp::kWarpsPerCta - 1) / warp::kWarpsPerCta, (int64_t)sm_count() * 16);
  return launch_part(big > 0, batch_solve_warp_kernel<TRANS>, ctas, 32 * warp::kWarpsPerCta,
                     (size_t)warp::kWarpsPerCta * 3 * limit * sizeof(double), st, s, limit);
}

// Right-hand sides per CTA: a second and a fourth column reuse the factor
// entries already loaded and the inverted blocks.
template <bool TRANS>
lu_status launch_batch_solve(cudaStream_t st, const SolveArgs& s, const int32_t* upto, int nmax) {
  if (s.nrhs == 1) return launch_sizes<TRANS, 1>(st, s, upto, nmax);
  if (s.nrhs == 2) return launch_sizes<TRANS, 2>(st, s, upto, nmax);
  return launch_sizes<TRANS, 4>(st, s, upto, nmax);
}

}  // namespace
}  // namespace lub

using namespace lub;

extern "C" {

LU_API lu_status lu_batch_solve_c(lu_batch_plan plan, lu_stream_t stream,
                                  const float* const* d_lu, const int32_t* d_ldlu,
                                  const float* const* d_a, const int32_t* d_lda,
                                  double* const* d_x, int32_t nrhs, int trans,
                                  int refine_iters) {
  if (!plan || nrhs < 0 || (trans != 0 && trans != 1) || refine_iters < 0)
    return LU_ERR_INVALID_ARG;
  const int64_t batch = batch_plan_size(plan);
  if (batch == 0 || nrhs == 0) return LU_SUCCESS;
  if (!d_lu || !d_x) return LU_ERR_INVALID_ARG;
  SolveArgs s;
  s.lu = d_lu;
  s.ldlu = d_ldlu;
  s.a = d_a;
  s.lda = d_lda;
  s.x = d_x;
  s.n = batch_plan_dev_n(plan);
  s.batch = batch;
  s.nrhs = nrhs;
  s.iters = d_a ? refine_iters : 0;
  s.order = batch_plan_dev_order(plan);
  const int32_t* upto = batch_plan_upto(plan);
  const int nmax = batch_plan_nmax(plan);
  return trans ? launch_batch_solve<true>((cudaStream_t)stream, s, upto, nmax)
               : launch_batch_solve<false>((cudaStream_t)stream, s, upto, nmax);
}

LU_API lu_status lu_batch_adjoint_c(lu_batch_plan plan, lu_stream_t stream,
                                    const float* const* d_lu, const int32_t* d_ldlu,
                                    const float* const* d_a, const int32_t* d_lda,
                                    double* const* d_x, double* const* d_g,
                                    float* const* d_da, const int32_t* d_ldda,
                                    int32_t nrhs, int refine_iters) {
  if (!plan || nrhs < 0 || refine_iters < 0) return LU_ERR_INVALID_ARG;
  const int64_t batch = batch_plan_size(plan);
  if (batch == 0 || nrhs == 0) return LU_SUCCESS;
  if (!d_lu || !d_x || !d_g) return LU_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  LUB_TRY(lu_batch_solve_c(plan, stream, d_lu, d_ldlu, d_a, d_lda, d_g, nrhs, 1,
                           refine_iters));
  if (d_da) {
    batch_outer_kernel<<<(unsigned)batch, kT, 0, st>>>(d_g, d_x, d_da, d_ldda,
                                                       batch_plan_dev_n(plan),
                                                       batch_plan_dev_order(plan), nrhs);
    LUB_LAUNCH_CHECK();
  }
  return LU_SUCCESS;
}

}  // extern "C"
