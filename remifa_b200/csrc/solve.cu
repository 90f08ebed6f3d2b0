// Triangular solves with the in-place L\U factors and the FP64 residual of
// iterative refinement.
//
// The reference solves on the host with LAPACK getrs and identity pivots
// (tests/testing_lu_gpu.hxx:1309-1313); its GPU solve is referenced but not
// shipped (tests/testing_lu_gpu.hxx:1353-1359).  Here the solves run on the
// device: the factors stay fp32 (4 bytes per element read per solve, the
// bandwidth that bounds a triangular solve), the right-hand sides and all
// arithmetic are fp64, so the solve adds no fp32 rounding on top of the
// factorization error -- what iterative refinement in fp64 needs.
//
// op(T) X = B, T = L (unit lower) or U (upper), op = identity or transpose,
// runs as one launch per triangle after a kernel that marks every entry of the
// solution pending, one for both triangles (a signalling-NaN pattern no arithmetic
// produces).  A CTA per (row block of 64 rows, group of 1, 2 or 8 right-hand
// sides); CTAs draw tickets in solve order (an atomic counter), so a CTA only
// ever waits for CTAs already running: no deadlock whatever the residency.
// Each warp of a CTA streams its share of the tiles op(T)[t, q] of the blocks
// solved earlier, reading the solution entries it needs straight from X
// (relaxed loads at GPU scope, re-read while pending; the solution IS the
// flag, so publishing a block costs one store, no fence and no counter).  The
// diagonal block is inverted in fp64 and the last tile is folded into W =
// Dinv op(T)[t, t-1] while the CTA waits, so the hand-over from block t-1 to
// block t is, per warp and without a CTA barrier: x_t = Dinv (b -
// sum_{q<t-1} op(T)[t,q] x_q) - W x_{t-1}.  trsv_kernel does this with FMAs
// and shuffles for 1 to 4 right-hand sides (groups of 1 or 2), trsv_mma_kernel
// on the FP64 matrix instruction for groups of 8.  On B200: one right-hand side,
// n = 10007, L and U 0.277 ms (0.344 without clusters), n = 16384 0.46 (0.58); 64
// right-hand sides, n = 8192 0.80, transposed 0.81 (1.36 with a counter per group
// and shared-memory tiles).  Bound by the chain of n / 64 hand-overs.
#include "common.cuh"
#include "kernels.cuh"
#include "mma64.cuh"
#include "solve.cuh"

#include <map>
#include <mutex>
#include <tuple>

namespace lub {
namespace {

constexpr int kT = 256;    // threads per CTA of the residual kernels

namespace trsv {

constexpr int BS = 64;                 // rows of a row block = columns of a tile
constexpr int kThreads = 256;          // 8 warps
constexpr unsigned long long kWaitNs = 4000000000ull;  // bound of one wait

struct Args {
  const float* lu;
  int64_t ld;
  double* X;        // solutions, all pending at the start
  int64_t ldx;
  double* B;        // right-hand sides
  int64_t ldb;
  int mark;         // leave B pending: the next pass publishes its solution there
  int early;        // LU and the sync words are ready before the kernel in front
                    // of this one ends: only B and X wait for it
  int64_t n;
  int64_t nrhs;
  int nblk;
  int ngroups;
  int forward;      // op(T) lower: L or U^T
  int unit;         // unit diagonal: L or L^T
  unsigned* sync;
  unsigned long long wait_ns;  // bound of one wait (kWaitNs)
  int withhold;     // self-test of the give-up path only: the row block solved
                    // first (ticket 0) does not publish its solution, -1: none
  int cluster;      // CTAs of a cluster of the warp kernel: kCluster or 1
};

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// cp.async with zero fill: copies src_bytes (0 .. size) and zeroes the rest.
__device__ __forceinline__ void cp16z(void* dst, const void* src, int src_bytes) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src),
               "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp4z(void* dst, const void* src, int src_bytes) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src),
               "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ int imin64(int64_t a, int b) { return a < b ? (int)a : b; }

// Shared layout of a full 64 x 64 tile of op(T) (rows r, columns k).  Not
// transposed: column k contiguous in r, by 16-byte chunks with chunk index
// (r/4) ^ (k & 7) (8 lanes reading one chunk of 8 consecutive columns hit 8
// bank groups).  Transposed: row-major.
template <bool TRANS>
__device__ __forceinline__ int tile_index(int r, int k) {
  return TRANS ? r * BS + k : k * BS + 4 * ((r >> 2) ^ (k & 7)) + (r & 3);
}

// Copy of the full tile op(T)[rows r0.., cols k0..] (rw x kw valid, the rest
// zero), all threads of the CTA.
template <bool TRANS, bool V16>
__device__ __forceinline__ void load_tile(float* dst, const Args& a, int64_t r0, int rw,
                                          int64_t k0, int kw) {
  const int tid = threadIdx.x;
  if (V16) {
#pragma unroll
    for (int m = 0; m < BS * BS / 4 / kThreads; ++m) {
      const int c = tid + m * kThreads;
      const int outer = c >> 4, q = c & 15;
      int64_t mcol, mrow;
      int valid;
      if (!TRANS) {
        mcol = k0 + outer; mrow = r0 + 4 * q;
        valid = outer < kw ? min(4, max(0, rw - 4 * q)) : 0;
      } else {
        mcol = r0 + outer; mrow = k0 + 4 * q;
        valid = outer < rw ? min(4, max(0, kw - 4 * q)) : 0;
      }
      const float* src = valid ? a.lu + mrow + mcol * a.ld : a.lu;
      float* d = TRANS ? dst + outer * BS + 4 * q : dst + outer * BS + 4 * (q ^ (outer & 7));
      cp16z(d, src, valid * 4);
    }
  } else {
#pragma unroll 4
    for (int m = 0; m < BS * BS / kThreads; ++m) {
      const int e = tid + m * kThreads;
      const int outer = e >> 6, inner = e & 63;
      if (!TRANS) {
        const bool ok = outer < kw && inner < rw;
        cp4z(dst + tile_index<false>(inner, outer),
             ok ? a.lu + (r0 + inner) + (k0 + outer) * a.ld : a.lu, ok ? 4 : 0);
      } else {
        const bool ok = outer < rw && inner < kw;
        cp4z(dst + tile_index<true>(outer, inner),
             ok ? a.lu + (k0 + inner) + (r0 + outer) * a.ld : a.lu, ok ? 4 : 0);
      }
    }
  }
}

// Copy of the diagonal block as plain fp32: memory column c, memory row r of
// the block at c * 64 + r (the rest zero), all threads of the CTA.
template <bool V16>
__device__ __forceinline__ void load_diag(float* dst, const Args& a, int64_t r0, int rw) {
  const int tid = threadIdx.x;
  if (V16) {
#pragma unroll
    for (int m = 0; m < BS * BS / 4 / kThreads; ++m) {
      const int c = tid + m * kThreads;
      const int outer = c >> 4, q = c & 15;
      const int valid = outer < rw ? min(4, max(0, rw - 4 * q)) : 0;
      const float* src = valid ? a.lu + (r0 + 4 * q) + (r0 + outer) * a.ld : a.lu;
      cp16z(dst + outer * BS + 4 * q, src, valid * 4);
    }
  } else {
#pragma unroll 4
    for (int m = 0; m < BS * BS / kThreads; ++m) {
      const int e = tid + m * kThreads;
      const int outer = e >> 6, inner = e & 63;
      const bool ok = outer < rw && inner < rw;
      cp4z(dst + outer * BS + inner, ok ? a.lu + (r0 + inner) + (r0 + outer) * a.ld : a.lu,
           ok ? 4 : 0);
    }
  }
}

// Inverse of the diagonal block of op(T) (fp32 in Dsrc as load_diag left it)
// by fp64 substitution with the reciprocals of the diagonal: column j by
// lanes 4j .. 4j+3, part p holding rows 4s + p.  Written row-major into
// Dinv[r * DS + j] (the same space as Dsrc; barriers separate the reads from
// the writes).  The block is converted to fp64 once, in place (column k at Dinv
// + 64 k): converting inside the substitution took most of its time.  Rows
// and columns past rw are the identity.  All threads.
template <bool TRANS, int DS = BS>
__device__ __forceinline__ void invert_diag(const float* Dsrc, double* Dinv, double* rdiag,
                                            int rw, bool fwd, bool unit) {
  const int tid = threadIdx.x, lane = tid & 31;
  {
    // thread: 4 x 4 elements of memory column 4 (tid / 16) + e, rows 4 (tid % 16) ..
    float v[4][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 u = *reinterpret_cast<const float4*>(Dsrc + (4 * (tid >> 4) + e) * BS +
                                                        4 * (tid & 15));
      v[e][0] = u.x; v[e][1] = u.y; v[e][2] = u.z; v[e][3] = u.w;
    }
    __syncthreads();
    const int mc = 4 * (tid >> 4), mr = 4 * (tid & 15);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      // op(T) row r, column k at Dinv[k * 64 + r]
      double* d = TRANS ? Dinv + (mr + e) * BS + mc : Dinv + (mc + e) * BS + mr;
      *reinterpret_cast<double2*>(d) = TRANS ? make_double2(v[0][e], v[1][e])
                                             : make_double2(v[e][0], v[e][1]);
      *reinterpret_cast<double2*>(d + 2) = TRANS ? make_double2(v[2][e], v[3][e])
                                                 : make_double2(v[e][2], v[e][3]);
    }
    __syncthreads();
  }
  auto D = [&](int r, int k) -> double { return Dinv[k * BS + r]; };
  if (tid < BS) rdiag[tid] = (unit || tid >= rw) ? 1.0 : 1.0 / D(tid, tid);
  __syncthreads();
  const int j = tid >> 2, p = tid & 3;
  double z[16];
#pragma unroll
  for (int s = 0; s < 16; ++s) z[s] = (4 * s + p == j) ? 1.0 : 0.0;
  if (fwd) {
#pragma unroll
    for (int k = 0; k < BS; ++k) {
      const bool live = k >= j;
      if (live && p == (k & 3)) z[k >> 2] *= rdiag[k];
      const double zk = __shfl_sync(0xffffffffu, z[k >> 2], (lane & ~3) | (k & 3));
      if (live) {
#pragma unroll
        for (int s = 0; s < 16; ++s)
          if (4 * s + p > k) z[s] = fma(-D(4 * s + p, k), zk, z[s]);
      }
    }
  } else {
#pragma unroll
    for (int k = BS - 1; k >= 0; --k) {
      const bool live = k <= j;
      if (live && p == (k & 3)) z[k >> 2] *= rdiag[k];
      const double zk = __shfl_sync(0xffffffffu, z[k >> 2], (lane & ~3) | (k & 3));
      if (live) {
#pragma unroll
        for (int s = 0; s < 16; ++s)
          if (4 * s + p < k) z[s] = fma(-D(4 * s + p, k), zk, z[s]);
      }
    }
  }
  __syncthreads();  // every read of the block precedes the overwrite
#pragma unroll
  for (int s = 0; s < 16; ++s) Dinv[(4 * s + p) * DS + j] = z[s];
  __syncthreads();
}

// Sum over the 32 lanes of each of 8 per-lane partial rows: three halving
// exchanges, then two full steps.  Lanes 4i .. 4i+3 end with row i.
__device__ __forceinline__ double row_reduce(double (&v)[8], int lane) {
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double send = b4 ? v[i] : v[i + 4];
    const double keep = b4 ? v[i + 4] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double send = b3 ? v[i] : v[i + 2];
    const double keep = b3 ? v[i + 2] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  double s;
  {
    const double send = b2 ? v[0] : v[1];
    const double keep = b2 ? v[1] : v[0];
    s = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s;
}

// ======================================================================
// Warp kernel (1 to 4 right-hand sides, in groups of 1 or 2).  X is marked pending by
// trsv_prepare_kernel; a solution entry is published by one store and read
// by relaxed loads at GPU scope, re-read while pending -- the solution is
// its own flag.
// ======================================================================

constexpr int S = 3;                   // stages of each warp's tile ring
// Row blocks solved one after another by the CTAs of one cluster: they hand
// their solutions over through distributed shared memory (0.6 us a block on
// B200, against 1.0 through L2 and 1.5 .. 2 from one cluster to the next, which
// is why 16 rather than the portable 8).  Where no cluster of 16 fits (few SMs in a
// processing cluster of the context), every CTA is its own.
constexpr int kCluster = 16;
constexpr int kWarpTile = 8 * BS;      // floats of a warp's share of a tile
// Marks a solution entry not yet published: a signalling-NaN payload that no
// arithmetic produces (published NaNs are stored as the canonical quiet NaN).
constexpr unsigned long long kPending = 0x7ff4dead5e1f5e1full;
constexpr unsigned long long kQuietNaN = 0x7ff8000000000000ull;

__host__ __device__ constexpr size_t warp_smem_bytes(int nr) {
  return (size_t)S * 8 * kWarpTile * 4    // per-warp tile rings (fp32)
         + (size_t)BS * BS * 8            // inverse of the diagonal block (fp64)
         + (size_t)BS * BS * 4            // tile of the previous block (fp32)
         + (size_t)BS * 8                 // reciprocals of the diagonal
         + (size_t)kCluster * nr * BS * 8 // solutions of the cluster's blocks
         + 64;                            // control words
}

__device__ __forceinline__ double ld_poll(const double* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return __longlong_as_double((long long)v);
}
__device__ __forceinline__ unsigned long long publish_bits(double x) {
  const unsigned long long v = (unsigned long long)__double_as_longlong(x);
  return (v & 0x7ff0000000000000ull) == 0x7ff0000000000000ull && (v & 0xfffffffffffffull)
             ? kQuietNaN : v;
}
__device__ __forceinline__ void st_publish(double* p, double x) {
  const unsigned long long v = publish_bits(x);
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Distributed shared memory: the cluster barrier, this CTA's rank, 8-byte and
// 4-byte stores to the same place in another CTA of the cluster.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
               "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ int cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}
__device__ __forceinline__ uint32_t map_rank(const void* p, int rank) {
  const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
  uint32_t d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(rank));
  return d;
}
__device__ __forceinline__ void st_remote64(const double* p, int rank, unsigned long long v) {
  asm volatile("st.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(map_rank(p, rank)), "l"(v)
               : "memory");
}
__device__ __forceinline__ void st_remote32(const int* p, int rank, int v) {
  asm volatile("st.relaxed.cluster.shared::cluster.b32 [%0], %1;" ::"r"(map_rank(p, rank)), "r"(v)
               : "memory");
}
__device__ __forceinline__ double ld_local64(const double* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.cluster.shared::cta.b64 %0, [%1];"
               : "=l"(v) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))) : "memory");
  return __longlong_as_double((long long)v);
}
__device__ __forceinline__ int ld_local32(const int* p) {
  int v;
  asm volatile("ld.relaxed.cluster.shared::cta.b32 %0, [%1];"
               : "=r"(v) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))) : "memory");
  return v;
}
__device__ __forceinline__ bool pending(double x) {
  return (unsigned long long)__double_as_longlong(x) == kPending;
}

// A warp's share of a tile.  Transposed (row share): rows 8w .. 8w+7 of the
// block, row-major [i][k] (each row of op(T) is 256 contiguous bytes of one
// factor column).  Not transposed (column share): columns 8w .. 8w+7 of the
// tile, [j][r] (each column 256 contiguous bytes).  Copied by the warp's
// own lanes.
template <bool TRANS, bool V16>
__device__ __forceinline__ void load_warp_tile(float* dst, const Args& a, int64_t r0, int rw,
                                               int64_t k0, int kw, int w, int lane) {
  const int b = 8 * w;
  if (V16) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int c = lane + 32 * m;
      const int o = c >> 4, q = c & 15;
      int valid;
      const float* src;
      if (!TRANS) {
        valid = b + o < kw ? min(4, max(0, rw - 4 * q)) : 0;
        src = valid ? a.lu + (r0 + 4 * q) + (k0 + b + o) * a.ld : a.lu;
      } else {
        valid = b + o < rw ? min(4, max(0, kw - 4 * q)) : 0;
        src = valid ? a.lu + (k0 + 4 * q) + (r0 + b + o) * a.ld : a.lu;
      }
      cp16z(dst + o * BS + 4 * q, src, valid * 4);
    }
  } else {
#pragma unroll 4
    for (int m = 0; m < 16; ++m) {
      const int e = lane + 32 * m;
      const int o = e >> 6, i = e & 63;
      bool ok;
      const float* src;
      if (!TRANS) {
        ok = b + o < kw && i < rw;
        src = ok ? a.lu + (r0 + i) + (k0 + b + o) * a.ld : a.lu;
      } else {
        ok = b + o < rw && i < kw;
        src = ok ? a.lu + (k0 + i) + (r0 + b + o) * a.ld : a.lu;
      }
      cp4z(dst + o * BS + i, src, ok ? 4 : 0);
    }
  }
}

// Solution entries of tile columns kb + h*ks (h < NX) of the group's
// columns (0 outside the matrix), as loaded -- possibly still pending.
template <int NX, int NR>
__device__ __forceinline__ void fetch_x(double (&x)[NX][NR], const Args& a, int64_t k0, int kw,
                                        int64_t c0, int nc, int kb, int ks) {
#pragma unroll
  for (int h = 0; h < NX; ++h)
#pragma unroll
    for (int c = 0; c < NR; ++c) {
      const int k = kb + h * ks;
      x[h][c] = (k < kw && c < nc) ? ld_poll(a.X + (k0 + k) + (c0 + c) * a.ldx) : 0.0;
    }
}
// Re-read the entries still pending until the whole warp has them.
// Bounded: after kWaitNs the pending entries become NaN and the count of
// expired waits is raised; every other wait of the solve then gives up at
// once, so a lost block costs one bound, not one per block, and its NaN
// propagates to every later block (a failed solve never looks like a
// result).
template <int NX, int NR>
__device__ __forceinline__ void settle_x(double (&x)[NX][NR], const Args& a, int64_t k0,
                                         int64_t c0, int kb, int ks, int lane) {
  bool ok = true;
#pragma unroll
  for (int h = 0; h < NX; ++h)
#pragma unroll
    for (int c = 0; c < NR; ++c) ok &= !pending(x[h][c]);
  if (__all_sync(0xffffffffu, ok)) return;
  const unsigned long long t0 = global_ns();
  for (;;) {
    ok = true;
#pragma unroll
    for (int h = 0; h < NX; ++h)
#pragma unroll
      for (int c = 0; c < NR; ++c)
        if (pending(x[h][c])) {
          x[h][c] = ld_poll(a.X + (k0 + kb + h * ks) + (c0 + c) * a.ldx);
          ok &= !pending(x[h][c]);
        }
    if (__all_sync(0xffffffffu, ok)) return;
    const bool expired = global_ns() - t0 > a.wait_ns;
    if (__any_sync(0xffffffffu, expired || *(volatile unsigned*)(a.sync + 1) != 0u)) {
#pragma unroll
      for (int h = 0; h < NX; ++h)
#pragma unroll
        for (int c = 0; c < NR; ++c)
          if (pending(x[h][c])) x[h][c] = __longlong_as_double((long long)kQuietNaN);
      if (lane == 0 && expired) atomicAdd(a.sync + 1, 1u);
      return;
    }
  }
}

// The same entries of a block that a CTA of this cluster solves, from the copy it
// writes into this CTA's shared memory (xin: [column][row]); the wait bounded
// as in settle_x.
template <int NX, int NR>
__device__ __forceinline__ void settle_local(double (&x)[NX][NR], const Args& a,
                                             const double* xin, int kw, int nc, int kb, int ks,
                                             int lane) {
#pragma unroll
  for (int h = 0; h < NX; ++h)
#pragma unroll
    for (int c = 0; c < NR; ++c)
      x[h][c] = (kb + h * ks < kw && c < nc) ? __longlong_as_double((long long)kPending) : 0.0;
  unsigned long long t0 = 0;
  for (unsigned it = 0;; ++it) {
    bool ok = true;
#pragma unroll
    for (int h = 0; h < NX; ++h)
#pragma unroll
      for (int c = 0; c < NR; ++c)
        if (pending(x[h][c])) {
          x[h][c] = ld_local64(xin + c * BS + kb + h * ks);
          ok &= !pending(x[h][c]);
        }
    if (__all_sync(0xffffffffu, ok)) return;
    if ((it & 31u) != 31u) continue;
    const unsigned long long now = global_ns();
    if (t0 == 0) t0 = now;
    const bool expired = now - t0 > a.wait_ns;
    if (__any_sync(0xffffffffu, expired || *(volatile unsigned*)(a.sync + 1) != 0u)) {
#pragma unroll
      for (int h = 0; h < NX; ++h)
#pragma unroll
        for (int c = 0; c < NR; ++c)
          if (pending(x[h][c])) x[h][c] = __longlong_as_double((long long)kQuietNaN);
      if (lane == 0 && expired) atomicAdd(a.sync + 1, 1u);
      return;
    }
  }
}

// settle_x for the matrix kernel's hand-over: entry e is row 8 (e / 2) + 2 lk +
// (e & 1) of one column.
__device__ __forceinline__ void settle_mma(double (&x)[16][1], const Args& a, int64_t k0,
                                           int64_t c, int lk, int lane) {
  bool ok = true;
#pragma unroll
  for (int e = 0; e < 16; ++e) ok &= !pending(x[e][0]);
  if (__all_sync(0xffffffffu, ok)) return;
  const unsigned long long t0 = global_ns();
  for (;;) {
    ok = true;
#pragma unroll
    for (int e = 0; e < 16; ++e)
      if (pending(x[e][0])) {
        x[e][0] = ld_poll(a.X + k0 + 8 * (e >> 1) + 2 * lk + (e & 1) + c * a.ldx);
        ok &= !pending(x[e][0]);
      }
    if (__all_sync(0xffffffffu, ok)) return;
    const bool expired = global_ns() - t0 > a.wait_ns;
    if (__any_sync(0xffffffffu, expired || *(volatile unsigned*)(a.sync + 1) != 0u)) {
#pragma unroll
      for (int e = 0; e < 16; ++e)
        if (pending(x[e][0])) x[e][0] = __longlong_as_double((long long)kQuietNaN);
      if (lane == 0 && expired) atomicAdd(a.sync + 1, 1u);
      return;
    }
  }
}

// One CTA per (row block, group): warps stream their shares of the tiles
// of all blocks but the previous one without CTA barriers; one barrier
// combines the partial sums into c = Dinv y; the hand-over x = c - W x_prev
// runs per warp (W = Dinv op(T)[block, previous block] in registers: rows
// 8 warp + i, columns lane and lane + 32).
template <bool TRANS, int NR, bool V16>
__global__ void __launch_bounds__(kThreads, 2)
trsv_kernel(Args a) {
  constexpr int PD = NR == 1 ? 3 : 2;     // tiles whose solution entries are fetched ahead
  constexpr int NX = TRANS ? 2 : 1;       // solution entries per lane per tile
  extern __shared__ __align__(16) unsigned char smem[];
  float* ring = reinterpret_cast<float*>(smem);
  double* Dinv = reinterpret_cast<double*>(smem + (size_t)S * 8 * kWarpTile * 4);
  float* Tw = reinterpret_cast<float*>(Dinv + BS * BS);
  double* rdiag = reinterpret_cast<double*>(Tw + BS * BS);
  double* xin = rdiag + BS;              // [block of the cluster][column][row]
  int* ctrl = reinterpret_cast<int*>(xin + kCluster * NR * BS);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (!a.early) dependency_wait();
  dependents_launch();
  // the cluster's ticket: its consecutive row blocks of one group
  const int rank = cluster_rank();
  for (int e = tid; e < kCluster * NR * BS; e += kThreads)
    xin[e] = __longlong_as_double((long long)kPending);
  if (tid == 0) ctrl[0] = -1;
  cluster_sync();   // every CTA runs and has its markers in place
  if (rank == 0 && tid < kCluster) {
    int tk = 0;
    if (tid == 0) tk = (int)atomicAdd(a.sync, 1u);
    tk = __shfl_sync((1u << kCluster) - 1, tk, 0);
    if (tid < a.cluster) st_remote32(ctrl, tid, tk);
  }
  if (tid == 0) {
    // the store is on its way; bounded like every wait
    int tk = -1;
    for (int it = 0; it < (1 << 24) && tk < 0; ++it) tk = ld_local32(ctrl);
    if (tk < 0) atomicAdd(a.sync + 1, 1u);
    ctrl[1] = tk;
  }
  __syncthreads();
  const int ticket = ctrl[1];
  const int base = ticket / a.ngroups * a.cluster;    // first block of the cluster
  const int t = base + rank, g = ticket % a.ngroups;
  if (ticket < 0 || t >= a.nblk) {
    cluster_sync();   // as at the end
    return;
  }
  const bool fwd = a.forward != 0;
  const int64_t r0 = (int64_t)(fwd ? t : a.nblk - 1 - t) * BS;
  const int rw = imin64(a.n - r0, BS);
  const int64_t c0 = (int64_t)g * NR;
  const int nc = imin64(a.nrhs - c0, NR);
  auto tile_k0 = [&](int q) -> int64_t { return (int64_t)(fwd ? q : a.nblk - 1 - q) * BS; };
  auto tile_kw = [&](int q) -> int { return imin64(a.n - tile_k0(q), BS); };
  const int nbulk = t > 1 ? t - 1 : 0;  // tiles before the previous block's
  const int nglob = nbulk < base ? nbulk : base;  // of them, solved by other clusters
  // tile columns whose solution entries this lane reads in the bulk phase
  const int kb = TRANS ? lane : 8 * warp + (lane & 7);
  const int ks = TRANS ? 32 : 0;

  // ---- set-up copies: diagonal block, previous block's tile, ring prologue
  float* Dsrc = reinterpret_cast<float*>(Dinv);
  load_diag<V16>(Dsrc, a, r0, rw);
  if (t >= 1) load_tile<TRANS, V16>(Tw, a, r0, rw, tile_k0(t - 1), tile_kw(t - 1));
  cp_commit();
  float* wring = ring + warp * S * kWarpTile;
  auto issue = [&](int q) {
    if (q < nbulk)
      load_warp_tile<TRANS, V16>(wring + (q % S) * kWarpTile, a, r0, rw, tile_k0(q),
                                 tile_kw(q), warp, lane);
    cp_commit();
  };
#pragma unroll
  for (int q = 0; q < S - 1; ++q) issue(q);
  double xq[PD][NX][NR];
  double bm[2][NR];   // right-hand sides of rows lane and lane + 32
  auto fetch_inputs = [&]() {
#pragma unroll
    for (int d = 0; d < PD; ++d)
      if (d < nglob) fetch_x<NX, NR>(xq[d], a, tile_k0(d), tile_kw(d), c0, nc, kb, ks);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        const int r = lane + 32 * h;
        bm[h][c] = (r < rw && c < nc) ? a.B[(r0 + r) + (c0 + c) * a.ldb] : 0.0;
      }
  };
  if (!a.early) fetch_inputs();

  cp_wait<S - 1>();
  __syncthreads();
  if (a.mark && warp == 0)   // every warp has its copy
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int c = 0; c < NR; ++c)
        if (lane + 32 * h < rw && c < nc)
          a.B[(r0 + lane + 32 * h) + (c0 + c) * a.ldb] = __longlong_as_double((long long)kPending);
  invert_diag<TRANS>(Dsrc, Dinv, rdiag, rw, fwd, a.unit != 0);

  // ---- W = Dinv * op(T)[block, previous block] ----
  double W[8][2];
#pragma unroll
  for (int i = 0; i < 8; ++i) W[i][0] = W[i][1] = 0.0;
  if (t >= 1) {
#pragma unroll 2
    for (int m4 = 0; m4 < BS / 4; ++m4) {
      float tk[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = lane + 32 * h;
        if (!TRANS) {
          const float4 u = *reinterpret_cast<const float4*>(Tw + tile_index<false>(4 * m4, k));
          tk[h][0] = u.x; tk[h][1] = u.y; tk[h][2] = u.z; tk[h][3] = u.w;
        } else {
#pragma unroll
          for (int mm = 0; mm < 4; ++mm) tk[h][mm] = Tw[tile_index<true>(4 * m4 + mm, k)];
        }
      }
#pragma unroll
      for (int mm = 0; mm < 4; ++mm)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const double d = Dinv[(8 * warp + i) * BS + 4 * m4 + mm];
          W[i][0] = fma(d, (double)tk[0][mm], W[i][0]);
          W[i][1] = fma(d, (double)tk[1][mm], W[i][1]);
        }
    }
  }

  if (a.early) {
    dependency_wait();
    fetch_inputs();
  }

  // ---- bulk: the tiles before the previous block's, per warp.
  // Transposed: rows 8 warp + i, per-lane partials over columns lane and
  // lane + 32.  Not transposed: columns 8 warp + j, per-lane partials of
  // rows lane and lane + 32 (the solution entry of column j broadcast from
  // lane j). ----
  constexpr int NA = TRANS ? 8 : 2;
  double acc[NA][NR];
#pragma unroll
  for (int i = 0; i < NA; ++i)
#pragma unroll
    for (int c = 0; c < NR; ++c) acc[i][c] = 0.0;
#pragma unroll 1
  for (int q = 0; q < nbulk; ++q) {
    double x[NX][NR];
#pragma unroll
    for (int h = 0; h < NX; ++h)
#pragma unroll
      for (int c = 0; c < NR; ++c) x[h][c] = xq[0][h][c];
#pragma unroll
    for (int d = 0; d + 1 < PD; ++d)
#pragma unroll
      for (int h = 0; h < NX; ++h)
#pragma unroll
        for (int c = 0; c < NR; ++c) xq[d][h][c] = xq[d + 1][h][c];
    if (q + PD < nglob)
      fetch_x<NX, NR>(xq[PD - 1], a, tile_k0(q + PD), tile_kw(q + PD), c0, nc, kb, ks);
    if (q < nglob) settle_x<NX, NR>(x, a, tile_k0(q), c0, kb, ks, lane);
    else settle_local<NX, NR>(x, a, xin + (q - base) * NR * BS, tile_kw(q), nc, kb, ks, lane);
    cp_wait<S - 2>();
    __syncwarp();
    issue(q + S - 1);
    const float* Ts = wring + (q % S) * kWarpTile;
    if (TRANS) {
#pragma unroll
      for (int h = 0; h < NX; ++h) {
        const int k = lane + 32 * h;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const double tv = (double)Ts[i * BS + k];
#pragma unroll
          for (int c = 0; c < NR; ++c) acc[i][c] = fma(tv, x[h][c], acc[i][c]);
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        double xj[NR];
#pragma unroll
        for (int c = 0; c < NR; ++c) xj[c] = __shfl_sync(0xffffffffu, x[0][c], j);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double tv = (double)Ts[j * BS + lane + 32 * h];
#pragma unroll
          for (int c = 0; c < NR; ++c) acc[h][c] = fma(tv, xj[c], acc[h][c]);
        }
      }
    }
  }
  cp_wait<0>();

  // the previous block's solution: fetched now, waited for after c
  double xf[2][NR];
  if (t >= 1 && rank == 0)
    fetch_x<2, NR>(xf, a, tile_k0(t - 1), tile_kw(t - 1), c0, nc, lane, 32);

  // ---- partial sums of the warps -> y = b - sum -> c = Dinv y ----
  // (each in its warp's ring, which is done with: two CTAs fit on an SM)
  auto part = [&](int w) { return reinterpret_cast<double*>(ring + w * S * kWarpTile); };
  __syncwarp();
  if (TRANS) {
#pragma unroll
    for (int c = 0; c < NR; ++c) {
      double v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = acc[i][c];
      const double s = row_reduce(v, lane);
      if ((lane & 3) == 0) part(warp)[c * 8 + (lane >> 2)] = s;
    }
  } else {
#pragma unroll
    for (int c = 0; c < NR; ++c)
#pragma unroll
      for (int h = 0; h < 2; ++h) part(warp)[c * BS + lane + 32 * h] = acc[h][c];
  }
  __syncthreads();
  double cv[NR];
#pragma unroll
  for (int c = 0; c < NR; ++c) {
    double y[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int m = lane + 32 * h;
      double s;
      if (TRANS) {
        s = part(m >> 3)[c * 8 + (m & 7)];
      } else {
        s = part(0)[c * BS + m];
#pragma unroll
        for (int w = 1; w < 8; ++w) s += part(w)[c * BS + m];
      }
      y[h] = bm[h][c] - s;
    }
    double v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      v[i] = fma(Dinv[(8 * warp + i) * BS + lane + 32], y[1],
                 Dinv[(8 * warp + i) * BS + lane] * y[0]);
    cv[c] = row_reduce(v, lane);
  }

  // ---- hand-over: x = c - W x_prev once the previous block is out ----
  if (t >= 1) {
    if (rank == 0) settle_x<2, NR>(xf, a, tile_k0(t - 1), c0, lane, 32, lane);
    else settle_local<2, NR>(xf, a, xin + (rank - 1) * NR * BS, tile_kw(t - 1), nc, lane, 32, lane);
#pragma unroll
    for (int c = 0; c < NR; ++c) {
      double v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = fma(W[i][1], xf[1][c], W[i][0] * xf[0][c]);
      cv[c] -= row_reduce(v, lane);
    }
  }
  // to the later CTAs of the cluster (a row's four lanes take turns), then to
  // the other clusters
  const int ri = 8 * warp + (lane >> 2);
  if (ri < rw && t != a.withhold) {
#pragma unroll
    for (int c = 0; c < NR; ++c)
      if (c < nc) {
#pragma unroll
        for (int h = 0; h < kCluster / 4; ++h) {
          const int to = rank + 1 + (lane & 3) + 4 * h;
          if (to < a.cluster && base + to < a.nblk)
            st_remote64(xin + (rank * NR + c) * BS + ri, to, publish_bits(cv[c]));
        }
        if ((lane & 3) == 0) st_publish(a.X + (r0 + ri) + (c0 + c) * a.ldx, cv[c]);
      }
  }
  // no CTA leaves while another may still write into its shared memory
  cluster_sync();
}

constexpr int kHeader = 4;   // words of a pass's sync area: ticket, expired waits, spare

// Clears the ticket and expiry words of both passes' sync areas and marks the
// n x nrhs solutions at Y (dense) pending; X given: moves X there first and
// marks X itself (one pass in place).
__global__ void trsv_prepare_kernel(int64_t n, int64_t nrhs, double* __restrict__ X,
                                    int64_t ldx, double* __restrict__ Y,
                                    unsigned* __restrict__ sync) {
  dependency_wait();
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e == 0) sync[0] = sync[1] = sync[kHeader] = sync[kHeader + 1] = 0;
  if (e >= n * nrhs) return;
  double* p = Y + e;
  if (X) {
    const int64_t c = e / n, i = e - c * n;
    p = X + i + c * ldx;
    Y[e] = *p;
  }
  *p = __longlong_as_double((long long)kPending);
}

// ======================================================================
// Matrix kernel (groups of 8 right-hand sides): the same scheme on mma64.
// Warp w takes columns 8w .. 8w + 7 of every tile for all 64 rows -- each tile
// element is loaded and converted once per CTA, straight from global memory to
// registers one tile ahead, and a lane reads only two solution entries per
// tile -- then rows 8w .. of Dinv y and of the hand-over.
//
// Bound by the FP64 rate (n = 8192, 64 right-hand sides: 2.1 G multiply-adds
// per triangle, 0.12 ms) and, as long, by the chain of n / 64 hand-overs.
// ======================================================================

constexpr int DS = BS + 4;   // row stride of Dinv: conflict-free fragment reads
constexpr int YS = 12;       // row stride of y, likewise

constexpr size_t mma_smem_bytes() {
  return (size_t)BS * DS * 8          // inverse of the diagonal block (fp64)
         + (size_t)BS * BS * 4        // tile of the previous block (fp32)
         + (size_t)8 * BS * 8 * 8     // the warps' partial sums
         + (size_t)BS * YS * 8        // y
         + (size_t)BS * 8             // reciprocals of the diagonal
         + 64;                        // control words
}

template <bool TRANS, bool V16>
__global__ void __launch_bounds__(kThreads, 2)
trsv_mma_kernel(Args a) {
  constexpr int PD = 3;     // tiles whose solution entries are fetched ahead
  extern __shared__ __align__(16) unsigned char smem[];
  double* Dinv = reinterpret_cast<double*>(smem);
  float* Tw = reinterpret_cast<float*>(Dinv + BS * DS);
  double* part = reinterpret_cast<double*>(Tw + BS * BS);
  double* ybuf = part + 8 * BS * 8;
  double* rdiag = ybuf + BS * YS;
  int* ctrl = reinterpret_cast<int*>(rdiag + BS);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lr = lane >> 2, lk = lane & 3;
  if (!a.early) dependency_wait();
  dependents_launch();
  if (tid == 0) ctrl[0] = (int)atomicAdd(a.sync, 1u);
  __syncthreads();
  const int ticket = ctrl[0];
  const int t = ticket / a.ngroups, g = ticket - t * a.ngroups;
  const bool fwd = a.forward != 0;
  const int64_t r0 = (int64_t)(fwd ? t : a.nblk - 1 - t) * BS;
  const int rw = imin64(a.n - r0, BS);
  const int64_t c0 = (int64_t)g * 8;
  const int nc = imin64(a.nrhs - c0, 8);
  auto tile_k0 = [&](int q) -> int64_t { return (int64_t)(fwd ? q : a.nblk - 1 - q) * BS; };
  auto tile_kw = [&](int q) -> int { return imin64(a.n - tile_k0(q), BS); };
  const int nbulk = t > 1 ? t - 1 : 0;  // tiles before the previous block's

  // ---- set-up copies: diagonal block, previous block's tile
  float* Dsrc = reinterpret_cast<float*>(Dinv);
  load_diag<V16>(Dsrc, a, r0, rw);
  if (t >= 1) load_tile<TRANS, V16>(Tw, a, r0, rw, tile_k0(t - 1), tile_kw(t - 1));
  cp_commit();

  // This warp's share of tile q: entry [m][s] is row 8 m + lr and column kk(s).
  // Rows past the matrix repeat the last one (their sums are dropped); only the
  // first tile of a backward solve has columns past it.
  auto kk = [&](int s) { return 8 * warp + (TRANS ? 2 * lk + s : 4 * s + lk); };
  auto load_a = [&](int q, float (&v)[8][2]) {
    const int64_t k0 = tile_k0(q);
    // not transposed, the limit stays here though only load_first needs it: without
    // it the kernel spills (n = 10007, 8 columns: 875 us, 818 with it)
    const int kw = TRANS ? BS : tile_kw(q);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int64_t r = r0 + (8 * m + lr < rw ? 8 * m + lr : rw - 1);
      if (TRANS && V16) {
        const float2 y = *reinterpret_cast<const float2*>(a.lu + k0 + kk(0) + r * a.ld);
        v[m][0] = y.x;
        v[m][1] = y.y;
      } else {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int64_t k = k0 + (kk(s) < kw ? kk(s) : kw - 1);
          v[m][s] = TRANS ? a.lu[k + r * a.ld] : a.lu[r + k * a.ld];
        }
      }
    }
  };
  // the first tile, columns past the matrix zero: they meet zeros of x, whose
  // products with an infinity would not be
  auto load_first = [&](float (&v)[8][2]) {
    const int64_t k0 = tile_k0(0);
    const int kw = tile_kw(0);
    if (kw == BS) return load_a(0, v);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int64_t r = r0 + (8 * m + lr < rw ? 8 * m + lr : rw - 1);
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int64_t k = k0 + kk(s);
        v[m][s] = kk(s) < kw ? (TRANS ? a.lu[k + r * a.ld] : a.lu[r + k * a.ld]) : 0.0f;
      }
    }
  };
  // Solution entries kb, kb + ks of column lr of the group, as loaded
  const int xs = TRANS ? 1 : 4;
  auto fetch = [&](double (&x)[2], int q) {
    const int64_t k0 = tile_k0(q);
    const int kw = tile_kw(q);
#pragma unroll
    for (int s = 0; s < 2; ++s)
      x[s] = (kk(s) < kw && lr < nc) ? ld_poll(a.X + k0 + kk(s) + (c0 + lr) * a.ldx) : 0.0;
  };
  float cur[8][2], nxt[8][2];
  double xq[PD][2];
  // right-hand side entries (row tid / 4, columns 2 (tid & 3) and the next)
  double bm[2];
  auto fetch_inputs = [&]() {
#pragma unroll
    for (int d = 0; d < PD; ++d)
      if (d < nbulk) fetch(xq[d], d);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = tid >> 2, c = 2 * (tid & 3) + h;
      double* p = a.B + (r0 + r) + (c0 + c) * a.ldb;
      bm[h] = 0.0;
      if (r < rw && c < nc) {
        bm[h] = *p;
        if (a.mark) *p = __longlong_as_double((long long)kPending);
      }
    }
  };
  if (!a.early) fetch_inputs();
  if (nbulk > 0) load_first(cur);
  cp_wait<0>();
  __syncthreads();
  invert_diag<TRANS, DS>(Dsrc, Dinv, rdiag, rw, fwd, a.unit != 0);

  // ---- W = Dinv op(T)[block, previous block], rows 8 warp + lr: columns 8 f +
  // 2 lk + h, which the hand-over takes as its k index
  double W[8][2];
#pragma unroll
  for (int f = 0; f < 8; ++f) W[f][0] = W[f][1] = 0.0;
  if (t >= 1) {
#pragma unroll 2
    for (int s = 0; s < BS / 4; ++s) {
      const int k = 4 * s + lk;
      const double d = Dinv[(8 * warp + lr) * DS + k];
#pragma unroll
      for (int f = 0; f < 8; ++f) mma64(W[f], d, (double)Tw[tile_index<TRANS>(k, 8 * f + lr)]);
    }
  }

  if (a.early) {
    dependency_wait();
    fetch_inputs();
  }

  // ---- bulk: the tiles before the previous block's
  double acc[8][2];
#pragma unroll
  for (int m = 0; m < 8; ++m) acc[m][0] = acc[m][1] = 0.0;
#pragma unroll 1
  for (int q = 0; q < nbulk; ++q) {
    double x[2][1] = {{xq[0][0]}, {xq[0][1]}};
#pragma unroll
    for (int d = 0; d + 1 < PD; ++d) {
      xq[d][0] = xq[d + 1][0];
      xq[d][1] = xq[d + 1][1];
    }
    if (q + PD < nbulk) fetch(xq[PD - 1], q + PD);
    if (q + 1 < nbulk) load_a(q + 1, nxt);
    settle_x<2, 1>(x, a, tile_k0(q), c0 + lr, kk(0), xs, lane);
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int m = 0; m < 8; ++m) mma64(acc[m], (double)cur[m][s], x[s][0]);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      cur[m][0] = nxt[m][0];
      cur[m][1] = nxt[m][1];
    }
  }

  // the previous block's solution: fetched now, waited for after c
  double xf[16][1];
  if (t >= 1) {
    const int64_t k0 = tile_k0(t - 1);
    const int kw = tile_kw(t - 1);
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const int k = 8 * (e >> 1) + 2 * lk + (e & 1);
      xf[e][0] = (k < kw && lr < nc) ? ld_poll(a.X + k0 + k + (c0 + lr) * a.ldx) : 0.0;
    }
  }

  // ---- partial sums of the warps -> y = b - sum -> c = Dinv y
#pragma unroll
  for (int m = 0; m < 8; ++m)
    *reinterpret_cast<double2*>(part + (warp * BS + 8 * m + lr) * 8 + 2 * lk) =
        make_double2(acc[m][0], acc[m][1]);
  __syncthreads();
  {
    const int r = tid >> 2, c = 2 * (tid & 3);
    double2 y = make_double2(0.0, 0.0);
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const double2 p = *reinterpret_cast<const double2*>(part + (w * BS + r) * 8 + c);
      y.x += p.x;
      y.y += p.y;
    }
    // rows past the matrix stay zero
    ybuf[r * YS + c] = r < rw ? bm[0] - y.x : 0.0;
    ybuf[r * YS + c + 1] = r < rw ? bm[1] - y.y : 0.0;
  }
  __syncthreads();
  double cv[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
  for (int s = 0; s < BS / 4; ++s)
    mma64(cv[s & 1], Dinv[(8 * warp + lr) * DS + 4 * s + lk], ybuf[(4 * s + lk) * YS + lr]);
  cv[0][0] += cv[1][0];
  cv[0][1] += cv[1][1];

  // ---- hand-over: x = c - W x_prev once the previous block is out
  if (t >= 1) {
    settle_mma(xf, a, tile_k0(t - 1), c0 + lr, lk, lane);
    double h[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
    for (int e = 0; e < 16; ++e) mma64(h[e & 1], W[e >> 1][e & 1], xf[e][0]);
    cv[0][0] -= h[0][0] + h[1][0];
    cv[0][1] -= h[0][1] + h[1][1];
  }
  const int row = 8 * warp + lr;
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (row < rw && 2 * lk + h < nc)
      st_publish(a.X + (r0 + row) + (c0 + 2 * lk + h) * a.ldx, cv[0][h]);
}

// Right-hand sides per CTA: from five on, the matrix kernel's 8; three or four as
// two groups of two (three, on B200: n = 2000 100 us, 8192 339, 10007 579, against
// 126, 464 and 636 with the matrix kernel).  Five in pairs gain little where the
// three groups fit (n = 2000 100 us against 132, 8192 482 against 498) and lose
// more where they do not (10007 862 against 703), so n is not in the rule.
int group_width(int64_t nrhs) { return nrhs >= 5 ? 8 : nrhs >= 2 ? 2 : 1; }

cudaLaunchAttribute cluster_attribute() {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = kCluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  return at;
}

// Whether clusters of kCluster CTAs of fn (a trsv_kernel) can run with this shared
// memory, asked once per kernel, device and amount (two columns have two).
bool clusters_fit(const void* fn, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<const void*, int, size_t>, bool> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_tuple(fn, dev, smem);
  const auto it = known.find(key);
  if (it != known.end()) return it->second;
  cudaLaunchAttribute at = cluster_attribute();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kCluster);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  // clusters of more than 8 CTAs are allowed per kernel
  int n = 0;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    n = 0;
  }
  return known[key] = n > 0;
}

template <bool TRANS, int NR, bool V16>
lu_status launch_one(cudaStream_t st, const Args& a) {
  size_t smem;
  void (*fn)(Args);
  if constexpr (NR <= 2) {
    // one group of two has the SMs for itself: a CTA each (n = 10007 409 us; 469
    // with two to an SM).  Two groups share them.
    smem = warp_smem_bytes(NR) + (NR == 2 && a.ngroups == 1 ? (size_t)8 * NR * BS * 8 : 0);
    fn = trsv_kernel<TRANS, NR, V16>;
    LUB_CUDA_TRY(set_smem_limit((const void*)fn, smem));
    Args b = a;
    if (a.cluster != 1) b.cluster = clusters_fit((const void*)fn, smem) ? kCluster : 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ceil_div(a.nblk, b.cluster) * b.cluster * a.ngroups));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1] = cluster_attribute();
    cfg.attrs = at;
    cfg.numAttrs = b.cluster > 1 ? 2 : 1;
    LUB_CUDA_TRY(launch_config(cfg, fn, b));
  } else {
    smem = mma_smem_bytes();
    fn = trsv_mma_kernel<TRANS, V16>;
    LUB_CUDA_TRY(set_smem_limit((const void*)fn, smem));
    LUB_CUDA_TRY(launch_dependent(fn, (unsigned)((int64_t)a.nblk * a.ngroups), kThreads, smem, st,
                                  a));
  }
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

template <bool TRANS, bool V16>
lu_status launch_nr(cudaStream_t st, const Args& a, int nr) {
  switch (nr) {
    case 8: return launch_one<TRANS, 8, V16>(st, a);
    case 2: return launch_one<TRANS, 2, V16>(st, a);
    default: return launch_one<TRANS, 1, V16>(st, a);
  }
}

}  // namespace trsv

// ---- residual r = b - A x (fp32 A, fp64 b, x, r) -------------------------
// Column chunks of kRC columns give partial dot products P[chunk][row]; a
// second pass adds them in chunk order, so the result does not depend on
// scheduling.  kRC also sizes the partial sums (n x ceil(n / kRC) doubles)
// and with them the compiled-in scratch of lu_refine_static_c
// (LU_REFINE_STATIC_SCRATCH_BYTES, checked against refine's layout at
// n = LU_REFINE_STATIC_MAX_N by a CPU test): a smaller kRC needs a larger
// array.
constexpr int kRC = 256;

__global__ void __launch_bounds__(kT)
residual_partial_kernel(int64_t n, const float* __restrict__ A, int64_t lda,
                        const double* __restrict__ x, double* __restrict__ P) {
  __shared__ double xs[kRC];
  dependency_wait();
  const int64_t c0 = (int64_t)blockIdx.y * kRC;
  const int cn = (int)((n - c0) < kRC ? (n - c0) : kRC);
  for (int k = threadIdx.x; k < cn; k += kT) xs[k] = x[c0 + k];
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x;
  if (i >= n) return;
  const float* col = A + i + c0 * lda;
  double acc = 0.0;
  // few CTAs at the sizes a single solve has: as many loads in flight per thread as
  // the kernel's registers hold
#pragma unroll 32
  for (int k = 0; k < cn; ++k) acc = fma((double)col[k * lda], xs[k], acc);
  P[(int64_t)blockIdx.y * n + i] = acc;
}

// r = b - sum_chunks P; also the row sums |A| once (rowsum != null) and the
// maxima needed for the backward error (atomicMax on non-negative doubles
// through their bit patterns).
__global__ void __launch_bounds__(kT)
residual_final_kernel(int64_t n, int nchunks, const double* __restrict__ P,
                      const double* __restrict__ b, const double* __restrict__ x,
                      double* __restrict__ r, unsigned long long* __restrict__ maxes) {
  dependency_wait();
  const int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x;
  double ri = 0.0, xi = 0.0, bi = 0.0;
  if (i < n) {
    double s = 0.0;
    for (int c = 0; c < nchunks; ++c) s += P[(int64_t)c * n + i];
    bi = b[i];
    ri = bi - s;
    r[i] = ri;
    xi = x[i];
  }
  // maxes[0] = max |r|, [1] = max |x|, [2] = max |b|
  double v[3] = {fabs(ri), fabs(xi), fabs(bi)};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    double m = v[q];
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&maxes[q], (unsigned long long)__double_as_longlong(m));
  }
}

// max_i sum_j |a_ij| (the infinity norm), same chunked scheme.
__global__ void __launch_bounds__(kT)
rowsum_partial_kernel(int64_t n, const float* __restrict__ A, int64_t lda,
                      double* __restrict__ P) {
  const int64_t c0 = (int64_t)blockIdx.y * kRC;
  const int cn = (int)((n - c0) < kRC ? (n - c0) : kRC);
  const int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x;
  if (i >= n) return;
  const float* col = A + i + c0 * lda;
  double acc = 0.0;
#pragma unroll 32
  for (int k = 0; k < cn; ++k) acc += fabs((double)col[k * lda]);
  P[(int64_t)blockIdx.y * n + i] = acc;
}

__global__ void __launch_bounds__(kT)
rowsum_final_kernel(int64_t n, int nchunks, const double* __restrict__ P,
                    unsigned long long* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x;
  double s = 0.0;
  if (i < n)
    for (int c = 0; c < nchunks; ++c) s += P[(int64_t)c * n + i];
  for (int o = 16; o > 0; o >>= 1) s = fmax(s, __shfl_xor_sync(0xffffffffu, s, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(s));
}

// X += D (n x nrhs, D dense): one launch for all columns.
__global__ void axpy_kernel(int64_t n, int64_t nrhs, const double* __restrict__ d,
                            double* __restrict__ x, int64_t ldx) {
  dependency_wait();
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n * nrhs) {
    const int64_t c = e / n;
    x[e - c * n + c * ldx] += d[e];
  }
}


// ---- residuals of several right-hand sides: R = B - op(A) X on the FP64
// matrix instruction.  A CTA computes RG x 16 rows of R for 8 NF right-hand
// sides; KS warps share each 16 rows, each taking its share RK of the KT values
// of the sum in a stage.  A goes straight from global memory to registers (fp32,
// converted there), one stage ahead; X is staged in shared memory by cp.async.
// The next stage's loads are spread over the steps of the current one: issued
// together after the barrier they held all warps' matrix instructions up.  The
// sums' order is fixed, so the result does not depend on scheduling.  maxes[3c ..
// 3c+2] receive max |r|, |x|, |b| of column c.
//
// Bound by the FP64 rate from 32 right-hand sides on (n = 8192, 64 columns: 4.3
// G multiply-adds, 0.24 ms at 64 per cycle and SM, 0.28 on the 128 SMs that 64
// rows per CTA fill), below that by reading A once, for which KS grows as NF
// shrinks: more, smaller CTAs in flight.  Eight column groups need 16 warps to
// cover the instruction's latency.  n = 8192, 64 columns on B200: 0.42 ms
// (transposed 0.37); 0.52 (0.47) with 8 warps and the loads together, 1.20 (1.86)
// with plain FMAs in groups of 8 columns.  n = 4096 with 32 rows per CTA: 0.139
// (0.128), against 0.263 (0.237) with 64.
// Bit pattern of |v|: ordered like the values, NaN above infinity.
__device__ __forceinline__ unsigned long long abs_bits(double v) {
  return (unsigned long long)__double_as_longlong(fabs(v));
}

constexpr int residual_kt(int nf) { return nf > 1 ? 512 / nf : 256; }  // values per stage

template <int NF, int KS, int RG>
constexpr size_t residual_smem() {
  const size_t x = (size_t)2 * 8 * NF * (residual_kt(NF) + 4);   // two stages of X
  const size_t p = (size_t)(KS - 1) * RG * 32 * 4 * NF;          // partial sums
  return (x > p ? x : p) * sizeof(double);
}

template <bool TRANS, int NF, int KS, int RG>
__global__ void __launch_bounds__(32 * KS * RG)
residual_multi_kernel(int64_t n, int64_t nrhs, const float* __restrict__ A, int64_t lda,
                      const double* __restrict__ B, int64_t ldb,
                      const double* __restrict__ X, int64_t ldx, double* __restrict__ R,
                      int64_t ldr, unsigned long long* __restrict__ maxes) {
  constexpr int NT = 32 * KS * RG, NC = 8 * NF, KT = residual_kt(NF);
  constexpr int RK = KT / KS, SK = RK / 4;  // values, steps of a warp per stage
  constexpr int S = KT + 4;   // column stride of the X stage: conflict-free fragment reads
  extern __shared__ __align__(16) double xs[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = warp % RG, kh = warp / RG, lr = lane >> 2, lk = lane & 3;
  const int64_t r0 = ((int64_t)blockIdx.x * RG + rg) * 16;
  const int64_t c0 = (int64_t)blockIdx.y * NC;
  const int nc = (int)((nrhs - c0) < NC ? (nrhs - c0) : NC);

  // op(A) rows r0 + lr and r0 + 8 + lr; rows past n repeat the last one (their
  // sums are dropped)
  const float* arow[2];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int64_t r = r0 + 8 * m + lr < n ? r0 + 8 * m + lr : n - 1;
    arow[m] = TRANS ? A + r * lda : A + r;
  }
  const bool vec = TRANS && ((reinterpret_cast<uintptr_t>(A) & 7) == 0) && (lda & 1) == 0;
  // entry s of a stage: this lane's k = 4 s + lk, or (transposed) 8 (s / 2) + 2
  // lk + (s & 1), so that a lane reads neighbours; k past n repeats the last
  // one against zeros of X
  auto load_a = [&](int s, int64_t kb, float (&v)[SK][2]) {
    if (!TRANS || s % 2 == 0)
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        if (TRANS) {
          const int64_t k = kb + 4 * s + 2 * lk;
          if (vec && k + 1 < n) {
            const float2 y = *reinterpret_cast<const float2*>(arow[m] + k);
            v[s][m] = y.x;
            v[s + 1][m] = y.y;
          } else {
            v[s][m] = arow[m][k < n ? k : n - 1];
            v[s + 1][m] = arow[m][k + 1 < n ? k + 1 : n - 1];
          }
        } else {
          const int64_t k = kb + 4 * s + lk;
          v[s][m] = arow[m][(k < n ? k : n - 1) * lda];
        }
      }
  };
  // this thread's entries of an X stage: value tid % KT of every (NT / KT)th
  // column, XE of them, an SKth per step
  constexpr int XC = NT / KT, XE = NC / XC;
  static_assert(NT % KT == 0 && XE % SK == 0, "X stage");
  const int xk = tid % KT, xc = tid / KT;
  const double* xsrc = X + xk + (c0 + xc) * ldx;
  const uint32_t xdst = static_cast<uint32_t>(__cvta_generic_to_shared(xs + xc * S + xk));
  auto load_x = [&](int s, int64_t k0, int buf) {
    const bool in = k0 + xk < n;
#pragma unroll
    for (int e = s * (XE / SK); e < (s + 1) * (XE / SK); ++e) {
      const bool ok = in && xc + e * XC < nc;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                       xdst + (uint32_t)((buf * NC + e * XC) * S * 8)),
                   "l"(ok ? xsrc + k0 + e * XC * ldx : X), "r"(ok ? 8 : 0)
                   : "memory");
    }
  };

  double acc[2][NF][2];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int f = 0; f < NF; ++f) acc[m][f][0] = acc[m][f][1] = 0.0;
  float cur[SK][2], nxt[SK][2];
#pragma unroll
  for (int s = 0; s < SK; ++s) {
    load_x(s, 0, 0);
    load_a(s, RK * kh, cur);
  }
  trsv::cp_commit();
  const int nst = (int)((n + KT - 1) / KT);
#pragma unroll 1
  for (int t = 0; t < nst; ++t) {
    const int64_t k1 = (int64_t)(t + 1) * KT;
    trsv::cp_wait<0>();
    __syncthreads();  // stage t is in, stage t - 1 read
    const double* x = xs + (t & 1) * NC * S + lr * S + RK * kh;
#pragma unroll
    for (int s = 0; s < SK; ++s) {
      const int k = TRANS ? 8 * (s >> 1) + 2 * lk + (s & 1) : 4 * s + lk;
      const double a0 = (double)cur[s][0], a1 = (double)cur[s][1];
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        const double b = x[8 * f * S + k];
        mma64(acc[0][f], a0, b);
        mma64(acc[1][f], a1, b);
      }
      if (t + 1 < nst) {  // the next stage, spread over the steps
        load_x(s, k1, (t + 1) & 1);
        load_a(s, k1 + RK * kh, nxt);
      }
    }
    trsv::cp_commit();
#pragma unroll
    for (int s = 0; s < SK; ++s) {
      cur[s][0] = nxt[s][0];
      cur[s][1] = nxt[s][1];
    }
  }
  // the KS partial sums of each row group, added in order
  if (KS > 1) {
    __syncthreads();
    double* part = xs + ((size_t)(kh > 0 ? kh - 1 : 0) * RG + rg) * 32 * 4 * NF;
    if (kh > 0) {
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int f = 0; f < NF; ++f)
#pragma unroll
          for (int h = 0; h < 2; ++h) part[((m * NF + f) * 2 + h) * 32 + lane] = acc[m][f][h];
    }
    __syncthreads();
    if (kh > 0) return;
    for (int q = 0; q < KS - 1; ++q) {
      const double* p = xs + ((size_t)q * RG + rg) * 32 * 4 * NF;
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int f = 0; f < NF; ++f)
#pragma unroll
          for (int h = 0; h < 2; ++h) acc[m][f][h] += p[((m * NF + f) * 2 + h) * 32 + lane];
    }
  }
#pragma unroll
  for (int f = 0; f < NF; ++f)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = 8 * f + 2 * lk + h;
      unsigned long long m[3] = {0ull, 0ull, 0ull};
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int64_t i = r0 + 8 * q + lr;
        if (i < n && c < nc) {
          const double b = B[i + (c0 + c) * ldb], x = X[i + (c0 + c) * ldx];
          const double r = b - acc[q][f][h];
          R[i + (c0 + c) * ldr] = r;
          m[0] = max(m[0], abs_bits(r));
          m[1] = max(m[1], abs_bits(x));
          m[2] = max(m[2], abs_bits(b));
        }
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) {
#pragma unroll
        for (int o = 16; o >= 4; o >>= 1)
          m[q] = max(m[q], __shfl_xor_sync(0xffffffffu, m[q], o));
        if (lr == 0 && c < nc) atomicMax(&maxes[3 * (c0 + c) + q], m[q]);
      }
    }
}

template <bool TRANS, int NF, int KS, int RG>
lu_status launch_residual_as(cudaStream_t st, int64_t n, int64_t nrhs, const float* A,
                             int64_t lda, const double* B, int64_t ldb, const double* X,
                             int64_t ldx, double* R, int64_t ldr, unsigned long long* maxes) {
  const int64_t groups = ceil_div(nrhs, 8 * NF);
  if (groups > 65535) return LU_ERR_INVALID_ARG;
  dim3 g((unsigned)ceil_div(n, 16 * RG), (unsigned)groups);
  constexpr size_t sm = residual_smem<NF, KS, RG>();
  LUB_CUDA_TRY(set_smem_limit((const void*)residual_multi_kernel<TRANS, NF, KS, RG>, sm));
  residual_multi_kernel<TRANS, NF, KS, RG><<<g, 32 * KS * RG, sm, st>>>(
      n, nrhs, A, lda, B, ldb, X, ldx, R, ldr, maxes);
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

// Right-hand sides per CTA: A is read once per group of columns.
template <bool TRANS>
lu_status launch_residual_nf(cudaStream_t st, int64_t n, int64_t nrhs, const float* A,
                             int64_t lda, const double* B, int64_t ldb, const double* X,
                             int64_t ldx, double* R, int64_t ldr, unsigned long long* maxes) {
  // 32 rows per CTA while that is one wave
  const bool few = n <= 32 * (int64_t)sm_count();
  const auto fn = nrhs <= 8    ? launch_residual_as<TRANS, 1, 8, 1>
                  : nrhs <= 16 ? launch_residual_as<TRANS, 2, 8, 1>
                  : nrhs <= 32 ? launch_residual_as<TRANS, 4, 4, 2>
                  : few        ? launch_residual_as<TRANS, 8, 8, 2>
                               : launch_residual_as<TRANS, 8, 4, 4>;
  return fn(st, n, nrhs, A, lda, B, ldb, X, ldx, R, ldr, maxes);
}
}  // namespace

size_t trsm_sync_bytes(int64_t nrhs) {
  (void)nrhs;
  return align_up((size_t)2 * trsv::kHeader * 4, 256);
}

size_t trsm_ws_bytes(int64_t n, int64_t nrhs) {
  return trsm_sync_bytes(nrhs) +
         align_up((size_t)(n < 0 ? 0 : n) * (size_t)(nrhs < 0 ? 0 : nrhs) * 8, 256);
}

namespace {
// One pass: op(T) X = B.
lu_status launch_pass(cudaStream_t st, int64_t n, const float* lu, int64_t ld, double* X,
                      int64_t ldx, double* B, int64_t ldb, int64_t nrhs, bool upper, bool trans,
                      unsigned* sync, bool mark, bool early, unsigned long long wait_ns,
                      int withhold, bool alone = false) {
  const int nr = trsv::group_width(nrhs);
  if (ceil_div(n, trsv::BS) * ceil_div(nrhs, nr) > 0x7fffffffll) return LU_ERR_INVALID_ARG;
  trsv::Args a;
  a.lu = lu;
  a.ld = ld;
  a.X = X;
  a.ldx = ldx;
  a.B = B;
  a.ldb = ldb;
  a.mark = mark;
  a.early = early;
  a.n = n;
  a.nrhs = nrhs;
  a.nblk = (int)ceil_div(n, trsv::BS);
  a.ngroups = (int)ceil_div(nrhs, nr);
  // op(T) is lower (forward substitution) for L and for U^T
  a.forward = upper == trans;
  a.unit = !upper;
  a.sync = sync;
  a.wait_ns = wait_ns > 0 ? wait_ns : trsv::kWaitNs;
  a.withhold = withhold;
  a.cluster = alone ? 1 : trsv::kCluster;
  const bool v16 = ((reinterpret_cast<uintptr_t>(lu) & 15) == 0) && (ld % 4 == 0);
  if (trans)
    return v16 ? trsv::launch_nr<true, true>(st, a, nr) : trsv::launch_nr<true, false>(st, a, nr);
  return v16 ? trsv::launch_nr<false, true>(st, a, nr) : trsv::launch_nr<false, false>(st, a, nr);
}

lu_status launch_prepare(cudaStream_t st, int64_t n, int64_t nrhs, double* X, int64_t ldx,
                         double* Y, unsigned* sync) {
  const int64_t blocks = ceil_div(n * nrhs, 256);
  LUB_CUDA_TRY(launch_dependent(trsv::trsv_prepare_kernel, (unsigned)blocks, 256, 0, st, n, nrhs,
                                X, ldx, Y, sync));
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}
}  // namespace

lu_status launch_trsm(cudaStream_t st, int64_t n, const float* lu, int64_t ld,
                      double* X, int64_t ldx, int64_t nrhs, bool upper,
                      bool trans, unsigned* sync, double* B,
                      unsigned long long wait_ns, int withhold, bool alone) {
  if (n <= 0 || nrhs <= 0) return LU_SUCCESS;
  if (!sync || !B) return LU_ERR_INVALID_ARG;
  LUB_TRY(launch_prepare(st, n, nrhs, X, ldx, B, sync));
  return launch_pass(st, n, lu, ld, X, ldx, B, n, nrhs, upper, trans, sync, false, false, wait_ns,
                     withhold, alone);
}

// The first pass takes its right-hand sides from X, leaves X pending and solves
// into Y; the second solves from Y into X.  So one preparing launch serves both,
// and the second pass may be placed while the first still runs: its set-up (the
// inverse of the diagonal block and its product with the neighbouring tile, ~14
// us) reads only the factors, which were complete before the first pass began
// (n = 10007: 297 -> 277.5 us; a preparing launch and a set-up per pass before).
lu_status launch_lu_solve(cudaStream_t st, int64_t n, const float* lu, int64_t ld,
                          double* X, int64_t ldx, int64_t nrhs, bool trans, unsigned* sync,
                          double* Y) {
  if (n <= 0 || nrhs <= 0) return LU_SUCCESS;
  if (!sync || !Y) return LU_ERR_INVALID_ARG;
  LUB_TRY(launch_prepare(st, n, nrhs, nullptr, 0, Y, sync));
  // L U x = b: L y = b, then U x = y; (L U)^T x = U^T L^T x = b: U^T y = b, then
  // L^T x = y
  LUB_TRY(launch_pass(st, n, lu, ld, Y, n, X, ldx, nrhs, trans, trans, sync, true, false, 0, -1));
  return launch_pass(st, n, lu, ld, X, ldx, Y, n, nrhs, !trans, trans, sync + trsv::kHeader, false,
                     true, 0, -1);
}

size_t residual_ws_bytes(int64_t n) {
  return align_up((size_t)ceil_div(n, kRC) * n * sizeof(double), 256) + 256;
}

lu_status launch_residual(cudaStream_t st, int64_t n, const float* A,
                          int64_t lda, const double* b, const double* x,
                          double* r, void* ws, unsigned long long* maxes) {
  const int nch = (int)ceil_div(n, kRC);
  double* P = static_cast<double*>(ws);
  LUB_CUDA_TRY(cudaMemsetAsync(maxes, 0, 3 * sizeof(unsigned long long), st));
  dim3 g((unsigned)ceil_div(n, kT), (unsigned)nch);
  LUB_CUDA_TRY(launch_dependent(residual_partial_kernel, g, kT, 0, st, n, A, lda, x, P));
  LUB_LAUNCH_CHECK();
  LUB_CUDA_TRY(launch_dependent(residual_final_kernel, (unsigned)ceil_div(n, kT), kT, 0, st, n, nch,
                                P, b, x, r, maxes));
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

lu_status launch_norm_inf(cudaStream_t st, int64_t n, const float* A,
                          int64_t lda, void* ws, unsigned long long* out) {
  const int nch = (int)ceil_div(n, kRC);
  double* P = static_cast<double*>(ws);
  LUB_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(unsigned long long), st));
  dim3 g((unsigned)ceil_div(n, kT), (unsigned)nch);
  rowsum_partial_kernel<<<g, kT, 0, st>>>(n, A, lda, P);
  LUB_LAUNCH_CHECK();
  rowsum_final_kernel<<<(unsigned)ceil_div(n, kT), kT, 0, st>>>(n, nch, P, out);
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

lu_status launch_residual_multi(cudaStream_t st, int64_t n, int64_t nrhs, const float* A,
                                int64_t lda, const double* B, int64_t ldb, const double* X,
                                int64_t ldx, double* R, int64_t ldr, bool trans,
                                unsigned long long* maxes) {
  if (n <= 0 || nrhs <= 0) return LU_SUCCESS;
  LUB_CUDA_TRY(cudaMemsetAsync(maxes, 0, (size_t)3 * nrhs * sizeof(unsigned long long), st));
  return trans ? launch_residual_nf<true>(st, n, nrhs, A, lda, B, ldb, X, ldx, R, ldr, maxes)
               : launch_residual_nf<false>(st, n, nrhs, A, lda, B, ldb, X, ldx, R, ldr, maxes);
}

lu_status launch_axpy(cudaStream_t st, int64_t n, int64_t nrhs, const double* d, double* x,
                      int64_t ldx) {
  if (n <= 0 || nrhs <= 0) return LU_SUCCESS;
  LUB_CUDA_TRY(launch_dependent(axpy_kernel, (unsigned)ceil_div(n * nrhs, 256), 256, 0, st, n, nrhs,
                                d, x, ldx));
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

}  // namespace lub
