// Panel kernels of the no-pivot LU (FP32 working precision).
//
// The reference factors each outer block column with an ib = 8 right-looking
// loop: per 8-column tile it factors the 8x8 diagonal tile (1/d then a
// multiply, fused rank-1 updates), eliminates the L rows below it and the U
// columns right of it, then applies a rank-8 GEMM update
// (src/lu_nopiv_inner_rl.hxx:104-196, src/lu_nopiv.cu:105-326).  Without
// pivoting the rows of L21 and the columns of U12 are independent of each
// other once the diagonal block is factored, so this file splits that loop
// into
//   diag_factor_kernel : the w x w diagonal block, one CTA, in registers (with
//                        the left-looking variant's Crout order as an option);
//   lupanel_kernel     : the L21 rows below the block and the U12 columns
//                        right of it, 32 or 64 rows or columns per CTA (one
//                        grid for both strips), optionally writing the K-major
//                        tensor-core operand copies of what it finishes;
//   lupanel_wide_kernel: the same for large launches beside tensor-core updates;
//   ref_panel_kernel   : remifa::lu_nopiv_panel<float,8> as a standalone
//                        entry point (lu_panel_c);
// each replaying, per element, the reference's exact operation sequence
// (the 8-column elimination, then rank-8 updates accumulated
// acc = fma(l, u, acc) over the 8 columns and subtracted once).
// The per-element order is fixed, so results match the CPU restatement bit
// for bit.
#include "common.cuh"
#include "kernels.cuh"

namespace lub {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ void ld8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  const float4 b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void st8(float* p, const float (&v)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}

// Factor the 8x8 tile whose rows live in lanes 0..7 of warp 0 (lane r holds
// row r in v[0..7]); tw <= 8 columns are factored.  Returns via v; writes
// 1/d into inv[].  Implements src/lu_nopiv.cu:123-171 for the tile.
__device__ __forceinline__ void factor_tile_warp(float (&v)[8], int tw,
                                                 float* inv, int64_t col0,
                                                 int* first_bad) {
  const int r = threadIdx.x & 31;
  const unsigned mask = 0xffffffffu;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (k < tw) {
      const float d = __shfl_sync(mask, v[k], k);
      const float iv = rcp_rn(d);  // correctly rounded 1/d
      if (r == 0) {
        inv[k] = iv;
        note_pivot(d, col0 + k, first_bad);
      }
      if (r > k && r < tw) v[k] = __fmul_rn(v[k], iv);
#pragma unroll
      for (int c = k + 1; c < 8; ++c) {
        const float ukc = __shfl_sync(mask, v[c], k);
        if (c < tw && r > k && r < 8) v[c] = __fmaf_rn(-v[k], ukc, v[c]);
      }
    }
  }
}

// The same tile factorization by a single thread, the tile held in
// registers (T points at its top-left element in shared memory, ld LD).
__device__ __noinline__ void factor_tile_thread(float* T, int LD, int tw,
                                                   float* inv, int64_t col0,
                                                   int* first_bad) {
  float v[8][8];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 8; ++c) v[r][c] = (r < tw && c < tw) ? T[r + c * LD] : 0.0f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (k < tw) {
      const float d = v[k][k];
      note_pivot(d, col0 + k, first_bad);
      const float iv = rcp_rn(d);  // correctly rounded 1/d
      inv[k] = iv;
#pragma unroll
      for (int r = k + 1; r < 8; ++r) v[r][k] = __fmul_rn(v[r][k], iv);
#pragma unroll
      for (int c = k + 1; c < 8; ++c)
#pragma unroll
        for (int r = k + 1; r < 8; ++r) v[r][c] = __fmaf_rn(-v[r][k], v[k][c], v[r][c]);
    }
  }
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (r < tw && c < tw) T[r + c * LD] = v[r][c];
}

// ---------------------------------------------------------------------------
// Diagonal block: w x w (w <= 128) at a (lda), factored in place by one CTA.
//
// The block lives in registers: 512 owner threads hold two 4 x 4 quads each
// (rows 4 tx, columns 4 ty and 64 + 4 ty), and one more warp factors the 8 x 8
// tiles.  Per tile t:
//   owners   : the rank-8 update of tile t to their quads (acc = fma chain
//              over the tile's 8 columns, one subtraction), then the rows and
//              columns of tile t+1 go to shared memory;
//   tile warp: the same update of tile t+1's own 8 x 8 block from a copy the
//              owners left one tile earlier, then its factorization by one
//              lane (src/lu_nopiv.cu:123-171);
//   barrier; one thread per row / column eliminates tile t+1's L rows and U
//   columns (src/lu_nopiv.cu:141-168, 304-316) into the strips the next
//   update reads, and stores them; barrier.
// CROUT (the left-looking order, src/lu_nopiv_inner_ll.hxx:197-370): the quads
// hold every element's running sum over the earlier tiles, carried along
// tile by tile and subtracted once, when the element's own tile comes.
// Either way each element gets the reference's operations in its order.
//
// What bounds it: the serial chain of w / 8 tiles, per tile the one-lane
// factorization (~730 cycles), its block's update (~280), one elimination
// (~220) and two barriers; for the first three tiles of a 128-wide block the
// rank-8 update of the owners.  w = 128 on B200, launches back to back: 20.7 us
// (CROUT 21); 22.7 with the block in shared memory, where every tile read
// and wrote the whole trailing block.
//
// The tile warp has an SM sub-partition to itself: the owners are the warps
// whose index is not a multiple of four (beside the owners its chain of
// dependent instructions took up to twice as long).  The other multiples of four
// do nothing but keep it so; with their registers the kernel fills an SM.
constexpr int kOwnerWarps = 16;
constexpr int kDiagLD = 132;           // leading dimension of CROUT's block
constexpr int kDiagThreads = 704;      // warps 0 .. 21: the tile warp, 16 owners

__device__ __forceinline__ void diag_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(32 * (kOwnerWarps + 1)) : "memory");
}

struct DiagSmem {
  float L[2][8 * 128];   // strips: column k of tile t's L rows, row r at [k * 128 + r]
  float U[2][8 * 128];   // row k of its U columns, column c at [k * 128 + c]
  float next[2][64];     // tile t+2's block after update t (CROUT: its sums)
  float tile[64];        // tile t+1, factored
  float inv[8];
};

__device__ __forceinline__ void ld4(const float* p, float (&v)[4]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}

// The tile warp: tile t+1's block and its factorization (see above).
template <bool CROUT>
__device__ __forceinline__ void diag_tile_warp(DiagSmem& sm, const float* D,
                                               float* __restrict__ a, int64_t lda, int w,
                                               int64_t col0, int* first_bad) {
  const int lane = threadIdx.x & 31;
  const int nt = (w + 7) / 8;
#pragma unroll 1
  for (int t = -1; t + 1 < nt; ++t) {
    const int c1 = 8 * (t + 1), tw = min(8, w - c1);
    const float* Ls = sm.L[t & 1] + c1;
    const float* Us = sm.U[t & 1] + c1;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = lane + 32 * h, i = e & 7, j = e >> 3;
      float x = sm.next[(t + 1) & 1][e], acc = CROUT ? x : 0.0f;
      if (CROUT) x = D[(c1 + j) * kDiagLD + c1 + i];
      if (t >= 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) acc = __fmaf_rn(Ls[k * 128 + i], Us[k * 128 + j], acc);
        x = __fsub_rn(x, acc);
      }
      sm.tile[e] = x;
    }
    __syncwarp();
    if (lane == 0 && !factor_tile8_fast(sm.tile, 8, sm.inv))
      factor_tile_thread(sm.tile, 8, tw, sm.inv, col0 + c1, first_bad);
    diag_sync();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = lane + 32 * h, i = e & 7, j = e >> 3;
      if (i < tw && j < tw) a[(c1 + i) + (c1 + j) * lda] = sm.tile[e];
    }
    diag_sync();
  }
}

// acc (+)= a tile's rank-8 product on a quad, strips at its first row / column.
__device__ __forceinline__ void quad_mul(const float* L, const float* U, float (&acc)[4][4]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    float l[4], u[4];
    ld4(L + k * 128, l);
    ld4(U + k * 128, u);
#pragma unroll
    for (int e = 0; e < 16; ++e)
      acc[e >> 2][e & 3] = __fmaf_rn(l[e >> 2], u[e & 3], acc[e >> 2][e & 3]);
  }
}
// The quad's elements v, or (CROUT) its running sums v: after tile t.
template <bool CROUT>
__device__ __forceinline__ void quad_update(const float* L, const float* U, float (&v)[4][4]) {
  if (CROUT) {
    quad_mul(L, U, v);
  } else {
    float acc[4][4];
#pragma unroll
    for (int e = 0; e < 16; ++e) acc[e >> 2][e & 3] = 0.0f;
    quad_mul(L, U, acc);
#pragma unroll
    for (int e = 0; e < 16; ++e)
      v[e >> 2][e & 3] = __fsub_rn(v[e >> 2][e & 3], acc[e >> 2][e & 3]);
  }
}
// The updated elements of a quad at (r, c): v, or (CROUT) the block's own
// elements in D less the sums v.
template <bool CROUT>
__device__ __forceinline__ void quad_value(const float (&v)[4][4], const float* D, int r, int c,
                                           float (&x)[4][4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (CROUT) ld4(D + (c + j) * kDiagLD + r, d);
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i][j] = CROUT ? __fsub_rn(d[i], v[i][j]) : v[i][j];
  }
}

// The 8 x 8 block of tile q (CROUT: its sums), from its owners' quads, for the
// tile warp.
__device__ __forceinline__ void put_block(DiagSmem& sm, int q, int nt, int tx, int ty,
                                          const float (&v)[2][4][4]) {
  const int c = 8 * q, dx = tx - (c >> 2), dy = ty - ((c & 63) >> 2);
  if (q < nt && (unsigned)dx <= 1u && (unsigned)dy <= 1u) {
    float* nx = sm.next[q & 1] + 4 * dy * 8 + 4 * dx;
    const bool hi = c >= 64;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) nx[j * 8 + i] = hi ? v[1][i][j] : v[0][i][j];
  }
}

// The owners (see above).
template <bool CROUT>
__device__ __forceinline__ void diag_owners(DiagSmem& sm, float* D, float* __restrict__ a,
                                            int64_t lda, int w, int warp) {
  const int lane = threadIdx.x & 31, tid = 32 * warp + lane;
  const int nt = (w + 7) / 8;
  const bool vec = ((reinterpret_cast<uintptr_t>(a) & 15) == 0) && (lda & 3) == 0;
  // 8 x 4 quads per warp: strip reads of 128 and 64 distinct bytes
  const int tx = (lane & 7) + 8 * (warp & 3), ty = (lane >> 3) + 4 * (warp >> 2);
  const int r = 4 * tx;

  float v[2][4][4];                 // quad b, element [row][column]
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int c = 64 * q + 4 * ty;
    if (vec && r + 4 <= w && c + 4 <= w) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 x = *reinterpret_cast<const float4*>(a + r + (c + j) * lda);
        v[q][0][j] = x.x; v[q][1][j] = x.y; v[q][2][j] = x.z; v[q][3][j] = x.w;
      }
    } else {  // past the edge: the identity
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          v[q][i][j] = (r + i < w && c + j < w) ? a[(r + i) + (c + j) * lda]
                                                : (r + i == c + j ? 1.0f : 0.0f);
    }
    if (CROUT) {  // the elements to D, the sums from zero
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        *reinterpret_cast<float4*>(D + (c + j) * kDiagLD + r) =
            make_float4(v[q][0][j], v[q][1][j], v[q][2][j], v[q][3][j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[q][i][j] = 0.0f;
      }
    }
  }
  put_block(sm, 0, nt, tx, ty, v);
  diag_sync();

#pragma unroll 1
  for (int t = -1; t + 1 < nt; ++t) {
    const int c1 = 8 * (t + 1);          // tile t+1
    const float* Ls = sm.L[t & 1];
    const float* Us = sm.U[t & 1];
    float* Ln = sm.L[(t + 1) & 1];
    float* Un = sm.U[(t + 1) & 1];
    // rank-8 update of tile t; a quad of finished rows or columns is left
    // out where the whole warp's are (elsewhere it takes values nobody
    // reads)
    if (t >= 0 && c1 <= 32 * (warp & 3) + 28) {
      if (c1 <= 16 * (warp >> 2) + 12) quad_update<CROUT>(Ls + r, Us + 4 * ty, v[0]);
      if (c1 <= 16 * (warp >> 2) + 76) quad_update<CROUT>(Ls + r, Us + 64 + 4 * ty, v[1]);
    }
    // tile t+1's rows below and columns right of its block
    const int dx = tx - (c1 >> 2), dy = ty - ((c1 & 63) >> 2);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int c = 64 * q + 4 * ty;
      const bool col = (c1 >> 6) == q && (unsigned)dy <= 1u && r >= c1 + 8;
      const bool row = (unsigned)dx <= 1u && c >= c1 + 8;
      if (col || row) {
        float x[4][4];
        quad_value<CROUT>(v[q], D, r, c, x);
        if (col) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(Ln + (4 * dy + j) * 128 + r) =
                make_float4(x[0][j], x[1][j], x[2][j], x[3][j]);
        }
        if (row) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<float4*>(Un + (4 * dx + i) * 128 + c) =
                make_float4(x[i][0], x[i][1], x[i][2], x[i][3]);
        }
      }
    }
    put_block(sm, t + 2, nt, tx, ty, v);
    diag_sync();
    // L rows (threads 0..127) and U columns (128..255) of tile t+1, in place
    const int q = tid & 127;
    if (tid < 256 && q >= c1 + 8 && q < w) {
      float x[8];
      if (tid < 128) {
#pragma unroll
        for (int c = 0; c < 8; ++c) x[c] = Ln[c * 128 + q];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          float u[8];
          ld8(sm.tile + c * 8, u);
#pragma unroll
          for (int k = 0; k < c; ++k) x[c] = __fmaf_rn(-x[k], u[k], x[c]);
          x[c] = __fmul_rn(x[c], sm.inv[c]);
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) Ln[c * 128 + q] = x[c];
#pragma unroll
        for (int c = 0; c < 8; ++c) a[q + (c1 + c) * lda] = x[c];
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = Un[i * 128 + q];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          float l[8];
          ld8(sm.tile + k * 8, l);
#pragma unroll
          for (int i = k + 1; i < 8; ++i) x[i] = __fmaf_rn(-l[i], x[k], x[i]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) Un[i * 128 + q] = x[i];
        float* d = a + c1 + q * lda;
        if (vec) {
          st8(d, x);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) d[i] = x[i];
        }
      }
    }
    diag_sync();
  }
}

// Two roles with the same barriers: one before the first tile (the tile warp
// has nothing to do before it), two per tile.
template <bool CROUT>
__global__ void __launch_bounds__(kDiagThreads, 1)
diag_factor_kernel(float* __restrict__ a, int64_t lda, int w, int64_t col0,
                   int* first_bad) {
  extern __shared__ __align__(16) float D[];   // CROUT: the block's elements
  __shared__ __align__(16) DiagSmem sm;
  const int warp = threadIdx.x >> 5;
  const int own = 3 * (warp >> 2) + (warp & 3) - 1;  // owner index of this warp
  dependency_wait();
  if (warp == 0) {
    diag_sync();
    diag_tile_warp<CROUT>(sm, D, a, lda, w, col0, first_bad);
  } else if ((warp & 3) != 0 && own < kOwnerWarps) {
    diag_owners<CROUT>(sm, D, a, lda, w, own);
  }
}

// ---------------------------------------------------------------------------
// L and U panels of one sub-panel, one launch.  `dg` is the factored w x w
// diagonal block (lda); M rows lie below it (L21), N columns right of it
// (U12).  A CTA owns ITEMS rows of L21 or columns of U12 ("items") of w
// positions each, and walks the 8-wide tiles t left to right:
//   (a) one thread per item eliminates tile t of its item: L rows
//       x_k *= 1/d_k, x_j -= x_k U[k][j] (src/lu_nopiv.cu:141-168); U
//       columns x_j -= L[j][k] x_k (src/lu_nopiv.cu:304-316), stores the
//       finished values and their low-precision operand copies;
//   (b) all threads apply the rank-8 update of tile t to the positions
//       right of it, acc = sum_k fma(x_k, F_k) over the tile's 8 columns
//       then one subtraction -- the reference's K = 8 GEMMs -- and hand the
//       positions of tile t+1 to (a).
// Each element receives the reference's operations in the reference's
// order.  Left-looking mode (src/lu_nopiv_inner_ll.hxx:225-300) keeps one
// running sum per element across the earlier tiles and subtracts it once,
// just before the element's tile is eliminated.
//
// The items live in registers: thread (tx, ty) holds items 4 tx .. 4 tx + 3 at
// positions 4 ty .. 4 ty + 3, so the update reads only the tile's item strip
// and the factor values from shared memory and writes nothing back, and the
// warps left of the current tile drop out.  8 threads per item, 32 items per CTA
// where that is at most one CTA per SM -- bound by the chain of w / 8 tiles; w =
// 128 on B200, launches back to back, 256 items of both strips 12.5 us, 16.6 with
// the items in shared memory -- and 64 in larger launches of the left-looking order
// or beside FP32 updates, bound by the FMA and shared-memory read rates (fp16
// storage, n = 8192: 4.33 ms, 4.48 with lupanel_wide_kernel and the running sums in
// shared memory; FP32 with nb = 128, n = 8192 14.4 and 15.6, n = 12000 40.9 and
// 46.6).  Larger launches beside tensor-core updates are lupanel_wide_kernel's.

// What one CTA works on: its items (row i: a + i, column i: a + i * lda) and
// the factor values that multiply item value k for position p, both as they
// lie in the diagonal block's columns: F[p * lf + k] = U[k][p] (L rows) or
// F[k * lf + p] = L[p][k] (U columns).
struct PanelStrip {
  float* a;
  int64_t lda;
  int w, nitems;
  const float* F;
  int lf;
  float* inv;    // reciprocals of the diagonal (L rows)
  float* X;      // tile t of the items, eliminated: [8][items + 4]
  float* P;      // tile t+1 of the items, updated
  void* pk[2];   // operand copies: item i's position p at pk[.][i * ldk + p]
  int64_t ldk[2];
  int64_t pk_lo[2];  // items below this one have no copy
  bool bf16;
};

template <bool IS_L, bool LEFT, int ITEMS>
__device__ __forceinline__ void lupanel_strip(const PanelStrip& s) {
  constexpr int XS = ITEMS + 4;     // stride of the tile strips X and P
  constexpr int WX = ITEMS / 32;    // warps across the items
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = (lane & 7) + 8 * (warp % WX), ty = (lane >> 3) + 4 * (warp / WX);
  const int w = s.w, nt = (w + 7) / 8;
  const int it = 4 * tx, p = 4 * ty;
  float v[4][4];                    // element [item][position]
  float sum[LEFT ? 4 : 1][4];
  if (((reinterpret_cast<uintptr_t>(s.a) & 15) == 0) && (s.lda & 3) == 0 &&
      it + 4 <= s.nitems && p + 4 <= w) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 x = *reinterpret_cast<const float4*>(
          IS_L ? s.a + it + (p + e) * s.lda : s.a + p + (it + e) * s.lda);
      const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int f = 0; f < 4; ++f) v[IS_L ? f : e][IS_L ? e : f] = xs[f];
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        v[i][j] = (it + i < s.nitems && p + j < w)
                      ? s.a[IS_L ? (it + i) + (p + j) * s.lda : (p + j) + (it + i) * s.lda]
                      : 0.0f;
  }
  if (LEFT) {
#pragma unroll
    for (int e = 0; e < 16; ++e) sum[LEFT ? e >> 2 : 0][e & 3] = 0.0f;
  }
  // tile 0 of the items
  if (ty < 2) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<float4*>(s.P + (p + j) * XS + it) =
          make_float4(v[0][j], v[1][j], v[2][j], v[3][j]);
  }
  cp_async_wait_all();
  __syncthreads();
  if (IS_L) {
    if (tid < ((w + 7) & ~7)) s.inv[tid] = (tid < w) ? rcp_rn(s.F[tid * s.lf + tid]) : 0.0f;
    __syncthreads();
  }
#pragma unroll 1
  for (int t = 0; t < nt; ++t) {
    const int t0 = 8 * t;
    if (tid < ITEMS) {
      const float* f = s.F + t0 * s.lf + t0;
      float x[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = s.P[k * XS + tid];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float fk[8];
        ld8(f + k * s.lf, fk);
        if (IS_L) {  // column k of U
#pragma unroll
          for (int m = 0; m < k; ++m) x[k] = __fmaf_rn(-x[m], fk[m], x[k]);
          x[k] = __fmul_rn(x[k], s.inv[t0 + k]);
        } else {     // column k of L
#pragma unroll
          for (int c = k + 1; c < 8; ++c) x[c] = __fmaf_rn(-fk[c], x[k], x[c]);
        }
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) s.X[k * XS + tid] = x[k];
    }
    __syncthreads();
    // rank-8 update of tile t to the positions right of it; where only part
    // of a warp's are, the others take values nobody reads
    const int p1 = t0 + 8;
    if (p1 < w && 16 * (warp / WX) + 12 >= p1) {
      const float* X = s.X + it;
      const float* F = IS_L ? s.F + t0 + p * s.lf : s.F + t0 * s.lf + p;
      float acc[4][4];
#pragma unroll
      for (int e = 0; e < 16; ++e) acc[e >> 2][e & 3] = 0.0f;
#pragma unroll
      for (int h = 0; h < 2; ++h) {   // columns 4 h .. 4 h + 3 of the tile
        float f[4][4];                // [column][position]
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float y[4];
          ld4(IS_L ? F + e * s.lf + 4 * h : F + (4 * h + e) * s.lf, y);
#pragma unroll
          for (int g = 0; g < 4; ++g) f[IS_L ? g : e][IS_L ? e : g] = y[g];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float x[4];
          ld4(X + (4 * h + k) * XS, x);
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float& y = LEFT ? sum[LEFT ? e >> 2 : 0][e & 3] : acc[e >> 2][e & 3];
            y = __fmaf_rn(x[e >> 2], f[k][e & 3], y);
          }
        }
      }
      if (!LEFT) {
#pragma unroll
        for (int e = 0; e < 16; ++e)
          v[e >> 2][e & 3] = __fsub_rn(v[e >> 2][e & 3], acc[e >> 2][e & 3]);
      }
      const int dy = ty - (p1 >> 2);
      if ((unsigned)dy <= 1u) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float y[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            y[i] = LEFT ? __fsub_rn(v[i][j], sum[LEFT ? i : 0][j]) : v[i][j];
          *reinterpret_cast<float4*>(s.P + (4 * dy + j) * XS + it) =
              make_float4(y[0], y[1], y[2], y[3]);
        }
      }
    }
    // the finished tile to global memory, one value per thread
    {
      const int ie = tid >> 3, e = tid & 7;
      const bool live = ie < s.nitems && t0 + e < w;
      const float y = s.X[e * XS + ie];
      if (IS_L) {
        const int i = tid % ITEMS, c = tid / ITEMS;
        if (i < s.nitems && t0 + c < w) s.a[i + (t0 + c) * s.lda] = s.X[c * XS + i];
      } else if (live) {
        s.a[(t0 + e) + ie * s.lda] = y;
      }
#pragma unroll
      for (int d = 0; d < 2; ++d)
        if (s.pk[d] && live && ie >= s.pk_lo[d])
          static_cast<uint16_t*>(s.pk[d])[ie * s.ldk[d] + t0 + e] =
              s.bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(y))
                     : __half_as_ushort(__float2half_rn(y));
    }
    __syncthreads();
  }
}

// F[c * lf + r] = dg[r + c * lda]: the upper triangle (and diagonal) of the
// w x w block, or the lower one; entries with r or c in [w, wp) zero, the
// rest of F is not read.
template <bool UPPER, int THREADS>
__device__ __forceinline__ void stage_triangle(float* F, int lf, const float* __restrict__ dg,
                                               int64_t lda, int w, int wp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (((reinterpret_cast<uintptr_t>(dg) & 15) == 0) && (lda & 3) == 0) {
    const int r = 4 * lane;
    for (int c = warp; c < w; c += THREADS / 32) {
      const float* src = dg + r + c * lda;
      float* dst = F + c * lf + r;
      if (UPPER ? r > c : r + 3 < c) continue;
      if (r + 4 <= w) {
        cp_async16(dst, src);
      } else {
        for (int e = 0; e < 4; ++e)
          if (r + e < w) cp_async4(dst + e, src + e);
      }
    }
  } else {
    for (int c = warp; c < w; c += THREADS / 32)
      for (int r = lane; r < w; r += 32)
        if (UPPER ? r <= c : r >= c) cp_async4(F + c * lf + r, dg + r + c * lda);
  }
  if (wp != w) {
    for (int i = threadIdx.x; i < wp * wp; i += THREADS) {
      const int r = i % wp, c = i / wp;
      if (r >= w || c >= w) F[c * lf + r] = 0.0f;
    }
  }
}

template <bool LEFT, int ITEMS>
__global__ void __launch_bounds__(8 * ITEMS, 2)
lupanel_kernel(float* __restrict__ dg, int64_t lda, int w, int64_t M,
               int64_t N, int nL, int64_t offL, int64_t offU, LuPack pk) {
  extern __shared__ __align__(16) float smem[];
  dependency_wait();
  const int wp = ((w + 7) / 8) * 8;  // padded width (zero filled)
  const int lf = wp + 4;
  // factor block; the update reads 128 columns whatever w is (the positions
  // past wp then take values nobody reads)
  float* F = smem;
  float* inv = F + (size_t)128 * lf;  // wp
  PanelStrip s;
  s.X = inv + wp;
  s.P = s.X + 8 * (ITEMS + 4);
  s.F = F;
  s.lf = lf;
  s.inv = inv;
  s.w = w;
  s.lda = lda;
  s.bf16 = pk.bf16 != 0;
  const bool is_l = (int)blockIdx.x < nL;
  const int64_t item0 = (int64_t)(is_l ? blockIdx.x : blockIdx.x - nL) * ITEMS;
  s.a = is_l ? dg + w + offL + item0 : dg + (w + offU + item0) * lda;
  s.nitems = (int)std::min<int64_t>(ITEMS, (is_l ? M : N) - item0);
  s.pk[0] = is_l ? pk.pa : pk.pb;
  s.pk[1] = is_l ? pk.pa2 : nullptr;
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    const int64_t base = (d == 1 ? pk.row02 : is_l ? pk.row0 : pk.col0) + item0;
    const int64_t ldk = d == 1 ? pk.ldk2 : pk.ldk;
    const int k0 = d == 1 ? pk.k02 : pk.k0;
    s.ldk[d] = ldk;
    s.pk_lo[d] = -base;  // rows above the copy's first one are skipped
    if (s.pk[d]) s.pk[d] = static_cast<uint16_t*>(s.pk[d]) + base * ldk + k0;
  }
  if (is_l) {
    stage_triangle<true, 8 * ITEMS>(F, lf, dg, lda, w, wp);
    lupanel_strip<true, LEFT, ITEMS>(s);
  } else {
    stage_triangle<false, 8 * ITEMS>(F, lf, dg, lda, w, wp);
    lupanel_strip<false, LEFT, ITEMS>(s);
  }
}

// ---------------------------------------------------------------------------
// The panels of large right-looking launches beside tensor-core updates: 64 items
// per CTA of 256 threads, in shared memory (S[item][pos]).  The item threads
// eliminate tile T+1 while the other warps still apply tile T's update (one barrier
// per tile), and the results leave at the end, whole rows of the operand copies at
// a time.  Alone it takes as long as the register variant with 64 items (27648
// items 39 us); beside the bulk update it is the faster one: whole factorizations
// on B200 with the register variant / this, n = 8192 e4m3 4.11 / 3.85 ms, n = 16384
// 9.88 / 9.2, n = 24576 23.0 / 21.7, n = 32768 46.8 / 44.2.
constexpr int kWideThreads = 256;
constexpr int kWideItems = 64;             // rows / columns per CTA
constexpr int kMicroI = 4, kMicroP = 8;    // register micro-tile

// Block copies between global memory and shared memory, by all threads
// of the CTA: warps take columns, lanes consecutive rows, so no index is
// divided by a runtime extent.  Both sides column-major unless noted.

// dst[r + c*ldd] = src[r + c*lds] asynchronously (complete with
// cp_async_wait_all); 16-byte copies when every column start is 16-byte
// aligned on both sides.
__device__ __forceinline__ void stage_cols_async(float* dst, int ldd, const float* src,
                                                 int64_t lds, int rows, int cols) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kNW = kWideThreads / 32;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0 &&
                   (lds & 3) == 0 && (ldd & 3) == 0 && (rows & 3) == 0;
  if (vec) {
    for (int c = warp; c < cols; c += kNW) {
      const float* s = src + (int64_t)c * lds;
      float* d = dst + c * ldd;
      for (int r = 4 * lane; r < rows; r += 128) cp_async16(d + r, s + r);
    }
  } else {
    for (int c = warp; c < cols; c += kNW) {
      const float* s = src + (int64_t)c * lds;
      float* d = dst + c * ldd;
      for (int r = lane; r < rows; r += 32) cp_async4(d + r, s + r);
    }
  }
}

// dst[r + c*ldd] = src[r + c*lds] (shared -> global), 16-byte stores when
// every column start is 16-byte aligned on both sides.
__device__ __forceinline__ void store_cols(float* dst, int64_t ldd, const float* src,
                                           int lds, int rows, int cols) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kNW = kWideThreads / 32;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0 &&
                   (ldd & 3) == 0 && (lds & 3) == 0 && (rows & 3) == 0;
  if (vec) {
    for (int c = warp; c < cols; c += kNW) {
      const float* s = src + c * lds;
      float* d = dst + (int64_t)c * ldd;
      for (int r = 4 * lane; r < rows; r += 128)
        *reinterpret_cast<float4*>(d + r) = *reinterpret_cast<const float4*>(s + r);
    }
  } else {
    for (int c = warp; c < cols; c += kNW) {
      const float* s = src + c * lds;
      float* d = dst + (int64_t)c * ldd;
      for (int r = lane; r < rows; r += 32) d[r] = s[r];
    }
  }
}

// Transposing load: dst[r*ldd + c] = src[r + c*lds] for r < rows, c < cols,
// and 0 for cols <= c < round4(cols).  Each thread reads four columns of
// one row (coalesced across the lanes) and writes them as one 16-byte
// shared store; dst 16-byte aligned, ldd % 4 == 0.
__device__ __forceinline__ void stage_rows_t(float* dst, int ldd, const float* src,
                                             int64_t lds, int rows, int cols) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kNW = kWideThreads / 32;
  const int nq = (cols + 3) >> 2;
  for (int q = warp; q < nq; q += kNW) {
    const int c0 = 4 * q;
    const float* s = src + (int64_t)c0 * lds;
#pragma unroll 2
    for (int r = lane; r < rows; r += 32) {
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = (c0 + e < cols) ? s[r + e * lds] : 0.0f;
      *reinterpret_cast<float4*>(dst + r * ldd + c0) = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
}

// Transposing store: dst[r + c*ldd] = src[r*lds + c] for r < rows,
// c < cols (16-byte shared reads; src 16-byte aligned, lds % 4 == 0).
__device__ __forceinline__ void store_rows_t(float* dst, int64_t ldd, const float* src,
                                             int lds, int rows, int cols) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kNW = kWideThreads / 32;
  const int nq = (cols + 3) >> 2;
  for (int q = warp; q < nq; q += kNW) {
    const int c0 = 4 * q;
    float* d = dst + (int64_t)c0 * ldd;
#pragma unroll 2
    for (int r = lane; r < rows; r += 32) {
      const float4 v4 = *reinterpret_cast<const float4*>(src + r * lds + c0);
      const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (c0 + e < cols) d[r + e * ldd] = v[e];
    }
  }
}

// Eliminate tile columns [t0, t0 + tw) of one item held in x[0..8):
// L rows x_c -= x_k U[k][c] (k < c), then x_c *= 1/d_c
// (src/lu_nopiv.cu:141-168); U columns x_c -= L[c][k] x_k
// (src/lu_nopiv.cu:304-316).
template <bool IS_L>
__device__ __forceinline__ void wide_elim(const float* F, int lf, const float* inv,
                                          int t0, int tw, float (&x)[8]) {
  if (tw == 8) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      float f[8];
      ld8(F + (t0 + c) * lf + t0, f);  // f[k] = U[k][c] (L) / L[c][k] (U)
      if (IS_L) {
#pragma unroll
        for (int k = 0; k < c; ++k) x[c] = __fmaf_rn(-x[k], f[k], x[c]);
        x[c] = __fmul_rn(x[c], inv[t0 + c]);
      } else {
#pragma unroll
        for (int k = 0; k < c; ++k) x[c] = __fmaf_rn(-f[k], x[k], x[c]);
      }
    }
  } else {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (c < tw) {
        const float* f = F + (t0 + c) * lf + t0;
        if (IS_L) {
#pragma unroll
          for (int k = 0; k < c; ++k) x[c] = __fmaf_rn(-x[k], f[k], x[c]);
          x[c] = __fmul_rn(x[c], inv[t0 + c]);
        } else {
#pragma unroll
          for (int k = 0; k < c; ++k) x[c] = __fmaf_rn(-f[k], x[k], x[c]);
        }
      }
    }
  }
}

// F[pos * lf + k]: the factor values that multiply item value k for
// position pos -- U[k][pos] (L blocks, F column-major) or L[pos][k] (U
// blocks, F row-major) -- so the 8 values of one tile are two float4.
// Per tile T, after one barrier:
//   warps 0-1 (one thread per item) apply tile T's rank-8 update to the
//     8 positions of tile T+1 and eliminate tile T+1 at once (look-ahead);
//   warps 2-7 apply tile T's rank-8 update to the positions right of tile
//     T+1 in register micro-tiles of 4 items x 8 positions (256 FMAs per 24
//     vector loads).
// Every element still receives acc = sum_k fma(x_k, F_k) over the tile's 8
// columns in k order, then one subtraction.
template <bool IS_L>
__device__ __forceinline__ void wide_strip(const float* F, int lf, const float* inv,
                                           float* S, int ls, int w) {
  constexpr int kIG = kWideItems / kMicroI;  // 16 item groups
  const int tid = threadIdx.x;
  const int nt = (w + 7) / 8;
  if (tid < kWideItems) {  // tile 0
    float* xr = S + tid * ls;
    float x[8];
    ld8(xr, x);
    wide_elim<IS_L>(F, lf, inv, 0, min(8, w), x);
    st8(xr, x);
  }
  __syncthreads();
  for (int T = 0; T + 1 < nt; ++T) {
    const int t0 = 8 * T, p0 = t0 + 8;
    if (tid < kWideItems) {
      float* xr = S + tid * ls;
      float xv[8], x[8], acc[8];
      ld8(xr + t0, xv);
      ld8(xr + p0, x);
#pragma unroll
      for (int b = 0; b < 8; ++b) acc[b] = 0.0f;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        float f[8];
        ld8(F + (p0 + b) * lf + t0, f);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[b] = __fmaf_rn(xv[k], f[k], acc[b]);
      }
#pragma unroll
      for (int b = 0; b < 8; ++b) x[b] = __fsub_rn(x[b], acc[b]);
      wide_elim<IS_L>(F, lf, inv, p0, min(8, w - p0), x);
      st8(xr + p0, x);
    } else {
      const int q0 = p0 + 8;
      const int npos = (w - q0 + kMicroP - 1) / kMicroP;
      for (int m = tid - kWideItems; m < npos * kIG; m += kWideThreads - kWideItems) {
        const int ig = m % kIG, pp = q0 + (m / kIG) * kMicroP;
        float xv[kMicroI][8];
#pragma unroll
        for (int a = 0; a < kMicroI; ++a) ld8(S + (ig + a * kIG) * ls + t0, xv[a]);
        float acc[kMicroI][kMicroP];
#pragma unroll
        for (int a = 0; a < kMicroI; ++a)
#pragma unroll
          for (int b = 0; b < kMicroP; ++b) acc[a][b] = 0.0f;
#pragma unroll
        for (int b = 0; b < kMicroP; ++b) {
          float f[8];
          ld8(F + (pp + b) * lf + t0, f);
#pragma unroll
          for (int k = 0; k < 8; ++k)
#pragma unroll
            for (int a = 0; a < kMicroI; ++a) acc[a][b] = __fmaf_rn(xv[a][k], f[k], acc[a][b]);
        }
#pragma unroll
        for (int a = 0; a < kMicroI; ++a) {
          float* row = S + (ig + a * kIG) * ls + pp;
          float c[8];
          ld8(row, c);
#pragma unroll
          for (int b = 0; b < kMicroP; ++b) c[b] = __fsub_rn(c[b], acc[a][b]);
          st8(row, c);
        }
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kWideThreads)
lupanel_wide_kernel(float* __restrict__ dg, int64_t lda, int w, int64_t M,
               int64_t N, int nL, int64_t offL, int64_t offU, LuPack pk) {
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x;
  dependency_wait();
  const int wp = ((w + 7) / 8) * 8;  // padded width (zero filled)
  const int ls = wp + 4;             // item stride (breaks bank aliasing)
  const int lf = wp + 4;             // leading dimension of F, same reason
  float* F = smem;                   // diagonal block, wp x wp
  float* inv = F + (size_t)wp * lf;  // wp
  float* S = inv + wp;               // kWideItems x ls
  const bool is_l = (int)blockIdx.x < nL;

  // Stage the factored diagonal block: column-major (F[c*lf + r]) for L
  // blocks, row-major (F[r*lf + c]) for U blocks; the padding rows and
  // columns [w, wp) are zero.
  if (is_l) stage_cols_async(F, lf, dg, lda, w, w);
  else stage_rows_t(F, lf, dg, lda, w, w);
  if (wp != w) {
    for (int idx = tid; idx < wp * wp; idx += kWideThreads) {
      const int r = idx % wp, c = idx / wp;
      if (r >= w || c >= (is_l ? w : ((w + 3) & ~3))) F[is_l ? c * lf + r : r * lf + c] = 0.0f;
    }
  }
  int64_t item0;
  float* A;
  int nitems;
  if (is_l) {
    item0 = (int64_t)blockIdx.x * kWideItems;
    A = dg + w + offL;               // first row of this launch's L rows
    nitems = (int)std::min<int64_t>(kWideItems, M - item0);
    // S[q*ls + c] = A[row item0 + q, column c]
    stage_rows_t(S, ls, A + item0, lda, nitems, w);
  } else {
    item0 = (int64_t)(blockIdx.x - nL) * kWideItems;
    A = dg + (w + offU) * lda;       // first column of this launch's U columns
    nitems = (int)std::min<int64_t>(kWideItems, N - item0);
    // S[q*ls + i] = A[row i, column item0 + q]
    stage_cols_async(S, ls, A + item0 * lda, lda, w, nitems);
  }
  // zero the positions [w, wp) of every item and the items past the end
  {
    const int wq = is_l ? ((w + 3) & ~3) : w;  // the L staging zeroed up to round4(w)
    const int padc = wp - wq;
    if (padc > 0)
      for (int idx = tid; idx < kWideItems * padc; idx += kWideThreads)
        S[(idx / padc) * ls + wq + idx % padc] = 0.0f;
    for (int idx = nitems * ls + tid; idx < kWideItems * ls; idx += kWideThreads) S[idx] = 0.0f;
  }
  cp_async_wait_all();
  __syncthreads();
  if (is_l) {
    for (int k = tid; k < wp; k += kWideThreads)
      inv[k] = (k < w) ? rcp_rn(F[k * lf + k]) : 0.0f;
    __syncthreads();
    wide_strip<true>(F, lf, inv, S, ls, w);
  } else {
    wide_strip<false>(F, lf, inv, S, ls, w);
  }
  if (is_l) store_rows_t(A + item0, lda, S, ls, nitems, w);
  else store_cols(A + item0 * lda, lda, S, ls, w, nitems);
  // the finished items as tensor-core operands: item qq's w values are
  // contiguous along K in both copies (consecutive threads, consecutive k)
  // destination 0: the tensor-core operand copy; 1: the second L copy
  for (int dsel = 0; dsel < 2; ++dsel) {
    void* dst = dsel == 0 ? (is_l ? pk.pa : pk.pb) : (is_l ? pk.pa2 : nullptr);
    if (!dst) continue;
    const int64_t lim = is_l ? M : N;
    const int64_t base = (dsel == 1 ? pk.row02 : is_l ? pk.row0 : pk.col0) + item0;
    const int64_t ldk = dsel == 1 ? pk.ldk2 : pk.ldk;
    const int k0 = dsel == 1 ? pk.k02 : pk.k0;
    if (w % 8 == 0 && ldk % 8 == 0 && k0 % 8 == 0) {
      // 8 values -> one 16-byte store
      const int w8 = w / 8;  // <= 16
      for (int idx = tid; idx < kWideItems * 16; idx += kWideThreads) {
        const int c8 = idx & 15, qq = idx >> 4;
        const int64_t pr = base + qq;
        if (c8 < w8 && item0 + qq < lim && pr >= 0) {
          float v[8];
          ld8(&S[qq * ls + 8 * c8], v);
          uint4 out;
          uint32_t* o32 = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (pk.bf16) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
              o32[e] = *reinterpret_cast<const uint32_t*>(&h);
            } else {
              const __half2 h = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
              o32[e] = *reinterpret_cast<const uint32_t*>(&h);
            }
          }
          *reinterpret_cast<uint4*>(static_cast<uint16_t*>(dst) + pr * ldk + k0 + 8 * c8) = out;
        }
      }
    } else {
      for (int idx = tid; idx < kWideItems * w; idx += kWideThreads) {
        const int c = idx % w, qq = idx / w;
        const int64_t pr = base + qq;
        if (item0 + qq < lim && pr >= 0) {
          const float v = S[qq * ls + c];
          const int64_t o = pr * ldk + k0 + c;
          if (pk.bf16) static_cast<__nv_bfloat16*>(dst)[o] = __float2bfloat16_rn(v);
          else static_cast<__half*>(dst)[o] = __float2half_rn(v);
        }
      }
    }
  }
  (void)nitems;
}

// ---------------------------------------------------------------------------
// Reference-compatible panel (remifa::lu_nopiv_panel<float,8>): n <= 8
// columns, the diagonal tile factored from the copy d by every CTA.
// blockIdx.y == 0: L rows [n, m); blockIdx.y == 1: U columns [n, m).
__global__ void __launch_bounds__(kThreads)
ref_panel_kernel(int64_t m, int n, const float* __restrict__ d, int64_t ldd,
                 float* __restrict__ l, int64_t ldl, float* __restrict__ u,
                 int64_t ldu, int* stat) {
  __shared__ float T[8][9];
  __shared__ float inv[8];
  const int tid = threadIdx.x;
  if (tid < 32) {
    float v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c)
      v[c] = (tid < n && c < n) ? d[tid + c * ldd] : 0.0f;
    factor_tile_warp(v, n, inv, 0, nullptr);
    if (tid < 8) {
#pragma unroll
      for (int c = 0; c < 8; ++c) T[tid][c] = v[c];
    }
  }
  __syncthreads();
  if (blockIdx.x == 0 && blockIdx.y == 0) {
    if (tid < 64) {
      const int r = tid % 8, c = tid / 8;
      if (r < n && c < n) l[r + c * ldl] = T[r][c];
    }
    if (tid == 0 && stat) *stat = n;
  }
  const int64_t q = (int64_t)blockIdx.x * kThreads + tid + n;
  if (q >= m) return;
  if (blockIdx.y == 0) {
    float row[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) row[c] = (c < n) ? l[q + c * ldl] : 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k < n) {
        row[k] = __fmul_rn(row[k], inv[k]);
#pragma unroll
        for (int c = k + 1; c < 8; ++c)
          if (c < n) row[c] = __fmaf_rn(-row[k], T[k][c], row[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (c < n) l[q + c * ldl] = row[c];
  } else {
    float col[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) col[r] = (r < n) ? u[r + q * ldu] : 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int r = k + 1; r < 8; ++r)
        if (k < n && r < n) col[r] = __fmaf_rn(-T[r][k], col[k], col[r]);
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < n) u[r + q * ldu] = col[r];
  }
}

// ---------------------------------------------------------------------------
// remifa::lu_nopiv_panel<half,8>: the same panel with fp16 storage and the
// reference's fp16 arithmetic (src/lu_nopiv.cu:105-326 instantiated for
// half, where nvcc contracts each a -= l * u into one fp16 fused multiply-add,
// which the reference's own outputs show): the pivot's reciprocal 1/d and
// the scaling l * (1/d) each rounded to fp16, and the update a - l * u
// rounded once.  The fp16 intrinsics below are the operations those
// expressions compile to.
__device__ __forceinline__ float h16_div1(float d) {
  return __half2float(__hdiv(__float2half(1.0f), __float2half(d)));
}
__device__ __forceinline__ float h16_mul(float a, float b) {
  return __half2float(__hmul(__float2half(a), __float2half(b)));
}
__device__ __forceinline__ float h16_sub_mul(float a, float l, float u) {
  return __half2float(__hfma(__hneg(__float2half(l)), __float2half(u), __float2half(a)));
}

__global__ void __launch_bounds__(kThreads)
ref_panel_f16_kernel(int64_t m, int n, const __half* __restrict__ d, int64_t ldd,
                     __half* __restrict__ l, int64_t ldl, __half* __restrict__ u,
                     int64_t ldu, int* stat) {
  __shared__ float T[8][9];
  __shared__ float inv[8];
  const int tid = threadIdx.x;
  if (tid < 64) {
    const int r = tid % 8, c = tid / 8;
    T[r][c] = (r < n && c < n) ? __half2float(d[r + c * ldd]) : 0.0f;
  }
  __syncthreads();
  if (tid == 0) {  // the 8 x 8 tile, right-looking, one thread (64 operations)
    for (int k = 0; k < n; ++k) {
      inv[k] = h16_div1(T[k][k]);
      for (int r = k + 1; r < n; ++r) T[r][k] = h16_mul(T[r][k], inv[k]);
      for (int c = k + 1; c < n; ++c)
        for (int r = k + 1; r < n; ++r) T[r][c] = h16_sub_mul(T[r][c], T[r][k], T[k][c]);
    }
  }
  __syncthreads();
  if (blockIdx.x == 0 && blockIdx.y == 0) {
    if (tid < 64) {
      const int r = tid % 8, c = tid / 8;
      if (r < n && c < n) l[r + c * ldl] = __float2half_rn(T[r][c]);
    }
    if (tid == 0 && stat) *stat = n;
  }
  const int64_t q = (int64_t)blockIdx.x * kThreads + tid + n;
  if (q >= m) return;
  if (blockIdx.y == 0) {
    float row[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) row[c] = (c < n) ? __half2float(l[q + c * ldl]) : 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k < n) {
        row[k] = h16_mul(row[k], inv[k]);
#pragma unroll
        for (int c = k + 1; c < 8; ++c)
          if (c < n) row[c] = h16_sub_mul(row[c], row[k], T[k][c]);
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (c < n) l[q + c * ldl] = __float2half_rn(row[c]);
  } else {
    float col[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) col[r] = (r < n) ? __half2float(u[r + q * ldu]) : 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int r = k + 1; r < 8; ++r)
        if (k < n && r < n) col[r] = h16_sub_mul(col[r], T[r][k], col[k]);
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < n) u[r + q * ldu] = __float2half_rn(col[r]);
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers

lu_status launch_diag_factor(cudaStream_t st, float* a, int64_t lda, int w,
                             int64_t col0, int* first_bad) {
  if (w <= 0 || w > 128) return LU_ERR_INVALID_ARG;
  LUB_CUDA_TRY(launch_dependent(diag_factor_kernel<false>, 1, kDiagThreads, 0, st, a, lda, w,
                                col0, first_bad));
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

lu_status launch_diag_crout(cudaStream_t st, float* a, int64_t lda, int w,
                            int64_t col0, int* first_bad) {
  if (w <= 0 || w > 128) return LU_ERR_INVALID_ARG;
  constexpr size_t sm = 128 * kDiagLD * sizeof(float);
  LUB_CUDA_TRY(set_smem_limit((const void*)diag_factor_kernel<true>, sm));
  LUB_CUDA_TRY(launch_dependent(diag_factor_kernel<true>, 1, kDiagThreads, sm, st, a, lda, w,
                                col0, first_bad));
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

template <bool LEFT, int ITEMS>
static lu_status launch_lupanel_items(cudaStream_t st, float* dg, int64_t lda, int w, int64_t M,
                                      int64_t N, int64_t offL, int64_t offU, const LuPack& pk) {
  const int64_t nL = ceil_div(M, ITEMS), nU = ceil_div(N, ITEMS);
  const size_t wp = (size_t)((w + 7) / 8) * 8;
  const size_t sm = (128 * (wp + 4) + wp + 2 * 8 * (ITEMS + 4)) * sizeof(float);
  LUB_CUDA_TRY(set_smem_limit((const void*)lupanel_kernel<LEFT, ITEMS>, sm));
  LUB_CUDA_TRY(launch_dependent(lupanel_kernel<LEFT, ITEMS>, (unsigned)(nL + nU), 8 * ITEMS, sm,
                                st, dg, lda, w, M, N, (int)nL, offL, offU, pk));
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

static lu_status launch_lupanel_wide(cudaStream_t st, float* dg, int64_t lda, int w, int64_t M,
                                     int64_t N, int64_t offL, int64_t offU, const LuPack& pk) {
  const int64_t nL = ceil_div(M, kWideItems), nU = ceil_div(N, kWideItems);
  const size_t wp = (size_t)((w + 7) / 8) * 8;
  const size_t sm = (wp * (wp + 4) + wp + (size_t)kWideItems * (wp + 4)) * sizeof(float);
  LUB_CUDA_TRY(set_smem_limit((const void*)lupanel_wide_kernel, sm));
  LUB_CUDA_TRY(launch_dependent(lupanel_wide_kernel, (unsigned)(nL + nU), kWideThreads, sm, st, dg,
                                lda, w, M, N, (int)nL, offL, offU, pk));
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

lu_status launch_lupanel(cudaStream_t st, float* dg, int64_t lda, int w,
                         int64_t M, int64_t N, bool left, int64_t offL, int64_t offU,
                         const LuPack* pack) {
  if (w <= 0 || w > 128) return LU_ERR_INVALID_ARG;
  M = std::max<int64_t>(M, 0);
  N = std::max<int64_t>(N, 0);
  if (M + N == 0) return LU_SUCCESS;
  const LuPack pk = pack ? *pack : LuPack{};
  // 32 items per CTA (a shorter chain per tile) while that is at most one CTA
  // per SM, else 64 (half the reads of the block)
  const bool small = ceil_div(M, 32) + ceil_div(N, 32) <= sm_count();
  const auto fn = left    ? (small ? launch_lupanel_items<true, 32> : launch_lupanel_items<true, 64>)
                  : small ? launch_lupanel_items<false, 32>
                  : pk.simt ? launch_lupanel_items<false, 64>
                            : launch_lupanel_wide;
  return fn(st, dg, lda, w, M, N, offL, offU, pk);
}

lu_status launch_ref_panel_f16(cudaStream_t st, int64_t m, int n, const __half* d,
                               int64_t ldd, __half* l, int64_t ldl, __half* u,
                               int64_t ldu, int* stat) {
  if (n <= 0 || n > 8 || m < n) return LU_ERR_INVALID_ARG;
  const int64_t rest = m - n;
  dim3 grid((unsigned)std::max<int64_t>(1, ceil_div(rest, kThreads)), 2);
  ref_panel_f16_kernel<<<grid, kThreads, 0, st>>>(m, n, d, ldd, l, ldl, u, ldu, stat);
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

lu_status launch_ref_panel(cudaStream_t st, int64_t m, int n, const float* d,
                           int64_t ldd, float* l, int64_t ldl, float* u,
                           int64_t ldu, int* stat) {
  if (n <= 0 || n > 8 || m < n) return LU_ERR_INVALID_ARG;
  const int64_t rest = m - n;
  dim3 grid((unsigned)std::max<int64_t>(1, ceil_div(rest, kThreads)), 2);
  ref_panel_kernel<<<grid, kThreads, 0, st>>>(m, n, d, ldd, l, ldl, u, ldu, stat);
  LUB_LAUNCH_CHECK();
  return LU_SUCCESS;
}

}  // namespace lub
