// Inner (ib = 8) elimination of a block column held in shared memory: the
// reference's per-element order (src/lu_nopiv.cu:105-326,
// src/lu_nopiv_inner_rl.hxx:104-196) -- the 8x8 diagonal tile (1/d correctly
// rounded, a multiply, fused a - l*u), the U columns right of it (forward
// substitution), the L rows below (row * 1/d and fused updates), then a rank-8
// update accumulated acc = fma(l, u, acc) and subtracted once.  Used by the
// batched LU (block columns of up to 512 rows).
//
// Per tile, two phases with a barrier after each:
//   eliminate: a thread per L row below the tile (two beyond NT rows) and per U
//              column right of it;
//   update   : warp 0 takes the next tile's own 8 x 8 block through the rank-8
//              update and factors it (one lane), while the other warps update
//              the rest in 4 x 8 blocks.
// What bounds it: that chain, per tile the elimination (~250 cycles), the
// block's update and one-lane factorization (~1000), two barriers -- and for
// blocks of more than ~250 rows the update's shared-memory traffic.  A warp that
// owned the tile's rows did its rows' whole update, the tile and the U strip in
// turn before: one CTA per SM, matrices of 64 / 256 / 360 rows took 19.8 / 140 /
// 291 us, now 11.3 / 112 / 250; 10000 matrices of 16 .. 511 rows 6.89 -> 5.81 ms.
#pragma once

#include "common.cuh"

namespace lub {
namespace rows {

__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  const float4 b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void store8(float* p, const float (&v)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}

// The tile at T (column-major, ld ldc), tw <= 8 columns, by one thread: the
// exact path of a partial tile, or of a pivot outside the fast range.
__device__ __noinline__ void tile_factor_exact(float* T, int ldc, int tw, float* inv, int* bad,
                                               int pbase) {
  float v[8][8];  // v[c][r]: tile column c
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    if (c < tw) {
      load8(T + c * ldc, v[c]);
    } else {
#pragma unroll
      for (int r = 0; r < 8; ++r) v[c][r] = 0.0f;
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (k < tw) {
      const float d = v[k][k];
      note_pivot(d, pbase + k, bad);
      const float iv = rcp_rn(d);  // correctly rounded 1/d
      inv[k] = iv;
#pragma unroll
      for (int r = k + 1; r < 8; ++r) v[k][r] = __fmul_rn(v[k][r], iv);
#pragma unroll
      for (int c = k + 1; c < 8; ++c)
#pragma unroll
        for (int r = k + 1; r < 8; ++r) v[c][r] = __fmaf_rn(-v[k][r], v[c][k], v[c][r]);
    }
  }
  // rows r >= tw of a partial tile lie below the matrix: never stored
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (c < tw && r < tw) T[r + c * ldc] = v[c][r];
}

// L rows at ra (and rb when TWO) of the tile's eight columns: fused updates
// with the tile's U part, then the 1/d multiply.  T: the tile, same ld.
template <bool TWO>
__device__ __forceinline__ void eliminate_rows(float* ra_p, float* rb_p, const float* T, int ldc,
                                               const float* inv) {
  float ra[8], rb[8], iv[8];
  load8(inv, iv);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    ra[c] = ra_p[c * ldc];
    rb[c] = TWO ? rb_p[c * ldc] : 0.0f;
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    float u[8];
    load8(T + c * ldc, u);  // u[k] = U[k][c]
#pragma unroll
    for (int k = 0; k < c; ++k) {
      ra[c] = __fmaf_rn(-ra[k], u[k], ra[c]);
      if (TWO) rb[c] = __fmaf_rn(-rb[k], u[k], rb[c]);
    }
    ra[c] = __fmul_rn(ra[c], iv[c]);
    if (TWO) rb[c] = __fmul_rn(rb[c], iv[c]);
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    ra_p[c * ldc] = ra[c];
    if (TWO) rb_p[c * ldc] = rb[c];
  }
}

// U column at p (the tile's eight rows): forward substitution.
__device__ __forceinline__ void eliminate_column(float* p, const float* T, int ldc) {
  float col[8];
  load8(p, col);
#pragma unroll
  for (int kk = 0; kk < 7; ++kk) {
    float l[8];
    load8(T + kk * ldc, l);  // tile column kk: l[r] = L[r][kk]
#pragma unroll
    for (int r = kk + 1; r < 8; ++r) col[r] = __fmaf_rn(-l[r], col[kk], col[r]);
  }
  store8(p, col);
}

// Rank-8 update of the 4 x 8 block at X: L rows at Lp (four rows, column k at
// Lp + k ldc), U columns at Up (eight rows, column j at Up + j ldc).
__device__ __forceinline__ void update_block(float* X, const float* Lp, const float* Up, int ldc) {
  float l[8][4];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float4 q = *reinterpret_cast<const float4*>(Lp + k * ldc);
    l[k][0] = q.x; l[k][1] = q.y; l[k][2] = q.z; l[k][3] = q.w;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float u[8], acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    load8(Up + j * ldc, u);
    float4 x = *reinterpret_cast<const float4*>(X + j * ldc);
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] = __fmaf_rn(l[k][i], u[k], acc[i]);
    x.x = __fsub_rn(x.x, acc[0]);
    x.y = __fsub_rn(x.y, acc[1]);
    x.z = __fsub_rn(x.z, acc[2]);
    x.w = __fsub_rn(x.w, acc[3]);
    *reinterpret_cast<float4*>(X + j * ldc) = x;
  }
}

// C: the block column's rows from global row c0 on at C + c0 (ldc a multiple of
// 4 with at least three rows of padding, 64 columns allocated: the update's
// blocks reach past row n and column wj).  inv: 8 floats (16-byte aligned) in
// shared memory; zero / non-finite pivots are reported to *bad as 1-based
// column pbase + k.  Ends with a CTA barrier on every path: the caller reads the
// block with another thread-to-row mapping.
template <int NT>
__device__ __forceinline__ void panel_block(float* C, int ldc, int n, int c0, int wj,
                                            float* inv, int* bad, int pbase) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int M = n - c0;
  const int nt = (wj + 7) >> 3;
  float* P = C + c0;
  if (tid == 0 && !(wj >= 8 && factor_tile8_fast(P, ldc, inv)))
    tile_factor_exact(P, ldc, min(8, wj), inv, bad, pbase);
  __syncthreads();
#pragma unroll 1
  for (int t = 0; t < nt; ++t) {
    const int t0 = 8 * t, t1 = t0 + 8;
    if (t1 > M) break;                       // a partial tile: nothing below it
    const float* T = P + t0 + t0 * ldc;
    {
      const int pa = t1 + tid, pb = pa + NT;
      if (pb < M) eliminate_rows<true>(P + pa + t0 * ldc, P + pb + t0 * ldc, T, ldc, inv);
      else if (pa < M) eliminate_rows<false>(P + pa + t0 * ldc, P + pa + t0 * ldc, T, ldc, inv);
      const int c = t1 + (NT - 1 - tid);     // the last warps: free of rows in small blocks
      if (c < wj) eliminate_column(P + t0 + c * ldc, T, ldc);
    }
    __syncthreads();
    if (t + 1 == nt) break;
    if (warp == 0) {
      const int tw = min(8, wj - t1);
      float* N = P + t1 + t1 * ldc;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = lane & 7, j = (lane >> 3) + 4 * h;
        const float* l = P + t1 + i + t0 * ldc;
        float u[8], acc = 0.0f;
        load8(P + t0 + (t1 + j) * ldc, u);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc = __fmaf_rn(l[k * ldc], u[k], acc);
        N[i + j * ldc] = __fsub_rn(N[i + j * ldc], acc);
      }
      __syncwarp();
      if (lane == 0 && !(tw == 8 && factor_tile8_fast(N, ldc, inv)))
        tile_factor_exact(N, ldc, tw, inv, bad, pbase + t1);
    } else {
      const int rg = (M - t1 + 3) >> 2, cg = (wj - t1 + 7) >> 3;
      for (int q = tid - 32; q < rg * cg; q += NT - 32) {
        const int jc = q / rg, ir = q - jc * rg;
        if (jc == 0 && ir < 2) continue;     // warp 0's
        const int r = t1 + 4 * ir, c = t1 + 8 * jc;
        update_block(P + r + c * ldc, P + r + t0 * ldc, P + t0 + c * ldc, ldc);
      }
    }
    __syncthreads();
  }
}

}  // namespace rows
}  // namespace lub
