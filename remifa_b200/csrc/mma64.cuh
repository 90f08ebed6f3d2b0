// FP64 matrix instruction (mma.sync m8n8k4): c += a b with fp64 products and
// sums.  Per lane: a = A[lane / 4][lane % 4], b = B[lane % 4][lane / 4], c = C[lane /
// 4][2 (lane % 4)] and the entry right of it.  One instruction does 256 fused
// multiply-adds at the FP64 pipe's rate (64 per cycle and SM) from two operand
// registers per lane, so operand loads and fp32 -> fp64 conversions (8 cycles
// each per warp) stay far below the arithmetic; the plain FMA form of the same
// sums is bound by them.
#pragma once

namespace lub {

__device__ __forceinline__ void mma64(double (&c)[2], double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

}  // namespace lub
