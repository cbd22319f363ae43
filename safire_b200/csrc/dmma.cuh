// The FP64 tensor instruction, mma.sync m8n8k4: C (8 x 8) += A (8 x 4) B (4 x 8).  With lane =
// 4 g + t, a lane holds A[g][t], B[t][g] and C[g][2t], C[g][2t + 1].
#pragma once

#include "common.cuh"

namespace afqmc {

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// the complex product step: (cr, ci) += a * b
__device__ __forceinline__ void zmma(double (&cr)[2], double (&ci)[2], c128 a, c128 b) {
  dmma(cr[0], cr[1], a.x, b.x);
  dmma(ci[0], ci[1], a.x, b.y);
  dmma(cr[0], cr[1], -a.y, b.y);
  dmma(ci[0], ci[1], a.y, b.x);
}

}  // namespace afqmc
