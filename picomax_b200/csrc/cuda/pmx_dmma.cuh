// FP64 tensor-core (mma.sync m8n8k4 .f64) helpers shared by the eigensolver and
// the FP64 contraction.
#pragma once

#include <cuda_runtime.h>

namespace pmx {
namespace dev {

// D += A B for one 8x8 (A 8x4 row-major, B 4x8 column-major) FP64 MMA.
// Fragments: a = A[lane/4][lane%4], b = B[lane%4][lane/4],
// d0/d1 = D[lane/4][2 (lane%4) + 0/1].
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// acc (re/im 8x8 block) += a * b in complex arithmetic, four real MMAs
__device__ __forceinline__ void cmma(double (&cr)[2], double (&ci)[2], double2 a, double2 b) {
  dmma(cr[0], cr[1], a.x, b.x);
  dmma(cr[0], cr[1], -a.y, b.y);
  dmma(ci[0], ci[1], a.x, b.y);
  dmma(ci[0], ci[1], a.y, b.x);
}

}  // namespace dev
}  // namespace pmx
