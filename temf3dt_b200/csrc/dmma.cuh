// D (8 x 8) += A (8 x 4) B (4 x 8) in FP64 on the tensor cores, by one warp:
// lane 4 g + q holds A(g, q), B(q, g) and D(g, 2 q), D(g, 2 q + 1).  The four
// products are added to D one FMA after the other, in ascending column of A.
#pragma once

namespace temf {

__device__ __forceinline__ void dmma_8x8x4(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

}  // namespace temf
