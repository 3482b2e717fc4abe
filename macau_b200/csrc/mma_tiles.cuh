// The FP64 warp matrix instruction.
#pragma once

namespace mg {

// D += A B with A 8 x 4 and B 4 x 8 in FP64.  Lane (g, t) = (lane / 4, lane % 4) holds A(g, t),
// B(t, g) and D(g, 2t), D(g, 2t + 1).
__device__ __forceinline__ void mma_f64(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

}  // namespace mg
