// Warp matrix instructions of the row samplers' Grams (sample_mma.cu).
#pragma once
#include <cstdint>

namespace mg {

// D += A B with A 8 x 4 and B 4 x 8 in FP64.  Lane (g, t) = (lane / 4, lane % 4) holds A(g, t),
// B(t, g) and D(g, 2t), D(g, 2t + 1).
__device__ __forceinline__ void mma_f64(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// D += A B with A 16 x 16 and B 16 x 8 in BF16, FP32 accumulation.  A's rows 0-7 and 8-15 are
// given as two 8-row blocks lo, hi and B as one, each as two words: word 0 holds elements
// (2t, 2t + 1) of the lane's index g along the sum, word 1 elements (2t + 8, 2t + 9), which is
// A's row g (or 8 + g) and B's column g alike.  D: (g, 2t), (g, 2t + 1), (8 + g, 2t), (8 + g, 2t + 1).
__device__ __forceinline__ void mma_bf16_f32(float (&d)[4], const uint32_t (&lo)[2],
                                             const uint32_t (&hi)[2], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(lo[0]), "r"(hi[0]), "r"(lo[1]), "r"(hi[1]), "r"(b[0]), "r"(b[1]));
}

}  // namespace mg
