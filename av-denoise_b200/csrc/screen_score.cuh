// The tensor-core step of the NL4D screen (collab_search.cu) and how far a screened score may be from the
// exact sum it stands for.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace avd {
namespace screen {

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, float c0,
                                        float c1, float c2, float c3) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}

constexpr float kUlp = 5.9604645e-8f;  // 2^-24, the rounding of one f32 operation

// One step sums an accumulator and 16 exact products in an order and with an alignment that are not
// documented. Measured against integers: at most 7.4 ulp (2^-24) of the largest of the accumulator, the
// products and the result, on sums made to lose the most (accumulators of 2^20 to 2^30 over products just
// below what they keep), and nothing at all while the magnitudes add up to less than 2^24. That is what
// cutting every product at half an ulp of the largest term does: 16 halves and one rounding of the sum,
// 10 ulp at most. The test of this header repeats the measurement against these two constants.
constexpr float kStepError = 10.0f * kUlp;
constexpr float kExactBelow = 16777216.0f;

// The largest error of a score over patches of 64 C samples of magnitude R at most, whose partial sums
// stay within `reach` = 3 * 64 C R^2: 4 C steps, and the 23 additions (after 24 C of an eighth the size,
// each) of the running sums of squares that the first step starts from.
template <int C>
__host__ __device__ constexpr float score_error(float reach) {
    return reach < kExactBelow ? 0.0f : reach * (4 * C * kStepError + (23 + 24 * C) * (kUlp / 3.0f));
}

}  // namespace screen
}  // namespace avd
