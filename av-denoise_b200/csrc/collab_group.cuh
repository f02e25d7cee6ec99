// What the NL4D group search (collab_search.cu) and the collaborative filter (collab.cu) share: the
// patch grid, the 8-lane group and the member words.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.h"

namespace avd {
namespace collab_detail {

constexpr int P = 8;
constexpr int STEP = 4;
constexpr int MAX_K = 8;
constexpr int kGroups = 16;  // reference patches per CTA
constexpr int kThreads = kGroups * 8;
constexpr float kUnfilled = 3.0e38f;
constexpr float kSelfPin = -1.0e38f;
constexpr float kReciprocalFloor = 1e-12f;
constexpr float kAccumClamp = 5.0f;
constexpr float kWeightGain = 5.0f;
constexpr float kVarianceFloor = 1.0e-20f;
constexpr float kFrac1Sqrt2 = 0.70710678118654752440f;
constexpr int kCurveBins = 16;

struct GroupCtx {
    unsigned mask;  // this group's 8 lanes of the warp
    int sub;        // lane within the group
};

__device__ __forceinline__ float reduce8(const GroupCtx& g, float v) {
    v += __shfl_xor_sync(g.mask, v, 1);
    v += __shfl_xor_sync(g.mask, v, 2);
    v += __shfl_xor_sync(g.mask, v, 4);
    return v;
}

__device__ __forceinline__ uint32_t pack_pos_t(uint32_t x, uint32_t y, uint32_t t) {
    return (t << 26) | (y << 13) | x;
}

__device__ __forceinline__ uint32_t clamp_top_left(int v, uint32_t max_pos) {
    return v < 0 ? 0u : (v > static_cast<int>(max_pos) ? max_pos : static_cast<uint32_t>(v));
}

// Member words per reference patch: 8 packed positions, then k_use | use_grid << 8.
constexpr int kMemberWords = 9;

}  // namespace collab_detail
}  // namespace avd
