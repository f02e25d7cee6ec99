// What the two tiles of the NLMeans adjoint (nlm_adjoint.cu, nlm_adjoint_cols.cu) share.
#pragma once

#include <cuda_runtime.h>

#include "kernels.h"
#include "nlm_tile.cuh"

namespace avd {

struct GradArgs {
    NlmLaunch a;  // the window as a ring: centre slot d, pair k's frames k and 2d - k
    const float* grad_out;
    const float* records;
    float* grad_window;
    float* partials;  // one per tile
    float h2;
};

// The records and the gradients of patch radii up to kColsMaxPatch (nlm_adjoint_cols.cu).
cudaError_t launch_adjoint_cols(const NlmLaunch& a, const nlm_tile_detail::RecordOut& rec, const GradArgs& g,
                                cudaStream_t s);

}  // namespace avd
