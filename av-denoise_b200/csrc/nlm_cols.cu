// The column-pair NLMeans tile (nlm_cols.cuh) of plain NLMeans: one strength, no noise offset, no confidence.

#include "nlm_cols.cuh"

namespace avd {

cudaError_t launch_nlm_cols_fast(const NlmLaunch& a, int split, cudaStream_t stream) {
    return a.channels == 1 ? nlm_cols_detail::launch_cols_s<true, 1, 0>(a, split, stream)
                           : nlm_cols_detail::launch_cols_s<true, 2, 0>(a, split, stream);
}

cudaError_t launch_nlm_cols_batch_fast(const NlmLaunch* jobs, const int* prefix, int njobs, int* counter, int channels,
                                     int patch_radius, int search_radius, bool shares, cudaStream_t stream) {
    return channels == 1 ? nlm_cols_detail::launch_cols_batch_s<true, 1, 0>(jobs, prefix, njobs, counter, patch_radius,
                                                                          search_radius, shares, stream)
                         : nlm_cols_detail::launch_cols_batch_s<true, 2, 0>(jobs, prefix, njobs, counter, patch_radius,
                                                                          search_radius, shares, stream);
}

}  // namespace avd
