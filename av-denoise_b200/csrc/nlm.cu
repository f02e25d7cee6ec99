// NLMeans / NLMeans-HQ windowed denoise for sm_100a: one launch per output frame and plane group.
//
// What it computes (av-denoise-core/src/nlmeans/kernels/fused.rs:138-530, accumulate.rs:152-202,
// launch order dispatch/mod.rs:665-679): for every pixel p, every temporal pair pass k (q_k = -d+k,
// forward frame centre+q_k read at p+q, backward frame centre-q_k read at p-q, all q in the
// (2a+1)^2 window), then the single-frame pass (all q != 0), the patch distance
//   D(p, q) = scale * sum over the (2s+1)^2 patch of sum_c (centre - neighbour)^2
// gives the Welsch weight w = exp(-max(D - offset, 0) * h2), optionally times a per-block
// confidence; the passes accumulate sum w*I(neighbour), sum w and max w, and the finish is
//   out = (I * wref * max_w + sum wI) / (wref * max_w + sum w)   (I if the denominator <= 1e-30).
//
// How (B200 layout). A CTA owns a 32 x TY output tile and keeps every running sum in registers,
// so accumulators never leave the SM; each frame tile is read from HBM once per pass. The work
// is walked in two-lane steps: lane 0 and lane 1 are two (neighbour tile, offset) pairs that run
// side by side in packed f32x2 arithmetic (Blackwell's FADD2/FMUL2/FFMA2 issue two fp32 ops per
// slot). A temporal pass pairs the forward frame at +q with the backward frame at -q; the
// single-frame pass pairs two consecutive offsets. Per step:
//   phase 1 - row runs: each thread owns 8 consecutive pixels of one tile row plus the 2s halo
//             (its centre values stay in registers for the whole kernel), forms the squared
//             differences of both lanes and their 8 horizontal box sums with running sums, and
//             stores the lane pairs to a double-buffered row-sum tile;
//   phase 2 - column strips: each thread owns V pixels of one column, forms the vertical box
//             sums of both lanes, two MUFU ex2 give the weights, one FFMA2 accumulates w*I and
//             one FADD2 the weight sums.
// One barrier per step. The max weight is tracked as the minimum distance (exp is monotonic, so
// this is exact) when every lane shares one strength and no offset or confidence applies.
//
// The box sums run in a different order from the reference's direct row-major patch sum and
// the two lanes are summed at the end, so results can differ from the reference in the last
// bits; the parity tests bound the effect on the quantised output.

#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.h"
#include "nlm_tile.cuh"
#include "smem_limit.h"

namespace avd {

namespace {

using namespace nlm_tile_detail;

template <int C, int S, bool FAST>
__global__ void __launch_bounds__(kThreads, C == 1 && FAST ? 5 : 4) nlm_window_kernel(NlmLaunch a) {
    nlm_tile<C, S, FAST>(a, blockIdx.x, blockIdx.y);
}

// Persistent batch: every CTA takes tiles from one counter until the batch's tiles run out. Tile t
// belongs to the job j with prefix[j] <= t < prefix[j + 1]; jobs are whole launch descriptions.
template <int C, int S, bool FAST>
__global__ void __launch_bounds__(kThreads, C == 1 && FAST ? 5 : 4)
    nlm_batch_kernel(const NlmLaunch* __restrict__ jobs, const int* __restrict__ prefix, int njobs, int* counter) {
    using K = Cfg<C, S>;
    __shared__ int tile_s;
    const int total = prefix[njobs];
    for (;;) {
        __syncthreads();  // the previous tile is done with shared memory and `tile_s`
        if (threadIdx.x == 0) tile_s = atomicAdd(counter, 1);
        __syncthreads();
        const int t = tile_s;
        if (t >= total) return;
        int lo = 0, hi = njobs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (prefix[mid] <= t) lo = mid;
            else hi = mid - 1;
        }
        const NlmLaunch& a = jobs[lo];
        const int local = t - prefix[lo];
        const int tiles_x = (a.width + kTX - 1) / kTX;
        nlm_tile<C, S, FAST>(a, local % tiles_x, local / tiles_x);
    }
}

template <int C, int S, bool FAST>
cudaError_t launch_csf(const NlmLaunch& a, cudaStream_t stream) {
    using K = Cfg<C, S>;
    if (cudaError_t e = allow_smem<nlm_window_kernel<C, S, FAST>>(200 * 1024)) return e;
    dim3 grid((a.width + kTX - 1) / kTX, (a.height + K::TY - 1) / K::TY);
    size_t smem = nlm_smem_bytes<C, S>(a.search_radius, a.pairs, false);
    nlm_window_kernel<C, S, FAST><<<grid, kThreads, smem, stream>>>(a);
    return cudaGetLastError();
}

template <int C, int S>
cudaError_t dispatch_s(const NlmLaunch& a, cudaStream_t stream) {
    if (a.patch_radius == S) return a.fast ? launch_csf<C, S, true>(a, stream) : launch_csf<C, S, false>(a, stream);
    if constexpr (S < 16) {
        return dispatch_s<C, S + 1>(a, stream);
    } else {
        return cudaErrorInvalidValue;
    }
}

template <int C, int S, bool FAST>
cudaError_t batch_csf(const NlmLaunch* jobs, const int* prefix, int njobs, int* counter, int max_a, int max_pairs,
                      cudaStream_t stream) {
    if (cudaError_t err = allow_smem<nlm_batch_kernel<C, S, FAST>>(200 * 1024)) return err;
    const size_t smem = nlm_smem_bytes<C, S>(max_a, max_pairs, false);
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, nlm_batch_kernel<C, S, FAST>, kThreads, smem);
    if (e != cudaSuccess) return e;
    nlm_batch_kernel<C, S, FAST><<<sms * (per_sm > 0 ? per_sm : 1), kThreads, smem, stream>>>(jobs, prefix, njobs,
                                                                                              counter);
    return cudaGetLastError();
}

template <int C, int S>
cudaError_t batch_s(int s, bool fast, const NlmLaunch* jobs, const int* prefix, int njobs, int* counter, int max_a,
                    int max_pairs, cudaStream_t stream) {
    if (s == S)
        return fast ? batch_csf<C, S, true>(jobs, prefix, njobs, counter, max_a, max_pairs, stream)
                    : batch_csf<C, S, false>(jobs, prefix, njobs, counter, max_a, max_pairs, stream);
    if constexpr (S < 16) {
        return batch_s<C, S + 1>(s, fast, jobs, prefix, njobs, counter, max_a, max_pairs, stream);
    } else {
        return cudaErrorInvalidValue;
    }
}

}  // namespace

// Cfg<C, S>::TY: the tile height depends on the patch radius alone.
int nlm_tile_rows(int /*channels*/, int patch_radius) {
    const int v = (32 - 2 * patch_radius) / 4;
    return 4 * (v >= 1 ? v : 1);
}

int nlm_tile_cols() { return kTX; }

namespace {
int frame_tiles(const NlmLaunch& a) {
    const int rows = nlm_tile_rows(a.channels, a.patch_radius);
    return ((a.width + kTX - 1) / kTX) * ((a.height + rows - 1) / rows);
}
// The rules on tiles below are part of what a launch computes (the order of its sums), so they take the
// SMs of the one GPU this library is built for, not those of the device it finds.
constexpr int kSms = 148;
}  // namespace

// The tile depends on the sizes alone, never on a timing: the two tiles add up the offsets in different
// orders. Past kColsMaxPatch only the offset-pair tile is built. It also takes a single frame's small
// window on a small frame, where the column-pair tile's CTAs of 64 threads have too little work to share
// (a = 2, s = 4, luma: 13 us against 16 at 320x180, 17 and 17 at 640x360, 25 and 21 at 957x539; a = 3,
// s = 1, chroma: 20 and 22 at 256x144, 24 and 30 at 640x360, 46 and 44 at 957x539), but for integer
// outputs only: the exact finish gives those the reference's order, while float outputs have to equal a
// batch's, which runs the column-pair tile.
bool runs_cols(const NlmLaunch& a) {
    if (a.patch_radius > kColsMaxPatch || (a.channels != 1 && a.channels != 2)) return false;
    return !(a.fix_count && a.pairs == 0 && a.search_radius <= 3 && frame_tiles(a) <= 2 * kSms);
}

int nlm_window_variants(const NlmLaunch& a) { return !a.ref_ring && runs_cols(a) ? 3 : 1; }

// How many CTAs of a cluster share a column-pair tile. A frame's tiles alone leave SMs idle below a few
// CTAs each: from 3 to an SM on, one CTA per tile (957x539 chroma a = 5, 690 tiles: 121 us alone, 129
// shared by two); under that, the fewest that reach it, up to the 8 of a portable cluster (640x360, 300
// tiles, a = 7: 88 us alone, 69 by two, 80 by four; 203x117, 35 tiles, d = 1 a = 5: 118 alone, 70, 45, 35
// by eight), as long as the window's rows leave each two after the four that a share's staging is worth
// (a = 2, one frame: 5 rows, 15 us alone and 17 by two at 256x144; a = 3, 7 rows: 24, 21 by two, 20 by
// four). Long windows are shared up to 10 tiles to an SM, where the last wave of whole tiles costs more
// than staging a frame twice (d = 4 a = 4 s = 4: 1100x620 595 us alone, 503 by two; 1279x719 678 and 613;
// 1920x1080, 2,700 tiles, 1,345 and 1,296).
int cols_split(const NlmLaunch& a) {
    const int tiles = frame_tiles(a), rows = (2 * a.pairs + 1) * (2 * a.search_radius + 1);
    int split = 1;
    while (split < 8 && ((tiles * split < 3 * kSms && rows >= 2 * split + 4) ||
                         (tiles * split < 10 * kSms && rows >= 40 * split)))
        split *= 2;
    return split;
}

cudaError_t launch_nlm_batch(const NlmLaunch* jobs, const int* prefix, int njobs, int* counter, int channels,
                             int patch_radius, bool fast, int max_search_radius, int max_pairs, bool shares,
                             cudaStream_t stream) {
    if (patch_radius <= kColsMaxPatch && (channels == 1 || channels == 2))
        return fast ? launch_nlm_cols_batch_fast(jobs, prefix, njobs, counter, channels, patch_radius,
                                                 max_search_radius, shares, stream)
                    : launch_nlm_cols_batch_hq(jobs, prefix, njobs, counter, channels, patch_radius, max_search_radius,
                                               shares, stream);
    if (channels == 1)
        return batch_s<1, kColsMaxPatch + 1>(patch_radius, fast, jobs, prefix, njobs, counter, max_search_radius, max_pairs, stream);
    if (channels == 2)
        return batch_s<2, kColsMaxPatch + 1>(patch_radius, fast, jobs, prefix, njobs, counter, max_search_radius, max_pairs, stream);
    return cudaErrorInvalidValue;
}

cudaError_t launch_nlm(const NlmLaunch& a, cudaStream_t stream) {
    if (a.pairs < 0 || a.pairs > kMaxPairs || a.search_radius < 0 || a.search_radius > 8 || a.patch_radius < 0 ||
        a.patch_radius > 16)
        return cudaErrorInvalidValue;
    if (a.ref_ring) return launch_nlm_ref(a, stream);
    if (runs_cols(a)) {
        const int split = cols_split(a);
        return a.fast ? launch_nlm_cols_fast(a, split, stream) : launch_nlm_cols_hq(a, split, stream);
    }
    if (a.channels == 1) return dispatch_s<1, 0>(a, stream);
    if (a.channels == 2) return dispatch_s<2, 0>(a, stream);
    return cudaErrorInvalidValue;
}

}  // namespace avd
