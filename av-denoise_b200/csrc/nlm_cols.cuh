// The forward NLMeans tile for patch radii up to kColsMaxS: what nlm.cu computes, with the two packed
// lanes of every f32x2 operation on two pixels 16 columns apart.
//
// What bounds it. Per (pixel, offset) the work is a squared difference, two running box sums, one
// exponential and three accumulations: about 11 FP32 operations (128 per clock and SM) and one MUFU
// (16 per clock and SM). The box sums cross threads through shared memory, and those bytes (128 per
// clock and SM) and the instructions around them are the bound. The tile of nlm_tile.cuh, whose lanes
// are two (frame, offset) pairs, moves 22 bytes and issues 18 instructions per (pixel, offset) at
// s = 2: 0.92 ms for a 1080p luma frame at d = 2, a = 5.
//
// How. A CTA of 64 threads owns 32 x TY pixels. Both lanes of a pair share the offset and the frame,
// so a staged sample pair (x, x + 16) is one 8-byte access, the centre values are pairs as they come,
// any number of offsets fills the lanes, and Q offsets side by side are taken per step:
//   phase 1 - a thread owns 8 consecutive pairs of one tile row plus the 2s halo (its centre pairs stay
//             in registers for the whole kernel), reads one row segment of 8 + 2s + Q - 1 sample pairs
//             for all Q offsets, and stores each offset's 8 horizontal box sums;
//   phase 2 - a thread owns V pairs of one column: vertical box sums, weights, accumulation.
// At s = 2 and Q = 3 that is 17.5 bytes and about 10 instructions per (pixel, offset): 0.725 ms for the
// frame above (the bytes alone take 0.60 ms at 128 per clock and SM); 1080p HQ d = 4 a = 4 s = 2
// 1.29 -> 1.02 ms, 960x540 chroma a = 5 0.113 -> 0.093 ms, the default s = 4, a = 2, d = 2 at 1080p
// 0.288 -> 0.271 ms. Small frames share a tile between the CTAs of a cluster (cols_split, nlm.cu).
//
// The order of every sum within a distance is the one of nlm_tile.cuh (runs from multiples of 8
// columns, strips of V rows). The samples are staged less a level (tile_level), which rounds those
// darker than it, so a distance may differ from that tile's in its last bits.

#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.h"
#include "nlm_tile.cuh"
#include "smem_limit.h"

namespace avd {
namespace nlm_cols_detail {

using nlm_tile_detail::add2;
using nlm_tile_detail::clampi;
using nlm_tile_detail::ex2_approx;
using nlm_tile_detail::f2;
using nlm_tile_detail::fma2;
using nlm_tile_detail::kLog2e;
using nlm_tile_detail::kRun;
using nlm_tile_detail::mul2;
using nlm_tile_detail::near_code_boundary;
using nlm_tile_detail::note_fix;
using nlm_tile_detail::sub2;

constexpr int kColsMaxS = kColsMaxPatch;
constexpr int kColsThreads = 64;
constexpr int kHalf = 16;      // columns between a pair's lanes
constexpr int kSmallA = 5, kMaxA = 8;
constexpr int kResidencies = 3;  // the tuner's choices of resident CTAs per SM: as many as fit, one or two fewer
constexpr int kHsPitch = 18;   // row sums: 9 x 16 bytes, an odd number, so 8 rows' stores miss each other

// Q offsets per step; BIG: search radii past 5.
template <int C, int S, int Q_, bool BIG>
struct Cols {
    static constexpr int V = nlm_tile_detail::Cfg<C, S>::V;
    static constexpr int TY = 4 * V;
    static constexpr int HR = TY + 2 * S;
    static constexpr int RUNW = kRun + 2 * S;
    // The sample tile's row pitch in pairs, fixed at the class's largest search radius so that every
    // access is an immediate offset from a few row pointers; odd, so 16 rows' reads of one column miss
    // each other.
    static constexpr int PITCH = (kHalf + 2 * S + 2 * (BIG ? kMaxA : kSmallA)) | 1;
    static constexpr int Q = Q_;
    __host__ __device__ static constexpr int rows(int a) { return HR + 2 * a; }
    // Pairs: the sample tile and the row sums; at the end of a shared tile, every thread's sums instead.
    __host__ __device__ static constexpr int tile_pairs(int a) { return rows(a) * PITCH * C; }
    static constexpr int HS_PAIRS = Q * HR * kHsPitch;
    static constexpr int SUM_PAIRS = (C + 2) * V * kColsThreads;
    // A CTA that takes the shares of a shared tile one after the other keeps their running sums as well.
    static constexpr int KEPT_PAIRS = (C + 1) * V * kColsThreads;
    __host__ __device__ static constexpr size_t smem_bytes(int a) {
        const int pairs = tile_pairs(a) + HS_PAIRS;
        return sizeof(float2) * static_cast<size_t>(pairs > SUM_PAIRS ? pairs : SUM_PAIRS);
    }
};

// A sample pair per channel.
template <int C>
struct Pair {
    float2 c[C];
};

template <int C>
__device__ __forceinline__ Pair<C> load_pair(const float2* p) {
    Pair<C> r;
    if (C == 1) {
        r.c[0] = p[0];
    } else {
        const float4 v = *reinterpret_cast<const float4*>(p);
        r.c[0] = f2(v.x, v.y);
        r.c[C - 1] = f2(v.z, v.w);
    }
    return r;
}

// The frame over the tile's window, coordinates clamped to the image (helpers.rs:20-32), as sample pairs
// less `mu` (per channel).
template <class K, int C>
__device__ __forceinline__ void load_cols(float2* tile, const float* __restrict__ frame, int x0, int y0, int rows,
                                          int cols, int W, int H, float2 mu) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = lane; c < cols; c += 32) {
        const int xa = clampi(x0 + c, 0, W - 1) * C, xb = clampi(x0 + c + kHalf, 0, W - 1) * C;
        float2* dst = tile + c * C;
#pragma unroll 8
        for (int r = warp; r < rows; r += kColsThreads / 32) {
            const float* row = frame + static_cast<int64_t>(clampi(y0 + r, 0, H - 1)) * W * C;
            if (C == 1) {
                dst[r * K::PITCH] = f2(__ldg(row + xa) - mu.x, __ldg(row + xb) - mu.x);
            } else {
                const float2 a = __ldg(reinterpret_cast<const float2*>(row + xa));
                const float2 b = __ldg(reinterpret_cast<const float2*>(row + xb));
                *reinterpret_cast<float4*>(dst + r * K::PITCH * C) = make_float4(a.x - mu.x, b.x - mu.x, a.y - mu.y, b.y - mu.y);
            }
        }
    }
}

// Per-thread state: the centre run, and per owned pair the running sums.
template <int C, class K>
struct ColsState {
    Pair<C> ctr[K::RUNW];
    float2 a[C][K::V];  // sum w * (I - level) per channel; with tracking, sum w * (I - the pixel's own)
    float2 ref[C][K::V];  // with tracking: the pixel's own value
    float2 ws[K::V];    // sum w
    float2 m[K::V];     // min distance (FAST) or max weight (HQ)
    int2 id[K::V];      // with tracking: the offset reaching m, the first in the forward's order
    float2 conf[K::V];
    const float2* run;           // tile: this thread's run at offset (0, 0)
    const float2* own;           // tile: this thread's first pixel pair at offset (0, 0)
    float2* hs_out;              // row sums: where the run's sums go
    const float2* hs_in;         // row sums: this thread's strip
};

// Keeps `v` and its offset's id where it beats the best so far, or ties it with an earlier id (frames
// are walked one after the other, the forward's order interleaves a pair's two).
template <bool LESS>
__device__ __forceinline__ void track(float& best, int& best_id, float v, int id) {
    if ((LESS ? v < best : v > best) || (v == best && id < best_id)) {
        best = v;
        best_id = id;
    }
}

// One step: the N offsets (dx .. dx + N - 1, dy), `at` = dy * pitch + dx in pairs. TRACK: the ids
// (id + q id_step) of the best are kept (the adjoint's records).
template <int C, int S, bool FAST, bool CONF, bool TRACK, class K, int N>
__device__ __forceinline__ void cols_step(ColsState<C, K>& z, int at, float2 kk, float2 scale2, const float (&off)[3],
                                          int id, int id_step) {
    constexpr int V = K::V, RUNW = K::RUNW;
    {
        const float2* n = z.run + at * C;
        float2 d[N][RUNW], run[N];
        float2 h[N][2];
#pragma unroll
        for (int i = 0; i < RUNW + N - 1; ++i) {
            const Pair<C> s = load_pair<C>(n + i * C);
#pragma unroll
            for (int q = 0; q < N; ++q) {
                const int k = i - q;  // the pair of the run this sample meets at offset q
                if (k < 0 || k >= RUNW) continue;
                const float2 du = sub2(z.ctr[k].c[0], s.c[0]);
                if (C == 1) {
                    d[q][k] = mul2(du, du);
                } else {
                    const float2 dv = sub2(z.ctr[k].c[C - 1], s.c[C - 1]);
                    d[q][k] = fma2(dv, dv, mul2(du, du));
                }
                if (k == 0) run[q] = d[q][0];
                else if (k <= 2 * S) run[q] = add2(run[q], d[q][k]);
                else run[q] = sub2(add2(run[q], d[q][k]), d[q][k - 2 * S - 1]);
                const int j = k - 2 * S;  // the run's sum complete now
                if (j >= 0) {
                    h[q][j & 1] = run[q];
                    if (j & 1)
                        *reinterpret_cast<float4*>(z.hs_out + q * (K::HR * kHsPitch) + j - 1) =
                            make_float4(h[q][0].x, h[q][0].y, h[q][1].x, h[q][1].y);
                }
            }
        }
    }
    __syncthreads();
    const float2* p = z.own + at * C;
#pragma unroll
    for (int q = 0; q < N; ++q) {
        const float2* hs = z.hs_in + q * (K::HR * kHsPitch);
        float2 hv[V + 2 * S];
#pragma unroll
        for (int i = 0; i < V + 2 * S; ++i) hv[i] = hs[i * kHsPitch];
        float2 dist = hv[0];
#pragma unroll
        for (int i = 1; i <= 2 * S; ++i) dist = add2(dist, hv[i]);
#pragma unroll
        for (int k = 0; k < V; ++k) {
            if (k > 0) dist = sub2(add2(dist, hv[k + 2 * S]), hv[k - 1]);
            float2 w;
            if (FAST) {
                const float2 e = mul2(dist, kk);
                w = f2(ex2_approx(e.x), ex2_approx(e.y));
                if (TRACK) {
                    track<true>(z.m[k].x, z.id[k].x, dist.x, id + q * id_step);
                    track<true>(z.m[k].y, z.id[k].y, dist.y, id + q * id_step);
                } else {
                    z.m[k] = f2(fminf(z.m[k].x, dist.x), fminf(z.m[k].y, dist.y));
                }
            } else {
                float2 x = fma2(dist, scale2, f2(-off[q], -off[q]));
                x = f2(fmaxf(x.x, 0.0f), fmaxf(x.y, 0.0f));
                const float2 e = mul2(x, kk);
                w = f2(ex2_approx(e.x), ex2_approx(e.y));
                if (CONF) w = mul2(w, z.conf[k]);
                if (TRACK) {
                    track<false>(z.m[k].x, z.id[k].x, w.x, id + q * id_step);
                    track<false>(z.m[k].y, z.id[k].y, w.y, id + q * id_step);
                } else {
                    z.m[k] = f2(fmaxf(z.m[k].x, w.x), fmaxf(z.m[k].y, w.y));
                }
            }
            const Pair<C> v = load_pair<C>(p + (k * K::PITCH + q) * C);
#pragma unroll
            for (int c = 0; c < C; ++c)
                z.a[c][k] = fma2(TRACK ? sub2(v.c[c], z.ref[c][k]) : v.c[c], w, z.a[c][k]);
            z.ws[k] = add2(z.ws[k], w);
        }
    }
    __syncthreads();
}

// Rows dy0 .. dy1 - 1 of one frame's window: `skip_centre` leaves out the offset 0 (the single-frame
// pass, whose noise offsets come from the table `lut`).
template <int C, int S, bool FAST, bool CONF, bool TRACK, class K>
__device__ __forceinline__ void cols_frame(ColsState<C, K>& z, int A, int dy0, int dy1, bool skip_centre,
                                           const float* __restrict__ lut, float off_pair, float2 kk, float2 scale2,
                                           int id_first, int id_step) {
    const int side = 2 * A + 1;
    for (int dy = dy0; dy < dy1; ++dy) {
        int dx = -A;
        while (dx <= A) {
            int left = A - dx + 1;  // offsets to go before the row's end or the left-out centre
            if (skip_centre && dy == 0 && dx <= 0) left = -dx;
            if (left == 0) {
                dx = 1;
                continue;
            }
            const int n = left == 4 || (K::Q == 2 && left > 2) ? 2 : min(left, K::Q);
            float off[3] = {off_pair, off_pair, off_pair};
            if (!FAST && skip_centre) {
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    off[q] = lut && q < n ? __ldg(lut + (dy + A) * side + dx + A + q) : 0.0f;
            }
            const int at = dy * K::PITCH + dx;
            const int o = (dy + A) * side + dx + A;
            const int id = TRACK ? id_first + id_step * (skip_centre && o > A * side + A ? o - 1 : o) : 0;
            if (K::Q == 3 && n == 3) cols_step<C, S, FAST, CONF, TRACK, K, K::Q>(z, at, kk, scale2, off, id, id_step);
            else if (n == 2) cols_step<C, S, FAST, CONF, TRACK, K, 2>(z, at, kk, scale2, off, id, id_step);
            else cols_step<C, S, FAST, CONF, TRACK, K, 1>(z, at, kk, scale2, off, id, id_step);
            dx += n;
        }
    }
}

// The level samples are staged relative to, per channel: just under the darkest pixel the tile owns. The
// weighted sum is then of smaller values and keeps bits that one running sum over several hundred offsets
// would lose, dark pixels' included. The level is a multiple of 1/256, so the subtraction is exact for
// samples at or above it. Darker ones (beside the tile, or in another frame) are rounded by up to 2^-25 =
// 3e-8, a sixtieth of the exact finish's band; the band's measurement (kernels.h) has hard edges in it.
// `two` is shared memory for two pairs; every thread calls it.
template <int C, class K>
__device__ __forceinline__ float2 tile_level(const float* __restrict__ centre, int X0, int Y0, int W, int H, float2* two) {
    const int tid = threadIdx.x, col = tid & (kHalf - 1), y0 = (tid / kHalf) * K::V;
    float2 mu = f2(1.0f, 1.0f);
#pragma unroll
    for (int k = 0; k < K::V; ++k)
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            const float* own = centre + (static_cast<int64_t>(min(Y0 + y0 + k, H - 1)) * W +
                                         min(X0 + col + l * kHalf, W - 1)) * C;
            mu = f2(fminf(mu.x, __ldg(own)), C == 2 ? fminf(mu.y, __ldg(own + 1)) : 0.0f);
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        mu = f2(fminf(mu.x, __shfl_xor_sync(0xffffffffu, mu.x, o)), fminf(mu.y, __shfl_xor_sync(0xffffffffu, mu.y, o)));
    if ((tid & 31) == 0) two[tid >> 5] = mu;
    __syncthreads();
    mu = f2(fminf(two[0].x, two[1].x), fminf(two[0].y, two[1].y));
    __syncthreads();
    return f2(mu.x > 0.0f && mu.x < 1.0f ? floorf(mu.x * 256.0f) * (1.0f / 256.0f) : 0.0f,
              mu.y > 0.0f && mu.y < 1.0f ? floorf(mu.y * 256.0f) * (1.0f / 256.0f) : 0.0f);
}

// A share's sums into the kept ones (`first`: they start them), the thread's own sums cleared.
template <int C, class K>
__device__ __forceinline__ void keep_sums(ColsState<C, K>& z, float2* kept, bool first) {
#pragma unroll
    for (int k = 0; k < K::V; ++k) {
#pragma unroll
        for (int c = 0; c <= C; ++c) {
            float2& own = c < C ? z.a[c < C ? c : 0][k] : z.ws[k];
            float2& sum = kept[(c * K::V + k) * kColsThreads];
            sum = first ? own : add2(sum, own);
            own = f2(0.0f, 0.0f);
        }
    }
}

extern __shared__ __align__(16) float2 cols_smem[];

// One output tile (tile_x, tile_y) of the launch `a`; the whole CTA calls it. With `split` > 1 the
// window's rows (frame by frame) are cut into that many shares, whose sums are added in order. CLUSTER:
// the CTAs of a cluster take one share each (`rank`) and CTA 0 adds and finishes; otherwise this CTA
// takes them all in turn, with the same sums (a batch's tile equals the frame denoised alone).
// REC: the adjoint's records instead of the output.
template <int C, int S, bool FAST, class K, bool CLUSTER, bool REC = false>
__device__ __forceinline__ void cols_tile(const NlmLaunch& a, int tile_x, int tile_y, int rank, int split,
                                          const nlm_tile_detail::RecordOut* rec = nullptr) {
    constexpr int V = K::V;
    const int A = a.search_radius, W = a.width, H = a.height;
    const int X0 = tile_x * 2 * kHalf, Y0 = tile_y * K::TY;
    const int tid = threadIdx.x, lane = tid & 31;
    const int col = tid & (kHalf - 1), y0 = (tid / kHalf) * V;
    // Phase 1: 16 rows by 2 runs per warp; a row past the last repeats it.
    const int run_row = min((tid >> 5) * 16 + (lane & 15), K::HR - 1), run_x = (lane >> 4) * kRun;

    float2* tile = cols_smem;
    float2* hs = tile + K::tile_pairs(A);
    ColsState<C, K> z;
    z.run = tile + ((run_row + A) * K::PITCH + run_x + A) * C;
    z.own = tile + ((y0 + S + A) * K::PITCH + col + S + A) * C;
    z.hs_out = hs + run_row * kHsPitch + run_x;
    z.hs_in = hs + y0 * kHsPitch + col;

    const float h2 = __ldg(a.derived + a.h2_word);
    const float off_pair = FAST ? 0.0f : __ldg(a.derived + a.offset_word);
    const float scale = C == 1 ? 3.0f : 1.5f;
    const float neg = -h2 * kLog2e;
    const float2 kk = FAST ? f2(scale * neg, scale * neg) : f2(neg, neg);
    const float2 scale2 = f2(scale, scale);
    const bool use_conf = !FAST && a.conf != nullptr;

#pragma unroll
    for (int k = 0; k < V; ++k) {
        z.ws[k] = f2(0.0f, 0.0f);
        z.m[k] = FAST ? f2(__int_as_float(0x7f800000), __int_as_float(0x7f800000)) : f2(0.0f, 0.0f);
        z.conf[k] = f2(1.0f, 1.0f);
        z.id[k] = make_int2(-1, -1);
#pragma unroll
        for (int c = 0; c < C; ++c) z.a[c][k] = f2(0.0f, 0.0f);
    }

    const float* centre = a.ring + a.slot_centre * a.frame_elems;
    const float2 mu = tile_level<C, K>(centre, X0, Y0, W, H, tile);
    const int cols = kHalf + 2 * S + 2 * A, side = 2 * A + 1;
    const int all = (2 * a.pairs + 1) * side;  // window rows of the whole tile
    float2* kept = hs + K::HS_PAIRS + tid;  // [(C + 1) V] of this thread, kColsThreads apart
    int share = CLUSTER ? rank : 0, held = -1;  // the frame the tile holds
    for (int step = 0; step <= 2 * a.pairs || (!CLUSTER && share + 1 < split); ++step) {
        if (step > 2 * a.pairs) {  // the next share, from the centre frame on
            keep_sums<C, K>(z, kept, share == 0);
            ++share;
            step = 0;
        }
        const int f = step;
        const int from = all * share / split, to = all * (share + 1) / split;
        // the centre frame first, by every CTA: its tile holds the centre runs
        const int dy0 = max(from - f * side, 0) - A, dy1 = min(to - f * side, side) - A;
        if (dy0 >= dy1 && (f > 0 || share > (CLUSTER ? rank : 0))) continue;
        const int pair = (f - 1) >> 1;
        const bool fwd = (f & 1) != 0;
        const int slot = f == 0 ? a.slot_centre : (fwd ? a.slot_fwd[pair] : a.slot_bwd[pair]);
        // The forward's order: pair by pair and offset by offset, the forward frame at q (an even id),
        // then the backward frame at -q; the single-frame pass last.
        const int id_first = 2 * pair * side * side + (fwd ? 0 : 2 * side * side - 1), id_step = fwd ? 2 : -2;
        if (CLUSTER || REC || f != held) {  // the next share may begin in the frame the last one ended in
            load_cols<K, C>(tile, a.ring + slot * a.frame_elems, X0 - S - A, Y0 - S - A, K::rows(A), cols, W, H, mu);
            __syncthreads();
            held = f;
        }
        if (f == 0) {
#pragma unroll
            for (int i = 0; i < K::RUNW; ++i) z.ctr[i] = load_pair<C>(z.run + i * C);
            if (REC) {
#pragma unroll
                for (int k = 0; k < V; ++k) {
                    const Pair<C> v = load_pair<C>(z.own + k * K::PITCH * C);
#pragma unroll
                    for (int c = 0; c < C; ++c) z.ref[c][k] = v.c[c];
                }
            }
            cols_frame<C, S, FAST, false, REC, K>(z, A, dy0, dy1, true, a.spatial_lut, off_pair, kk, scale2,
                                                  2 * a.pairs * side * side, 1);
        } else if (use_conf) {
            const float* cf = a.conf + (fwd ? a.conf_fwd_off[pair] : a.conf_bwd_off[pair]);
            const int bc0 = min(min(X0 + col, W - 1) / a.conf_step, a.blocks_x - 1);
            const int bc1 = min(min(X0 + col + kHalf, W - 1) / a.conf_step, a.blocks_x - 1);
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const int br = min(min(Y0 + y0 + k, H - 1) / a.conf_step, a.blocks_y - 1);
                z.conf[k] = f2(__ldg(cf + br * a.blocks_x + bc0), __ldg(cf + br * a.blocks_x + bc1));
            }
            cols_frame<C, S, FAST, !FAST, REC, K>(z, A, dy0, dy1, false, nullptr, off_pair, kk, scale2, id_first, id_step);
        } else {
            cols_frame<C, S, FAST, false, REC, K>(z, A, dy0, dy1, false, nullptr, off_pair, kk, scale2, id_first, id_step);
        }
        __syncthreads();  // every thread is done with this frame's tile
    }
    if (!CLUSTER && split > 1) {
        keep_sums<C, K>(z, kept, false);
#pragma unroll
        for (int k = 0; k < V; ++k) {
#pragma unroll
            for (int c = 0; c < C; ++c) z.a[c][k] = kept[(c * V + k) * kColsThreads];
            z.ws[k] = kept[(C * V + k) * kColsThreads];
        }
    }
    if (CLUSTER && split > 1) {
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
        float2* sums = cols_smem + tid;  // [(C + 2) V] of this thread, kColsThreads apart
        if (rank != 0) {
#pragma unroll
            for (int k = 0; k < V; ++k) {
#pragma unroll
                for (int c = 0; c < C; ++c) sums[(c * V + k) * kColsThreads] = z.a[c][k];
                sums[(C * V + k) * kColsThreads] = z.ws[k];
                sums[((C + 1) * V + k) * kColsThreads] = z.m[k];
            }
        }
        cluster.sync();
        if (rank == 0) {
            for (int r = 1; r < split; ++r) {
                const float2* other = cluster.map_shared_rank(sums, r);
#pragma unroll
                for (int k = 0; k < V; ++k) {
#pragma unroll
                    for (int c = 0; c < C; ++c) z.a[c][k] = add2(z.a[c][k], other[(c * V + k) * kColsThreads]);
                    z.ws[k] = add2(z.ws[k], other[(C * V + k) * kColsThreads]);
                    const float2 m = other[((C + 1) * V + k) * kColsThreads];
                    z.m[k] = FAST ? f2(fminf(z.m[k].x, m.x), fminf(z.m[k].y, m.y))
                                  : f2(fmaxf(z.m[k].x, m.x), fmaxf(z.m[k].y, m.y));
                }
            }
        }
        cluster.sync();  // the others' shared memory stays until it is read
        if (rank != 0) return;
    }

    if constexpr (REC) {
        // accumulate.rs:175-201 differentiated at each pixel, as the offset-pair tile records it, but for
        // the output, which is recorded less the tile's level: dL/dh2 sums w (I - out) over every pixel and
        // offset with much cancellation, and the rounding of `out` was most of its error (the sum of
        // w (I - own), divided by the denominator, keeps it to the last bits of the difference).
#pragma unroll
        for (int l = 0; l < 2; ++l)
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const int gx = X0 + col + l * kHalf, gy = Y0 + y0 + k;
                if (gx >= W || gy >= H) continue;
                const int64_t px = static_cast<int64_t>(gy) * W + gx;
                const float m = l ? z.m[k].y : z.m[k].x;
                const float self_weight = a.wref * (FAST ? ex2_approx(m * kk.x) : m);
                const float den = self_weight + (l ? z.ws[k].y : z.ws[k].x);
                const float* g = rec->grad_out + px * C;
                float* gc = rec->grad_centre + px * C;
                float* r = rec->records + px * nlm_tile_detail::kRecordWords;
                const bool live = den > 1e-30f;
                const float inv = live ? 1.0f / den : 0.0f;
                float gm = 0.0f;
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const float away = (l ? z.a[c][k].y : z.a[c][k].x) * inv;  // out - own
                    gc[c] = live ? g[c] * self_weight * inv : g[c];
                    gm -= g[c] * a.wref * away * inv;
                    r[c] = (l ? z.ref[c][k].y : z.ref[c][k].x) + away;
                }
                r[2] = inv;
                r[3] = gm;
                r[4] = __int_as_float(live ? (l ? z.id[k].y : z.id[k].x) : -1);
            }
        return;
    }

    // Finish (accumulate.rs:175-201), written straight to the output frame.
    const bool flags = a.fix_count != nullptr;
    const float band = a.code_max * (a.fix_band + kFixBandPerH2 * h2);
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        const int gx = X0 + col + l * kHalf;
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const int gy = Y0 + y0 + k;
            bool near = false;
            if (gx < W && gy < H) {
                const float m = l ? z.m[k].y : z.m[k].x;
                const float max_w = FAST ? ex2_approx(m * kk.x) : m;
                const float wsum = l ? z.ws[k].y : z.ws[k].x;
                const float* orig = centre + (static_cast<int64_t>(gy) * W + gx) * C;
                const float self_weight = __fmul_rn(a.wref, max_w);
                const float denom = __fadd_rn(self_weight, wsum);
                float* dst = a.out + (static_cast<int64_t>(gy) * W + gx) * C;
                if (denom > 1e-30f) {
                    const float inv = __frcp_rn(denom);
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        const float sum_wi = l ? z.a[c][k].y : z.a[c][k].x;
                        const float level = c == 0 ? mu.x : mu.y;
                        const float own = __ldg(orig + c) - level;
                        const float v = __fadd_rn(__fmul_rn(__fadd_rn(__fmul_rn(own, self_weight), sum_wi), inv), level);
                        dst[c] = v;
                        if (flags) near |= near_code_boundary(v, a.code_max, band);
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < C; ++c) dst[c] = __ldg(orig + c);  // passes through exactly
                }
            }
            if (flags) note_fix(near, static_cast<int64_t>(gy) * W + gx, a.fix_list, a.fix_count);
        }
    }
}

// Resident CTAs per SM asked of each instance, and the registers that leaves: 8 (128 registers) for
// luma of s <= 2 without offsets, 6 (168) where the noise offset's state or a longer run would spill
// at 128 (HQ s = 2, 1080p d = 4 a = 4: 1.02 ms at 6, 1.06 at 8), 5 for two channels.
template <int C, int S, bool FAST>
constexpr int cols_minb() {
    return C == 2 ? 5 : (S == 4 && FAST ? 5 : (S <= 2 && FAST ? 8 : 6));
}

// Q = 3 offsets per step for luma, 2 where two channels' samples fill the registers (luma at s = 2,
// 1080p d = 2 a = 5: 0.725 ms at 3, 0.767 at 2).
template <int C, int S, bool BIG>
using ColsOf = Cols<C, S, C == 1 ? 3 : 2, BIG>;

template <int C, int S, bool FAST, bool BIG>
__global__ void __launch_bounds__(kColsThreads, cols_minb<C, S, FAST>()) nlm_cols_kernel(NlmLaunch a, int split) {
    cols_tile<C, S, FAST, ColsOf<C, S, BIG>, true>(a, blockIdx.x / split, blockIdx.y, blockIdx.x % split, split);
}

// Persistent batch: every CTA takes tiles from one counter until the batch's tiles run out. Tile t
// belongs to the job j with prefix[j] <= t < prefix[j + 1]; jobs are whole launch descriptions, with the
// shares a lone launch would cut a tile into (cols_split) in `variant`.
template <int C, int S, bool FAST, bool BIG>
__global__ void __launch_bounds__(kColsThreads, cols_minb<C, S, FAST>())
    nlm_cols_batch_kernel(const NlmLaunch* __restrict__ jobs, const int* __restrict__ prefix, int njobs, int* counter) {
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
        const int tiles_x = (a.width + 2 * kHalf - 1) / (2 * kHalf);
        cols_tile<C, S, FAST, ColsOf<C, S, BIG>, false>(a, local % tiles_x, local / tiles_x, 0, a.variant);
    }
}

template <int C, int S, bool FAST, bool BIG>
cudaError_t launch_cols_one(const NlmLaunch& a, int split, cudaStream_t stream) {
    using K = ColsOf<C, S, BIG>;
    // Shared memory that leaves room for `n` CTAs on an SM (228 KB, 1 KB of it the runtime's per CTA).
    constexpr auto room = [](int n) { return static_cast<size_t>(228 / n - 1) * 1024; };
    constexpr int kMinb = cols_minb<C, S, FAST>();
    constexpr size_t kFewest = room(kMinb - (kResidencies - 1));
    constexpr size_t kMost = kFewest > K::smem_bytes(kMaxA) ? kFewest : K::smem_bytes(kMaxA);
    if (cudaError_t e = allow_smem<nlm_cols_kernel<C, S, FAST, BIG>>(kMost)) return e;
    size_t smem = K::smem_bytes(a.search_radius);
    if (a.variant > 0 && a.variant < kResidencies) {
        const size_t least = room(kMinb - a.variant);
        smem = smem > least ? smem : least;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((a.width + 2 * kHalf - 1) / (2 * kHalf) * split, (a.height + K::TY - 1) / K::TY);
    cfg.blockDim = dim3(kColsThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute cluster[1];
    cluster[0].id = cudaLaunchAttributeClusterDimension;
    cluster[0].val.clusterDim.x = static_cast<unsigned>(split);
    cluster[0].val.clusterDim.y = 1;
    cluster[0].val.clusterDim.z = 1;
    cfg.attrs = cluster;
    cfg.numAttrs = split > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, nlm_cols_kernel<C, S, FAST, BIG>, a, split);
}

template <int C, int S, bool FAST, bool BIG>
cudaError_t launch_cols_batch_one(const NlmLaunch* jobs, const int* prefix, int njobs, int* counter, int a,
                                  bool shares, cudaStream_t stream) {
    using K = ColsOf<C, S, BIG>;
    if (cudaError_t err = allow_smem<nlm_cols_batch_kernel<C, S, FAST, BIG>>(K::smem_bytes(kMaxA) +
                                                                             sizeof(float2) * K::KEPT_PAIRS))
        return err;
    const size_t smem = shares ? sizeof(float2) * (K::tile_pairs(a) + K::HS_PAIRS + K::KEPT_PAIRS) : K::smem_bytes(a);
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, nlm_cols_batch_kernel<C, S, FAST, BIG>, kColsThreads,
                                                          smem);
    if (e != cudaSuccess) return e;
    nlm_cols_batch_kernel<C, S, FAST, BIG><<<sms * (per_sm > 0 ? per_sm : 1), kColsThreads, smem, stream>>>(
        jobs, prefix, njobs, counter);
    return cudaGetLastError();
}

template <bool FAST, int C, int S>
cudaError_t launch_cols_s(const NlmLaunch& a, int split, cudaStream_t stream) {
    if (a.patch_radius == S)
        return a.search_radius > kSmallA ? launch_cols_one<C, S, FAST, true>(a, split, stream)
                                         : launch_cols_one<C, S, FAST, false>(a, split, stream);
    if constexpr (S < kColsMaxS) return launch_cols_s<FAST, C, S + 1>(a, split, stream);
    else return cudaErrorInvalidValue;
}

template <bool FAST, int C, int S>
cudaError_t launch_cols_batch_s(const NlmLaunch* jobs, const int* prefix, int njobs, int* counter, int s, int a,
                                bool shares, cudaStream_t stream) {
    if (s == S)
        return a > kSmallA ? launch_cols_batch_one<C, S, FAST, true>(jobs, prefix, njobs, counter, a, shares, stream)
                           : launch_cols_batch_one<C, S, FAST, false>(jobs, prefix, njobs, counter, a, shares, stream);
    if constexpr (S < kColsMaxS) return launch_cols_batch_s<FAST, C, S + 1>(jobs, prefix, njobs, counter, s, a, shares, stream);
    else return cudaErrorInvalidValue;
}

}  // namespace nlm_cols_detail
}  // namespace avd
