// The NLMeans adjoint on the column-pair tile (nlm_cols.cuh) for patch radii up to kColsMaxPatch: what
// nlm_adjoint.cu computes, with the two packed lanes of every f32x2 operation on two pixels 16 columns
// apart and one frame and offset per step.
//
// What bounds it. Per (pixel, offset) the forward's distance and weight are formed again, dL/dD is box
// summed back over the patch (as many additions as the forward's box sums) and two products are added
// into the neighbour frame's gradient: shared-memory accesses and the instructions around them. On the
// offset-pair tile that took 83 instructions per (pixel, offset): two scalar accesses and an address per
// lane, and shared atomics in the single-frame pass, whose two lanes add into one tile. Here a lane pair
// is one 8-byte access at an immediate offset, and as both lanes share the offset every pixel's cell is
// its own, so nothing is atomic before the tile is flushed.
//
// How. A CTA of 64 threads owns 32 x TY pixels and walks the frames one after the other. Per offset:
//   1 - row runs of the squared differences (the forward's), to shared memory;
//   2 - column strips: distance, weight, dL/dw; w times the upstream gradient added into the neighbour
//       frame's gradient tile; dL/dD stored;
//   3 - the vertical box of dL/dD on the tile's rows and their s halo;
//   4 - the horizontal box, on the row runs of phase 1: a run's 8 columns reach exactly the 8 + 2s cells
//       whose centre and neighbour samples the thread read there, so both are still in its registers. The
//       distance terms go to the centre frame's gradient (registers, for the whole kernel) and to the
//       neighbour's tile.
// Neighbouring runs and the two lanes' halves overlap by 2s cells, where each adds its own share: the
// terms are linear in dL/dD. A frame's gradient tile is added to global memory once, at the clamped pixels.
//
// Measured at 1280x720, luma, d = 2, a = 5, s = 2: records 0.53 -> 0.48 ms, gradient 2.77 -> 1.40 ms (43
// instructions per pixel and offset). The gradient kernel holds two pixel columns' centre samples, centre
// gradients and outputs in registers: at six CTAs per SM it spilled (1.60 ms), four leave it 255.

#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.h"
#include "nlm_adjoint.cuh"
#include "nlm_cols.cuh"

namespace avd {
namespace {

using namespace nlm_cols_detail;
using nlm_tile_detail::kRecordWords;
using nlm_tile_detail::RecordOut;

// The adjoint takes one offset per step.
template <int C, int S, bool BIG>
struct GradTile : Cols<C, S, 1, BIG> {
    using K = Cols<C, S, 1, BIG>;
    static constexpr int EH = K::TY + 2 * S;          // extended rows: the tile plus its s halo
    static constexpr int RPS = (EH + 3) / 4;          // extended rows per column strip
    static constexpr int ETOP = 2 * S + 1;            // zero rows above the stored dL/dD
    static constexpr int ET_PAIRS = (ETOP + 4 * RPS) * kHalf;
    static constexpr int GVW = kHalf + 1;             // odd, so 16 rows' reads of one column miss each other
    static constexpr int GV_PAIRS = 4 * RPS * GVW;
    __host__ __device__ static constexpr size_t grad_bytes(int a) {
        return sizeof(float2) * static_cast<size_t>(2 * K::tile_pairs(a) + K::HS_PAIRS + ET_PAIRS + GV_PAIRS);
    }
};

template <int C, int S, bool FAST, bool BIG>
__global__ void __launch_bounds__(kColsThreads, C == 1 ? 6 : 4) nlm_record_cols_kernel(NlmLaunch a, RecordOut r) {
    cols_tile<C, S, FAST, ColsOf<C, S, BIG>, false, true>(a, blockIdx.x, blockIdx.y, 0, 1, &r);
}

template <int C>
__device__ __forceinline__ void store_pair(float2* p, const Pair<C>& v) {
    if (C == 1) p[0] = v.c[0];
    else *reinterpret_cast<float4*>(p) = make_float4(v.c[0].x, v.c[0].y, v.c[C - 1].x, v.c[C - 1].y);
}

// Adds a frame's gradient tile into its gradient, at the clamped pixels the tile was staged from (border
// duplicates fold onto the edge pixels), and clears it.
template <int C, class K>
__device__ __forceinline__ void flush_cols(float2* tile, int rows, int cols, float* grad_frame, int x0, int y0, int W,
                                           int H) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = lane; c < cols; c += 32) {
        const int xa = clampi(x0 + c, 0, W - 1), xb = clampi(x0 + c + kHalf, 0, W - 1);
        for (int r = warp; r < rows; r += kColsThreads / 32) {
            float2* cell = tile + (r * K::PITCH + c) * C;
            const Pair<C> v = load_pair<C>(cell);
            float* row = grad_frame + static_cast<int64_t>(clampi(y0 + r, 0, H - 1)) * W * C;
            Pair<C> zero;
#pragma unroll
            for (int ch = 0; ch < C; ++ch) {
                zero.c[ch] = f2(0.0f, 0.0f);
                if (v.c[ch].x != 0.0f) atomicAdd(row + xa * C + ch, v.c[ch].x);
                if (v.c[ch].y != 0.0f) atomicAdd(row + xb * C + ch, v.c[ch].y);
            }
            store_pair<C>(cell, zero);
        }
    }
}

template <int C, int S, bool FAST, bool BIG>
__global__ void __launch_bounds__(kColsThreads, 4) nlm_grad_cols_kernel(GradArgs g) {
    using T = GradTile<C, S, BIG>;
    using K = typename T::K;
    constexpr int V = K::V, RUNW = K::RUNW, EH = T::EH, RPS = T::RPS, GVW = T::GVW;
    const NlmLaunch& a = g.a;
    const int A = a.search_radius, W = a.width, H = a.height;
    const int X0 = blockIdx.x * 2 * kHalf, Y0 = blockIdx.y * K::TY;
    const int tid = threadIdx.x, lane = tid & 31;
    const int col = tid & (kHalf - 1), strip = tid / kHalf, y0 = strip * V;
    const int run_row = min((tid >> 5) * 16 + (lane & 15), K::HR - 1), run_x = (lane >> 4) * kRun;

    float2* tile = cols_smem;
    float2* gt = tile + K::tile_pairs(A);
    float2* hs = gt + K::tile_pairs(A);
    // dL/dD * 2 scale, rows -ETOP .. -1 and TY .. 4 RPS - 1 held at zero so the vertical box reads them
    // unguarded; then its vertical box on the extended rows.
    float2* et_raw = hs + K::HS_PAIRS;
    float2* et = et_raw + T::ETOP * kHalf;
    float2* gv = et_raw + T::ET_PAIRS;
    for (int i = tid; i < T::ET_PAIRS + T::GV_PAIRS; i += kColsThreads) et_raw[i] = f2(0.0f, 0.0f);
    for (int i = tid; i < K::tile_pairs(A); i += kColsThreads) gt[i] = f2(0.0f, 0.0f);

    const float2* run = tile + ((run_row + A) * K::PITCH + run_x + A) * C;
    const int own = ((y0 + S + A) * K::PITCH + col + S + A) * C;
    float2* hs_out = hs + run_row * kHsPitch + run_x;
    const float2* hs_in = hs + y0 * kHsPitch + col;
    const bool run_live = (tid >> 5) * 16 + (lane & 15) < K::HR;  // a repeated last row adds nothing

    const float h2 = g.h2;
    const float off_pair = FAST ? 0.0f : __ldg(a.derived + a.offset_word);
    const float scale = C == 1 ? 3.0f : 1.5f;
    const float neg = -h2 * kLog2e;
    const float2 kk = FAST ? f2(scale * neg, scale * neg) : f2(neg, neg);
    const float2 scale2 = f2(scale, scale);
    const float2 e_scale = f2(-h2 * 2.0f * scale, -h2 * 2.0f * scale);
    const float* centre = a.ring + a.slot_centre * a.frame_elems;

    const float2 mu = tile_level<C, K>(centre, X0, Y0, W, H, tile);  // the recorded outputs' level
    // Per owned pixel: upstream gradient over the denominator, output less the level, dL/dM and the max
    // weight's offset.
    float2 gamma[C][V], out[C][V], gm[V];
    int2 arg[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
        float gmv[2];
        int av[2];
        float ga[2][C], ov[2][C];
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            const int gx = X0 + col + l * kHalf, gy = Y0 + y0 + k;
            const bool in = gx < W && gy < H;
            const int64_t px = in ? static_cast<int64_t>(gy) * W + gx : 0;
            const float* r = g.records + px * kRecordWords;
            gmv[l] = in ? r[3] : 0.0f;
            av[l] = in ? __float_as_int(r[4]) : -1;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                ga[l][c] = in ? g.grad_out[px * C + c] * r[2] : 0.0f;  // 1/den is 0 where the pixel passes through
                ov[l][c] = in ? r[c] : 0.0f;
            }
        }
        gm[k] = f2(gmv[0], gmv[1]);
        arg[k] = make_int2(av[0], av[1]);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            gamma[c][k] = f2(ga[0][c], ga[1][c]);
            out[c][k] = f2(ov[0][c], ov[1][c]);
        }
    }
    // The centre frame's distance gradient on the cells of this thread's run.
    float2 gcen[RUNW][C];
#pragma unroll
    for (int i = 0; i < RUNW; ++i)
#pragma unroll
        for (int c = 0; c < C; ++c) gcen[i][c] = f2(0.0f, 0.0f);
    float2 gh2 = f2(0.0f, 0.0f);

    Pair<C> ctr[RUNW];
    const int cols = kHalf + 2 * S + 2 * A, side = 2 * A + 1;
    const float2 zero2 = f2(0.0f, 0.0f);
    for (int f = 0; f <= 2 * a.pairs; ++f) {
        // the centre frame first: its tile holds the centre runs
        const int pair = (f - 1) >> 1;
        const bool fwd = (f & 1) != 0;
        const int slot = f == 0 ? a.slot_centre : (fwd ? a.slot_fwd[pair] : a.slot_bwd[pair]);
        const int id_first = f == 0 ? 2 * a.pairs * side * side : 2 * pair * side * side + (fwd ? 0 : 2 * side * side - 1);
        const int id_step = f == 0 ? 1 : (fwd ? 2 : -2);
        load_cols<K, C>(tile, a.ring + slot * a.frame_elems, X0 - S - A, Y0 - S - A, K::rows(A), cols, W, H, mu);
        __syncthreads();
        if (f == 0) {
#pragma unroll
            for (int i = 0; i < RUNW; ++i) ctr[i] = load_pair<C>(run + i * C);
        }
        for (int dy = -A; dy <= A; ++dy)
            for (int dx = -A; dx <= A; ++dx) {
                const int o = (dy + A) * side + dx + A, mid = A * side + A;
                if (f == 0 && o == mid) continue;
                const int id = id_first + id_step * (f == 0 && o > mid ? o - 1 : o);
                const int at = (dy * K::PITCH + dx) * C;
                const float off = FAST ? 0.0f : (f == 0 ? (a.spatial_lut ? __ldg(a.spatial_lut + o) : 0.0f) : off_pair);
                // 1: the row box sums of the squared differences. Luma keeps the run's samples for phase 4;
                // two channels' would not fit the registers and are read again.
                Pair<C> kept[C == 1 ? RUNW : 1];
                {
                    float2 d[RUNW], sum = zero2, h[2];
#pragma unroll
                    for (int k = 0; k < RUNW; ++k) {
                        const Pair<C> s = load_pair<C>(run + at + k * C);
                        if (C == 1) kept[C == 1 ? k : 0] = s;
                        const float2 du = sub2(ctr[k].c[0], s.c[0]);
                        if (C == 1) {
                            d[k] = mul2(du, du);
                        } else {
                            const float2 dv = sub2(ctr[k].c[C - 1], s.c[C - 1]);
                            d[k] = fma2(dv, dv, mul2(du, du));
                        }
                        if (k == 0) sum = d[0];
                        else if (k <= 2 * S) sum = add2(sum, d[k]);
                        else sum = sub2(add2(sum, d[k]), d[k - 2 * S - 1]);
                        const int j = k - 2 * S;
                        if (j >= 0) {
                            h[j & 1] = sum;
                            if (j & 1)
                                *reinterpret_cast<float4*>(hs_out + j - 1) = make_float4(h[0].x, h[0].y, h[1].x, h[1].y);
                        }
                    }
                }
                __syncthreads();
                // 2: distances, weights, dL/dw, the weighted-sum term, dL/dD.
                {
                    float2 hv[V + 2 * S];
#pragma unroll
                    for (int i = 0; i < V + 2 * S; ++i) hv[i] = hs_in[i * kHsPitch];
                    float2 dist = hv[0];
#pragma unroll
                    for (int i = 1; i <= 2 * S; ++i) dist = add2(dist, hv[i]);
                    const float2* p = tile + own + at;
                    float2* q = gt + own + at;
#pragma unroll
                    for (int k = 0; k < V; ++k) {
                        if (k > 0) dist = sub2(add2(dist, hv[k + 2 * S]), hv[k - 1]);
                        float2 x, w;
                        if (FAST) {
                            x = mul2(dist, scale2);
                            const float2 e = mul2(dist, kk);
                            w = f2(ex2_approx(e.x), ex2_approx(e.y));
                        } else {
                            x = fma2(dist, scale2, f2(-off, -off));
                            const float2 e = mul2(f2(fmaxf(x.x, 0.0f), fmaxf(x.y, 0.0f)), kk);
                            w = f2(ex2_approx(e.x), ex2_approx(e.y));
                        }
                        const Pair<C> n = load_pair<C>(p + k * K::PITCH * C);
                        Pair<C> sum = load_pair<C>(q + k * K::PITCH * C);
                        float2 gw = f2(id == arg[k].x ? gm[k].x : 0.0f, id == arg[k].y ? gm[k].y : 0.0f);
#pragma unroll
                        for (int c = 0; c < C; ++c) {
                            gw = fma2(gamma[c][k], sub2(n.c[c], out[c][k]), gw);
                            sum.c[c] = fma2(gamma[c][k], w, sum.c[c]);
                        }
                        store_pair<C>(q + k * K::PITCH * C, sum);
                        gw = mul2(gw, w);
                        // nothing passes where the offset clips the distance
                        gw = f2(x.x > 0.0f ? gw.x : 0.0f, x.y > 0.0f ? gw.y : 0.0f);
                        gh2 = fma2(gw, x, gh2);
                        et[(y0 + k) * kHalf + col] = mul2(gw, e_scale);
                    }
                }
                __syncthreads();
                // 3: the vertical box of dL/dD onto this strip's extended rows.
                {
                    const float2* ec = et + strip * RPS * kHalf + col;
                    float2 sum = ec[-2 * S * kHalf];
#pragma unroll
                    for (int r = 1 - 2 * S; r <= 0; ++r) sum = add2(sum, ec[r * kHalf]);
                    float2* gc = gv + strip * RPS * GVW + col;
                    gc[0] = sum;
#pragma unroll
                    for (int i = 1; i < RPS; ++i) {
                        sum = sub2(add2(sum, ec[i * kHalf]), ec[(i - 2 * S - 1) * kHalf]);
                        if (EH % RPS == 0 || strip * RPS + i < EH) gc[i * GVW] = sum;
                    }
                }
                __syncthreads();
                // 4: the horizontal box of the run's 8 columns onto its cells, then the distance terms.
                {
                    const float2* gr = gv + run_row * GVW + run_x;
                    float2* q = gt + (run - tile) + at;
                    float2 e[kRun];
#pragma unroll
                    for (int k = 0; k < kRun; ++k) e[k] = gr[k];
                    float2 G = zero2;
#pragma unroll
                    for (int k = 0; k < RUNW; ++k) {
                        // The last 2s cells are the next run's first, whose thread is in this warp and has
                        // added its share by then.
                        if (k == kRun) __syncwarp();
                        if (k == 0) G = e[0];
                        else if (k <= 2 * S && k < kRun) G = add2(G, e[k]);
                        else if (k < kRun) G = sub2(add2(G, e[k]), e[k - 2 * S - 1]);
                        else if (k - 2 * S - 1 >= 0) G = sub2(G, e[k - 2 * S - 1]);
                        const Pair<C> n = C == 1 ? kept[C == 1 ? k : 0] : load_pair<C>(run + at + k * C);
                        if (run_live) {
                            Pair<C> sum = load_pair<C>(q + k * C);
#pragma unroll
                            for (int c = 0; c < C; ++c) {
                                const float2 term = mul2(G, sub2(ctr[k].c[c], n.c[c]));
                                gcen[k][c] = add2(gcen[k][c], term);
                                sum.c[c] = sub2(sum.c[c], term);
                            }
                            store_pair<C>(q + k * C, sum);
                        }
                    }
                }
            }
        __syncthreads();
        flush_cols<C, K>(gt, K::rows(A), cols, g.grad_window + slot * a.frame_elems, X0 - S - A, Y0 - S - A, W, H);
        __syncthreads();
    }

    // The owned centre cells, at their clamped pixels.
    float* grad_centre = g.grad_window + a.slot_centre * a.frame_elems;
    auto flush_cell = [&](int ey, int ex, const float2 (&acc)[C]) {
        const int gy = clampi(Y0 - S + ey, 0, H - 1);
        float* row = grad_centre + static_cast<int64_t>(gy) * W * C;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (acc[c].x != 0.0f) atomicAdd(row + clampi(X0 - S + ex, 0, W - 1) * C + c, acc[c].x);
            if (acc[c].y != 0.0f) atomicAdd(row + clampi(X0 - S + ex + kHalf, 0, W - 1) * C + c, acc[c].y);
        }
    };
    if (run_live) {
#pragma unroll
        for (int i = 0; i < RUNW; ++i) flush_cell(run_row, run_x + i, gcen[i]);
    }
    // dL/dh2 of the tile, summed in a fixed order.
    __shared__ float red[kColsThreads / 32];
    float total = -(gh2.x + gh2.y);
#pragma unroll
    for (int i = 16; i > 0; i >>= 1) total += __shfl_xor_sync(0xffffffffu, total, i);
    if (lane == 0) red[tid >> 5] = total;
    __syncthreads();
    if (tid == 0) g.partials[blockIdx.y * gridDim.x + blockIdx.x] = red[0] + red[1];
}

template <int C, int S, bool FAST, bool BIG>
cudaError_t launch_one(const NlmLaunch& a, const RecordOut& rec, const GradArgs& g, cudaStream_t s) {
    using K = ColsOf<C, S, BIG>;
    using T = GradTile<C, S, BIG>;
    if (cudaError_t e = allow_smem<nlm_record_cols_kernel<C, S, FAST, BIG>>(K::smem_bytes(kMaxA))) return e;
    if (cudaError_t e = allow_smem<nlm_grad_cols_kernel<C, S, FAST, BIG>>(T::grad_bytes(kMaxA))) return e;
    const dim3 grid((a.width + 2 * kHalf - 1) / (2 * kHalf), (a.height + K::TY - 1) / K::TY);
    nlm_record_cols_kernel<C, S, FAST, BIG><<<grid, kColsThreads, K::smem_bytes(a.search_radius), s>>>(a, rec);
    nlm_grad_cols_kernel<C, S, FAST, BIG><<<grid, kColsThreads, T::grad_bytes(a.search_radius), s>>>(g);
    return cudaGetLastError();
}

template <int C, int S>
cudaError_t dispatch(const NlmLaunch& a, const RecordOut& rec, const GradArgs& g, cudaStream_t s) {
    if (a.patch_radius == S) {
        if (a.search_radius > kSmallA)
            return a.fast ? launch_one<C, S, true, true>(a, rec, g, s) : launch_one<C, S, false, true>(a, rec, g, s);
        return a.fast ? launch_one<C, S, true, false>(a, rec, g, s) : launch_one<C, S, false, false>(a, rec, g, s);
    }
    if constexpr (S < kColsMaxPatch) return dispatch<C, S + 1>(a, rec, g, s);
    else return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_adjoint_cols(const NlmLaunch& a, const nlm_tile_detail::RecordOut& rec, const GradArgs& g,
                                cudaStream_t s) {
    return a.channels == 1 ? dispatch<1, 0>(a, rec, g, s) : dispatch<2, 0>(a, rec, g, s);
}

}  // namespace avd
