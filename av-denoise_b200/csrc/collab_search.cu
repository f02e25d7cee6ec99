// NL4D group search for sm_100a: the best 8 positions of the centre frame's spatial window for every
// reference patch (fused/centre.rs:213-258), then the volumes along the neighbour frames' motion
// (fused/trajectory.rs). Two launches per pass, joined by the member words.
//
// The centre search. The members are the 8 smallest (distance, visiting index) pairs, the distance
// being an f32 sum in the restatement's own order, so those bits decide. Scoring all (2r+1)^2
// candidates that way costs 192 unfused f32 operations each and bounded the pass (4K luma, r = 16:
// 1,089 candidates, about 9 of the search's 14.0 ms; 1080p luma, r = 9: 0.97 of 1.70 ms). The scoring
// below takes 2.67 and 0.44 ms (chroma of the 4K frame 1.3). But only a dozen candidates are ever near
// the best eight, and telling the rest apart needs no exact bits. So the candidates are first scored on
// the tensor cores: with samples c, n in units of codes around the middle code, exact in f16,
//     sum c^2 - D = 2 sum c n - sum n^2
// is a contraction over the 64 (128) samples of a patch whose f32 accumulation is the integer itself
// or within a measured bound of it. The larger of it ranks the smaller distance. Every thread keeps the
// largest score of its own share of a patch's candidates (64 shares to a patch); the eighth largest of
// those shares' maxima is reached by at least eight candidates, so a candidate whose score lies below
// it by more than the error of both scores cannot be among the best eight. A second round of the same
// products lists the candidates at or above that line, and the 8-lane group of the patch scores the
// listed ones (nine or ten of 1,089 on noisy frames) in the exact order.
//
// Clean areas. Past 8 bits the samples are taken less the middle of the tile's, so that a tile of a narrow
// range has exact scores whatever the depth, and lists real ties alone. A patch whose list still overflows
// (hundreds of equal patches) and every patch of a tile whose samples overrun f16 falls back on exact
// sums: where eight candidates seem to equal the patch, the window's first 48 until eight do (constant
// areas); then the window in bands of rows, up to the first band that leaves eight equal patches in the
// list. The groups without such a patch take a part of another's window. Streams of six frames, all
// kernels, ms with the exact search of every candidate, with a full search per overflow, and so: 1080p
// 8-bit r = 9 constant 22.0, 21.5, 15.8, dithered 32.6, 33.0, 25.2, flat shapes 24.1, 23.8, 18.8; 10-bit
// 4:2:0 r = 16 constant 39.4, 46.6, 24.7, dithered 53.9, 62.8, 35.6, shapes 44.4, 52.5, 34.5 (noisy 43.3,
// 25.4, 25.5). What gains least is a flat area with one sample in a hundred off, whose ties are not the
// patch's equals and need every exact sum: 31.0, 31.3, 29.8 and 54.1, 62.7, 54.3; float chroma at 720p
// 20.5, 22.1, 22.4.
//
// The error of a score, in units of squared codes: the tensor core's accumulation and the sums of squares
// (screen_score.cuh, which also says what that rests on), the f32 distance's own rounding (1e-5 of it),
// where the ring holds codes the rounding of their quotients (2^-24 of the largest code per sample), and
// where it holds floats the samples' rounding to f16: |sqrt(D) - sqrt(D~)| is at most the norm of the
// rounding of both patches.
//
// How. A CTA owns 8 x 4 reference patches (step 4), four groups of 8 (4 x 2) that share a staged tile of
// 16-byte chunks, chunk (x, y) holding the eight samples x..x+7 of row y: patch row r of candidate
// (x, y) is chunk (x, y + r), so ldmatrix gathers sixteen candidates' rows (the instruction's 16 rows)
// straight from it, and the eight patches of a group (times 2, its 8 columns) stay in registers. Warps
// take the window's rows in turn.

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "collab_group.cuh"
#include "kernels.h"
#include "screen_score.cuh"
#include "smem_limit.h"

namespace avd {

namespace {

using namespace collab_detail;
using screen::mma_f16;

// The lane's share of the distance from `ref` (its 8 x C column) to the candidate at (x, y).
template <int C>
__device__ __forceinline__ float column_ssd(const float (&ref)[P * C], const float* __restrict__ frame, int width,
                                            uint32_t x, uint32_t y, int sub) {
    float s = 0.0f;
    const float* p = frame + (static_cast<size_t>(y) * width + x + sub) * C;
#pragma unroll
    for (int r = 0; r < P; ++r) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            float d = ref[r * C + c] - __ldg(p + static_cast<size_t>(r) * width * C + c);
            s = __fadd_rn(s, __fmul_rn(d, d));
        }
    }
    return s;
}

__device__ __forceinline__ uint32_t covering_lo(uint32_t patch_start, uint32_t blksize, uint32_t step) {
    const uint32_t overhang = max(patch_start + P, blksize) - blksize;
    return (overhang + step - 1) / step;
}

// Keyed top-8 insert: the reference visits the window row by row and keeps ties in visiting order
// (fused/plane_ops.rs:38-53), so its list is the 8 smallest (distance, visiting index) pairs. The
// search here visits columns, comparing the pair, which keeps exactly the same list.
__device__ __forceinline__ bool key_less(float d, uint32_t i, float bd, uint32_t bi) {
    return d < bd || (d == bd && i < bi);
}

__device__ __forceinline__ void shift_insert8_key(const GroupCtx& g, float& best_d, uint32_t& best_i, float d,
                                                  uint32_t i) {
    const float prev_d = __shfl_up_sync(g.mask, best_d, 1, 8);
    const uint32_t prev_i = __shfl_up_sync(g.mask, best_i, 1, 8);
    if (key_less(d, i, best_d, best_i)) {
        if (g.sub == 0 || !key_less(d, i, prev_d, prev_i)) {
            best_d = d;
            best_i = i;
        } else {
            best_d = prev_d;
            best_i = prev_i;
        }
    }
}

// The group sums of eight candidates at once, each lane's eight column distances in `v`: the same
// pairwise tree as reduce8 (partners xor 1, then 2, then 4), each level keeping half the candidates
// on each side, so every total has the bits reduce8 gives it. Lane `sub` ends with the total of
// candidate (sub & 1) * 4 + (sub & 2) + ((sub >> 2) & 1).
__device__ __forceinline__ float reduce_scatter8(const GroupCtx& g, const float (&v)[8]) {
    const bool b0 = g.sub & 1, b1 = g.sub & 2, b2 = g.sub & 4;
    float u[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float give = b0 ? v[j] : v[4 + j];
        const float keep = b0 ? v[4 + j] : v[j];
        u[j] = __fadd_rn(keep, __shfl_xor_sync(g.mask, give, 1));
    }
    float w[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const float give = b1 ? u[j] : u[2 + j];
        const float keep = b1 ? u[2 + j] : u[j];
        w[j] = __fadd_rn(keep, __shfl_xor_sync(g.mask, give, 2));
    }
    const float give = b2 ? w[0] : w[1];
    const float keep = b2 ? w[1] : w[0];
    return __fadd_rn(keep, __shfl_xor_sync(g.mask, give, 4));
}

__device__ __forceinline__ int scattered_candidate(int sub) { return (sub & 1) * 4 + (sub & 2) + ((sub >> 2) & 1); }

// One candidate per lane into the group's list, where `in` and it beats the list's worst key, one at a
// time and in any order (the list is the 8 smallest (distance, visiting index) pairs whatever the order
// they arrive in).
__device__ __forceinline__ void take_winners(const GroupCtx& g, bool in, float d, uint32_t i, float& best_d,
                                             uint32_t& best_i, float& worst_d, uint32_t& worst_i) {
    const bool wins = in && d < kUnfilled && key_less(d, i, worst_d, worst_i);
    unsigned m = __ballot_sync(g.mask, wins) & g.mask;
    while (m) {
        const int src = __ffs(m) - 1;
        m &= m - 1;
        const float dd = __shfl_sync(g.mask, d, src);
        const uint32_t ii = __shfl_sync(g.mask, i, src);
        if (key_less(dd, ii, worst_d, worst_i)) {  // uniform: every lane holds the same words
            shift_insert8_key(g, best_d, best_i, dd, ii);
            worst_d = __shfl_sync(g.mask, best_d, 7, 8);
            worst_i = __shfl_sync(g.mask, best_i, 7, 8);
        }
    }
}

// A patch and its clipped window (fused/centre.rs:213-258). `cur` is the lane's column of the patch.
template <int C>
struct PatchWindow {
    float cur[P * C];
    uint32_t rx, ry, left, top, ww, hh;
    __device__ __forceinline__ uint32_t self() const { return (ry - top) * ww + (rx - left); }
};

template <int C>
__device__ __forceinline__ PatchWindow<C> patch_window(const CollabLaunch& a, const float* __restrict__ centre,
                                                       uint32_t rx, uint32_t ry, int sub) {
    PatchWindow<C> p;
    const uint32_t max_x = a.width - P, max_y = a.height - P;
    const int R = a.spatial_radius;
    p.rx = rx;
    p.ry = ry;
    p.left = clamp_top_left(static_cast<int>(rx) - R, max_x);
    p.top = clamp_top_left(static_cast<int>(ry) - R, max_y);
    p.ww = clamp_top_left(static_cast<int>(rx) + R, max_x) - p.left + 1;
    p.hh = clamp_top_left(static_cast<int>(ry) + R, max_y) - p.top + 1;
#pragma unroll
    for (int r = 0; r < P; ++r)
#pragma unroll
        for (int c = 0; c < C; ++c)
            p.cur[r * C + c] = __ldg(centre + ((static_cast<size_t>(ry) + r) * a.width + rx + sub) * C + c);
    return p;
}

// The 8-lane group's list, one member per lane, and its worst key.
struct TopEight {
    float d = kUnfilled;
    uint32_t i = 0xFFFFFFFFu;
    float worst_d = kUnfilled;
    uint32_t worst_i = 0xFFFFFFFFu;
    // The patch itself, before any other candidate.
    __device__ __forceinline__ void pin(const GroupCtx& g, uint32_t self) {
        if (g.sub == 0) {
            d = kSelfPin;
            i = self;
        }
    }
    __device__ __forceinline__ void take(const GroupCtx& g, bool in, float dist, uint32_t index) {
        take_winners(g, in, dist, index, d, i, worst_d, worst_i);
    }
    // Eight candidates of which none can be beaten but by an earlier one.
    __device__ __forceinline__ bool settled() const { return worst_d <= 0.0f; }
};

// The 15 samples a lane reads for eight candidate rows from window row jb of a column (rows past the
// window's last repeat it), and the distance of candidate jb + scattered_candidate(sub): its column sums
// in row order, the group's pairwise sum (reduce8's tree), times the channel scale.
template <int C>
struct ColumnBand {
    float rows[15][C];
    __device__ __forceinline__ void load(const PatchWindow<C>& p, const float* __restrict__ centre, int width,
                                         uint32_t col, uint32_t jb, int sub) {
        const float* colp = centre + static_cast<size_t>(p.left + col + sub) * C;
        const uint32_t last = p.top + p.hh + P - 2;
#pragma unroll
        for (int r = 0; r < 15; ++r)
#pragma unroll
            for (int c = 0; c < C; ++c)
                rows[r][c] = __ldg(colp + static_cast<size_t>(min(p.top + jb + r, last)) * width * C + c);
    }
    __device__ __forceinline__ float distance(const GroupCtx& g, const float (&cur)[P * C], float scale) const {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float sum = 0.0f;
#pragma unroll
            for (int r = 0; r < P; ++r)
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const float d = cur[r * C + c] - rows[k + r][c];
                    sum = __fadd_rn(sum, __fmul_rn(d, d));
                }
            v[k] = sum;
        }
        return reduce_scatter8(g, v) * scale;
    }
};

// Window columns [c0, c1) in the exact order, in bands of eight candidate rows. A band holds every earlier
// visiting index than the next one's, so the search ends with the first that leaves the list settled.
template <int C>
__device__ __noinline__ TopEight centre_columns(const GroupCtx& g, const PatchWindow<C>& p,
                                                const float* __restrict__ centre, int width, uint32_t c0,
                                                uint32_t c1, float scale) {
    TopEight best;
    const uint32_t self_col = p.rx - p.left, self_row = p.ry - p.top;
    if (self_col >= c0 && self_col < c1) best.pin(g, p.self());
    for (uint32_t jb = 0; jb < p.hh && !best.settled(); jb += 8) {
        const uint32_t j = jb + static_cast<uint32_t>(scattered_candidate(g.sub));
        for (uint32_t col = c0; col < c1; ++col) {
            ColumnBand<C> band;
            band.load(p, centre, width, col, jb, g.sub);
            best.take(g, j < p.hh && !(col == self_col && j == self_row), band.distance(g, p.cur, scale), j * p.ww + col);
        }
    }
    return best;
}

// `n` candidates in the exact order, eight at a time: candidate k at the position `at(k)`. ORDERED: in
// visiting order, and only until the list is settled.
template <int C, bool ORDERED, class At>
__device__ __forceinline__ void centre_listed(const GroupCtx& g, const PatchWindow<C>& p,
                                              const float* __restrict__ centre, int width, int n, float scale, At at,
                                              TopEight& best) {
    for (int j0 = 0; j0 < n && !(ORDERED && best.settled()); j0 += 8) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint2 c = at(min(j0 + k, n - 1));
            v[k] = column_ssd<C>(p.cur, centre, width, c.x, c.y, g.sub);
        }
        const int j = j0 + scattered_candidate(g.sub);
        const float d = reduce_scatter8(g, v) * scale;
        const uint2 c = at(min(j, n - 1));
        best.take(g, j < n && !(c.x == p.rx && c.y == p.ry), d, (c.y - p.top) * p.ww + (c.x - p.left));
    }
}

// The patch's members and group size from the group's list, into the member words.
__device__ __forceinline__ void write_members(const GroupCtx& g, uint32_t* words, uint32_t best_i, uint32_t left,
                                              uint32_t top, uint32_t ww, uint32_t hh, int k_max) {
    const uint32_t n_live = ww * hh;
    int k_use = 1;
    while (static_cast<uint32_t>(k_use * 2) <= n_live && k_use * 2 <= k_max) k_use *= 2;
    words[g.sub] = best_i == 0xFFFFFFFFu ? 0u : pack_pos_t(left + best_i % ww, top + best_i / ww, 0);
    if (g.sub == 0) words[MAX_K] = static_cast<uint32_t>(k_use);
}

constexpr int kRefsX = 8, kRefsY = 4, kRefs = kRefsX * kRefsY;  // reference patches of one CTA
constexpr int kWarps = 8, kScreenThreads = 32 * kWarps;         // one 8-lane group per patch
constexpr int kList = 48;                                       // candidates listed per patch
constexpr int kShares = kWarps * 8;                             // shares of a patch's candidates
constexpr int kProbe = 48;                                      // first candidates tried for eight equal ones
constexpr int kMaxParts = 8;                                    // groups that share one window's columns
constexpr int kMaxRadius = 16;
constexpr float kRound = 12582912.0f;  // 1.5 * 2^23
constexpr float kOutside = -1e30f;

// Tile sizes for spatial radius r: candidate columns (whole 16s), candidate rows, staged rows.
__host__ __device__ inline int screen_tiles(int r) { return (4 * (kRefsX - 1) + 1 + 2 * r + 15) / 16; }
__host__ __device__ inline int screen_pitch(int r) { return 16 * screen_tiles(r) + 1; }
__host__ __device__ inline int screen_rows(int r) { return 4 * (kRefsY - 1) + 1 + 2 * r; }

template <int C>
__host__ __device__ inline size_t screen_smem(int r) {
    const size_t rows = screen_rows(r) + 7, cp = screen_pitch(r);
    const size_t shares = static_cast<size_t>(kRefs) * kShares, sums = rows * cp;
    return 16 * C * rows * cp + sizeof(float) * (sums > shares ? sums : shares) +
           sizeof(float) * screen_rows(r) * cp + sizeof(float) * kRefs + sizeof(int) * kRefs +
           sizeof(uint16_t) * kRefs * kList;
}

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

extern __shared__ __align__(16) unsigned char screen_raw[];

// One round over the CTA's candidates: `visit(nt, e, cell, score)` for every candidate inside the window
// of patch e of group nt held by this thread (cell = row * 64 + column of the tile).
template <int C, class Visit>
__device__ __forceinline__ void score_round(const CollabLaunch& a, uint32_t chunk_addr, const float* __restrict__ sums,
                                            int tiles, int cp, int rows_staged, const uint32_t (&b)[4][8 * C],
                                            const int (&px)[4][2], const int (&py)[4], const int (&first_x)[2],
                                            const int (&last_x)[2], const int (&first_y)[2], const int (&last_y)[2],
                                            Visit visit) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2;
    const int r2 = 2 * a.spatial_radius;
    const int crows = screen_rows(a.spatial_radius);
    // This lane's row of the instruction's matrices: matrix l / 8 is (row half, patch row of the pair).
    const int half = (lane >> 3) & 1, k_sel = lane >> 4;
    const uint32_t base = chunk_addr + 16u * static_cast<uint32_t>(k_sel * cp + (lane & 7) + 8 * half);
    for (int cr = warp; cr < crows; cr += kWarps) {
        for (int ct = 0; ct < tiles; ++ct) {
            uint32_t m[4 * C][4];
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                    ldmatrix4(m[4 * c + ks], base + 16u * static_cast<uint32_t>((c * rows_staged + cr + 2 * ks) * cp + 16 * ct));
            const int c0 = 16 * ct + g;
            const float s0 = sums[cr * cp + c0], s1 = sums[cr * cp + c0 + 8];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const int nx = nt & 1, ny = nt >> 1;
                if (16 * ct + 15 < first_x[nx] || 16 * ct > last_x[nx] + r2 || cr < first_y[ny] || cr > last_y[ny] + r2)
                    continue;
                float d[4];
                mma_f16(d, m[0], b[nt][0], b[nt][1], s0, s0, s1, s1);
#pragma unroll
                for (int ks = 1; ks < 4 * C; ++ks)
                    mma_f16(d, m[ks], b[nt][2 * ks], b[nt][2 * ks + 1], d[0], d[1], d[2], d[3]);
                const bool row_in = static_cast<unsigned>(cr - py[nt]) <= static_cast<unsigned>(r2);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const bool in0 = row_in && static_cast<unsigned>(c0 - px[nt][e]) <= static_cast<unsigned>(r2);
                    const bool in1 = row_in && static_cast<unsigned>(c0 + 8 - px[nt][e]) <= static_cast<unsigned>(r2);
                    visit(nt, e, cr * 64 + c0, in0 ? d[e] : kOutside, in1 ? d[2 + e] : kOutside);
                }
            }
        }
    }
}

template <int C>
__global__ void __launch_bounds__(kScreenThreads, C == 1 ? 2 : 1) collab_screen_kernel(CollabLaunch a) {
    const int R = a.spatial_radius;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gq = lane >> 2, t4 = lane & 3;
    const int max_x = a.width - P, max_y = a.height - P;
    const int refs_x = (a.width - P + STEP - 1) / STEP + 1, refs_y = (a.height - P + STEP - 1) / STEP + 1;
    const int ix0 = blockIdx.x * kRefsX, iy0 = blockIdx.y * kRefsY;
    const int ox = min(ix0 * STEP, max_x), oy = min(iy0 * STEP, max_y);  // the tile's first patch
    const int tiles = screen_tiles(R), cp = screen_pitch(R), crows = screen_rows(R), rows = crows + 7;
    const float* centre = a.ring + static_cast<size_t>(a.centre_slot) * a.frame_elems;

    uint4* chunks = reinterpret_cast<uint4*>(screen_raw);  // [C][rows][cp]
    float* squares = reinterpret_cast<float*>(chunks + C * rows * cp);  // row sums, then the shares' maxima
    const int sq = max(rows * cp, kRefs * kShares);
    float* sums = squares + sq;                      // [crows][cp]: minus the patch's sum of squares
    float* line = sums + crows * cp;                 // [kRefs]: the score a listed candidate reaches
    int* count = reinterpret_cast<int*>(line + kRefs);
    uint16_t* list = reinterpret_cast<uint16_t*>(count + kRefs);

    // ---- stage: 8 chunks of one row per task; consecutive lanes take consecutive rows, whose odd pitch
    // spreads the 16-byte stores over the banks ----
    const bool codes = a.ring_code_max > 0.0f && a.ring_code_max <= 4095.0f;
    const float to_code = codes ? a.ring_code_max : 1023.0f;
    // What the samples are taken less. 8-bit codes: the middle of their range, where every score is exact.
    // Others: the middle of 32 samples spread over the tile, per channel (every warp finds it for itself), a
    // whole number, for codes one that leaves every code within the 2,048 that f16 holds exactly.
    float mid[C];
#pragma unroll
    for (int c = 0; c < C; ++c) mid[c] = 128.0f;
    if (!codes || to_code > 255.0f) {
        const int gx = min(max(ox - R + (lane & 7) * (16 * tiles + 6) / 7, 0), a.width - 1);
        const int gy = min(max(oy - R + (lane >> 3) * (rows - 1) / 3, 0), a.height - 1);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            float lo = __ldg(centre + (static_cast<size_t>(gy) * a.width + gx) * C + c), hi = lo;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            }
            const float m = rintf(0.5f * (lo + hi) * to_code);
            mid[c] = fabsf(m) <= 65536.0f ? m : 512.0f;  // NaN and infinities: the tile is searched in full
            if (codes) mid[c] = fminf(fmaxf(mid[c], to_code - 2048.0f), 2048.0f);
        }
    }
    float worst = 0.0f;
    bool bad = false;
    const int segs = 2 * tiles;
    for (int task = tid; task < rows * segs; task += kScreenThreads) {
        const int seg = task / rows, y = task - seg * rows;
        const int x0 = 8 * seg;
        const int gy = min(max(oy - R + y, 0), a.height - 1);
        const float* src = centre + static_cast<size_t>(gy) * a.width * C;
        float part[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) part[i] = 0.0f;
        float v[C][16];
#pragma unroll
        for (int i = 0; i < 15; ++i) {
            const int gx = min(max(ox - R + x0 + i, 0), a.width - 1);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const float s = __ldg(src + static_cast<size_t>(gx) * C + c);
                // codes: rounded to the code; floats: rounded to f16
                const float x = codes ? fmaf(s, to_code, kRound - mid[c]) - kRound
                                      : __half2float(__float2half_rn(fmaf(s, to_code, -mid[c])));
                bad |= !(fabsf(x) <= 2048.0f);
                worst = fmaxf(worst, fabsf(x));
                v[c][i] = x;
            }
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            v[c][15] = 0.0f;
            float run = 0.0f;
#pragma unroll
            for (int i = 0; i < 7; ++i) run = fmaf(v[c][i], v[c][i], run);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                run = fmaf(v[c][i + 7], v[c][i + 7], run);
                part[i] += run;
                run = fmaf(-v[c][i], v[c][i], run);
            }
            uint32_t even[8], odd[7];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const __half2 h = __floats2half2_rn(v[c][2 * i], v[c][2 * i + 1]);
                even[i] = *reinterpret_cast<const uint32_t*>(&h);
            }
#pragma unroll
            for (int i = 0; i < 7; ++i) odd[i] = __funnelshift_r(even[i], even[i + 1], 16);
            uint4* dst = chunks + (c * rows + y) * cp + x0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t* w = (i & 1) ? odd + i / 2 : even + i / 2;
                dst[i] = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) squares[y * cp + x0 + i] = part[i];
    }
    __shared__ int pending[kRefs], npending;
    __shared__ bool even[kRefs];  // eight candidates may equal the patch
    if (tid < kRefs) count[tid] = 0;
    if (tid == 0) npending = 0;
    bad = __syncthreads_or(bad);
    for (int task = tid; task < ((crows + 7) / 8) * 16 * tiles; task += kScreenThreads) {
        const int run_y = task / (16 * tiles), x = task - run_y * 16 * tiles;
        const int y0 = 8 * run_y;
        const int gx = ox - R + x;
        float run = 0.0f;
#pragma unroll
        for (int i = 0; i < 7; ++i) run += squares[(y0 + i) * cp + x];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (y0 + i < crows) {
                run += squares[(y0 + i + 7) * cp + x];
                const int gy = oy - R + y0 + i;
                const bool in = gx >= 0 && gx <= max_x && gy >= 0 && gy <= max_y;
                sums[(y0 + i) * cp + x] = in ? -run : kOutside;
                run -= squares[(y0 + i) * cp + x];
            }
        }
    }
    __syncthreads();

    // The group's patch (column n of the instruction) and this thread's two (columns 2 t4, 2 t4 + 1), as
    // positions in the tile: a patch's window starts at its own position less the tile's first patch.
    const uint32_t chunk_addr = static_cast<uint32_t>(__cvta_generic_to_shared(chunks));
    bool over = bad;  // some list of the CTA overflowed, or there are none
    if (!bad) {
        uint32_t b[4][8 * C];
        int px[4][2], py[4], first_x[2], last_x[2], first_y[2], last_y[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            first_x[h] = min((ix0 + 4 * h) * STEP, max_x) - ox;
            last_x[h] = min((ix0 + 4 * h + 3) * STEP, max_x) - ox;
            first_y[h] = min((iy0 + 2 * h) * STEP, max_y) - oy;
            last_y[h] = min((iy0 + 2 * h + 1) * STEP, max_y) - oy;
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            const int nx = nt & 1, ny = nt >> 1;
            const int qx = min((ix0 + 4 * nx + (gq & 3)) * STEP, max_x) - ox + R;
            const int qy = min((iy0 + 2 * ny + (gq >> 2)) * STEP, max_y) - oy + R;
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const uint32_t word =
                        reinterpret_cast<const uint32_t*>(chunks + (c * rows + qy + r) * cp + qx)[t4];
                    const __half2 h = *reinterpret_cast<const __half2*>(&word);
                    const __half2 h2x = __hadd2(h, h);
                    b[nt][8 * c + r] = *reinterpret_cast<const uint32_t*>(&h2x);
                }
#pragma unroll
            for (int e = 0; e < 2; ++e) px[nt][e] = min((ix0 + 4 * nx + (2 * t4 & 3) + e) * STEP, max_x) - ox;
            py[nt] = min((iy0 + 2 * ny + (t4 >> 1)) * STEP, max_y) - oy;
        }

        // ---- round 1: the largest score of every share ----
        float top[4][2];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) top[nt][0] = top[nt][1] = kOutside;
        score_round<C>(a, chunk_addr, sums, tiles, cp, rows, b, px, py, first_x, last_x, first_y, last_y,
                       [&](int nt, int e, int, float s0, float s1) { top[nt][e] = fmaxf(top[nt][e], fmaxf(s0, s1)); });
        __syncthreads();  // the row sums are no longer read; the shares take their place
        float* shares = squares;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int ref = (2 * (nt >> 1) + (t4 >> 1)) * kRefsX + 4 * (nt & 1) + (2 * t4 & 3) + e;
                shares[ref * kShares + warp * 8 + gq] = top[nt][e];
            }
        // the tile's largest sample
        __shared__ float worst_warp[kWarps];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) worst = fmaxf(worst, __shfl_xor_sync(0xffffffffu, worst, o));
        if (lane == 0) worst_warp[warp] = worst;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kWarps; ++w) worst = fmaxf(worst, worst_warp[w]);
        {
            // The eighth largest share of the group's own patch, then the line.
            const int ref = tid >> 3, sub = tid & 7;
            const unsigned mask = 0xFFu << (lane & ~7);
            float own[kShares / 8];
#pragma unroll
            for (int i = 0; i < kShares / 8; ++i) own[i] = shares[ref * kShares + sub * (kShares / 8) + i];
            float eighth = kOutside;
            for (int round = 0; round < 8; ++round) {
                float m = own[0];
#pragma unroll
                for (int i = 1; i < kShares / 8; ++i) m = fmaxf(m, own[i]);
                float all = m;
                all = fmaxf(all, __shfl_xor_sync(mask, all, 1));
                all = fmaxf(all, __shfl_xor_sync(mask, all, 2));
                all = fmaxf(all, __shfl_xor_sync(mask, all, 4));
                eighth = all;
                const unsigned holders = __ballot_sync(mask, m == all) & mask;
                if (lane == __ffs(holders) - 1) {
                    bool taken = false;
#pragma unroll
                    for (int i = 0; i < kShares / 8; ++i) {
                        const bool take = !taken && own[i] == all;
                        taken |= take;
                        if (take) own[i] = kOutside;
                    }
                }
            }
            if (sub == 0) {
                const int qx = min((ix0 + ref % kRefsX) * STEP, max_x) - ox + R;
                const int qy = min((iy0 + ref / kRefsX) * STEP, max_y) - oy + R;
                const float n = 64.0f * C;
                const float reach = 3.0f * n * worst * worst;  // no partial sum is larger
                const float dist = fmaxf(-sums[qy * cp + qx] - eighth, 0.0f);
                // Codes below kExactBelow have whole scores: an allowance under a half keeps to real ties.
                const float fixed = (codes ? 1e-3f : 4.0f) + screen::score_error<C>(reach);
                const float dist1 = dist + fixed;
                // |D - D~| <= 2 sqrt(D) times the norm of the quotients' rounding, 2 * 2^-24 to_code a sample.
                const float quotients = (codes ? 4.0f * screen::kUlp * to_code * sqrtf(n * dist1) : 0.0f) + 1e-5f * dist1;
                // f16 rounds at 2^-11 of the sample, and at 2^-25 near zero.
                const float halves = codes ? 0.0f : 2.0f * sqrtf(n) * (worst * 4.9e-4f + 3e-8f);
                const float slack = 2.0f * (fixed + quotients) + 4.0f * halves * (sqrtf(dist1) + halves);
                line[ref] = fmaxf(eighth - slack, -1e29f);
                even[ref] = dist <= fixed;
            }
        }
        __syncthreads();
        // ---- round 2: list the candidates at or above the line ----
        float bar[4][2];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                bar[nt][e] = line[(2 * (nt >> 1) + (t4 >> 1)) * kRefsX + 4 * (nt & 1) + (2 * t4 & 3) + e];
        score_round<C>(a, chunk_addr, sums, tiles, cp, rows, b, px, py, first_x, last_x, first_y, last_y,
                       [&](int nt, int e, int cell, float s0, float s1) {
                           if (fmaxf(s0, s1) >= bar[nt][e]) {
                               const int ref = (2 * (nt >> 1) + (t4 >> 1)) * kRefsX + 4 * (nt & 1) + (2 * t4 & 3) + e;
                               if (s0 >= bar[nt][e]) {
                                   const int at = atomicAdd(count + ref, 1);
                                   if (at < kList) list[ref * kList + at] = static_cast<uint16_t>(cell);
                                   over |= at >= kList;
                               }
                               if (s1 >= bar[nt][e]) {
                                   const int at = atomicAdd(count + ref, 1);
                                   if (at < kList) list[ref * kList + at] = static_cast<uint16_t>(cell + 8);
                                   over |= at >= kList;
                               }
                           }
                       });
        over = __syncthreads_or(over);
    }

    // ---- the listed candidates in the exact order, one 8-lane group per patch ----
    GroupCtx g;
    g.sub = tid & 7;
    g.mask = 0xFFu << (lane & ~7);
    const int group = tid >> 3;
    const float scale = C == 1 ? 3.0f : 1.5f;
    auto window_of = [&](int ref) {
        return patch_window<C>(a, centre, min((ix0 + ref % kRefsX) * STEP, max_x), min((iy0 + ref / kRefsX) * STEP, max_y),
                               g.sub);
    };
    auto write = [&](int ref, const PatchWindow<C>& p, const TopEight& best) {
        const int ix = ix0 + ref % kRefsX, iy = iy0 + ref / kRefsX;
        write_members(g, a.members + static_cast<size_t>(iy * refs_x + ix) * kMemberWords, best.i, p.left, p.top, p.ww,
                      p.hh, a.k_max);
    };
    if (ix0 + group % kRefsX < refs_x && iy0 + group / kRefsX < refs_y) {
        const PatchWindow<C> p = window_of(group);
        TopEight best;
        best.pin(g, p.self());
        const int listed = bad ? kList + 1 : count[group];
        if (listed <= kList) {
            centre_listed<C, false>(g, p, centre, a.width, listed, scale,
                                    [&](int k) {
                                        const int cell = list[group * kList + k];
                                        return make_uint2(ox - R + (cell & 63), oy - R + (cell >> 6));
                                    },
                                    best);
        } else {
            const int probe = bad || even[group] ? min(static_cast<int>(p.ww * p.hh), kProbe) : 0;
            centre_listed<C, true>(g, p, centre, a.width, probe, scale,
                                   [&](int k) { return make_uint2(p.left + k % p.ww, p.top + k / p.ww); }, best);
        }
        if (listed <= kList || best.settled()) write(group, p, best);
        else if (g.sub == 0) pending[atomicAdd(&npending, 1)] = group;
    }
    if (!over) return;  // the same for the whole CTA

    // ---- the patches left: each window's columns in as many parts as there are groups for it ----
    __syncthreads();
    const int n = npending;
    if (n == 0) return;
    const int parts = min(kRefs / n, kMaxParts), part = group / n;
    struct Member {
        float d;
        uint32_t i;
    };
    Member* found = reinterpret_cast<Member*>(squares);  // [kRefs][8]
    TopEight best;
    if (part < parts) {
        const PatchWindow<C> p = window_of(pending[group % n]);
        best = centre_columns<C>(g, p, centre, a.width, p.ww * part / parts, p.ww * (part + 1) / parts, scale);
        found[group * 8 + g.sub] = Member{best.d, best.i};
    }
    __syncthreads();
    if (part > 0) return;
    for (int q = 1; q < parts; ++q) {
        const Member m = found[(group + q * n) * 8 + g.sub];
        best.take(g, true, m.d, m.i);
    }
    write(pending[group], window_of(pending[group]), best);
}

// One block of a refine rectangle: up to 5 x 5 candidates from (x0, y0), each scored in the exact order.
// `minus` is the lane's anchor column negated. A lane reads a candidate column once for all its candidate
// rows: 60 loads for 25 candidates, where one candidate at a time takes 200 and a group sum of its own
// each. Candidate c of the block is column c / 5, row c % 5; lane `sub` ends with candidates
// 8 b + scattered_candidate(sub), b = 0..2, and lane 0 with candidate 24, in d[b] (kUnfilled outside).
constexpr int kBlk = 5;

template <int C>
__device__ __forceinline__ void score_block(const GroupCtx& g, const float (&minus)[P * C],
                                            const float* __restrict__ frame, int width, uint32_t x0, uint32_t y0,
                                            uint32_t right, uint32_t bottom, float scale, float (&d)[4]) {
    float v[kBlk * kBlk];
    const uint32_t last = bottom + P - 1;  // the last row any candidate reads
#pragma unroll
    for (int q = 0; q < kBlk; ++q) {
        const float* p = frame + static_cast<size_t>(min(x0 + q, right) + g.sub) * C;
        float rows[kBlk + P - 1][C];
#pragma unroll
        for (int r = 0; r < kBlk + P - 1; ++r) {
            const size_t off = static_cast<size_t>(min(y0 + r, last)) * width * C;
#pragma unroll
            for (int c = 0; c < C; ++c) rows[r][c] = __ldg(p + off + c);
        }
#pragma unroll
        for (int k = 0; k < kBlk; ++k) {
            float sum = 0.0f;
#pragma unroll
            for (int r = 0; r < P; ++r)
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    // candidate - anchor: the negated difference has the same square
                    const float diff = __fadd_rn(rows[k + r][c], minus[r * C + c]);
                    sum = __fadd_rn(sum, __fmul_rn(diff, diff));
                }
            v[kBlk * q + k] = sum;
        }
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int c = b < 3 ? 8 * b + scattered_candidate(g.sub) : 24;
        float total;
        if (b < 3) {
            const float part[8] = {v[8 * (b % 3)], v[8 * (b % 3) + 1], v[8 * (b % 3) + 2], v[8 * (b % 3) + 3],
                                   v[8 * (b % 3) + 4], v[8 * (b % 3) + 5], v[8 * (b % 3) + 6], v[8 * (b % 3) + 7]};
            total = reduce_scatter8(g, part) * scale;
        } else {
            total = reduce8(g, v[24]) * scale;
        }
        const uint32_t cx = x0 + c / kBlk, cy = y0 + c % kBlk;
        d[b] = cx <= right && cy <= bottom && (b < 3 || g.sub == 0) ? total : kUnfilled;
    }
}

// The volumes (fused/trajectory.rs, clipped walk): each anchor's walk through the neighbour frames. Per
// frame, the best candidate over one refine rectangle per covering motion block (blocks under c_min
// skipped, rectangles already searched and positions the earlier volumes hold skipped) joins the
// volume's sorted tail; a full grid replaces the members. The reference visits a rectangle row by row
// and keeps the first of equal distances: the least (distance, visiting index) of the candidates not
// skipped, taken if it beats the frame's best so far. Lane `sub` holds grid slot `sub`; the rectangles
// searched so far and the held positions are in the group's shared memory, so the volumes, frames and
// rectangles are loops around one copy of the scoring: 4.67 -> 3.97 ms per 4K luma pass (d = 3), 0.73 ->
// 0.56 at 1080p (d = 2), against one candidate at a time in fully unrolled rectangles. The distances' 600
// unfused f32 operations per rectangle and lane, which must keep their order, bound it; packed f32x2
// takes the pipe as long. Four CTAs per SM: 3.97 ms, five (96 registers, spills) 4.32.
constexpr int kMaxRects = 16;  // four covering blocks per axis

template <int C>
__global__ void __launch_bounds__(kThreads, 4) collab_walk_kernel(CollabLaunch a, int gf) {
    __shared__ uint4 rects[kGroups][kMaxRects];
    __shared__ uint32_t held[kGroups][MAX_K];
    const int lane = threadIdx.x & 31, group = threadIdx.x >> 3;
    GroupCtx g;
    g.sub = threadIdx.x & 7;
    g.mask = 0xFFu << (lane & ~7);
    const uint32_t refs_x = (a.width - P + STEP - 1) / STEP + 1;
    const uint32_t ix = blockIdx.x * kGroups + group;
    if (ix >= refs_x) return;  // the group's 8 lanes leave together; no barrier spans groups
    uint32_t* words = a.members + static_cast<size_t>(blockIdx.y * refs_x + ix) * kMemberWords;
    if ((words[MAX_K] & 0xFFu) != MAX_K) return;  // a smaller group keeps its members
    const uint32_t member = words[g.sub];
    const uint32_t max_x = a.width - P, max_y = a.height - P;
    const float scale = C == 1 ? 3.0f : 1.5f;
    const float* centre = a.ring + static_cast<size_t>(a.centre_slot) * a.frame_elems;
    float grid_d = kUnfilled;
    uint32_t grid_pos = 0;
    for (int first = 0; first < MAX_K; first += gf) {
        const uint32_t anchor_packed = __shfl_sync(g.mask, member, first / gf, 8);
        const uint32_t ax = anchor_packed & 0x1FFFu, ay = (anchor_packed >> 13) & 0x1FFFu;
        if (g.sub == first) {
            grid_pos = anchor_packed;
            grid_d = 0.0f;
        }
        held[group][g.sub] = grid_pos;
        __syncwarp(g.mask);
        float minus[P * C];
#pragma unroll
        for (int r = 0; r < P; ++r)
#pragma unroll
            for (int c = 0; c < C; ++c)
                minus[r * C + c] = -__ldg(centre + ((static_cast<size_t>(ay) + r) * a.width + ax + g.sub) * C + c);
        const uint32_t bx_hi = min(ax / a.blk_step, static_cast<uint32_t>(a.blocks_x - 1));
        const uint32_t by_hi = min(ay / a.blk_step, static_cast<uint32_t>(a.blocks_y - 1));
        const uint32_t bx_lo = min(covering_lo(ax, a.blksize, a.blk_step), bx_hi);
        const uint32_t by_lo = min(covering_lo(ay, a.blksize, a.blk_step), by_hi);
        for (int t = 0; t < 2 * a.radius; ++t) {
            const int slot = static_cast<int>(__ldg(a.neighbour_slots + t));
            const float* frame = a.ring + static_cast<size_t>(slot) * a.frame_elems;
            const uint32_t packed_t = static_cast<uint32_t>(t + 1) << 26;
            float frame_d = kUnfilled;
            uint32_t frame_pos = 0;
            int searched = 0;
            for (uint32_t by = by_lo; by <= by_hi && by < by_lo + 4; ++by)
                for (uint32_t bx = bx_lo; bx <= bx_hi && bx < bx_lo + 4; ++bx) {
                    const uint32_t block = by * a.blocks_x + bx;
                    if (!(__ldg(a.confidence + t * a.conf_stride + block) >= a.c_min)) continue;
                    const int mvx = __ldg(a.mv_field + t * a.mv_stride + block * 2);
                    const int mvy = __ldg(a.mv_field + t * a.mv_stride + block * 2 + 1);
                    const uint32_t left = clamp_top_left(static_cast<int>(ax) + mvx - a.refine, max_x);
                    const uint32_t right = clamp_top_left(static_cast<int>(ax) + mvx + a.refine, max_x);
                    const uint32_t top = clamp_top_left(static_cast<int>(ay) + mvy - a.refine, max_y);
                    const uint32_t bottom = clamp_top_left(static_cast<int>(ay) + mvy + a.refine, max_y);
                    bool contained = false;
                    for (int i = 0; i < searched; ++i) {
                        const uint4 r = rects[group][i];
                        contained |= left >= r.x && right <= r.y && top >= r.z && bottom <= r.w;
                    }
                    if (contained) continue;
                    // The rectangle's best candidate that is not skipped, this lane's share of it first.
                    float best_d = kUnfilled;
                    uint32_t best_key = 0xFFFFFFFFu;  // the visiting order: (row, column)
                    for (uint32_t y0 = top; y0 <= bottom; y0 += kBlk)
                        for (uint32_t x0 = left; x0 <= right; x0 += kBlk) {
                            float d[4];
                            score_block<C>(g, minus, frame, a.width, x0, y0, right, bottom, scale, d);
#pragma unroll
                            for (int b = 0; b < 4; ++b) {
                                const int c = b < 3 ? 8 * b + scattered_candidate(g.sub) : 24;
                                const uint32_t cx = x0 + c / kBlk, cy = y0 + c % kBlk;
                                const uint32_t key = cy << 13 | cx;
                                if (!key_less(d[b], key, best_d, best_key)) continue;
                                bool skip = false;
                                for (int i = 0; i < searched; ++i) {
                                    const uint4 r = rects[group][i];
                                    skip |= cx >= r.x && cx <= r.y && cy >= r.z && cy <= r.w;
                                }
                                for (int k = 0; k < first; ++k) skip |= held[group][k] == (packed_t | key);
                                if (skip) continue;
                                best_d = d[b];
                                best_key = key;
                            }
                        }
                    __syncwarp(g.mask);
#pragma unroll
                    for (int o = 1; o < 8; o <<= 1) {
                        const float other_d = __shfl_xor_sync(g.mask, best_d, o);
                        const uint32_t other_key = __shfl_xor_sync(g.mask, best_key, o);
                        if (key_less(other_d, other_key, best_d, best_key)) {
                            best_d = other_d;
                            best_key = other_key;
                        }
                    }
                    if (best_d < frame_d) {
                        frame_d = best_d;
                        frame_pos = packed_t | best_key;
                    }
                    if (g.sub == 0) rects[group][searched] = make_uint4(left, right, top, bottom);
                    ++searched;
                    __syncwarp(g.mask);
                }
            // Sorted insert into lanes first + 1 .. first + gf - 1, as the reference carries it: what a slot
            // gives up moves on and passes an equal one that is held.
            float carry_d = frame_d;
            uint32_t carry_pos = frame_pos;
            for (int j = first + 1; j < first + gf; ++j) {
                const float held_d = __shfl_sync(g.mask, grid_d, j, 8);
                const uint32_t held_pos = __shfl_sync(g.mask, grid_pos, j, 8);
                if (!(carry_d < held_d)) continue;
                if (g.sub == j) {
                    grid_d = carry_d;
                    grid_pos = carry_pos;
                }
                carry_d = held_d;
                carry_pos = held_pos;
            }
        }
    }
    // Every volume's last slot filled: the grid replaces the members.
    const bool open = (g.sub + 1) % gf == 0 && !(grid_d < kUnfilled);
    if (__ballot_sync(g.mask, open) & g.mask) return;
    words[g.sub] = grid_pos;
    if (g.sub == 0) words[MAX_K] = static_cast<uint32_t>(MAX_K) | 0x100u;
}

template <int C>
cudaError_t launch_centre(const CollabLaunch& a, cudaStream_t stream) {
    const int refs_x = (a.width - P + STEP - 1) / STEP + 1, refs_y = (a.height - P + STEP - 1) / STEP + 1;
    if (a.spatial_radius < 0 || a.spatial_radius > kMaxRadius) return cudaErrorInvalidValue;
    if (cudaError_t e = allow_smem<collab_screen_kernel<C>>(screen_smem<C>(kMaxRadius))) return e;
    const dim3 grid((refs_x + kRefsX - 1) / kRefsX, (refs_y + kRefsY - 1) / kRefsY);
    collab_screen_kernel<C><<<grid, kScreenThreads, screen_smem<C>(a.spatial_radius), stream>>>(a);
    return cudaGetLastError();
}

template <int C>
cudaError_t launch_c(const CollabLaunch& a, cudaStream_t stream) {
    const cudaError_t e = launch_centre<C>(a, stream);
    if (e != cudaSuccess || a.radius == 0 || a.k_max != MAX_K) return e;
    const int refs_x = (a.width - P + STEP - 1) / STEP + 1, refs_y = (a.height - P + STEP - 1) / STEP + 1;
    const dim3 grid((refs_x + kGroups - 1) / kGroups, refs_y);
    collab_walk_kernel<C><<<grid, kThreads, 0, stream>>>(a, a.radius == 1 ? 2 : 4);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_collab_search(const CollabLaunch& a, cudaStream_t stream) {
    return a.channels == 1 ? launch_c<1>(a, stream) : launch_c<2>(a, stream);
}

}  // namespace avd
