"""The error of the NL4D screen's scores (csrc/screen_score.cuh): the tensor-core step and whole scores
against integers, at the extremes of what the codes of every depth can bring. The header is compiled here,
with a kernel that runs its step on given operands."""

import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parent.parent / "av-denoise_b200" / "csrc"

PROGRAM = r"""
#include <cuda_fp16.h>
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <random>
#include <vector>
#include "screen_score.cuh"

using namespace avd::screen;

// Problem p: a[16][16 steps] b[16 steps][8] + c[16][8], `steps` of them in turn, by one warp.
__global__ void run(const __half* A, const __half* B, const float* Cin, float* D, int steps) {
    const int p = blockIdx.x, lane = threadIdx.x, g = lane >> 2, t = lane & 3, K = 16 * steps;
    const __half* a = A + static_cast<size_t>(p) * 16 * K;
    const __half* b = B + static_cast<size_t>(p) * 8 * K;
    auto pack = [](__half x, __half y) {
        __half2 h = __halves2half2(x, y);
        return *reinterpret_cast<uint32_t*>(&h);
    };
    const float* c = Cin + p * 128;
    float d[4] = {c[g * 8 + 2 * t], c[g * 8 + 2 * t + 1], c[(g + 8) * 8 + 2 * t], c[(g + 8) * 8 + 2 * t + 1]};
    for (int s = 0; s < steps; ++s) {
        uint32_t m[4];
        for (int l = 0; l < 4; ++l) {
            const __half* q = a + (g + 8 * (l & 1)) * K + 16 * s + 8 * (l >> 1) + 2 * t;
            m[l] = pack(q[0], q[1]);
        }
        const __half* q = b + (16 * s + 2 * t) * 8 + g;
        mma_f16(d, m, pack(q[0], q[8]), pack(q[64], q[72]), d[0], d[1], d[2], d[3]);
    }
    float* o = D + p * 128;
    o[g * 8 + 2 * t] = d[0];
    o[g * 8 + 2 * t + 1] = d[1];
    o[(g + 8) * 8 + 2 * t] = d[2];
    o[(g + 8) * 8 + 2 * t + 1] = d[3];
}

std::mt19937_64 rng(11);
long uni(long lo, long hi) { return lo + static_cast<long>(rng() % static_cast<uint64_t>(hi - lo + 1)); }
constexpr int kProblems = 1024;

struct Set {
    int steps;
    std::vector<long> a, b;
    std::vector<float> c, d;
    Set(int n, std::function<long(int)> fa, std::function<long(int)> fb, std::function<long()> fc)
        : steps(n), a(kProblems * 256 * n), b(kProblems * 128 * n), c(kProblems * 128), d(kProblems * 128) {
        const int K = 16 * n;
        for (int p = 0; p < kProblems; ++p) {
            for (int i = 0; i < 16 * K; ++i) a[p * 16 * K + i] = fa(i % K);
            for (int i = 0; i < 8 * K; ++i) b[p * 8 * K + i] = fb(i / 8);
        }
        for (float& v : c) v = static_cast<float>(fc());
    }
    bool launch() {
        std::vector<__half> ha(a.size()), hb(b.size());
        for (size_t i = 0; i < a.size(); ++i) ha[i] = __float2half(static_cast<float>(a[i]));
        for (size_t i = 0; i < b.size(); ++i) hb[i] = __float2half(static_cast<float>(b[i]));
        __half *da, *db;
        float *dc, *dd;
        if (cudaMalloc(&da, ha.size() * 2) || cudaMalloc(&db, hb.size() * 2) || cudaMalloc(&dc, c.size() * 4) ||
            cudaMalloc(&dd, d.size() * 4))
            return false;
        cudaMemcpy(da, ha.data(), ha.size() * 2, cudaMemcpyHostToDevice);
        cudaMemcpy(db, hb.data(), hb.size() * 2, cudaMemcpyHostToDevice);
        cudaMemcpy(dc, c.data(), c.size() * 4, cudaMemcpyHostToDevice);
        run<<<kProblems, 32>>>(da, db, dc, dd, steps);
        const bool ok = cudaMemcpy(d.data(), dd, d.size() * 4, cudaMemcpyDeviceToHost) == cudaSuccess;
        cudaFree(da);
        cudaFree(db);
        cudaFree(dc);
        cudaFree(dd);
        return ok;
    }
    // visit(row, column, |error|, largest of accumulator, products and sum, sum of magnitudes)
    void each(std::function<void(int, int, int, double, double, double)> visit) const {
        const int K = 16 * steps;
        for (int p = 0; p < kProblems; ++p)
            for (int i = 0; i < 16; ++i)
                for (int j = 0; j < 8; ++j) {
                    long sum = static_cast<long>(c[p * 128 + i * 8 + j]);
                    double large = std::labs(sum), all = large;
                    for (int k = 0; k < K; ++k) {
                        const long q = a[(p * 16 + i) * K + k] * b[(p * K + k) * 8 + j];
                        sum += q;
                        all += std::labs(q);
                        large = std::max(large, static_cast<double>(std::labs(q)));
                    }
                    large = std::max(large, static_cast<double>(std::labs(sum)));
                    visit(p, i, j, std::fabs(static_cast<double>(d[p * 128 + i * 8 + j]) - static_cast<double>(sum)), large, all);
                }
    }
};

int bad = 0;

// One step: at most kStepError of the largest magnitude, exact while the magnitudes stay below kExactBelow.
void step(const char* name, std::function<long(int)> fa, std::function<long(int)> fb, std::function<long()> fc) {
    Set s(1, fa, fb, fc);
    if (!s.launch()) std::exit(2);
    double worst = 0;
    long inexact = 0;
    s.each([&](int, int, int, double e, double large, double all) {
        if (large > 0) worst = std::max(worst, e / large);
        if (all < kExactBelow && e != 0) ++inexact;
    });
    std::printf("%s: %.2f ulp of the largest magnitude, %ld small sums inexact\n", name, worst / kUlp, inexact);
    if (worst > kStepError || inexact) ++bad;
}

// Whole scores of patches of 64 C samples up to R: 2 sum c n - sum n^2 with n within `spread` of c.
template <int C>
void score(long lo, long hi, long spread) {
    const int K = 64 * C;
    const long R = std::max(std::labs(lo), std::labs(hi));
    Set s(4 * C, [&](int) { return 0l; }, [&](int) { return 0l; }, [] { return 0l; });
    for (int p = 0; p < kProblems; ++p)
        for (int k = 0; k < K; ++k) {
            const long v = uni(lo, hi);
            for (int j = 0; j < 8; ++j) s.b[(p * K + k) * 8 + j] = 2 * std::clamp(v + uni(-spread, spread), lo, hi);
            for (int i = 0; i < 16; ++i) s.a[(p * 16 + i) * K + k] = std::clamp(v + uni(-spread, spread), lo, hi);
        }
    for (int p = 0; p < kProblems; ++p)
        for (int i = 0; i < 16; ++i) {
            long squares = 0;
            for (int k = 0; k < K; ++k) squares += s.a[(p * 16 + i) * K + k] * s.a[(p * 16 + i) * K + k];
            for (int j = 0; j < 8; ++j) s.c[p * 128 + i * 8 + j] = -static_cast<float>(squares);
        }
    if (!s.launch()) std::exit(2);
    const double bound = score_error<C>(3.0f * K * static_cast<float>(R * R));
    double worst = 0;
    s.each([&](int, int, int, double e, double, double) { worst = std::max(worst, e); });
    std::printf("scores of %d samples in %ld..%ld: error %.0f, bound %.0f\n", K, lo, hi, worst, bound);
    if (worst > bound) ++bad;
}

int main() {
    auto none = [](int) { return 1l; };
    auto big = [] { return (rng() & 1 ? 1 : -1) * ((1l << uni(20, 30)) + uni(0, 1 << 20)); };
    step("random codes", [](int) { return uni(-2048, 2048); }, [](int) { return 2 * uni(-2047, 2047); },
         [] { return -uni(0, 1 << 28); });
    step("same sign", [](int) { return uni(2030, 2047); }, [](int) { return 2 * uni(2030, 2047); },
         [] { return -uni(1 << 26, 1 << 28); });
    step("small under a large accumulator", [](int) { return uni(1, 63); }, [](int) { return uni(1, 63); }, big);
    step("middling under a large accumulator", [](int) { return uni(1, 181); }, [](int) { return uni(1, 181); }, big);
    step("ones under a large accumulator", none, none, big);
    step("one large product", [](int k) { return k == 5 ? 2047l : uni(1, 3); },
         [](int k) { return k == 5 ? 4094l : uni(1, 3); }, [] { return uni(-1000, 1000); });
    step("8-bit codes", [](int) { return uni(-255, 255); }, [](int) { return 2 * uni(-255, 255); },
         [] { return -uni(0, 10000000); });
    score<1>(-2048, 2047, 40);
    score<1>(2040, 2047, 2);
    score<2>(-2048, -2040, 2);
    score<2>(-2048, 2047, 400);
    score<1>(-512, 511, 20);
    score<2>(500, 511, 3);
    score<1>(-128, 127, 255);
    score<2>(-128, 127, 255);
    return bad ? 1 : 0;
}
"""


def test_scores_stay_within_the_stated_error(tmp_path):
    src, exe = tmp_path / "score.cu", tmp_path / "score"
    src.write_text(PROGRAM)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", f"-I{CSRC}", str(src),
                    "-ccbin", "/usr/bin/g++", "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    print(done.stdout)
    assert done.returncode == 0, done.stdout + done.stderr
