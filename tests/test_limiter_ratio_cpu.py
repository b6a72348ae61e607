"""Venkatakrishnan's coefficient from the least ratio (LeastRatio, hcc_stage_impl.cuh) against the minimum over every
slot's own coefficient, bit for bit: the kernel's source compiled for the host, ratios spread, zero, equal up to a few
units of round-off, inside the window around the least one, and products out of range."""
import pathlib
import subprocess

import pytest

SOURCE = pathlib.Path(__file__).resolve().parent.parent / "hypercloudcore.jl_gb300" / "csrc" / "hcc_stage_impl.cuh"
HEAD = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#define __device__
#define __forceinline__ inline
enum { HCC_LIMITER_BJ_SOFT = 1, HCC_LIMITER_BJ_HARD = 2, VK = 3 };
static long long __double_as_longlong(double x) { long long r; std::memcpy(&r, &x, 8); return r; }
static int __double2hiint(double x) { return int(__double_as_longlong(x) >> 32); }
template <class T> T vmin(T x, T y) { return std::isnan(x) || std::isnan(y) ? T(NAN) : (y < x ? y : x); }
template <class T> T vmax(T x, T y) { return std::isnan(x) || std::isnan(y) ? T(NAN) : (y > x ? y : x); }
"""
MAIN = r"""
template <class T> long run(long trials, unsigned seed) {
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> u(0, 1);
    const bool d = sizeof(T) == 8;
    long bad = 0;
    for (long t = 0; t < trials; ++t) {
        const int n = 1 + g() % 40, mode = g() % 6;
        const double base = u(g) * 2.3, scale = mode == 5 ? std::pow(10.0, (d ? -150 : -12) * u(g)) : 1.0;
        T phi = 1, want = 1;
        LeastRatio<T> least;
        for (int k = 0; k < n; ++k) {
            const double r = mode == 0 ? u(g) * 2.01 : mode == 1 ? base * (1 + (int(g() % 9) - 4) * (d ? 1.1e-16 : 6e-8))
                           : mode == 2 ? base * (1 + (u(g) - 0.5) * (d ? 4e-13 : 4e-5)) : mode == 3 ? (g() % 3 ? u(g) : 0.0)
                           : mode == 4 ? std::pow(10.0, -12 * u(g)) : u(g);
            const T rc = T((mode == 1 && g() % 2 ? 0.5 : 0.1 + u(g)) * scale), rm = T(r * rc);
            if (!(rc > 0) || rm >= T(2.01) * rc) continue;
            want = vmin(want, limiter_phi<T>(VK, rm / rc));
            least.add(VK, rm, rc, phi);
        }
        least.finish(VK, phi);
        bad += !(phi == want);
    }
    return bad;
}
int main() { std::printf("%ld %ld\n", run<double>(300000, 1), run<float>(300000, 2)); }
"""


def test_least_ratio_gives_the_least_coefficient(tmp_path):
    text = SOURCE.read_text()
    start = text.index("template <typename T>\n__device__ __forceinline__ T limiter_phi(int lim, T r) {")
    (tmp_path / "t.cpp").write_text(HEAD + text[start:text.index("template <typename T> __device__ __forceinline__ T eps16();")] + MAIN)
    try:
        subprocess.run(["g++", "-O1", "-ffp-contract=off", "-std=c++17", "t.cpp", "-o", "t"], cwd=tmp_path, check=True)
    except FileNotFoundError:
        pytest.skip("no host compiler")
    assert subprocess.run(["./t"], cwd=tmp_path, check=True, capture_output=True, text=True).stdout.split() == ["0", "0"]
