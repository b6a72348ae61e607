"""The buffers a context keeps (csrc/hcc_buffers.h) over an allocator with a limit, compiled for the host: what is reused,
what a smaller cloud gives back, and what is released before a failure is reported."""
import pathlib
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "hypercloudcore.jl_gb300" / "csrc"
MAIN = r"""
#include "hcc_buffers.h"
#include <cstdio>
#include <cstdlib>
#include <map>
static std::map<void *, size_t> live;
static size_t used, limit, allocations;
struct Memory {
    int allocate(void **p, size_t bytes) {
        if (used + bytes > limit) return 2;
        *p = std::malloc(bytes);
        live[*p] = bytes;
        used += bytes;
        ++allocations;
        return 0;
    }
    void release(void *p) {
        if (!live.count(p)) { std::puts("released twice"); std::exit(1); }
        used -= live[p];
        live.erase(p);
        std::free(p);
    }
};
static int bad;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s (used %zu)\n", __LINE__, #x, used); ++bad; } } while (0)
int main() {
    hcc::KeptBuffers<Memory> kept;
    double *state = nullptr;
    int *lists = nullptr;
    float *weights = nullptr;
    auto rebuild = [&](size_t n, size_t slots, size_t spare) {
        kept.begin(0);
        int e = kept.reserve(&state, n, 0, 0);
        kept.begin(1);
        if (!e) e = kept.reserve(&lists, slots, spare, 1);
        kept.begin(2);
        if (!e) e = kept.reserve(&weights, 2 * slots, 2 * spare, 2);
        return e;
    };
    limit = 1000000;
    CHECK(rebuild(1000, 4000, 0) == 0 && used == 13000 && allocations == 3);
    void *before = lists;
    CHECK(rebuild(1000, 3600, 0) == 0 && lists == before && allocations == 3);       // room, and at most a quarter too much
    CHECK(rebuild(1000, 2000, 0) == 0 && used == 7000);                              // far too large: replaced
    CHECK(rebuild(400, 800, 0) == 0 && used == 2800);                                // a smaller cloud gives memory back
    CHECK(rebuild(400, 800, 200) == 0 && used == 2800);
    CHECK(rebuild(400, 900, 200) == 0 && used == 400 + 1100 + 2200);                 // grown with the spare slots
    CHECK(rebuild(400, 850, 200) == 0 && used == 400 + 1100 + 2200);
    // fewer lists, more particles: fits once what is replaced has been released
    CHECK(rebuild(100, 20000, 0) == 0 && used == 60100);
    limit = 61000;
    CHECK(rebuild(50000, 3000, 0) == 0 && used == 59000);
    // the spare slots are wanted, not needed
    limit = 59500;
    CHECK(rebuild(50000, 3100, 5000) == 0 && used == 59300);
    // what does not fit at all: the allocator's error, nothing held for it, and the next cloud is served
    CHECK(rebuild(70000, 10, 0) == 2 && state == nullptr && used == 0);
    CHECK(rebuild(1000, 4000, 0) == 0 && used == 13000);
    // only what is to be rebuilt is given up
    limit = 13500;
    kept.begin(2);
    CHECK(kept.reserve(&weights, 30000, 0, 2) == 2 && weights == nullptr && state && lists && used == 5000);
    std::puts(bad ? "bad" : "ok");
}
"""


def test_kept_buffers(tmp_path):
    (tmp_path / "t.cpp").write_text(MAIN)
    try:
        subprocess.run(["g++", "-O2", "-Wall", "-std=c++17", f"-I{CSRC}", "t.cpp", "-o", "t"], cwd=tmp_path, check=True)
    except FileNotFoundError:
        pytest.skip("no host compiler")
    assert subprocess.run(["./t"], cwd=tmp_path, capture_output=True, text=True).stdout.strip() == "ok"
