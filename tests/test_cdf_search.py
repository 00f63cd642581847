"""CPU checks of the device code's searches of a cached prefix
(csrc/cdf_search.cuh, built with a host compiler): the same index as a linear
definition, and no read outside the arrays, for rows at every offset in their
tile, sector and group, of one edge to several groups, with ties, zero edges,
no mass and an infinite total; and for rows of close to 2^31 edges, whose
positions do not fit 32-bit signed arithmetic (the arrays are untouched
zero pages)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <sys/mman.h>
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#define __device__
#define __forceinline__ inline
using std::max;
using std::min;
static inline float __int_as_float(int i) { float f; memcpy(&f, &i, 4); return f; }
static inline int __float_as_int(float f) { int i; memcpy(&i, &f, 4); return i; }
// every read must lie in one of the arrays
static struct { const float *lo, *hi; } spans[3];
static inline float __ldg(const float *p) {
    for (auto &s : spans)
        if (p >= s.lo && p < s.hi) return *p;
    std::printf("read outside the arrays\n");
    std::exit(2);
}
namespace csaw {
struct DevGraph { const float *cdf, *cdf1, *cdf2; };
static inline float its_target(uint32_t x, float T) {
    float t = (float)(x >> 8) * 5.9604644775390625e-8f * T;
    if (!(t < T)) t = __int_as_float(__float_as_int(T) - 1);
    return t;
}
}
#include "cdf_search.cuh"
using namespace csaw;

static uint64_t st = 88172645463325252ull;
static uint32_t rnd() { st ^= st << 13; st ^= st >> 7; st ^= st << 17; return (uint32_t)(st >> 16); }

static float *pages(int64_t n) {   // 32-byte aligned zero pages, touched where written
    void *p = mmap(nullptr, (size_t)n * 4, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (p == MAP_FAILED) { std::printf("mmap\n"); std::exit(3); }
    return (float *)p;
}

static void fail(const char *what, long long beg, long long d, unsigned x, long long got, long long want) {
    std::printf("%s beg %lld d %lld x %u: %lld, expected %lld\n", what, beg, d, x, got, want);
    std::exit(1);
}

static void small_rows() {
    for (int round = 0; round < 400; ++round) {
        const int lead = (int)(rnd() % 2100), d = 1 + (int)(round % 3 == 0 ? rnd() % 70 : rnd() % 6000);
        const int64_t E = lead + d + rnd() % 40, n1 = (E + 31) >> 5, n2 = (E + 1023) >> 10;
        const int64_t Ep = (E + 8) & ~7ll;
        std::vector<float> mem(Ep + 8), c1(n1), c2(n2);
        float *cdf = mem.data();
        while ((uintptr_t)cdf & 31) ++cdf;
        for (int64_t i = 0; i < E; ++i) cdf[i] = (float)(rnd() % 1000);   // other rows' values
        float P = 0.f;
        const int kind = round % 5;   // uniform, many ties, one edge, none, overflow to infinity
        const int one = (int)(rnd() % d);
        for (int i = 0; i < d; ++i) {
            float w = kind == 0 ? 1e-3f + (rnd() % 1000) : kind == 1 ? (float)(rnd() % 20 == 0) : kind == 2 ? (float)(i == one)
                    : kind == 3 ? 0.f : 3e38f;
            P += w;
            cdf[lead + i] = P;
        }
        for (int64_t k = 0; k < n1; ++k) c1[k] = 32 * k + 31 < E ? cdf[32 * k + 31] : 0.f;
        for (int64_t u = 0; u < n2; ++u) c2[u] = 1024 * u + 1023 < E ? cdf[1024 * u + 1023] : 0.f;
        spans[0] = {cdf, cdf + Ep};
        spans[1] = {c1.data(), c1.data() + n1};
        spans[2] = {c2.data(), c2.data() + n2};
        const DevGraph g{cdf, c1.data(), c2.data()};
        const float T = cdf[lead + d - 1];
        for (int q = 0; q < 60; ++q) {
            const uint32_t x = q == 0 ? 0u : q == 1 ? ~0u : rnd() * 2654435761u;
            const float t = its_target(x, T);
            int want = 0;
            while (want < d - 1 && !(cdf[lead + want] > t)) ++want;
            const int a = cdf_find(g, lead, d, x, T), b = cdf_find_far(g, lead, d, x, T);
            if (!(T > 0.f)) {   // callers replace the index: only the reads and its range matter
                if (a < 0 || a >= d || b < 0 || b >= d) fail("no mass", lead, d, x, a, b);
                continue;
            }
            if (a != want) fail("cdf_find", lead, d, x, a, want);
            if (b != want) fail("cdf_find_far", lead, d, x, b, want);
        }
    }
}

static void long_rows() {
    const int64_t E = (1ll << 31) + 4096, n1 = (E + 31) >> 5, n2 = (E + 1023) >> 10;
    float *cdf = pages(E), *c1 = pages(n1), *c2 = pages(n2);
    spans[0] = {cdf, cdf + E};
    spans[1] = {c1, c1 + n1};
    spans[2] = {c2, c2 + n2};
    const DevGraph g{cdf, c1, c2};
    for (int64_t beg : {0ll, 5ll, 31ll, 32ll, 700ll, 1023ll, 1024ll, 1900ll}) {
        for (int64_t d : {(1ll << 31) - 1, (1ll << 31) - 20, (1ll << 31) - 1000, (1ll << 31) - 1100}) {
            // all mass on one edge near the row's end, or its middle
            for (int64_t at : {d - 1, d - 2, d - 33, d - 900, d / 2, (int64_t)0}) {
                const int64_t from = beg + at, to = std::min<int64_t>(beg + d, beg + at + 3000);
                // mass at `at`: the prefix is 0 before, 1 from there to the row's end.  Only the entries a
                // search can meet are written: around `at`, the row's last, and the index entries past it.
                std::vector<int64_t> e1, e2;
                for (int64_t i = from; i < to; ++i) cdf[i] = 1.f;
                for (int64_t i = std::max(from, beg + d - 2000); i < beg + d; ++i) cdf[i] = 1.f;
                for (int64_t u = from >> 10; u <= (beg + d - 1) >> 10; ++u)
                    if (1024 * u + 1023 >= from && 1024 * u + 1023 < beg + d) c2[u] = 1.f, e2.push_back(u);
                for (int64_t k = from >> 5; k <= std::min((beg + d - 1) >> 5, (from >> 5) + 64); ++k)
                    if (32 * k + 31 >= from && 32 * k + 31 < beg + d) c1[k] = 1.f, e1.push_back(k);
                for (uint32_t x : {0u, 0x80000000u, ~0u}) {
                    const int a = cdf_find(g, beg, (int)d, x, 1.f), b = cdf_find_far(g, beg, (int)d, x, 1.f);
                    if (a != at) fail("cdf_find", beg, d, x, a, at);
                    if (b != at) fail("cdf_find_far", beg, d, x, b, at);
                }
                const RowSpan r = row_span(beg, (int)d);
                const int k = (int)((beg + at - r.b0) >> 5);
                const int64_t lo = (int64_t)tile_at(r, k) + tile_lo(r, k), hi = (int64_t)tile_at(r, k) + tile_hi(r, k);
                if (!(lo <= at && at < hi && lo >= 0 && hi <= d)) fail("tile", beg, d, 0, lo, hi);
                for (int64_t i = from; i < to; ++i) cdf[i] = 0.f;
                for (int64_t i = std::max(from, beg + d - 2000); i < beg + d; ++i) cdf[i] = 0.f;
                for (int64_t k2 : e1) c1[k2] = 0.f;
                for (int64_t u : e2) c2[u] = 0.f;
            }
        }
    }
}

int main(int argc, char **argv) {
    if (argc > 1) long_rows(); else small_rows();
    std::printf("ok\n");
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("cdf_search")
    (d / "t.cpp").write_text(SOURCE)
    exe = d / "t"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "c-saw_b200", "csrc"), str(d / "t.cpp"), "-o",
                    str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("which", ["small", "long"])
def test_cached_prefix_searches(program, which):
    r = subprocess.run([program] + ([which] if which == "long" else []), capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
