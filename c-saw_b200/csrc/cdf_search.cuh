// cdf_search.cuh -- per-thread searches of a cached per-vertex prefix through
// its two index levels.  Index arithmetic and loads only, so that a host
// compiler can build it too (with stand-ins for DevGraph, its_target and
// __ldg) and check every read against an array's bounds.
#pragma once

#include <cstdint>

namespace csaw {

// The eight floats of a 32-byte sector.
__device__ __forceinline__ void load_sector(const float *p, float v[8]) {
#ifdef __CUDACC__
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(p));
#else
    for (int i = 0; i < 8; ++i) v[i] = __ldg(p + i);
#endif
}

// First i in [lo, hi) with line[i] > t (line[hi - 1] > t is known and not
// read) of a 32-entry line of a cached prefix or of its index: the last
// entries of the line's first three 32-byte sectors are probed together, then
// the sector found is searched (it is cached by then, but for the fourth).
// Three loads in flight and three short ones after them, where a binary
// search would wait for two or three sectors in turn.
struct LineProbes {
    float p0, p1, p2;
};
__device__ __forceinline__ LineProbes line_probes(const float *line, int lo, int hi) {
    const float none = __int_as_float(0x7f800000);   // at or past the last entry: the answer lies before
    const unsigned n = (unsigned)(hi - 1 - lo);
    LineProbes r;
    r.p0 = 7 < lo ? -none : none;
    r.p1 = 15 < lo ? -none : none;
    r.p2 = 23 < lo ? -none : none;
    if ((unsigned)(7 - lo) < n) r.p0 = __ldg(line + 7);
    if ((unsigned)(15 - lo) < n) r.p1 = __ldg(line + 15);
    if ((unsigned)(23 - lo) < n) r.p2 = __ldg(line + 23);
    return r;
}
__device__ __forceinline__ int line_find(const float *line, const LineProbes &r, int lo, int hi, float t) {
    const int s = (r.p0 <= t ? 8 : 0) + (r.p1 <= t ? 8 : 0) + (r.p2 <= t ? 8 : 0);
    int at = s > lo ? s : lo;
    const int end = s + 7 < hi - 1 ? s + 7 : hi - 1;
#pragma unroll
    for (int step = 4; step >= 1; step >>= 1) {
        const int i = at + step - 1;
        if (i < end && !(__ldg(line + i) > t)) at += step;
    }
    return at;
}

// First i in [0, d) with P[i] > its_target(x, T) for the row [beg, beg + d) of
// a cached prefix, through its two index levels: the row's 1024-edge groups
// in cdf2 (E/1024 floats, L2-resident), the group's 32-edge tiles in cdf1,
// the tile in cdf (each of these one line).  Every probe lies inside the row;
// the last candidate of each level is known to exceed the target (it ends the
// row, or ends the previous level's pick).  Positions are relative to the row
// in 32 bits, and only rows of several groups loop, so lanes on different
// rows stay converged; the first tile line's probes do not wait for T.
__device__ __forceinline__ int cdf_find(const DevGraph &g, int64_t beg, int d, uint32_t x, float T) {
    const int o1 = (int)(beg & 31), o2 = (int)(beg & 1023);   // the row's start in its tile and group
    const int last = d - 1;                                   // row positions and tiles times 32 wrap in 32 bits
    const float *c1 = g.cdf1 + ((beg >> 10) << 5);            // the tiles of the row's first group
    const int kend = (int)(((unsigned)o2 + (unsigned)last) >> 5);                        // its last tile, from there
    int lo = o2 >> 5, hi = kend < 31 ? kend + 1 : 32;
    LineProbes r = line_probes(c1, lo, hi);
    const float t = its_target(x, T);
    int top = (int)(((unsigned)o2 + (unsigned)last) >> 10);
    if (top > 0) {
        const float *c2 = g.cdf2 + (beg >> 10);
        int u = 0;
#pragma unroll 1
        while (u < top) {
            const int mid = (u + top) >> 1;
            if (__ldg(c2 + mid) > t) top = mid; else u = mid + 1;
        }
        if (u > 0) {
            c1 += u << 5;
            lo = 0;
            hi = kend - (u << 5) < 31 ? kend - (u << 5) + 1 : 32;
            r = line_probes(c1, lo, hi);
        }
        top = u;
    }
    const int k = (top << 5) + line_find(c1, r, lo, hi, t) - (o2 >> 5);   // the tile, from the row's first
    const float *line = g.cdf + (beg - o1) + ((uint32_t)k << 5);
    const int e0 = (int)(((uint32_t)k << 5) - (uint32_t)o1);               // its first edge, from the row's
    const int a = e0 < 0 ? -e0 : 0, b = last - e0 < 31 ? last - e0 + 1 : 32;
    return e0 + line_find(line, line_probes(line, a, b), a, b, t);
}

// The row [beg, beg + d) from the start b0 of its first 1024-edge group: its
// first and last edge there.  A row of close to 2^31 edges ends above 2^31
// edges from there, so positions from b0 are unsigned.
struct RowSpan {
    int64_t b0;
    uint32_t o2, last;
};
__device__ __forceinline__ RowSpan row_span(int64_t beg, int d) {
    RowSpan r;
    r.o2 = (uint32_t)beg & 1023u;
    r.last = r.o2 + (uint32_t)d - 1u;
    r.b0 = beg - r.o2;
    return r;
}
// The row's edges [lo, hi) of tile k (32 edges, from b0), and the row position
// of the tile's first edge (below 0 if the row begins inside it).
__device__ __forceinline__ int tile_lo(const RowSpan &r, int k) {
    const uint32_t e0 = (uint32_t)k << 5;
    return r.o2 > e0 ? (int)(r.o2 - e0) : 0;
}
__device__ __forceinline__ int tile_hi(const RowSpan &r, int k) {
    const uint32_t left = r.last - ((uint32_t)k << 5);
    return left < 31u ? (int)left + 1 : 32;
}
__device__ __forceinline__ int tile_at(const RowSpan &r, int k) { return (int)(((uint32_t)k << 5) - r.o2); }

// cdf_find for a row whose prefix may lie in host memory (its index levels
// and its total T are on the device): what counts there is the number of
// 32-byte sectors asked for over the link.  The tile's end values are index
// entries, so the target's place between them says which sector of the tile
// line to ask for first; it decides, or its neighbor does.  One sector and a
// half for uniform weights, where cdf_find asks for three or four and the
// total is one more: R-MAT 24 through a 1 GiB budget, 18.4 -> 14.0 ms.  The
// prefix has to be 32-byte aligned as its edges are numbered (host arrays
// are; a partition's device copy need not be and is searched by cdf_find).
__device__ __forceinline__ int cdf_find_far(const DevGraph &g, int64_t beg, int d, uint32_t x, float T) {
    if ((reinterpret_cast<uintptr_t>(g.cdf) & 31) != 0) return cdf_find(g, beg, d, x, T);
    const float t = its_target(x, T);
    const RowSpan r = row_span(beg, d);
    int u = 0;
    {
        const float *c2 = g.cdf2 + (r.b0 >> 10);
        int top = (int)(r.last >> 10);
#pragma unroll 1
        while (u < top) {
            const int mid = (u + top) >> 1;
            if (__ldg(c2 + mid) > t) top = mid; else u = mid + 1;
        }
    }
    u <<= 5;
    const float *c1 = g.cdf1 + (r.b0 >> 5);
    const int kfirst = (int)(r.o2 >> 5), klast = (int)(r.last >> 5);
    int lo = max(kfirst - u, 0), hi = min(klast - u, 31) + 1;
    const int k = u + line_find(c1 + u, line_probes(c1 + u, lo, hi), lo, hi, t);
    const float vlo = k > kfirst ? __ldg(c1 + k - 1) : 0.f, vhi = k < klast ? __ldg(c1 + k) : T;
    lo = tile_lo(r, k);
    hi = tile_hi(r, k);                                      // the answer lies in [lo, hi)
    const float *line = g.cdf + r.b0 + ((uint32_t)k << 5);
    int at = lo;
    if (vhi > vlo) at += (int)(fminf(fmaxf((t - vlo) / (vhi - vlo), 0.f), 1.f) * (float)(hi - lo));
    at = min(at, hi - 2);
    while (lo < hi - 1) {   // entry hi - 1 is known to exceed t, those before lo not to
        const int s = max(at, lo) & ~7, from = max(lo, s), to = min(hi - 1, s + 8);
        float v[8];
        load_sector(line + s, v);
        int c = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) c += s + i >= from && s + i < to && v[i] <= t ? 1 : 0;
        if (from + c == to) {            // all at or below t
            lo = at = to;
        } else if (c > 0 || from == lo) {
            lo = from + c;
            break;
        } else {                         // the first one read exceeds t: the sector before decides
            hi = from + 1;
            at = from - 1;
        }
    }
    return tile_at(r, k) + lo;
}

}  // namespace csaw
