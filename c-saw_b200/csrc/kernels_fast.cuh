// kernels_fast.cuh -- batched-form level expansion and walk kernels (sm_100a).
//
// Same output as kernels_sample.cuh (the canonical prefix, draw keys and slot
// resolver are shared), scheduled for latency.  On power-law graphs most
// frontier items have d <= N and take every neighbor, so the work is a chain
// of dependent loads, not arithmetic:
//   - queue items carry their own row begin and degree, and every edge has a
//     materialised neighbor record (row begin, degree of col[e]), so a pushed
//     child or a walk's next vertex needs no rowptr round trip;
//   - a warp takes a batch of up to 32 items (lane-parallel loads), reserves
//     output and next-queue space for the whole batch with one atomic each,
//     then expands all take-all items together: lanes stride over the batch's
//     edges, find the owning item by a shuffle binary search over the
//     inclusive prefix of degrees, and issue every column load at once;
//   - items with d > N are selected one at a time by the whole warp: biases,
//     prefix and column ids in registers when d <= 32 (shuffle scans and a
//     5-step shuffle search), biases preloaded into shared memory in batches
//     of 8 tiles when d <= WF, the CTA kernel beyond;
//   - batch size shrinks on small levels so every warp gets work.
#pragma once

#include "kernels_sample.cuh"

namespace csaw {

constexpr int WF = 512;  // per-warp shared prefix capacity of the fast kernels
// Resident CTAs per SM the group kernel is compiled for (register budget).
#ifndef CSAW_GROUP_MIN_BLOCKS
#define CSAW_GROUP_MIN_BLOCKS 6
#endif
// Cached items with N <= 16 and d >= this many times N go to the group pass
// (3: a phase-1 rejection is rare enough that its refill stays cheap; N =
// 17..32, one item a warp, measured slower on the power-law batch, N = 20:
// 0.26 -> 0.34 ms, as few rows are that long and each level pays for the
// pass's launches).
#ifndef CSAW_PAIR_MIN_RATIO
#define CSAW_PAIR_MIN_RATIO 3
#endif

constexpr int FAST_THREADS = 256;

// Canonical prefix of a single tile held one element per lane (w = 0 for
// lanes >= d): identical to warp_canon_prefix for d <= 32.
__device__ __forceinline__ float tile_prefix(float w, int d, int lane) {
    float v = warp_ks_sum(w, lane);
    float p = lane < d ? __fadd_rn(0.f, __fadd_rn(0.f, v)) : 0.f;
    return fmaxf(warp_max_scan(p, lane), 0.f);
}

// First lane whose P exceeds t (P monotone across lanes, P[31] > t).
__device__ __forceinline__ int shfl_search(float P, float t) {
    int lo = 0;
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        float pv = __shfl_sync(FULL, P, lo + s - 1);
        if (!(pv > t)) lo += s;
    }
    return lo;
}

// First lane whose inclusive count exceeds e (incl monotone, incl[31] > e).
__device__ __forceinline__ int shfl_search_int(int incl, int e) {
    int lo = 0;
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        int pv = __shfl_sync(FULL, incl, lo + s - 1);
        if (!(pv > e)) lo += s;
    }
    return lo;
}

__device__ __forceinline__ int warp_incl_scan(int x, int lane) {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        int up = __shfl_up_sync(FULL, x, off);
        if (lane >= off) x += up;
    }
    return x;
}

// Neighbor of edge e with its row begin and degree: one 128-bit record load
// with the neighbor records, else the column and two rowptr loads.
template <typename I>
__device__ __forceinline__ NbrRec edge_rec(const DevGraph &g, int64_t e) {
    if (g.nrec) return load_rec(g.nrec, e);
    NbrRec r;
    r.col = __ldg(g.v.col + e);
    r.beg = row_begin<I>(g, r.col);
    r.deg = (int32_t)(row_begin<I>(g, r.col + 1) - r.beg);
    return r;
}

// Row begin and degree of u = Update(col[e]): the record's when Update kept
// the neighbor, else from rowptr.
template <typename I>
__device__ __forceinline__ void row_of(const DevGraph &g, const NbrRec &r, int32_t u, int64_t &beg, int32_t &deg) {
    if (u == r.col) {
        beg = r.beg;
        deg = r.deg;
    } else {
        beg = row_begin<I>(g, u);
        deg = (int32_t)(row_begin<I>(g, u + 1) - beg);
    }
}

// Loads the biases of edges [beg, beg+d) into W, 8 tiles per round trip.
template <typename I, int BIAS>
__device__ __forceinline__ void preload_bias(const DevGraph &g, int64_t beg, int d, float *W, int lane) {
    for (int i0 = 0; i0 < d; i0 += 256) {
        float r[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            int i = i0 + u * 32 + lane;
            r[u] = i < d ? edge_bias<I, BIAS>(g, beg + i) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            int i = i0 + u * 32 + lane;
            if (i < d) W[i] = r[u];
        }
    }
    __syncwarp();
}

// Speculative resolver of the batched kernels (same result as resolve_slots).
// A rejection phase allows REJECT_ATTEMPTS = 4 draws per slot, and the four
// words of one Philox block are exactly the next four draws of a slot, so
// every pending lane computes the candidates of its next four draws at once
// (four independent searches, overlapped) and a round of rejections costs a
// match and two ballots instead of a search.
struct Spec4 {
    int j = 0;          // warp uniform: current slot
    int a = 1;          // lane: draws its slot has used in this window (cand is draw a - 1)
    int have = 4;       // warp uniform: candidates computed ahead per lane (4, or 1 when lazy)
    int base = 0;       // lane: draw index of the window's first draw (a multiple of 4)
    int sel = -1, cand = -1;
    int c1 = -1, c2 = -1, c3 = -1;
};

// Windows of lanes [from, N): lane `from` starts at draw from_base, later
// lanes at draw 0, all on the current prefix.  Warp-uniform.
// lazy: compute only the first candidate of each window; later ones are
// computed on demand for the rejected slots (where rejections are rare, e.g.
// d >= 4N).
template <typename CandFn>
__device__ __forceinline__ void spec_fill(Spec4 &st, int from, int N, int lane, const DrawCtx &dc, SlotRng &rng,
                                          CandFn cand_of, int from_base, bool lazy) {
    const bool act = lane >= from && lane < N;
    const int base = lane == from ? from_base : 0;
    st.a = 1;
    if (act) st.base = base;
    if (lazy) {
        const uint32_t x0 = act ? rng.word(dc, lane, base) : 0u;
        const int n0 = cand_of(x0, act);
        if (act) st.cand = n0;
        st.have = 1;
        return;
    }
    uint32_t x0 = 0, x1 = 0, x2 = 0, x3 = 0;
    if (act) {
        x0 = rng.word(dc, lane, base);
        x1 = rng.word(dc, lane, base + 1);
        x2 = rng.word(dc, lane, base + 2);
        x3 = rng.word(dc, lane, base + 3);
    }
    const int n0 = cand_of(x0, act), n1 = cand_of(x1, act), n2 = cand_of(x2, act), n3 = cand_of(x3, act);
    if (act) {
        st.cand = n0;
        st.c1 = n1;
        st.c2 = n2;
        st.c3 = n3;
    }
    st.have = 4;
}

__device__ __forceinline__ void fill_smallest(Spec4 &st, int j, int lane) {
    int i = 0;
    while (__ballot_sync(FULL, lane < j && st.sel == i)) ++i;
    if (lane == j) st.sel = i;
}

// 0: all N slots accepted; 1: slot st.j needs a phase rebuild.  Rounds as in
// resolve_slots: every slot whose candidate repeats an accepted selection
// goes on to its next draw in the same round.
template <typename CandFn>
__device__ __forceinline__ int resolve4(Spec4 &st, int N, int lane, const DrawCtx &dc, SlotRng &rng, CandFn cand_of) {
    while (st.j < N) {
        const int j0 = st.j;
        const int v = lane < j0 ? st.sel : (lane < N ? st.cand : -2 - lane);
        const unsigned lower = __match_any_sync(FULL, v) & ((1u << lane) - 1u);
        const bool dup = lane >= j0 && lane < N && lower != 0u;
        const unsigned db = __ballot_sync(FULL, dup);
        const int f = db ? __ffs(db) - 1 : N;
        if (lane >= j0 && lane < f) st.sel = v;
        st.j = f;
        if (f == N) return 0;
        if (__shfl_sync(FULL, st.base + st.a, f) == MAX_SLOT_DRAWS) {
            fill_smallest(st, f, lane);
            st.j = f + 1;
            continue;
        }
        const bool again = dup && (lower & ((1u << f) - 1u)) != 0u && st.a < REJECT_ATTEMPTS;
        if (!((__ballot_sync(FULL, again) >> f) & 1u)) return 1;   // slot f's window ran out
        if (st.have == 4) {
            if (again) st.cand = st.a == 1 ? st.c1 : (st.a == 2 ? st.c2 : st.c3);
        } else {   // lazy windows: the next draws of the rejected slots
            const uint32_t x = again ? rng.word(dc, lane, st.base + st.a) : 0u;
            const int nc = cand_of(x, again);
            if (again) st.cand = nc;
        }
        if (again) st.a++;
    }
    return 0;
}

// Generic driver: cand_of(x, act) maps a draw word to a candidate (warp-
// uniform call); rebuild(st, j) zeroes the selections of slots < j out of the
// prefix and returns false when no positive mass is left.
// j0 > 0 resumes an item whose first phase failed at slot j0 (lane m < j0
// passes its accepted index in sel0): slot j0 has used its draws
// 0..REJECT_ATTEMPTS-1, so the run goes on exactly as it would after that
// phase -- rebuild without the j0 selections, slot j0 from draw
// REJECT_ATTEMPTS, later slots from draw 0.
template <typename CandFn, typename RebuildFn>
__device__ __forceinline__ int select_spec(int N, int lane, const DrawCtx &dc, bool zero, CandFn cand_of,
                                           RebuildFn rebuild, bool lazy = false, int j0 = 0, int sel0 = -1) {
    SlotRng rng;
    Spec4 st;
    bool again = j0 > 0;   // a phase failed: rebuild without the selections so far
    int from = again ? j0 : 0, base = again ? REJECT_ATTEMPTS : 0;
    if (again) st.sel = lane < j0 ? sel0 : -1;
    st.j = from;
    for (;;) {
        if (again && !rebuild(st, from)) zero = true;
        if (zero) {
            for (int jj = from; jj < N; ++jj) fill_smallest(st, jj, lane);
            break;
        }
        spec_fill(st, from, N, lane, dc, rng, cand_of, base, lazy);
        if (resolve4(st, N, lane, dc, rng, cand_of) == 0) break;
        from = st.j;
        base = __shfl_sync(FULL, st.base, from) + REJECT_ATTEMPTS;
        again = true;
    }
    return st.sel;
}

// Selection for N < d <= 32 entirely in registers.
template <typename I, int BIAS>
__device__ __forceinline__ int select_reg(const DevGraph &g, int64_t beg, int d, int N, const DrawCtx &dc,
                                          int lane) {
    const float w = lane < d ? edge_bias<I, BIAS>(g, beg + lane) : 0.f;
    float P = tile_prefix(w, d, lane);
    float T = __shfl_sync(FULL, P, 31);
    auto cand_of = [&](uint32_t x, bool act) -> int {
        const float t = act ? its_target(x, T) : 0.f;
        return shfl_search(P, t);
    };
    auto rebuild = [&](const Spec4 &st, int j) -> bool {
        const unsigned zm = __reduce_or_sync(FULL, lane < j ? (1u << st.sel) : 0u);
        P = tile_prefix(((zm >> lane) & 1u) ? 0.f : w, d, lane);
        T = __shfl_sync(FULL, P, 31);
        return T > 0.f;
    };
    return select_spec(N, lane, dc, !(T > 0.f), cand_of, rebuild);
}

// Selection for 32 < d with the canonical prefix in P (shared or a cached
// CDF); W holds the raw biases for rebuilds (shared), zb a rebuild bitmap.
__device__ __forceinline__ int select_smem(const float *W, int d, int N, const DrawCtx &dc, float *P,
                                           uint32_t *zb, int lane) {
    auto wfn = [&](int64_t i) { return W[i]; };
    float T = warp_canon_prefix(wfn, d, P, nullptr, lane);
    auto cand_of = [&](uint32_t x, bool act) -> int {
        return act ? search_upper32(P, d, its_target(x, T)) : -1;
    };
    auto rebuild = [&](const Spec4 &st, int j) -> bool {
        const int nwords = (d + 31) >> 5;
        for (int w = lane; w < nwords; w += 32) zb[w] = 0u;
        __syncwarp();
        if (lane < j) atomicOr(&zb[st.sel >> 5], 1u << (st.sel & 31));
        __syncwarp();
        T = warp_canon_prefix(wfn, d, P, zb, lane);
        return T > 0.f;
    };
    return select_spec(N, lane, dc, !(T > 0.f), cand_of, rebuild, d >= 4 * N);
}

// Selection for 32 < d <= WF from the cached canonical prefix: the row's
// prefix is copied to shared P (one coalesced pass, no scan); a rebuild reads
// the raw biases from global memory.  Same draws and result as select_smem,
// since the cache holds exactly the prefix it would compute.
template <typename I, int BIAS>
__device__ __forceinline__ int select_cached(const DevGraph &g, int64_t beg, int d, int N, const DrawCtx &dc,
                                             float *P, uint32_t *zb, int lane, int j0 = 0, int sel0 = -1) {
    const float *cp = g.cdf + beg;
    const bool lazy = d >= 4 * N;
    // a row of few edges per slot needs rebuilds: its raw biases come to L2
    // while the first phase runs
    if constexpr (BIAS == CSAW_BIAS_EDGE_WEIGHT || BIAS == CSAW_BIAS_DEGREE) {
        constexpr int PER_LINE = BIAS == CSAW_BIAS_EDGE_WEIGHT ? 32 : 8;
        if (!lazy && lane * PER_LINE < d) {
            const void *at = BIAS == CSAW_BIAS_EDGE_WEIGHT ? (const void *)(g.v.weight + beg + lane * PER_LINE)
                                                           : (const void *)(g.nrec + beg + lane * PER_LINE);
            if (BIAS == CSAW_BIAS_EDGE_WEIGHT || g.nrec) asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
        }
    }
    // a resumed item (j0 > 0) starts with a rebuild, which writes all of P
    for (int i0 = 0; i0 < (j0 > 0 ? 0 : d); i0 += 256) {
        float r[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = i0 + u * 32 + lane;
            r[u] = i < d ? __ldg(cp + i) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = i0 + u * 32 + lane;
            if (i < d) P[i] = r[u];
        }
    }
    __syncwarp();
    float T = j0 > 0 ? 1.f : P[d - 1];
    auto cand_of = [&](uint32_t x, bool act) -> int {
        return act ? search_upper32(P, d, its_target(x, T)) : -1;
    };
    auto rebuild = [&](const Spec4 &st, int j) -> bool {
        const int nwords = (d + 31) >> 5;
        for (int w = lane; w < nwords; w += 32) zb[w] = 0u;
        __syncwarp();
        if (lane < j) atomicOr(&zb[st.sel >> 5], 1u << (st.sel & 31));
        __syncwarp();
        auto wfn = [&](int64_t i) { return edge_bias<I, BIAS>(g, beg + i); };
        T = warp_canon_prefix(wfn, d, P, zb, lane);
        return T > 0.f;
    };
    return select_spec(N, lane, dc, !(T > 0.f), cand_of, rebuild, lazy, j0, sel0);
}

// Unbiased selection (no prefix): index ranks over the non-excluded range.
__device__ __forceinline__ int select_unbiased(int64_t d, int N, const DrawCtx &dc, int *zs, int lane) {
    int nZ = 0;
    auto cand_of = [&](uint32_t x, bool act) -> int {
        return act ? kth_not_excluded(mulhi(x, (uint32_t)(d - nZ)), zs, nZ) : -1;
    };
    auto rebuild = [&](const Spec4 &st, int j) -> bool {
        int rank = 0;
        for (int m = 0; m < j; ++m) {
            const int sm = __shfl_sync(FULL, st.sel, m);
            if (sm < st.sel) ++rank;
        }
        __syncwarp();
        if (lane < j) zs[rank] = st.sel;
        __syncwarp();
        nZ = j;
        return true;
    };
    return select_spec(N, lane, dc, false, cand_of, rebuild);
}

// Seeds -> level-0 queue with row begin and degree.
template <typename I>
__global__ void k_init_queue_fast(DevGraph g, const int32_t *seeds, uint32_t n, int F, int s0, int32_t *qv,
                                  int32_t *qs, uint32_t *qp, I *qb, int32_t *qd, uint32_t *qn, int *err) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *qn = n;
    if (i >= n) return;
    int32_t v = seeds[i];
    if (v < 0 || v >= g.v.n_vertices) {
        atomicOr(err, ERR_SEED_RANGE);
        v = 0;
    }
    const int64_t b = row_begin<I>(g, v);
    qv[i] = v;
    qs[i] = s0 + (int32_t)(i / (uint32_t)F);
    qp[i] = i % (uint32_t)F;
    qb[i] = (I)b;
    qd[i] = (int32_t)(row_begin<I>(g, v + 1) - b);
}

// Emitting an edge: emit_load reads the selected neighbor (its record on
// inner levels), emit_finish writes the output edge and, on inner levels,
// the child queue item; emit_edge does both.
template <typename I>
__device__ __forceinline__ NbrRec emit_load(const DevGraph &g, const LevelArgs &a, int64_t e) {
    NbrRec r;
    if (a.push) r = edge_rec<I>(g, e);   // the child's adjacency range comes with it
    else r.col = __ldg(g.v.col + e);     // last level: the column alone (4-byte stride over a row)
    return r;
}

// The stores of an emitted edge whose neighbor (record) r was loaded by emit_load.
template <typename I>
__device__ __forceinline__ void emit_finish(const DevGraph &g, const LevelArgs &a, const NbrRec &r, int32_t v,
                                            int32_t s, uint32_t child_p, int64_t pos, uint32_t q) {
    int32_t dst = Update(&g.v, r.col, v);
    if (dst < 0 || dst >= g.v.n_vertices) {
        atomicOr(a.err, ERR_UPDATE_RANGE);
        dst = 0;
    }
    if (pos < a.cap) {
        a.o_src[pos] = v;
        a.o_dst[pos] = dst;
        if (a.o_smp) a.o_smp[pos] = s;
        if (a.o_dep) a.o_dep[pos] = a.depth;
    }
    if (a.push) {
        int64_t nb;
        int32_t nd;
        row_of<I>(g, r, dst, nb, nd);
        a.out_v[q] = dst;
        a.out_s[q] = s;
        a.out_p[q] = child_p;
        ((I *)a.out_beg)[q] = (I)nb;
        a.out_deg[q] = nd;
    }
}

template <typename I>
__device__ __forceinline__ void emit_edge(const DevGraph &g, const LevelArgs &a, int64_t e, int32_t v, int32_t s,
                                          uint32_t child_p, int64_t pos, uint32_t q) {
    emit_finish<I>(g, a, emit_load<I>(g, a, e), v, s, child_p, pos, q);
}

// Level expansion, part 1 (every item): batches of up to 32 items per warp,
// output and next-queue slots reserved for the whole batch, take-all items
// (d <= N) expanded cooperatively, items needing a draw appended with their
// reserved slots to the warp list (or the CTA list when biased and d > WF).
template <typename I, int BIAS>
__device__ __forceinline__ void coop_body(const DevGraph &g, const LevelArgs &a) {
    constexpr bool BIASED = BIAS != CSAW_BIAS_UNBIASED;
    constexpr int NW = FAST_THREADS / 32;
    // per reservation (output, next queue, warp, thread, group and hub list,
    // four CTA lists): each warp's count, then its range's start
    __shared__ uint32_t s_cnt[9][NW], s_at[9][NW];
    __shared__ unsigned long long s_ob[NW];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const uint32_t n = __ldcg(a.n_in);
    const int N = a.N;
    const bool cached = BIASED && g.cdf && g.cdf_bias == BIAS;
    const bool routed = BIASED && a.sched && a.sched->mode != SCHED_THRESHOLD;
    const bool thr_ok = BIASED && a.thread_list != nullptr;
    const int nout = 2 + (a.o_smp != nullptr) + (a.o_dep != nullptr);
    const unsigned long long per_edge = 4ull + 4ull * nout + (a.push ? 12ull + 2 * (sizeof(I) + 4) : 0ull);
    uint32_t bs = (n + nw - 1) / nw;
    bs = bs < 1 ? 1 : (bs > 32 ? 32 : bs);
    unsigned long long my_bytes = 0, my_items = 0;
    for (uint32_t cta = blockIdx.x * NW * bs; cta < n; cta += nw * bs) {
        const uint32_t it = cta + wib * bs + lane;
        const bool valid = lane < (int)bs && it < n;
        int32_t v = 0, s = 0;
        uint32_t p = 0;
        int64_t beg = 0, d = 0;
        if (valid) {
            v = __ldcg(a.in_v + it);
            s = __ldcg(a.in_s + it);
            p = __ldcg(a.in_p + it);
            beg = (int64_t)__ldcg((const I *)a.in_beg + it);
            d = __ldcg(a.in_deg + it);
        }
        const int k = (valid && d > 0) ? (int)(d < N ? d : N) : 0;
        const bool drawn = k > 0 && d > N;
        // execution class of items that need draws: degree rule, or learned
        int cls = 1;
        if (drawn && BIASED) cls = rule_class(d, N, n, WF, cached, thr_ok, a.thread_force);
        if (routed && a.sched_tab) {   // trained model: one table load per item
            if (drawn) cls = table_class(a.sched_tab, d, a.sched->vstats[v], N, WF, cached);
        } else if (routed) {
            float2 st = make_float2(0.f, 0.f);
            if (drawn) st = a.sched->vstats[v];
            unsigned dm = __ballot_sync(FULL, drawn);
            while (dm) {
                const int b = __ffs(dm) - 1;
                dm &= dm - 1;
                const int64_t db = __shfl_sync(FULL, d, b);
                const float2 sb = make_float2(__shfl_sync(FULL, st.x, b), __shfl_sync(FULL, st.y, b));
                uint32_t hb = (uint32_t)__shfl_sync(FULL, s, b) * 0x9E3779B1u ^ __shfl_sync(FULL, p, b) * 0x85EBCA77u ^
                              (uint32_t)a.depth * 0xC2B2AE3Du ^ a.k0;
                hb ^= hb >> 15;
                hb *= 0x2C1B3C6Du;
                hb ^= hb >> 13;
                const int c = choose_class(a.sched, a.sched->wq, db, N, sb, n, a.depth, hb, WF, cached, thr_ok, lane);
                if (lane == b) cls = c;
            }
        }
        // thread class: one item per thread (valid only with a thread list)
        const bool thr = drawn && cls == CLS_THREAD;
        const bool heavy = drawn && cls >= 2 && !thr;
        // cached items with few slots and a rare rebuild run 32 / N per warp;
        // other warp-class items above WF search the cached prefix in their own list
        const bool pair = drawn && !heavy && !thr && cached && N <= 16 && d >= CSAW_PAIR_MIN_RATIO * N && a.pair_list;
        const bool hub = drawn && !heavy && !thr && cached && d > WF && !pair;
        const int incl = warp_incl_scan(k, lane);
        const int excl = incl - k;
        const int K = __shfl_sync(FULL, incl, 31);
        // Items that need draws go to one list each, with their reserved
        // slots.  The CTA reserves its warps' output and queue slots and their
        // ranges in every list together, a counter a thread: every warp of the
        // GPU adds to the same few words, and an add per warp and counter was
        // half of the pass's time.
        const bool to_sel = drawn && !heavy && !hub && !pair && !thr;
        const unsigned sm = __ballot_sync(FULL, to_sel);
        const unsigned tm = __ballot_sync(FULL, thr);
        const unsigned pbm = __ballot_sync(FULL, pair);
        const unsigned hbm = __ballot_sync(FULL, hub);
        unsigned cm[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) cm[c] = __ballot_sync(FULL, heavy && cls == 2 + c);
        if (lane == 0) {
            s_cnt[0][wib] = (uint32_t)K;
            s_cnt[1][wib] = (uint32_t)__popc(sm);
            s_cnt[2][wib] = (uint32_t)__popc(tm);
            s_cnt[3][wib] = (uint32_t)__popc(pbm);
            s_cnt[4][wib] = (uint32_t)__popc(hbm);
#pragma unroll
            for (int c = 0; c < 4; ++c) s_cnt[5 + c][wib] = (uint32_t)__popc(cm[c]);
        }
        __syncthreads();
        if (threadIdx.x < 10) {   // 0: the output; 1..8: the lists; 9: the next queue
            const int k9 = threadIdx.x == 9 ? 0 : threadIdx.x;
            uint32_t tot = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) tot += s_cnt[k9][w];
            if (threadIdx.x == 0) {
                unsigned long long at = tot ? atomicAdd(a.o_count, (unsigned long long)tot) : 0ull;
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    s_ob[w] = at;
                    at += s_cnt[0][w];
                }
            } else {
                uint32_t *ctr = threadIdx.x == 1   ? a.n_sel
                                : threadIdx.x == 2 ? a.n_thread
                                : threadIdx.x == 3 ? a.n_pair
                                : threadIdx.x == 4 ? a.n_hub
                                : threadIdx.x == 9 ? a.n_out
                                                   : a.n_cta + (threadIdx.x - 5);
                uint32_t at = tot && (threadIdx.x != 9 || a.push) ? atomicAdd(ctr, tot) : 0u;
                uint32_t *to = threadIdx.x == 9 ? s_at[0] : s_at[threadIdx.x];
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    to[w] = at;
                    at += s_cnt[k9][w];
                }
            }
        }
        __syncthreads();
        const unsigned long long ob = s_ob[wib];
        const uint32_t qb = s_at[0][wib];
        const unsigned below = (1u << lane) - 1u;
        const SelEntry en{it, qb + (uint32_t)excl, ob + excl, v, s, p, (int32_t)d, (long long)beg, cls, 0};
        {
            if (to_sel) {
                a.sel_list[s_at[1][wib] + __popc(sm & below)] = en;
            } else if (thr) {
                a.thread_list[s_at[2][wib] + __popc(tm & below)] = en;
            } else if (pair) {
                a.pair_list[s_at[3][wib] + __popc(pbm & below)] = en;
            } else if (hub) {
                a.hub_list[s_at[4][wib] + __popc(hbm & below)] = en;
            } else if (heavy) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (cls == 2 + c) a.cta_list[c][s_at[5 + c][wib] + __popc(cm[c] & below)] = en;
            }
        }
        if (valid) {
            my_items++;
            my_bytes += 12 + sizeof(I) + 4 + (k > 0 && d <= N ? per_edge * k : 0ull);
        }
        // take-all items: all lanes stride over their edges together
        const int ks = (k > 0 && d <= N) ? k : 0;
        const int incl_s = warp_incl_scan(ks, lane);
        const int Ks = __shfl_sync(FULL, incl_s, 31);
        for (int e0 = 0; e0 < Ks; e0 += 32) {
            const int e = e0 + lane;
            const bool act = e < Ks;
            const int b = shfl_search_int(incl_s, act ? e : 0);
            const int32_t vb = __shfl_sync(FULL, v, b);
            const int32_t sb = __shfl_sync(FULL, s, b);
            const uint32_t pb = __shfl_sync(FULL, p, b);
            const int64_t begb = __shfl_sync(FULL, beg, b);
            const int exb = __shfl_sync(FULL, excl, b);
            const int j = e - (__shfl_sync(FULL, incl_s, b) - __shfl_sync(FULL, ks, b));
            if (act)
                emit_edge<I>(g, a, begb + j, vb, sb, pb * (uint32_t)N + (uint32_t)j, (int64_t)ob + exb + j,
                             qb + (uint32_t)(exb + j));
        }
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        my_bytes += __shfl_xor_sync(FULL, my_bytes, off);
        my_items += __shfl_xor_sync(FULL, my_items, off);
    }
    if (lane == 0 && my_items) {
        atomicAdd(&a.bytes[0], my_bytes);
        atomicAdd(&a.items[0], my_items);
    }
}

template <typename I, int BIAS>
__global__ void __launch_bounds__(FAST_THREADS)
k_coop_fast(DevGraph g, LevelArgs a) {
    coop_body<I, BIAS>(g, a);
}

// Level expansion, part 2: one warp per listed item (N < d <= WF when
// biased); writes into the slots reserved by part 1.  CACHED: the graph holds
// the prefix cache for BIAS, so no shared copy of the raw biases is kept
// (half the shared memory, more resident warps).
template <typename I, int BIAS, bool CACHED>
__device__ __forceinline__ void select_fast_body(const DevGraph &g, const LevelArgs &a) {
    constexpr bool BIASED = BIAS != CSAW_BIAS_UNBIASED;
    constexpr int NW = FAST_THREADS / 32;
    __shared__ float s_W[BIASED && !CACHED ? NW * WF : 1];
    __shared__ float s_P[BIASED ? NW * WF : 1];
    __shared__ uint32_t s_z[BIASED ? NW * (WF / 32) : 1];
    __shared__ int s_zs[NW * 32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    float *W = s_W + (BIASED && !CACHED ? wib * WF : 0);
    float *P = s_P + (BIASED ? wib * WF : 0);
    uint32_t *zb = s_z + (BIASED ? wib * (WF / 32) : 0);
    int *zs = s_zs + wib * 32;
    const uint32_t n = __ldcg(a.n_sel);
    const uint32_t n_level = __ldcg(a.n_in);
    const int N = a.N;
    constexpr bool cached = BIASED && CACHED;
    const int nout = 2 + (a.o_smp != nullptr) + (a.o_dep != nullptr);
    unsigned long long my_bytes = 0, my_items = 0;
    for (uint32_t i = gw; i < n; i += nw) {
        const SelEntry en = load_sel(a.sel_list + i);
        const int32_t v = en.v, s = en.s;
        const uint32_t p = en.p;
        const int64_t beg = en.beg, d = en.d;
        const DrawCtx dc{a.k0, a.k1, p, (uint32_t)s, (uint32_t)a.depth};
        const bool rec = a.sched && a.sched->mode == SCHED_RECORD;
        long long t0 = 0;
        if (rec) t0 = clock64();
        int sel;
        if constexpr (!BIASED) {
            sel = select_unbiased(d, N, dc, zs, lane);
        } else {
            if (en.cls == 0) {
                sel = select_reg<I, BIAS>(g, beg, (int)d, N, dc, lane);
            } else if constexpr (CACHED) {
                if (d <= WF) {
                    // a pair item whose first phase failed (en.pad = its pair
                    // index + 1): its failing slot and accepted indices wait
                    // in the consumed pair entry
                    int j0 = 0, sel0 = -1;
                    if (en.pad > 0 && a.pair_list) {
                        const uint16_t *ps = reinterpret_cast<const uint16_t *>(a.pair_list + (en.pad - 1));
                        j0 = __ldcg(ps);
                        if (j0 >= N) j0 = 0;
                        if (lane < j0) sel0 = __ldcg(ps + 1 + lane);
                    }
                    sel = select_cached<I, BIAS>(g, beg, (int)d, N, dc, P, zb, lane, j0, sel0);
                } else {   // hubs are listed for k_select_hub; kept for completeness
                    sel = select_warp<I, BIAS>(g, beg, d, N, dc, P, zb, zs, lane, WF);
                    if (sel == -2) {   // needs a rebuild that does not fit: retried by the CTA pass
                        if (lane == 0) a.retry_list[atomicAdd(a.n_retry, 1u)] = en;
                        continue;
                    }
                }
            } else {
                preload_bias<I, BIAS>(g, beg, (int)d, W, lane);
                sel = select_smem(W, (int)d, N, dc, P, zb, lane);
            }
        }
        if (lane < N)
            emit_edge<I>(g, a, beg + sel, v, s, p * (uint32_t)N + (uint32_t)lane, (int64_t)en.ob + lane,
                         en.q + (uint32_t)lane);
        if (rec) {
            __syncwarp();
            if (lane == 0) record_profile(a.sched, d, N, a.sched->vstats[v], n_level, a.depth, en.cls, clock64() - t0);
        }
        if (lane == 0) {
            my_items++;
            my_bytes += 16 + (BIASED && !(cached && d > WF) ? 4ull * d : 0ull) +   // weights, or cached prefix row
                        (unsigned long long)N * (4ull + 4ull * nout + (a.push ? 12ull + 2 * (sizeof(I) + 4) : 0ull));
        }
    }
    if (lane == 0 && my_items) {
        atomicAdd(&a.bytes[5], my_bytes);
        atomicAdd(&a.items[5], my_items);
    }
}

template <typename I, int BIAS, bool CACHED>
__global__ void __launch_bounds__(FAST_THREADS, 4)
k_select_fast(DevGraph g, LevelArgs a) {
    select_fast_body<I, BIAS, CACHED>(g, a);
}

// ------------------------------------------------ thread-per-item selection
// One thread runs one item with N < d <= 32 (biased) through the whole
// selection, serially in slot order, exactly as the semantics define it:
// the row's canonical prefix lives in 32 registers (the same Kogge-Stone
// additions and running max as the warp's tile scan, so the same bits), a
// draw's index is the number of prefix values <= t (the prefix is monotone),
// selected indices are a 32-bit mask, a slot that has drawn REJECT_ATTEMPTS
// times in a phase rebuilds the prefix with the selected neighbors zeroed,
// and zero mass or MAX_SLOT_DRAWS takes the smallest unselected index.  The
// slots' indices go to shared memory and the edges are emitted afterwards,
// four slots at a time, so an item's neighbor gathers are in flight together
// instead of one per slot.  A warp thus carries 32 items instead of one.

constexpr int THREAD_SEL_SLOTS = 32;   // N < d <= 32

// Canonical prefix of the (at most 32) biases of row [beg, beg + d), the
// neighbors in zmask counted as zero; returns T.
template <typename I, int BIAS>
__device__ __forceinline__ float thread_tile_prefix(const DevGraph &g, int64_t beg, int d, uint32_t zmask,
                                                    float (&P)[32]) {
#pragma unroll
    for (int i = 0; i < 32; ++i) P[i] = (i < d && !((zmask >> i) & 1u)) ? edge_bias<I, BIAS>(g, beg + i) : 0.f;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
#pragma unroll
        for (int i = 31; i >= off; --i) P[i] = __fadd_rn(P[i], P[i - off]);
    }
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const float pi = i < d ? __fadd_rn(0.f, __fadd_rn(0.f, P[i])) : 0.f;
        m = fmaxf(m, pi);
        P[i] = m;
    }
    return P[31];
}

// Selects the item's N slots; slot j's neighbor index goes to sidx[j * stride].
template <typename I, int BIAS>
__device__ __forceinline__ void select_thread_item(const DevGraph &g, const LevelArgs &a, const SelEntry &en, int N,
                                                   uint8_t *sidx, int stride) {
    const int64_t beg = en.beg;
    const int d = en.d;
    const DrawCtx dc{a.k0, a.k1, en.p, (uint32_t)en.s, (uint32_t)a.depth};
    float P[32];
    float T = thread_tile_prefix<I, BIAS>(g, beg, d, 0u, P);
    uint32_t selmask = 0;
    for (int j = 0; j < N; ++j) {
        SlotRng rng;
        int A = 0, ph = 0, idx = 0;
        for (;;) {
            if (!(T > 0.f) || A == MAX_SLOT_DRAWS) {   // no mass left, or the slot's draw guard
                idx = __ffs(~selmask) - 1;
                break;
            }
            if (ph == REJECT_ATTEMPTS) {   // new phase: the selected neighbors zeroed out of the prefix
                T = thread_tile_prefix<I, BIAS>(g, beg, d, selmask, P);
                ph = 0;
                continue;
            }
            const float t = its_target(rng.word(dc, j, A), T);
            ++A;
            ++ph;
            idx = 0;
#pragma unroll
            for (int i = 0; i < 32; ++i) idx += P[i] <= t ? 1 : 0;
            if (!((selmask >> idx) & 1u)) break;
        }
        selmask |= 1u << idx;
        sidx[j * stride] = (uint8_t)idx;
    }
}

#ifndef CSAW_THREAD_SEL_MIN_BLOCKS
#define CSAW_THREAD_SEL_MIN_BLOCKS 3
#endif

template <typename I, int BIAS>
__device__ __forceinline__ void select_thread_body(const DevGraph &g, const LevelArgs &a) {
    __shared__ uint8_t s_idx[THREAD_SEL_SLOTS * FAST_THREADS];   // [slot][thread]
    const int lane = threadIdx.x & 31;
    const uint32_t n = __ldcg(a.n_thread);
    const uint32_t n_level = __ldcg(a.n_in);
    const int N = a.N;
    const int nout = 2 + (a.o_smp != nullptr) + (a.o_dep != nullptr);
    const bool rec = a.sched && a.sched->mode == SCHED_RECORD;
    uint8_t *sidx = s_idx + threadIdx.x;
    unsigned long long my_bytes = 0, my_items = 0;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        long long t0 = 0;
        if (rec) t0 = clock64();
        select_thread_item<I, BIAS>(g, a, load_sel(a.thread_list + i), N, sidx, FAST_THREADS);
        // the entry again (an L1/L2 hit): its emission fields stay out of the
        // selection loop's registers
        const SelEntry en = load_sel(a.thread_list + i);
        for (int j0 = 0; j0 < N; j0 += 4) {
            NbrRec r[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (j0 + u < N) r[u] = emit_load<I>(g, a, en.beg + sidx[(j0 + u) * FAST_THREADS]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (j0 + u < N)
                    emit_finish<I>(g, a, r[u], en.v, en.s, en.p * (uint32_t)N + (uint32_t)(j0 + u),
                                   (int64_t)en.ob + j0 + u, en.q + (uint32_t)(j0 + u));
        }
        if (rec) record_profile(a.sched, en.d, N, a.sched->vstats[en.v], n_level, a.depth, en.cls, clock64() - t0);
        my_items++;
        my_bytes += 16 + 4ull * en.d +
                    (unsigned long long)N * (4ull + 4ull * nout + (a.push ? 12ull + 2 * (sizeof(I) + 4) : 0ull));
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        my_bytes += __shfl_xor_sync(FULL, my_bytes, o);
        my_items += __shfl_xor_sync(FULL, my_items, o);
    }
    if (lane == 0 && my_items) {
        atomicAdd(&a.bytes[10], my_bytes);
        atomicAdd(&a.items[10], my_items);
    }
}

template <typename I, int BIAS>
__global__ void __launch_bounds__(FAST_THREADS, CSAW_THREAD_SEL_MIN_BLOCKS)
k_select_thread(DevGraph g, LevelArgs a) {
    select_thread_body<I, BIAS>(g, a);
}

// Level expansion, part 2 for items over a cached prefix with N <= 16 and
// d >= 3N (a rebuild is rare): 32 / N items per warp, slot s of the warp's
// item i on lane i * N + s.  All items of a warp run the same instructions:
// their entries, first draws and searches (cdf_find), then rounds as in
// resolve_slots -- one match over the warp finds every repeated candidate,
// each item's lanes look at their own, and the repeats of all items draw
// again together -- until no item has one.  Items that need a rebuild go on
// from their failed first phase (its state kept in the consumed entry): rows
// up to WF edges by k_select_fast on the refill list (written over the
// consumed warp list), larger ones by the CTA pass.
//
// What bounds it: dependent sector gathers (entry, total and tile line, edge
// line, column) and the instructions of the rounds, about equally: 55% issue
// active, 3.9 TB/s of DRAM, 20 cycles between a warp's instructions, 11 of
// them waiting for loads (level 2 at R-MAT scale 22).  An item costs 285 warp
// instructions; two items a warp in halves of their own, their rows staged
// in shared memory by the bulk copy engine, cost 550, as the halves diverged
// in draws and refinements and paid the staging per item.  The gathers need
// no shared memory, so registers set the occupancy: 40 a thread, six CTAs
// (48 and five: 4% slower), which is why a slot's later draw words and the
// recording clock wait in shared memory and the entry is read again when its
// edges are emitted.  Scale-25 step: 23.4 -> 18.4 ms; an 8192-seed [15,10,5]
// request on R-MAT 22: 0.55 -> 0.43 ms.
template <typename I, int BIAS>
__device__ __forceinline__ void group_body(const DevGraph &g, const LevelArgs &a) {
    static_assert(REJECT_ATTEMPTS == 4, "a first phase's draws are one Philox block");
    __shared__ uint32_t s_word[3 * FAST_THREADS];        // per thread: its slot's draws 1..3 of the phase
    __shared__ long long s_t0[FAST_THREADS / 32];        // recording: when the warp's items began
    const int lane = threadIdx.x & 31;
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const uint32_t n = __ldcg(a.n_pair);
    const int N = a.N;
    const int nout = 2 + (a.o_smp != nullptr) + (a.o_dep != nullptr);
    const uint32_t G = 32 / N;
    const uint32_t gi = (uint32_t)lane / (uint32_t)N;
    const int first = (int)gi * N, sl = lane - first;   // the item's first lane, the lane's slot
    const unsigned gmask = gi < G ? ((1u << N) - 1u) << first : 0u;   // N <= 16
    const unsigned below = gmask & ((1u << lane) - 1u);
    const bool rec = a.sched && a.sched->mode == SCHED_RECORD;
    uint32_t my_items = 0, my_probes = 0;
#pragma unroll 1
    for (uint32_t base = gw * G; base < n; base += nw * G) {
        const uint32_t i = base + gi;
        bool act = gi < G && i < n;
        if (rec && lane == 0) s_t0[threadIdx.x >> 5] = clock64();
        // what the draws need of the entry; the rest is read again when the
        // edges are emitted, so it does not hold registers over the search
        int64_t beg = 0;
        int d = 0;
        float T = 0.f;
        uint32_t x = 0;
        int cand = -2 - lane, used = 0;
        if (act) {
            const int4 *q = reinterpret_cast<const int4 *>(a.pair_list + i);
            const int4 y = __ldcg(q + 1);
            beg = __ldcg(reinterpret_cast<const long long *>(q + 2));
            d = y.w;
            T = __ldg(g.cdf + beg + d - 1);
            // the slot's draws of the first phase are one block's words
            const uint4 blk = philox(make_uint4((uint32_t)y.z, (uint32_t)y.y, (TAG_SAMPLE << 24) | (uint32_t)a.depth,
                                                (uint32_t)sl << 16), a.k0, a.k1);
            x = blk.x;
            s_word[threadIdx.x] = blk.y;
            s_word[FAST_THREADS + threadIdx.x] = blk.z;
            s_word[2 * FAST_THREADS + threadIdx.x] = blk.w;
        }
        bool draw = act;
#pragma unroll 1
        for (;;) {
            if (draw) {
                if (used) x = s_word[(used - 1) * FAST_THREADS + threadIdx.x];
                cand = cdf_find(g, beg, d, x, T);
                if (!(T > 0.f)) cand = sl;   // no mass: the slots take indices 0..N-1
                ++used;
            }
            // lanes of the item holding the same candidate, before this one;
            // an accepted slot never has any, so the first slot with one is
            // the item's current slot and the slots before it are accepted
            const unsigned lower = __match_any_sync(FULL, cand) & below;
            const unsigned db = __ballot_sync(FULL, lower != 0u);
            if (db == 0u) break;
            const unsigned mine = db & gmask;
            const int f = __ffs(mine) - 1;   // -1: the item is done
            draw = (lower & ((1u << (f & 31)) - 1u)) != 0u && used < REJECT_ATTEMPTS;
            const unsigned ab = __ballot_sync(FULL, draw);
            if (mine && !((ab >> f) & 1u)) {
                // slot f's draws of the first phase ran out: a whole warp
                // (rows) or CTA (hubs) rebuilds the prefix and goes on.  The
                // failing slot and the accepted indices (16-bit) go into the
                // item's entry, which nothing reads any more.
                const bool keep = d <= RESUME_MAX_DEG && i < 0x7FFFFFFFu;
                if (sl == 0) {
                    const int4 *q = reinterpret_cast<const int4 *>(a.pair_list + i);
                    int4 *o = reinterpret_cast<int4 *>(
                        d <= WF ? a.refill_list + atomicAdd(a.n_refill, 1u) : a.retry_list + atomicAdd(a.n_retry, 1u));
                    o[0] = __ldcg(q);
                    o[1] = __ldcg(q + 1);
                    int4 z = __ldcg(q + 2);
                    if (keep) z.w = (int)(i + 1);   // pad: where its first phase's state waits
                    o[2] = z;
                }
                __syncwarp(gmask);   // the entry is read before its first bytes are overwritten
                if (keep) {
                    uint16_t *ps = reinterpret_cast<uint16_t *>(a.pair_list + i);
                    if (lane < f) ps[1 + sl] = (uint16_t)cand;
                    if (sl == 0) ps[0] = (uint16_t)(f - first);
                }
                act = draw = false;
                cand = -2 - lane;
            }
        }
        if (act) {
            const SelEntry en = load_sel(a.pair_list + i);
            emit_edge<I>(g, a, beg + cand, en.v, en.s, en.p * (uint32_t)N + (uint32_t)sl, (int64_t)en.ob + sl,
                         en.q + (uint32_t)sl);
            if (sl == 0) {
                ++my_items;
                my_probes += 32 - __clz(d);
            }
        }
        if (rec) {
            __syncwarp();
            if (act && sl == 0) {
                const SelEntry en = load_sel(a.pair_list + i);
                record_profile(a.sched, d, N, a.sched->vstats[en.v], __ldcg(a.n_in), a.depth, en.cls,
                               clock64() - s_t0[threadIdx.x >> 5]);
            }
            __syncwarp();
        }
    }
    // counted bytes: per item its entry's 16, per draw one 4-byte prefix probe
    // per halving of the row and the edge's records
    unsigned long long my_bytes = (unsigned long long)my_probes * N * 4ull +
                                  (unsigned long long)my_items *
                                      (16ull + (unsigned long long)N * (4ull + 4ull * nout +
                                                                        (a.push ? 12ull + 2 * (sizeof(I) + 4) : 0ull)));
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        my_bytes += __shfl_xor_sync(FULL, my_bytes, o);
        my_items += __shfl_xor_sync(FULL, my_items, o);
    }
    if (lane == 0 && my_items) {
        atomicAdd(&a.bytes[7], my_bytes);
        atomicAdd(&a.items[7], (unsigned long long)my_items);
    }
}

template <typename I, int BIAS>
__global__ void __launch_bounds__(FAST_THREADS, CSAW_GROUP_MIN_BLOCKS)
k_select_group(DevGraph g, LevelArgs a) {
    group_body<I, BIAS>(g, a);
}

// Level expansion, part 2 for hub items (d > WF) over a cached prefix: one
// warp per item, each draw a search of the prefix through its index
// (cdf_find) taken one attempt at a time, since a search costs dependent
// loads; no shared memory.  An item whose draws need a rebuild of its prefix
// goes to the retry list (the CTA pass rebuilds it in global scratch).
template <typename I, int BIAS>
__device__ __forceinline__ void hub_body(const DevGraph &g, const LevelArgs &a) {
    const int lane = threadIdx.x & 31;
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const uint32_t n = __ldcg(a.n_hub);
    const uint32_t n_level = __ldcg(a.n_in);
    const int N = a.N;
    const int nout = 2 + (a.o_smp != nullptr) + (a.o_dep != nullptr);
    unsigned long long my_bytes = 0, my_items = 0;
    for (uint32_t i = gw; i < n; i += nw) {
        const SelEntry en = load_sel(a.hub_list + i);
        const DrawCtx dc{a.k0, a.k1, en.p, (uint32_t)en.s, (uint32_t)a.depth};
        const bool rec = a.sched && a.sched->mode == SCHED_RECORD;
        long long t0 = 0;
        if (rec) t0 = clock64();
        const int sel = select_warp<I, BIAS>(g, en.beg, en.d, N, dc, nullptr, nullptr, nullptr, lane, 0);
        if (sel == -2) {
            if (lane == 0) a.retry_list[atomicAdd(a.n_retry, 1u)] = en;
            continue;
        }
        if (lane < N)
            emit_edge<I>(g, a, en.beg + sel, en.v, en.s, en.p * (uint32_t)N + (uint32_t)lane, (int64_t)en.ob + lane,
                         en.q + (uint32_t)lane);
        if (rec) {
            __syncwarp();
            if (lane == 0)
                record_profile(a.sched, en.d, N, a.sched->vstats[en.v], n_level, a.depth, en.cls, clock64() - t0);
        }
        if (lane == 0) {
            my_items++;
            // per draw: one 4-byte prefix probe per halving of the row (the
            // index levels split the same search), then the edge's records
            my_bytes += 16 + (unsigned long long)N * (4ull * (64 - __clzll((unsigned long long)en.d)) + 4ull +
                                                      4ull * nout + (a.push ? 12ull + 2 * (sizeof(I) + 4) : 0ull));
        }
    }
    if (lane == 0 && my_items) {
        atomicAdd(&a.bytes[6], my_bytes);
        atomicAdd(&a.items[6], my_items);
    }
}

template <typename I, int BIAS>
__global__ void __launch_bounds__(FAST_THREADS, 4)
k_select_hub(DevGraph g, LevelArgs a) {
    hub_body<I, BIAS>(g, a);
}

// Biased walks: one warp per walk.  A step with d <= 32 is one round trip:
// the biases, column ids and neighbor records of all neighbors load together,
// the prefix and search run in registers, and the chosen lane's record gives
// the next vertex's adjacency range.  Lane l computes the Philox block of step
// t0 + l, so one warp-wide Philox serves 32 steps, and lane l holds the edge
// of step t0 + l until 32 records are written out together.
template <typename I, int BIAS>
__global__ void __launch_bounds__(FAST_THREADS, 4)
k_walk_fast(DevGraph g, WalkArgs a) {
    constexpr int NW = FAST_THREADS / 32;
    __shared__ float s_W[NW * WF];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    float *W = s_W + wib * WF;
    const bool cached = BIAS != CSAW_BIAS_UNBIASED && g.cdf && g.cdf_bias == BIAS;
    const bool mat = BIAS == CSAW_BIAS_EDGE_WEIGHT || BIAS == CSAW_BIAS_DEGREE;
    const unsigned long long obytes = 4ull * (2 + (a.o_smp != nullptr) + (a.o_dep != nullptr));
    const unsigned long long rec = 4ull + sizeof(I) + 4ull;   // col + neighbor record
    unsigned long long steps = 0, bytes = 0;
    uint32_t rounds = 0;   // 5 x the 32-way search rounds of this warp's cached steps
    for (int w = gw; w < a.n; w += nw) {
        int32_t v = a.seeds[w];
        if (v < 0 || v >= g.v.n_vertices) {
            if (lane == 0) atomicOr(a.err, ERR_SEED_RANGE);
            continue;
        }
        int64_t beg = row_begin<I>(g, v);
        int32_t d = (int32_t)(row_begin<I>(g, v + 1) - beg);
        bytes += 2 * sizeof(I);
        uint32_t xw = 0;
        int32_t rs = 0, rd = 0;
        int t0 = 0, nrec = 0;
        auto flush = [&]() {
            if (nrec == 0) return;
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(a.o_count, (unsigned long long)nrec);
            base = __shfl_sync(FULL, base, 0);
            const int64_t pos = (int64_t)base + lane;
            if (lane < nrec && pos < a.cap) {
                a.o_src[pos] = rs;
                a.o_dst[pos] = rd;
                if (a.o_smp) a.o_smp[pos] = a.base + w;
                if (a.o_dep) a.o_dep[pos] = t0 + lane;
            }
            nrec = 0;
        };
        for (int t = 0; t < a.len; ++t) {
            if ((t & 31) == 0) {
                flush();
                t0 = t;
                xw = philox(make_uint4(0u, (uint32_t)(a.base + w), (TAG_SAMPLE << 24) | (uint32_t)(t + lane), 0u), a.k0,
                            a.k1).x;
            }
            if (d <= 0) break;
            const uint32_t x = __shfl_sync(FULL, xw, t & 31);
            int64_t e = beg;
            int32_t u = 0, nd = 0;
            int64_t nb = 0;
            bool have = false;
            if (d == 1) {
            } else if (BIAS == CSAW_BIAS_UNBIASED) {
                e = beg + mulhi(x, (uint32_t)d);
            } else if (cached) {
                // every round's probes are loaded together, the first round's
                // with the total, the last round's with the records of the
                // edges it decides between: one round trip for a row of one
                // tile, two up to 1024 edges, three or four beyond
                const float *cp = g.cdf + beg;
                int lo = 0, n = d;        // the answer lies in row positions [lo, lo + n), n <= 32 at the end
                float T, tt;
                NbrRec r{};
                float pv;
                if (d <= 1024) {
                    const int step = (d + 31) >> 5;
                    const int at = (lane + 1) * step - 1 < d - 1 ? (lane + 1) * step - 1 : d - 1;
                    pv = __ldg(cp + at);
                    if (step == 1 && lane < d && g.nrec) r = load_rec(g.nrec, beg + lane);
                    T = __shfl_sync(FULL, pv, 31);   // the last probe is the row's last entry
                    tt = its_target(x, T);
                    if (step > 1) {
                        const int k = __ffs(__ballot_sync(FULL, at == d - 1 || pv > tt)) - 1;
                        lo = k * step;
                        n = d - lo < step ? d - lo : step;
                    }
                } else {
                    const RowSpan row = row_span(beg, d);
                    const float *c2 = g.cdf2 + (row.b0 >> 10);
                    int u = 0, m = (int)(row.last >> 10) + 1;
                    T = __ldg(cp + d - 1);
                    do {   // the last group's entry is never read: it is known to exceed the target
                        const int st = (m + 31) >> 5, q = u + (lane + 1) * st - 1;
                        pv = q < u + m - 1 ? __ldg(c2 + q) : 0.f;
                        tt = its_target(x, T);
                        const int k = __ffs(__ballot_sync(FULL, q >= u + m - 1 || pv > tt)) - 1;
                        m = m - k * st < st ? m - k * st : st;
                        u += k * st;
                    } while (m > 1);
                    const int ka = max(u << 5, (int)(row.o2 >> 5));   // its tiles
                    const int kb = min((u << 5) + 31, (int)(row.last >> 5));
                    const int q = ka + lane;
                    pv = q < kb ? __ldg(g.cdf1 + (row.b0 >> 5) + q) : 0.f;
                    const int k = ka + __ffs(__ballot_sync(FULL, q >= kb || pv > tt)) - 1;
                    lo = tile_at(row, k) + tile_lo(row, k);
                    n = tile_hi(row, k) - tile_lo(row, k);
                }
                const bool mine = lane < n;
                if (d > 32) {
                    pv = mine ? __ldg(cp + lo + lane) : 0.f;
                    if (mine && g.nrec) r = load_rec(g.nrec, beg + lo + lane);
                }
                int idx = __ffs(__ballot_sync(FULL, lane >= n - 1 || pv > tt)) - 1;
                if (!(T > 0.f)) {   // no mass: the row's first edge
                    idx = 0;
                    lo = 0;
                    if (g.nrec) r = load_rec(g.nrec, beg);
                }
                e = beg + lo + idx;
                u = __shfl_sync(FULL, r.col, idx);
                nb = __shfl_sync(FULL, r.beg, idx);
                nd = __shfl_sync(FULL, r.deg, idx);
                have = g.nrec != nullptr;
                rounds += 36 - __clz(d);
            } else if (d <= 32) {
                float wl = 0.f;
                int32_t ul = 0, dl = 0;
                int64_t bl = 0;
                if (lane < d) {
                    if (g.nrec) {   // one 128-bit record per lane, coalesced
                        const NbrRec r = load_rec(g.nrec, beg + lane);
                        ul = r.col;
                        dl = r.deg;
                        bl = r.beg;
                        wl = BIAS == CSAW_BIAS_DEGREE ? __int2float_rn(dl) : edge_bias<I, BIAS>(g, beg + lane);
                    } else {
                        wl = edge_bias<I, BIAS>(g, beg + lane);
                        ul = __ldg(g.v.col + beg + lane);
                    }
                }
                // canonical prefix of one tile; the first lane above t is the
                // same with or without the running max, and T is the max
                const float v = warp_ks_sum(wl, lane);
                const float P = lane < d ? __fadd_rn(0.f, __fadd_rn(0.f, v)) : 0.f;
                const float T = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(P)));
                int idx = 0;
                if (T > 0.f) idx = __ffs(__ballot_sync(FULL, P > its_target(x, T))) - 1;
                e = beg + idx;
                u = __shfl_sync(FULL, ul, idx);
                nb = __shfl_sync(FULL, bl, idx);
                nd = __shfl_sync(FULL, dl, idx);
                have = g.nrec != nullptr;
                bytes += (mat ? 4ull : 4ull + 2ull * sizeof(I)) * d + rec * (d - 1);
            } else if (d <= WF) {
                preload_bias<I, BIAS>(g, beg, d, W, lane);
                auto wfn = [&](int64_t i) { return W[i]; };
                const float T = warp_canon_prefix(wfn, d, W, nullptr, lane);
                e = beg + (T > 0.f ? search_upper(W, d, its_target(x, T)) : 0);
                __syncwarp();
                bytes += (mat ? 4ull : 4ull + 2ull * sizeof(I)) * d;
            } else {
                if (d > a.scratch_stride) {
                    if (lane == 0) atomicOr(a.err, ERR_SCRATCH);
                    break;
                }
                float *buf = a.scratch + (int64_t)gw * a.scratch_stride;
                auto wfn = [&](int64_t i) { return edge_bias<I, BIAS>(g, beg + i); };
                const float T = warp_canon_prefix(wfn, (int64_t)d, buf, nullptr, lane);
                e = beg + (T > 0.f ? search_upper(buf, d, its_target(x, T)) : 0);
                bytes += (mat ? 4ull : 4ull + 2ull * sizeof(I)) * d;
            }
            if (!have) {
                if (g.nrec) {
                    const NbrRec r = load_rec(g.nrec, e);
                    u = r.col;
                    nb = r.beg;
                    nd = r.deg;
                } else {
                    u = __ldg(g.v.col + e);
                }
            }
            int32_t dst = Update(&g.v, u, v);
            if (dst < 0 || dst >= g.v.n_vertices) {
                if (lane == 0) atomicOr(a.err, ERR_UPDATE_RANGE);
                dst = 0;
            }
            if (!g.nrec || dst != u) {
                nb = row_begin<I>(g, dst);
                nd = (int32_t)(row_begin<I>(g, dst + 1) - nb);
            }
            if (lane == (t & 31)) {
                rs = v;
                rd = dst;
            }
            ++nrec;
            v = dst;
            beg = nb;
            d = nd;
            ++steps;
        }
        flush();
    }
    if (lane == 0 && steps) {
        atomicAdd(&a.bytes[2], bytes + steps * (obytes + rec) + 128ull * (rounds / 5));   // 32 probes a round
        atomicAdd(&a.items[2], steps);
    }
    counters_out(a.done);
}

// Walks with one thread per walk, for many walks: unbiased steps take one
// round trip via the neighbor records; biased steps search the cached prefix
// (the graph must hold it for BIAS) through its index, so a warp keeps 32
// walks in flight instead of one.  Same draws as the warp kernels: step t of
// walk w uses word x of Philox(0, w, t).
//
// A step is a dependent gather or three, so nothing else may stand in a
// walk's chain.  A thread keeps the vertices of WALK_KEEP steps in shared
// memory; the warp then reserves their output range with one atomic and
// writes them a step later, when the reservation has come back beside the
// step's own loads.  (Staging 64 edges a warp and waiting for the atomic of
// each flush took 531 us for 262,144 unbiased walks of 40 on R-MAT 22; this
// takes 318, and 247 by columns, 4.8 TB/s of DRAM in 32- and 64-byte
// accesses: 99 bytes read a step.)
constexpr int WALK_KEEP = 8;

template <typename I, int BIAS>
__global__ void __launch_bounds__(WALK_THREADS, BIAS == CSAW_BIAS_UNBIASED ? 8 : 6)
k_walk_thread_fast(DevGraph g, WalkArgs a) {
    constexpr bool BIASED = BIAS != CSAW_BIAS_UNBIASED;
    __shared__ int32_t s_dst[WALK_KEEP * WALK_THREADS];   // [step][thread]
    const int lane = threadIdx.x & 31;
    int32_t *mine = s_dst + threadIdx.x;
    const int stride = gridDim.x * blockDim.x;
    unsigned long long steps = 0;
    uint32_t probes = 0;   // of one walk at most a.len x 33
    unsigned long long tot_probes = 0;
    for (int base = blockIdx.x * blockDim.x; base < a.n; base += stride) {
        const int w = base + threadIdx.x;
        bool alive = w < a.n;
        int32_t v = 0;
        int64_t beg = 0;
        int32_t d = 0;
        if (alive) {
            v = a.seeds[w];
            if (v < 0 || v >= g.v.n_vertices) {
                atomicOr(a.err, ERR_SEED_RANGE);
                alive = false;
            } else {
                beg = row_begin<I>(g, v);
                d = (int32_t)(row_begin<I>(g, v + 1) - beg);
            }
        }
        int32_t first = v;                  // source of the kept steps' first edge
        int kept = 0, t0 = 0;               // steps kept by this thread, the first one's number
        unsigned long long out = 0;         // lane 0: the range reserved for them
        // writes the kept steps of every lane, step by step
        auto flush = [&]() {
            unsigned long long pos0 = __shfl_sync(FULL, out, 0);
            int32_t src = first;
            for (int k = 0; k < WALK_KEEP; ++k) {
                const unsigned m = __ballot_sync(FULL, k < kept);
                if (m == 0u) break;
                if (k < kept) {
                    const int32_t dst = mine[k * WALK_THREADS];
                    const int64_t pos = (int64_t)pos0 + __popc(m & ((1u << lane) - 1u));
                    if (pos < a.cap) {
                        a.o_src[pos] = src;
                        a.o_dst[pos] = dst;
                        if (a.o_smp) a.o_smp[pos] = a.base + w;
                        if (a.o_dep) a.o_dep[pos] = t0 + k;
                    }
                    src = dst;
                }
                pos0 += __popc(m);
            }
        };
        auto reserve = [&]() {
            const unsigned n = __reduce_add_sync(FULL, (unsigned)kept);
            if (lane == 0 && n) out = atomicAdd(a.o_count, (unsigned long long)n);
        };
        // the step's draw; unbiased, computed beside the load of the step before
        // (biased walks have no register to hold it)
        auto draw = [&](int t) -> uint32_t {
            return philox(make_uint4(0u, (uint32_t)(a.base + w), (TAG_SAMPLE << 24) | (uint32_t)t, 0u), a.k0, a.k1).x;
        };
        uint32_t x = BIASED ? 0u : draw(0);
        bool full = false;   // WALK_KEEP steps kept, their range reserved
        for (int t = 0; t < a.len; ++t) {
            if (alive && d <= 0) alive = false;
            if (!__any_sync(FULL, alive)) break;
            int32_t dst = 0;
            if (alive) {
                uint32_t idx = 0;
                if (d > 1) {
                    if constexpr (BIASED) {
                        const float T = __ldg(g.cdf + beg + d - 1);
                        idx = (uint32_t)cdf_find(g, beg, d, draw(t), T);
                        if (!(T > 0.f)) idx = 0;
                        probes += 33 - __clz(d);
                    } else {
                        idx = mulhi(x, (uint32_t)d);
                    }
                }
                NbrRec r;
                if (a.by_col) {
                    r.col = __ldg(g.v.col + beg + idx);
                    r.beg = row_begin<I>(g, r.col);
                    r.deg = (int32_t)(row_begin<I>(g, r.col + 1) - r.beg);
                } else {
                    r = edge_rec<I>(g, beg + idx);
                }
                if (!BIASED) x = draw(t + 1);
                dst = Update(&g.v, r.col, v);
                if (dst < 0 || dst >= g.v.n_vertices) {
                    atomicOr(a.err, ERR_UPDATE_RANGE);
                    dst = 0;
                }
                int64_t nb;
                int32_t nd;
                row_of<I>(g, r, dst, nb, nd);
                beg = nb;
                d = nd;
                ++steps;
            }
            if (full) {
                flush();
                full = false;
                kept = 0;
                first = v;
                t0 = t;
            }
            if (alive) {
                mine[(t - t0) * WALK_THREADS] = dst;
                ++kept;
                v = dst;
            }
            if (t - t0 == WALK_KEEP - 1) {
                reserve();
                full = true;
            }
        }
        if (!full) reserve();
        flush();
        if (BIASED) {
            tot_probes += probes;
            probes = 0;
        }
    }
    unsigned long long tot = steps, pr = tot_probes;
    for (int off = 16; off; off >>= 1) {
        tot += __shfl_xor_sync(FULL, tot, off);
        pr += __shfl_xor_sync(FULL, pr, off);
    }
    if (lane == 0) {
        // the column and a record's row range, or (by_col) two row offsets
        unsigned long long per = 4 + sizeof(I) + (a.by_col ? sizeof(I) : 4) +
                                 4ull * (2 + (a.o_smp != nullptr) + (a.o_dep != nullptr));
        atomicAdd(&a.bytes[8], tot * per + 4 * pr);   // + prefix probes (biased)
        atomicAdd(&a.items[8], tot);
    }
    counters_out(a.done);
}

// MDRW with a frontier of at most 32 vertices: one warp per sample, slot i on
// lane i with its vertex, row and bias in registers.  A step's chain is the
// neighbor's load alone where the graph has neighbor records (a column and
// two row offsets otherwise): the biases of the unchanged slots, which a
// frontier in shared memory gathered again every step, stay where they are,
// lane l computes the draws of step t0 + l, and 32 steps' edges are written
// together.  4000 samples F4 x 3: 18.6 -> 14.7 us on the device, 51 -> 48 a
// call.
template <typename I, int BIAS>
__global__ void __launch_bounds__(WALK_THREADS)
k_mdrw_warp(DevGraph g, WalkArgs a) {
    const int lane = threadIdx.x & 31;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const int F = a.F;
    unsigned long long steps = 0, visits = 0;
    auto bias_of = [&](int32_t v, int32_t deg) -> float {
        if constexpr (BIAS == CSAW_BIAS_UNBIASED) return 1.f;
        else if constexpr (BIAS == CSAW_BIAS_DEGREE) return __int2float_rn(deg);
        else return VertexBias(v, &g.v);
    };
    for (int s = gw; s < a.n; s += nw) {
        int32_t v = 0, d = 0;
        int64_t beg = 0;
        float w = 0.f;
        if (lane < F) {
            v = a.seeds[(int64_t)s * F + lane];
            if (v < 0 || v >= g.v.n_vertices) {
                atomicOr(a.err, ERR_SEED_RANGE);
                v = 0;
            }
            beg = row_begin<I>(g, v);
            d = (int32_t)(row_begin<I>(g, v + 1) - beg);
            w = bias_of(v, d);
        }
        uint4 x = make_uint4(0u, 0u, 0u, 0u);
        int32_t rs = 0, rd = 0;   // lane l: the edge of step t0 + l, if it has one
        bool have = false;
        for (int t0 = 0; t0 < a.len; t0 += 32) {
            x = philox(make_uint4(0u, (uint32_t)(a.base + s), (TAG_MDRW << 24) | (uint32_t)(t0 + lane), 0u), a.k0, a.k1);
            have = false;
            const int m = a.len - t0 < 32 ? a.len - t0 : 32;
            for (int k = 0; k < m; ++k) {
                int slot = 0;
                if (F > 1) {
                    const float P = tile_prefix(w, F, lane);
                    const float T = __shfl_sync(FULL, P, 31);
                    const float t = its_target(__shfl_sync(FULL, x.x, k), T);
                    if (T > 0.f) slot = __ffs(__ballot_sync(FULL, lane >= F - 1 || P > t)) - 1;
                }
                const uint32_t y = __shfl_sync(FULL, x.y, k);
                int32_t dst = 0;
                const int32_t src = v;
                if (lane == slot && d > 0) {
                    const NbrRec r = edge_rec<I>(g, beg + mulhi(y, (uint32_t)d));
                    dst = Update(&g.v, r.col, v);
                    if (dst < 0 || dst >= g.v.n_vertices) {
                        atomicOr(a.err, ERR_UPDATE_RANGE);
                        dst = 0;
                    }
                    row_of<I>(g, r, dst, beg, d);
                    v = dst;
                    w = bias_of(v, d);
                    ++steps;
                    dst = ~dst;   // an edge (negative) or none (0)
                }
                const int32_t es = __shfl_sync(FULL, src, slot), ed = __shfl_sync(FULL, dst, slot);
                if (lane == k) {
                    rs = es;
                    rd = ~ed;
                    have = ed < 0;
                }
            }
            visits += m;
            const unsigned hm = __ballot_sync(FULL, have);
            unsigned long long base = 0;
            if (lane == 0 && hm) base = atomicAdd(a.o_count, (unsigned long long)__popc(hm));
            base = __shfl_sync(FULL, base, 0);
            const int64_t pos = (int64_t)base + __popc(hm & ((1u << lane) - 1u));
            if (have && pos < a.cap) {
                a.o_src[pos] = rs;
                a.o_dst[pos] = rd;
                if (a.o_smp) a.o_smp[pos] = a.base + s;
                if (a.o_dep) a.o_dep[pos] = t0 + lane;
            }
        }
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) steps += __shfl_xor_sync(FULL, steps, off);
    if (lane == 0 && visits) {
        // per step its slot's row range; per edge the neighbor and the edge written
        atomicAdd(&a.bytes[3], visits * 2ull * sizeof(I) + steps * (4ull + 4ull * (2 + (a.o_smp != nullptr) + (a.o_dep != nullptr))));
        atomicAdd(&a.items[3], steps);
    }
    counters_out(a.done);
}

template <typename I>
__global__ void k_nbr_records(DevGraph g, NbrRec *rec) {
    const I *r = (const I *)g.v.rowptr;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < g.v.n_edges;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t u = __ldg(g.v.col + e);
        const I b = __ldg(r + u);
        const unsigned long long ub = (unsigned long long)(long long)b;
        reinterpret_cast<int4 *>(rec)[e] =
            make_int4(u, (int32_t)(__ldg(r + u + 1) - b), (int32_t)(uint32_t)ub, (int32_t)(uint32_t)(ub >> 32));
    }
}

}  // namespace csaw
