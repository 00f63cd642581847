// kernels_tree.cuh -- whole sample trees in one launch (sm_100a).
//
// The trees of different seeds are independent (without dedup), so a neighbor
// job needs no level-wide order: a CTA takes a chunk of consecutive roots, the
// samples' seeds, and runs all levels of their trees, the frontier queue in
// shared memory, with CTA barriers between levels.  The
// per-level passes (kernels_fast.cuh) cost 6-8 launches a level, each several
// microseconds however few items it finds; a small or middle-sized job is
// nothing but those launches.  Here it is one launch whose length is the
// dependent chain of one chunk.  Per level:
//   scan    every item's edge count, items that need draws (d > N) listed; the
//           chunk's output range is reserved by one atomic, whose round trip
//           the first selections hide (edges are written past a second barrier)
//   draw    listed items 32 / N a warp (group_select) where N <= 16 and few
//           first phases fail -- d >= 3N over a cached prefix, d >= 2N unbiased,
//           any d for N <= 4 -- or a warp each, taken from shared counters so
//           that warps that meet long items take fewer.  (A warp each for
//           unbiased and for short rows of few slots: 200,000 seeds [2] on the
//           power-law graph, edge weights, 119 us, 80 so; 1024 unbiased seeds
//           [15,10,5] on R-MAT 22 119 and 69.)
//   expand  take-all items by flattened batches, as the take-all pass does
//   retry   cached hubs whose first phase failed, the whole CTA on each
// A selected edge's child goes straight to the next level's queue slot (the
// output offset is the slot), so nothing between the seeds and the edges
// touches global memory but the graph.
//
// What bounds it: the chain of dependent accesses of the longest chunk, about
// 0.9 us for each one that misses L2: seed, row range, then per level prefix
// total and lines, neighbor record, and the launch itself; 64 seeds [25,10]
// take 27 us, 12 of them before the first draw is written.  64 registers a
// thread keep 1024 threads an SM resident, at the price of some spilled
// values in the biased kernels (128 registers: 66 us a call for 64 seeds against
// 69, but 93 against 79 for 1024).
//
// Selections are those of the other passes (the same device functions, draw
// keys and canonical prefix), so the edges are the same.
#pragma once

#include "kernels_fast.cuh"

namespace csaw {

constexpr int TREE_MAX_LEVELS = 8;
constexpr int TREE_MAX_ITEMS = 4096;   // queue entries of a chunk, all levels (shared memory; 16-bit lists)

struct TreeArgs {
    LevelArgs lv;                          // outputs, keys, counters, scratch, fan, D (queue fields unused)
    const int32_t *seeds;
    int n_roots, F, base, per_chunk, n_chunks;   // roots: the samples' seeds, F a sample
    uint32_t qoff[TREE_MAX_LEVELS + 1];    // first queue entry of level l; [D] the chunk's total
    uint32_t wmax;                         // entries of the widest level
    CounterOut done;
};

// Byte offsets of the dynamic shared memory of k_tree for nw warps.
struct TreeSmem {
    uint32_t zb, qb, qv, qs, qp, qd, qo, list, glist, retry, bytes;
};
__host__ __device__ __forceinline__ TreeSmem tree_smem(int nw, uint32_t qtot, uint32_t wmax, uint32_t isz, bool biased) {
    TreeSmem m;
    uint32_t at = biased ? (uint32_t)nw * WF * 4u : (uint32_t)nw * 32u * 4u;   // rows / sorted exclusions per warp
    if (biased && at < (uint32_t)sizeof(HeavyShared)) at = (uint32_t)sizeof(HeavyShared);
    at = (at + 15u) & ~15u;
    m.zb = at;
    at += biased ? (uint32_t)nw * (WF / 32) * 4u : 0u;
    m.qb = at;
    at += (qtot * isz + 15u) & ~15u;
    m.qv = at;
    at += qtot * 4u;
    m.qs = at;
    at += qtot * 4u;
    m.qp = at;
    at += qtot * 4u;
    m.qd = at;
    at += qtot * 4u;
    m.qo = at;
    at += wmax * 4u;
    m.list = at;
    at += (wmax * 2u + 3u) & ~3u;
    m.glist = at;
    at += (wmax * 2u + 3u) & ~3u;
    m.retry = at;
    at += biased ? (wmax * 2u + 3u) & ~3u : 0u;
    m.bytes = at;
    return m;
}

// First phase of 32 / N items, slot sl of the lane's item on lane first + sl
// (lanes of gmask), as the group pass runs it; biased ones over a cached
// prefix.  cand: the lane's index.  Returns -1, or the slot of the lane's item
// whose draws ran out (the slots before it are accepted).
template <bool BIASED>
__device__ __forceinline__ int group_select(const DevGraph &g, int64_t beg, int d, int N, const DrawCtx &dc, bool act,
                                            unsigned gmask, int first, int sl, int lane, int &cand) {
    const unsigned below = gmask & ((1u << lane) - 1u);
    float T = 0.f;
    uint4 blk = make_uint4(0u, 0u, 0u, 0u);
    int used = 0, fail = -1, c = -2 - lane;
    if (act) {
        if (BIASED) T = __ldg(g.cdf + beg + d - 1);
        blk = philox(make_uint4(dc.p, dc.s, (TAG_SAMPLE << 24) | dc.l, (uint32_t)sl << 16), dc.k0, dc.k1);
    }
    bool draw = act;
#pragma unroll 1
    for (;;) {
        if (draw) {
            if (BIASED) {
                c = cdf_find(g, beg, d, word_of(blk, used), T);
                if (!(T > 0.f)) c = sl;
            } else {
                c = (int)mulhi(word_of(blk, used), (uint32_t)d);
            }
            ++used;
            cand = c;
        }
        const unsigned lower = __match_any_sync(FULL, c) & below;
        const unsigned db = __ballot_sync(FULL, lower != 0u);
        if (db == 0u) return fail;
        const unsigned mine = db & gmask;
        const int f = __ffs(mine) - 1;
        draw = (lower & ((1u << (f & 31)) - 1u)) != 0u && used < REJECT_ATTEMPTS;
        const unsigned ab = __ballot_sync(FULL, draw);
        if (mine && !((ab >> f) & 1u)) {   // the item is out: its lanes hold values of their own
            fail = f - first;
            draw = false;
            c = -2 - lane;
        }
    }
}

template <typename I, int BIAS>
__global__ void __launch_bounds__(512, 2)
k_tree(const __grid_constant__ DevGraph g, const __grid_constant__ TreeArgs t) {
    constexpr bool BIASED = BIAS != CSAW_BIAS_UNBIASED;
    extern __shared__ __align__(16) unsigned char s_tree[];
    __shared__ uint32_t s_w[32], s_wi[32];
    __shared__ unsigned long long s_ob;
    __shared__ uint32_t s_ndraw, s_ngroup, s_next, s_nextg, s_nretry;
    __shared__ unsigned long long s_bytes[4];   // kinds: take-all, selection, hub, CTA retry
    __shared__ uint32_t s_items[4];
    const LevelArgs &a = t.lv;
    const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
    const TreeSmem m = tree_smem(nw, t.qoff[a.D], t.wmax, sizeof(I), BIASED);
    float *P = reinterpret_cast<float *>(s_tree) + warp * WF;
    int *zs = reinterpret_cast<int *>(s_tree) + warp * 32;
    uint32_t *zb = reinterpret_cast<uint32_t *>(s_tree + m.zb) + warp * (WF / 32);
    HeavyShared &sh = *reinterpret_cast<HeavyShared *>(s_tree);   // the rows are free during retries
    I *qb = reinterpret_cast<I *>(s_tree + m.qb);
    int32_t *qv = reinterpret_cast<int32_t *>(s_tree + m.qv), *qs = reinterpret_cast<int32_t *>(s_tree + m.qs);
    uint32_t *qp = reinterpret_cast<uint32_t *>(s_tree + m.qp);
    int32_t *qd = reinterpret_cast<int32_t *>(s_tree + m.qd);
    uint32_t *qo = reinterpret_cast<uint32_t *>(s_tree + m.qo);
    uint16_t *list = reinterpret_cast<uint16_t *>(s_tree + m.list);
    uint16_t *glist = reinterpret_cast<uint16_t *>(s_tree + m.glist);
    uint16_t *retry = reinterpret_cast<uint16_t *>(s_tree + m.retry);
    const int nout = 2 + (a.o_smp != nullptr) + (a.o_dep != nullptr);
    if (tid < 4) {
        s_bytes[tid] = 0ull;
        s_items[tid] = 0u;
    }
    if (tid == 0) s_ndraw = s_ngroup = s_next = s_nextg = s_nretry = 0u;
    uint32_t my_bytes = 0, my_items = 0;   // a chunk's bytes are below 2^23 (TREE_MAX_ITEMS)

    for (int chunk = blockIdx.x; chunk < t.n_chunks; chunk += gridDim.x) {
        const int c0 = chunk * t.per_chunk;
        uint32_t n = (uint32_t)(t.n_roots - c0 < t.per_chunk ? t.n_roots - c0 : t.per_chunk);
        for (uint32_t i = tid; i < n; i += T) {
            const uint32_t root = (uint32_t)c0 + i;
            int32_t v = __ldg(t.seeds + root);
            if (v < 0 || v >= g.v.n_vertices) {
                atomicOr(a.err, ERR_SEED_RANGE);
                v = 0;
            }
            const int64_t b = row_begin<I>(g, v);
            qv[i] = v;
            qs[i] = t.base + (int32_t)(root / (uint32_t)t.F);
            qp[i] = root % (uint32_t)t.F;
            qb[i] = (I)b;
            qd[i] = (int32_t)(row_begin<I>(g, v + 1) - b);
        }
        __syncthreads();
        for (int l = 0; l < a.D && n > 0; ++l) {
            const int N = a.fan[l];
            const bool push = l + 1 < a.D;
            const uint32_t Q = t.qoff[l], Qn = t.qoff[l + 1];
            const uint32_t per_edge = 4u + 4u * (uint32_t)nout + (push ? 12u + 2u * ((uint32_t)sizeof(I) + 4u) : 0u);
            // ---- scan: output offsets and the lists of items that need draws
            // (unbiased items that are no more than the warps take one each: there
            // are no rounds to share, and a failed first phase starts over.  1000
            // seeds [2,2] on R-MAT 16: 42.2 us a call in groups, 40.7 so)
            const bool grouped = N <= 16 && (BIASED || n > (uint32_t)nw);
            const int dgroup = N <= 4 ? N + 1 : (BIASED ? CSAW_PAIR_MIN_RATIO * N : 2 * N);
            uint32_t total = 0;
            for (uint32_t b0 = 0; b0 < n; b0 += T) {
                const uint32_t i = b0 + tid;
                uint32_t excl = 0;
                if (n > 32 || warp == 0) {
                    const int d = i < n ? qd[Q + i] : 0;
                    const int k = d < N ? d : N;
                    const int incl = warp_incl_scan(k, lane);
                    excl = (uint32_t)(incl - k);
                    if (lane == 31) s_w[warp] = (uint32_t)incl;
                    const bool drawn = d > N, grp = drawn && grouped && d >= dgroup;
                    const unsigned gm = __ballot_sync(FULL, grp), wm = __ballot_sync(FULL, drawn && !grp);
                    uint32_t pg = 0, pw = 0;
                    if (n <= 32) {
                        if (lane == 0) {
                            s_ngroup = (uint32_t)__popc(gm);
                            s_ndraw = (uint32_t)__popc(wm);
                        }
                    } else if (lane == 0) {
                        if (gm) pg = atomicAdd(&s_ngroup, (uint32_t)__popc(gm));
                        if (wm) pw = atomicAdd(&s_ndraw, (uint32_t)__popc(wm));
                    }
                    pg = __shfl_sync(FULL, pg, 0);
                    pw = __shfl_sync(FULL, pw, 0);
                    const unsigned lt = (1u << lane) - 1u;
                    if (grp) glist[pg + __popc(gm & lt)] = (uint16_t)i;
                    else if (drawn) list[pw + __popc(wm & lt)] = (uint16_t)i;
                    if (i < n) {
                        if (n <= 32) qo[i] = excl;
                        my_items++;
                        my_bytes += 12u + (uint32_t)sizeof(I) + 4u + (!drawn ? per_edge * (uint32_t)k : 0u);
                    }
                }
                __syncthreads();
                if (n <= 32) {   // one warp's scan is the chunk's
                    total = s_w[0];
                    break;
                }
                if (warp == 0) s_wi[lane] = (uint32_t)warp_incl_scan(lane < nw ? (int)s_w[lane] : 0, lane);
                __syncthreads();
                if (i < n) qo[i] = total + (warp ? s_wi[warp - 1] : 0u) + excl;
                total += s_wi[31];
            }
            // the output range: its reservation is waited for by the last warp
            // alone until the level barrier below
            if (tid == T - 32) s_ob = total ? atomicAdd(a.o_count, (unsigned long long)total) : 0ull;
            if (n > 32) __syncthreads();   // every item's offset
            const uint32_t ndraw = s_ndraw, ngroup = s_ngroup;
            // The barrier after which s_ob is there, passed by every thread
            // once a level.  It follows loads under `if (act)`, after which
            // the source alone does not say that the warp has converged, so it
            // is the form that does not ask for it (bar.sync does).
            bool met = false;   // the same in all lanes of a warp
            auto meet = [&]() {
                if (!met) {
                    __syncwarp();
                    asm volatile("barrier.sync 1, %0;" ::"r"(T) : "memory");
                }
                met = true;
            };
            // edge j of queue item i, its neighbor at offset off of the row:
            // written at the item's output offset + j and, on inner levels,
            // its child at that queue slot of the next level.  The neighbor's
            // load is in flight while the warp meets the others.
            auto emit = [&](bool act, uint32_t i, int j, int off) {
                NbrRec r{};
                int32_t v = 0;
                if (act) {
                    const int64_t e = (int64_t)qb[Q + i] + off;
                    v = qv[Q + i];
                    if (push) r = edge_rec<I>(g, e);
                    else r.col = __ldg(g.v.col + e);
                }
                meet();
                if (!act) return;
                int32_t dst = Update(&g.v, r.col, v);
                if (dst < 0 || dst >= g.v.n_vertices) {
                    atomicOr(a.err, ERR_UPDATE_RANGE);
                    dst = 0;
                }
                const int32_t s = qs[Q + i];
                const uint32_t o = qo[i] + (uint32_t)j;
                const int64_t pos = (int64_t)s_ob + o;
                if (pos < a.cap) {
                    a.o_src[pos] = v;
                    a.o_dst[pos] = dst;
                    if (a.o_smp) a.o_smp[pos] = s;
                    if (a.o_dep) a.o_dep[pos] = l;
                }
                if (push) {
                    int64_t nb;
                    int32_t nd;
                    row_of<I>(g, r, dst, nb, nd);
                    const uint32_t c = Qn + o;
                    qv[c] = dst;
                    qs[c] = s;
                    qp[c] = qp[Q + i] * (uint32_t)N + (uint32_t)j;
                    qb[c] = (I)nb;
                    qd[c] = nd;
                }
            };
            // ---- items that need draws: 32 / N a warp while there are such,
            // then a warp each.  An item of a group whose first phase failed
            // goes on in its warp from there (a row) or waits for the CTA (a hub).
            {
                const int G = 32 / N, gi = lane / N, first = gi * N, sl = lane - first;
                const unsigned gmask = gi < G ? (N == 32 ? FULL : ((1u << N) - 1u)) << first : 0u;
                unsigned pend = 0u;      // failed rows of the warp's last group, by first lane
                uint32_t ig = 0u;        // the lane's item, index and failing slot in it
                int cg = -1, fg = -1;
                bool groups = ngroup > 0u;
                for (;;) {
                    bool act;
                    uint32_t i;
                    int j, off;
                    if (pend == 0u && groups) {
                        uint32_t x = 0;
                        if (lane == 0) x = atomicAdd(&s_nextg, 1u) * (uint32_t)G;
                        x = __shfl_sync(FULL, x, 0);
                        if (x >= ngroup) {
                            groups = false;
                            continue;
                        }
                        act = gi < G && x + (uint32_t)gi < ngroup;
                        ig = act ? glist[x + gi] : 0u;
                        const int d = qd[Q + ig];
                        const DrawCtx dc{a.k0, a.k1, qp[Q + ig], (uint32_t)qs[Q + ig], (uint32_t)l};
                        fg = group_select<BIASED>(g, (int64_t)qb[Q + ig], d, N, dc, act, gmask, first, sl, lane, cg);
                        const bool failed = act && fg >= 0;
                        if (BIASED && failed && sl == 0 && d > WF) retry[atomicAdd(&s_nretry, 1u)] = (uint16_t)ig;
                        pend = __ballot_sync(FULL, failed && sl == 0 && (!BIASED || d <= WF));
                        act = act && !failed;
                        i = ig;
                        j = sl;
                        off = cg;
                    } else {
                        int j0 = 0, sel = -1;
                        if (pend) {
                            const int ld = __ffs(pend) - 1;
                            pend &= pend - 1;
                            i = __shfl_sync(FULL, ig, ld);
                            if (BIASED) {   // unbiased items start over
                                j0 = __shfl_sync(FULL, fg, ld);
                                sel = __shfl_sync(FULL, cg, (ld + lane) & 31);
                            }
                        } else {
                            uint32_t x = 0;
                            if (lane == 0) x = atomicAdd(&s_next, 1u);
                            x = __shfl_sync(FULL, x, 0);
                            if (x >= ndraw) break;
                            i = list[x];
                        }
                        const int d = qd[Q + i];
                        const int64_t beg = (int64_t)qb[Q + i];
                        const DrawCtx dc{a.k0, a.k1, qp[Q + i], (uint32_t)qs[Q + i], (uint32_t)l};
                        if constexpr (!BIASED) {
                            sel = select_unbiased(d, N, dc, zs, lane);
                        } else {
                            if (d <= 32 && j0 == 0) sel = select_reg<I, BIAS>(g, beg, d, N, dc, lane);
                            else if (d <= WF) sel = select_cached<I, BIAS>(g, beg, d, N, dc, P, zb, lane, j0, sel);
                            else sel = select_warp<I, BIAS>(g, beg, d, N, dc, nullptr, nullptr, nullptr, lane, 0);
                            if (sel == -2) {   // a cached hub that needs a rebuild: the whole CTA redoes it
                                if (lane == 0) retry[atomicAdd(&s_nretry, 1u)] = (uint16_t)i;
                                continue;
                            }
                        }
                        act = lane < N;
                        j = lane;
                        off = sel;
                    }
                    emit(act, i, j, off);
                    if (act && j == 0) {
                        const int d = qd[Q + i];
                        const int kind = BIASED && d > WF ? 2 : 1;
                        const unsigned long long search =
                            !BIASED ? 0ull : (d <= WF ? 4ull * d : (unsigned long long)N * 4ull * (32 - __clz(d)));
                        atomicAdd(&s_bytes[kind], 16ull + search + (uint32_t)N * per_edge);
                        atomicAdd(&s_items[kind], 1u);
                    }
                }
            }
            // ---- take-all items: lanes stride over a batch's edges together
            uint32_t bs = (n + nw - 1) / nw;
            bs = bs > 32 ? 32 : bs;
            for (uint32_t b0 = warp * bs; b0 < n; b0 += nw * bs) {
                const uint32_t i = b0 + lane;
                int ks = 0, d = 0;
                if (lane < (int)bs && i < n) {
                    d = qd[Q + i];
                    if (d <= N) ks = d;
                }
                const int incl = warp_incl_scan(ks, lane);
                const int K = __shfl_sync(FULL, incl, 31);
                for (int e0 = 0; e0 < K; e0 += 32) {
                    const int e = e0 + lane;
                    const bool act = e < K;
                    const int b = shfl_search_int(incl, act ? e : 0);
                    const int j = e - (__shfl_sync(FULL, incl, b) - __shfl_sync(FULL, ks, b));
                    emit(act, b0 + (uint32_t)b, j, j);
                }
            }
            meet();
            __syncthreads();
            // ---- cached hubs that need a rebuild: the CTA takes them in turn
            if constexpr (BIASED) {
                const uint32_t nretry = s_nretry;
                for (uint32_t x = 0; x < nretry; ++x) {
                    const uint32_t i = retry[x];
                    const int32_t d = qd[Q + i];
                    unsigned long long rebuild_bytes = 0;
                    if (heavy_need(d) > a.heavy_stride) {
                        if (tid == 0) atomicOr(a.err, ERR_SCRATCH);
                        continue;
                    }
                    const DrawCtx dc{a.k0, a.k1, qp[Q + i], (uint32_t)qs[Q + i], (uint32_t)l};
                    const int sel = heavy_select<I, BIAS, false>(g, qv[Q + i], (int64_t)qb[Q + i], d, N, dc,
                                                                 a.heavy_scratch + (int64_t)blockIdx.x * a.heavy_stride,
                                                                 sh, 0, -1, rebuild_bytes);
                    if (warp == 0) emit(lane < N, i, lane, sel);
                    if (tid == 0) {
                        s_bytes[3] += 12 + 2 * sizeof(I) + rebuild_bytes + (uint32_t)N * per_edge +
                                      (unsigned long long)N * 4ull * (32 - __clz(d));
                        s_items[3] += 1u;
                    }
                    __syncthreads();   // the shared state and scratch are free for the next
                }
            }
            if (tid == 0) s_ndraw = s_ngroup = s_next = s_nextg = s_nretry = 0u;
            n = push ? total : 0u;
            __syncthreads();
        }
        if (my_bytes >= 1u << 31) {
            atomicAdd(&s_bytes[0], (unsigned long long)my_bytes);
            my_bytes = 0u;
        }
    }
    unsigned long long warp_bytes = my_bytes;
#pragma unroll
    for (int off = 16; off; off >>= 1) warp_bytes += __shfl_xor_sync(FULL, warp_bytes, off);
    my_items = __reduce_add_sync(FULL, my_items);
    if (lane == 0 && my_items) {
        atomicAdd(&s_bytes[0], warp_bytes);
        atomicAdd(&s_items[0], my_items);
    }
    __syncthreads();
    if (tid < 4 && s_items[tid]) {
        const int kind = tid == 0 ? 0 : (tid == 1 ? 5 : (tid == 2 ? 6 : 1));
        atomicAdd(&a.bytes[kind], s_bytes[tid]);
        atomicAdd(&a.items[kind], (unsigned long long)s_items[tid]);
    }
    counters_out(t.done);
}

}  // namespace csaw
