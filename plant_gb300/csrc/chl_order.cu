// Plain vertex orderings computed on the GPU (no reference counterpart: the
// reference reads its order from a file produced by outside tools; its own
// degree tool is distributed_memory/degree.cpp:62-67).
//
//   degree      : Graph::get_degree(v) (shared_memory/graph.hpp:324)
//                 descending; ties by a seeded permutation (tie_key).
//   betweenness : Brandes dependencies from `sources` seeded sources over
//                 forward shortest paths, descending; same tie break.
//
// Both sort with the stable radix sort: first by the tie key, then by the
// primary key, so equal primary keys keep tie-key order.
#include "chl_dev.cuh"

#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

namespace chl {

namespace {

constexpr uint32_t kInfD = 0x7FFFFFFFu;

__device__ __forceinline__ uint64_t d_mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__global__ void tie_keys(uint32_t n, uint64_t seed, uint64_t *key, uint32_t *val) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        key[v] = d_mix64(seed * 0x9E3779B97F4A7C15ull + (uint64_t)v);
        val[v] = v;
    }
}

// primary key descending == ~primary ascending
__global__ void degree_keys(uint32_t n, const uint64_t *off_out, const uint64_t *off_in,
                            const uint32_t *vals, uint64_t *key) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t v = vals[i];
        const uint64_t deg = (off_out[v + 1] - off_out[v]) + (off_in[v + 1] - off_in[v]);
        key[i] = ~deg;
    }
}

__global__ void bc_keys(uint32_t n, const double *bc, const uint32_t *vals, uint64_t *key) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint64_t bits = (uint64_t)__double_as_longlong(bc[vals[i]]);
        key[i] = ~bits;
    }
}

__global__ void pack_arcs(uint64_t m, const uint32_t *head, const int32_t *len, uint2 *arc) {
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x)
        arc[e] = make_uint2(head[e], (uint32_t)len[e]);
}

// One block per source, in three phases; every one is bound by the latency of
// its chain of gathers per step, so what counts is few steps.
//  1. Distances, label-correcting in distance windows [.., thr): every vertex
//     whose distance fell is relaxed again until none below thr falls, then
//     the next window is taken from the far pile.  Windows are as wide as to
//     hold about kWindow vertices (256 sources of a 1024-square grid: 123 ms
//     with 1,024, 117 with 2,048, 115 with 4,096 and 8,192; the order as a
//     whole, against 8 s with one lane per source), distance and queue mark
//     falling in one 64-bit minimum (115 -> 101 ms).  (Settling only vertices that are final by
//     the IN criterion of Crauser et al. took about 8 vertices a step on
//     road-like graphs and 43 ms for a 256-square grid.)
//  2. Path counts sigma in waves over the shortest-path graph: a wave holds
//     the vertices whose predecessors are all counted.
//  3. Dependencies delta over the waves in reverse.
// Every sum of 2 and 3 runs in adjacency order with explicitly rounded
// operations (no contraction), matching the CPU restatement bit for bit.  The
// order of a 256-square grid by 256 sources takes 7.5 ms, 308 with one lane
// per source and a binary heap.
// A vertex of up to kLight arcs belongs to one thread, half of its arcs in
// flight at a time; others to one warp.  Which arcs of a short list lie on
// shortest paths is found once and kept as two bytes beside the vertex's
// distance: phases 2 and 3 gather no distances, a trip less in either chain
// (9.0 -> 7.5 ms).
constexpr int kOrdThreads = 512;
constexpr uint32_t kOrdWarps = kOrdThreads / 32;
constexpr int kLight = 8;
constexpr int kGroup = kLight / 2;
constexpr uint32_t kWindow = 4096;

constexpr uint32_t kFarMark = 0xFFFFFFFFu;   // above every pass
constexpr uint32_t kShort = 0x80000000u;     // both lists have at most kLight arcs, see the words below
static_assert(kLight == 8, "a byte of a word says which arcs of a list count");

// Passes and waves of at most kNarrow vertices (a lane each), none with a long
// list, are run by warp 0 alone, one after the other, while the block waits at
// one barrier.  Such steps cost their barriers and dependent accesses (an L2
// atomic takes 500 cycles, a load 300), and graphs one or two vertices wide
// consist of them: the queue stays in shared memory with what the next step
// wants to know of its vertices, two arcs at a time keep the loops short, a
// lone vertex needs no atomics, and phase 3 reads ahead for all waves among
// the next 32 vertices.  16 sources of a path of 3,000 vertices 13.6 -> 4.7 ms
// (6.1 with a lane per source, whose heap and lists one thread's L1 serves), a
// ladder of 3,000 rungs 18.1 -> 9.6 (13.9), a directed cycle of 5,000 24.2 ->
// 7.6 (8.1).
constexpr uint32_t kNarrow = 32;
constexpr std::integral_constant<int, 2> kTwo{};
constexpr std::integral_constant<int, 4> kFour{};

struct OrdShared {
    uint32_t nn, npile, nkeep, heavy, lo, kmin, kmax;
    uint32_t a, b, c;   // state that warp 0 hands back
    uint32_t stale;     // a queued vertex's distance fell again in the same pass
    uint32_t q[kNarrow * kLight], qx[kNarrow * kLight];   // vertices; their distances or marks
};

__global__ void __launch_bounds__(kOrdThreads) brandes_kernel(uint32_t n, const uint64_t *off_out, const uint2 *arc_out,
                                                              const uint64_t *off_in, const uint2 *arc_in,
                                                              const uint32_t *src, unsigned long long *ws_word,
                                                              uint32_t *ws_list, double *ws_sigma, double *deltas) {
    __shared__ OrdShared sh;
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    const uint32_t j = blockIdx.x;
    // word of a vertex: distance in the high half; in the low one the last pass
    // it was queued in (phase 1), then (phases 2 and 3) the predecessors not yet
    // counted and, where both its lists are short, which of their arcs lie on
    // shortest paths: kShort | out-arcs << 16 | in-arcs << 8 | predecessors
    unsigned long long *word = ws_word + (size_t)j * n;
    auto dist_at = [&](uint32_t v) -> uint32_t { return __ldcg((const uint32_t *)(word + v) + 1); };
    auto mark_at = [&](uint32_t v) -> uint32_t * { return (uint32_t *)(word + v); };
    uint32_t *front = ws_list + (size_t)j * 2 * n, *fnext = front + n;
    double *sigma = ws_sigma + (size_t)j * n;
    uint32_t *pile = (uint32_t *)sigma, *pile2 = pile + n;   // phase 1 only
    double *delta = deltas + (size_t)j * n;
    const uint32_t s = src[j];
    for (uint32_t v = tid; v < n; v += kOrdThreads) {
        __stcg(&word[v], (unsigned long long)(v == s ? 0u : kInfD) << 32 | kFarMark);
        __stcg(&delta[v], 0.0);
    }
    if (tid == 0) {
        __stcg(&front[0], s);
        sh.npile = 0;
        sh.lo = kInfD;
    }
    __syncthreads();
    // run body(v) by whole warps for the listed vertices that are long(v)
    auto for_heavy = [&](const uint32_t *list, uint32_t cnt, auto is_long, auto body) {
        for (uint32_t i0 = warp * 32; i0 < cnt; i0 += kOrdThreads) {
            uint32_t v = 0;
            bool h = false;
            if (i0 + lane < cnt) {
                v = __ldcg(&list[i0 + lane]);
                h = is_long(v);
            }
            for (uint32_t m = __ballot_sync(kFull, h); m; m &= m - 1) body(__shfl_sync(kFull, v, __ffs(m) - 1));
        }
    };

    // ---- phase 1: distances
    uint32_t nf = 1, thr = 1, width = 0, pass = 0, members = 0;
    while (true) {
        // passes over the window until no distance below thr falls
        uint32_t lo = kInfD;   // smallest distance at or past thr this thread has set
        // one minimum over distance and mark: the smaller distance wins and
        // brings its mark
        // (alone: no other thread of the block is at work)
        auto lower = [&](uint32_t w, uint32_t dd, bool alone) {
            const unsigned long long now = (unsigned long long)dd << 32 | (dd < thr ? pass : kFarMark);
            if (!alone) return atomicMin(&word[w], now);
            const unsigned long long was = word[w];
            if (now < was) word[w] = now;
            return was;
        };
        // the lists that w joins, whose word was `was` before
        auto settle = [&](uint32_t w, uint32_t dd, unsigned long long was, auto push) {
            const uint32_t stamp = dd < thr ? pass : kFarMark;
            const uint32_t old = (uint32_t)(was >> 32), mark = (uint32_t)was;
            if (dd > old || (dd == old && stamp >= mark)) return;
            if (dd < thr) {
                // a vertex of the far pile whose distance falls below thr
                // leaves a stale entry there; an equal distance only takes
                // the mark of a vertex the sweep queued: queued again
                if (mark != pass) push(atomicAdd(&sh.nn, 1u), w);
                else sh.stale = 1;
            } else {
                lo = min(lo, dd);
                if (old == kInfD) __stcg(&pile[atomicAdd(&sh.npile, 1u)], w);
            }
        };
        while (nf) {
            if (nf <= kNarrow) {
                if (warp == 0) {
                    uint32_t cnt = nf, v = lane < cnt ? __ldcg(&front[lane]) : s, dv = dist_at(v);
                    bool heavy;
                    while (true) {
                        const bool on = lane < cnt;
                        const uint64_t ob = on ? off_out[v] : 0, oe = on ? off_out[v + 1] : 0;
                        heavy = __any_sync(kFull, oe - ob > kLight);
                        if (heavy) break;
                        ++pass;
                        if (lane == 0) sh.nn = sh.stale = 0;
                        __syncwarp();
                        // no read first, and two minima on their way together
#pragma unroll 1
                        for (uint64_t e = ob; e < oe; e += 2) {
                            const uint2 x = arc_out[e], y = e + 1 < oe ? arc_out[e + 1] : make_uint2(v, kInfD);
                            const uint32_t dx = dv + x.y, dy = dv + y.y;
                            const unsigned long long wx = dx < kInfD ? lower(x.x, dx, cnt == 1) : 0ull;
                            const unsigned long long wy = dy < kInfD ? lower(y.x, dy, cnt == 1) : 0ull;
                            auto queue = [&](uint32_t w, uint32_t dd, unsigned long long was) {
                                if (dd < kInfD)
                                    settle(w, dd, was, [&](uint32_t i, uint32_t) {
                                        sh.q[i] = w;
                                        sh.qx[i] = dd;
                                    });
                            };
                            queue(x.x, dx, wx);
                            queue(y.x, dy, wy);
                        }
                        __syncwarp();
                        members += cnt;
                        cnt = sh.nn;
                        if (cnt == 0 || cnt > kNarrow) break;
                        v = lane < cnt ? sh.q[lane] : s;
                        dv = sh.stale ? dist_at(v) : sh.qx[lane];
                        __syncwarp();   // the queue is read before the next pass writes it
                    }
                    if (heavy) {
                        if (lane < cnt) __stcg(&front[lane], v);
                    } else {
                        for (uint32_t i = lane; i < cnt; i += 32) __stcg(&front[i], sh.q[i]);
                    }
                    if (lane == 0) {
                        sh.a = cnt;
                        sh.b = pass;
                        sh.c = members;
                        sh.heavy = heavy ? 1u : 0u;
                    }
                }
                __syncthreads();
                nf = sh.a;
                pass = sh.b;
                members = sh.c;
                const bool heavy = sh.heavy != 0;
                __syncthreads();   // the state is read before it changes
                if (!heavy) continue;
            }
            ++pass;
            if (tid == 0) {
                sh.nn = 0;
                sh.heavy = 0;
            }
            __syncthreads();
            auto relax = [&](uint32_t w, uint32_t dd, uint32_t seen) {
                // distances only fall: a read no larger than dd proves the atomic idle
                if (dd < seen) settle(w, dd, lower(w, dd, false), [&](uint32_t i, uint32_t x) { __stcg(&fnext[i], x); });
            };
            for (uint32_t i = tid; i < nf; i += kOrdThreads) {
                const uint32_t v = __ldcg(&front[i]);
                const uint64_t ob = off_out[v], oe = off_out[v + 1];
                const uint32_t dv = dist_at(v);
                if (oe - ob > kLight) {
                    sh.heavy = 1;
                    continue;
                }
#pragma unroll
                for (int h = 0; h < kLight; h += kGroup) {
                    if (ob + h >= oe) break;
                    uint2 hl[kGroup];
                    uint32_t dw[kGroup];
#pragma unroll
                    for (int q = 0; q < kGroup; ++q)
                        hl[q] = ob + h + q < oe ? arc_out[ob + h + q] : make_uint2(v, 1u);
#pragma unroll
                    for (int q = 0; q < kGroup; ++q) dw[q] = ob + h + q < oe ? dist_at(hl[q].x) : 0u;
#pragma unroll
                    for (int q = 0; q < kGroup; ++q) relax(hl[q].x, dv + hl[q].y, dw[q]);
                }
            }
            __syncthreads();
            if (sh.heavy) {
                for_heavy(front, nf, [&](uint32_t v) { return off_out[v + 1] - off_out[v] > kLight; }, [&](uint32_t v) {
                    const uint32_t dv = dist_at(v);
                    for (uint64_t a = off_out[v] + lane; a < off_out[v + 1]; a += 32) {
                        const uint2 hl = arc_out[a];
                        relax(hl.x, dv + hl.y, dist_at(hl.x));
                    }
                    __syncwarp();
                });
            }
            __syncthreads();
            members += nf;
            nf = sh.nn;
            uint32_t *t = front;
            front = fnext;
            fnext = t;
            __syncthreads();   // the counters are read before the next pass clears them
        }
        lo = __reduce_min_sync(kFull, lo);
        if (lane == 0 && lo != kInfD) atomicMin(&sh.lo, lo);
        __syncthreads();
        if (sh.npile == 0) break;
        if (width == 0) {
            // the first width: the spread of the source's neighbours
            if (tid == 0) {
                sh.kmin = kInfD;
                sh.kmax = 0;
            }
            __syncthreads();
            uint32_t mn = kInfD, mx = 0;
            for (uint32_t i = tid; i < sh.npile; i += kOrdThreads) {
                const uint32_t d = dist_at(__ldcg(&pile[i]));
                mn = min(mn, d);
                mx = max(mx, d);
            }
            mn = __reduce_min_sync(kFull, mn);
            mx = __reduce_max_sync(kFull, mx);
            if (lane == 0) {
                atomicMin(&sh.kmin, mn);
                atomicMax(&sh.kmax, mx);
            }
            __syncthreads();
            width = max(sh.kmax - sh.kmin, 1u);
        } else if (members > 2 * kWindow) {
            width = max(width / 2, 1u);
        } else if (members < kWindow / 2) {
            width = width < 0x20000000u ? 2 * width : 0x3FFFFFFFu;
        }
        members = 0;
        // next window: pile entries below the old thr are stale (they joined a
        // window), those below the new one are taken, the rest are kept.  lo is
        // a lower bound of the live entries, exact after one such sweep, so a
        // second sweep always takes some.
        while (nf == 0 && sh.npile) {
            const uint32_t t_old = thr, np = sh.npile;
            thr = sh.lo + width < kInfD ? sh.lo + width : kInfD;
            __syncthreads();
            if (tid == 0) {
                sh.nn = 0;
                sh.nkeep = 0;
                sh.lo = kInfD;
            }
            __syncthreads();
            uint32_t lo = kInfD;
            for (uint32_t i0 = 0; i0 < np; i0 += kOrdThreads) {
                const uint32_t i = i0 + tid;
                const uint32_t x = i < np ? __ldcg(&pile[i]) : 0u;
                const uint32_t d = i < np ? dist_at(x) : 0u;
                const bool take = i < np && d >= t_old && d < thr, keep = i < np && d >= thr;
                const uint32_t tm = __ballot_sync(kFull, take), km = __ballot_sync(kFull, keep);
                uint32_t tb = 0, kb = 0;
                if (lane == 0) {
                    if (tm) tb = atomicAdd(&sh.nn, (uint32_t)__popc(tm));
                    if (km) kb = atomicAdd(&sh.nkeep, (uint32_t)__popc(km));
                }
                tb = __shfl_sync(kFull, tb, 0);
                kb = __shfl_sync(kFull, kb, 0);
                if (take) __stcg(&front[tb + __popc(tm & lanemask_lt())], x);
                if (keep) {
                    __stcg(&pile2[kb + __popc(km & lanemask_lt())], x);
                    lo = min(lo, d);
                }
            }
            lo = __reduce_min_sync(kFull, lo);
            if (lane == 0 && lo != kInfD) atomicMin(&sh.lo, lo);
            __syncthreads();
            nf = sh.nn;
            if (tid == 0) sh.npile = sh.nkeep;
            uint32_t *t = pile;
            pile = pile2;
            pile2 = t;
            __syncthreads();
        }
        if (nf == 0) break;   // only stale entries were left
    }
    __syncthreads();

    // ---- phase 2: tight arcs of every reached vertex, then the waves
    for (uint32_t v0 = warp * 32; v0 < n; v0 += kOrdThreads) {
        const uint32_t v = v0 + lane;
        bool h = false;
        if (v < n) {
            const uint32_t dv = dist_at(v);
            uint32_t mark = 0;
            if (dv != kInfD) {
                const uint64_t ib = off_in[v], ie = off_in[v + 1], ob = off_out[v], oe = off_out[v + 1];
                h = ie - ib > kLight || oe - ob > kLight;
#pragma unroll
                for (int g = 0; g < kLight; g += kGroup) {
                    if (h || (ib + g >= ie && ob + g >= oe)) break;
                    uint2 hi[kGroup], ho[kGroup];   // past an end: d(v) + 1 != d(v)
#pragma unroll
                    for (int q = 0; q < kGroup; ++q) {
                        hi[q] = ib + g + q < ie ? arc_in[ib + g + q] : make_uint2(v, 1u);
                        ho[q] = ob + g + q < oe ? arc_out[ob + g + q] : make_uint2(v, 1u);
                    }
#pragma unroll
                    for (int q = 0; q < kGroup; ++q) {
                        const uint32_t dw = dist_at(ho[q].x);
                        if (dist_at(hi[q].x) + hi[q].y == dv) mark += 1u | 1u << (8 + g + q);
                        if (dw != kInfD && dv + ho[q].y == dw) mark |= 1u << (16 + g + q);
                    }
                }
                mark |= kShort;
            }
            if (!h) __stcg(mark_at(v), mark);
        }
        for (uint32_t m = __ballot_sync(kFull, h); m; m &= m - 1) {
            const uint32_t x = v0 + __ffs(m) - 1;
            const uint32_t dx = dist_at(x);
            uint32_t c = 0;
            for (uint64_t a = off_in[x] + lane; a < off_in[x + 1]; a += 32) {
                const uint2 hl = arc_in[a];
                c += dist_at(hl.x) + hl.y == dx ? 1u : 0u;
            }
            c = __reduce_add_sync(kFull, c);
            if (lane == 0) __stcg(mark_at(x), c);
        }
    }
    uint32_t *seq = ws_list + (size_t)j * 2 * n, *wave = seq + n;   // vertices in wave order; each wave's first
    if (tid == 0) __stcg(&seq[0], s);
    uint32_t begin = 0, end = 1, waves = 0;
    __syncthreads();
    auto is_long = [&](uint32_t v) { return !(__ldcg(mark_at(v)) & kShort); };
    // one predecessor of w is counted: the next wave takes w after its last
    // (push gets its place there and w's mark)
    auto count_down = [&](uint32_t w, bool alone, auto push) {
        const uint32_t mark = alone ? *mark_at(w) : atomicSub(mark_at(w), 1u);
        if (alone) *mark_at(w) = mark - 1u;
        if ((mark & kShort ? mark & 0xFFu : mark) == 1u) push(atomicAdd(&sh.nn, 1u), mark);
    };
    // the first G bits of m, taken from it: arc numbers, or kLight past the last
    auto take = [](auto &at, uint32_t &m) {
#pragma unroll
        for (int &q : at) {
            q = m ? __ffs(m) - 1 : kLight;
            m &= m - 1;
        }
    };
    // sigma(v) and the vertices it completes, for a vertex of short lists, G
    // arcs of each at a time
    auto count_paths = [&](auto group, uint32_t v, uint32_t mark, bool alone, auto push) {
        constexpr int G = decltype(group)::value;
        const uint64_t ib = off_in[v], ob = off_out[v];
        double acc = 0.0;
#pragma unroll 1
        for (uint32_t im = mark >> 8 & 0xFFu, om = mark >> 16 & 0xFFu; im | om;) {
            int ai[G], ao[G];
            uint32_t p[G], w[G];
            double sp[G];
            take(ai, im);
            take(ao, om);
#pragma unroll
            for (int q = 0; q < G; ++q) {
                p[q] = ai[q] < kLight ? arc_in[ib + ai[q]].x : v;
                w[q] = ao[q] < kLight ? arc_out[ob + ao[q]].x : v;
            }
#pragma unroll
            for (int q = 0; q < G; ++q) sp[q] = ai[q] < kLight ? sigma[p[q]] : 0.0;
#pragma unroll
            for (int q = 0; q < G; ++q)
                if (ao[q] < kLight) count_down(w[q], alone, [&](uint32_t i, uint32_t m) { push(i, w[q], m); });
#pragma unroll
            for (int q = 0; q < G; ++q)
                if (ai[q] < kLight) acc = __dadd_rn(acc, sp[q]);
        }
        sigma[v] = v == s ? 1.0 : acc;
    };
    while (begin < end) {
        if (end - begin <= kNarrow) {
            if (warp == 0) {
                uint32_t cnt = end - begin, v = lane < cnt ? __ldcg(&seq[begin + lane]) : s;
                uint32_t mark = __ldcg(mark_at(v));
                bool heavy;
                while (true) {
                    heavy = __any_sync(kFull, lane < cnt && !(mark & kShort));
                    if (heavy) break;
                    if (lane == 0) {
                        __stcg(&wave[waves], begin);
                        sh.nn = 0;
                    }
                    __syncwarp();
                    if (lane < cnt)
                        count_paths(kTwo, v, mark, cnt == 1, [&](uint32_t i, uint32_t w, uint32_t m) {
                            sh.q[i] = w;
                            sh.qx[i] = m;
                            __stcg(&seq[end + i], w);
                        });
                    __syncwarp();
                    ++waves;
                    begin = end;
                    cnt = sh.nn;
                    end += cnt;
                    if (cnt == 0 || cnt > kNarrow) break;
                    v = lane < cnt ? sh.q[lane] : s;
                    mark = sh.qx[lane];
                    __syncwarp();   // the queue is read before the next wave writes it
                }
                if (lane == 0) {
                    sh.a = begin;
                    sh.b = end;
                    sh.c = waves;
                    sh.heavy = heavy ? 1u : 0u;
                }
            }
            __syncthreads();
            begin = sh.a;
            end = sh.b;
            waves = sh.c;
            const bool heavy = sh.heavy != 0;
            __syncthreads();   // the state is read before it changes
            if (!heavy) continue;
        }
        if (tid == 0) {
            __stcg(&wave[waves], begin);
            sh.nn = 0;
            sh.heavy = 0;
        }
        __syncthreads();
        auto push = [&](uint32_t i, uint32_t w, uint32_t) { __stcg(&seq[end + i], w); };
        for (uint32_t i = begin + tid; i < end; i += kOrdThreads) {
            const uint32_t v = __ldcg(&seq[i]), mark = __ldcg(mark_at(v));
            if (mark & kShort) count_paths(kFour, v, mark, false, push);
            else sh.heavy = 1;
        }
        __syncthreads();
        if (sh.heavy) {
            for_heavy(seq + begin, end - begin, is_long, [&](uint32_t v) {
                const uint32_t dv = dist_at(v);
                const uint64_t ie = off_in[v + 1];
                double acc = 0.0;
                for (uint64_t a = off_in[v]; a < ie; a += 32) {
                    double sp = 0.0;
                    if (a + lane < ie) {
                        const uint2 hl = arc_in[a + lane];
                        if (dist_at(hl.x) + hl.y == dv) sp = sigma[hl.x];
                    }
                    for (uint32_t m = __ballot_sync(kFull, sp != 0.0); m; m &= m - 1)
                        acc = __dadd_rn(acc, __shfl_sync(kFull, sp, __ffs(m) - 1));
                }
                if (lane == 0) sigma[v] = v == s ? 1.0 : acc;
                for (uint64_t a = off_out[v] + lane; a < off_out[v + 1]; a += 32) {
                    const uint2 hl = arc_out[a];
                    const uint32_t dw = dist_at(hl.x);
                    if (dw != kInfD && dv + hl.y == dw)
                        count_down(hl.x, false, [&](uint32_t i, uint32_t m) { push(i, hl.x, m); });
                }
                __syncwarp();
            });
        }
        __syncthreads();
        begin = end;
        end += sh.nn;
        ++waves;
        __syncthreads();   // the counter is read before the next wave clears it
    }

    // ---- phase 3: dependencies over the waves in reverse, successors in out order
    auto depend = [&](uint32_t v, uint32_t mark) {   // delta(v), short lists
        constexpr int G = kGroup;
        const uint64_t ob = off_out[v];
        const double sv = sigma[v];
        double acc = 0.0;
#pragma unroll 1
        for (uint32_t om = mark >> 16 & 0xFFu; om;) {
            int ao[G];
            uint32_t w[G];
            double sw[G], dw[G];
            take(ao, om);
#pragma unroll
            for (int q = 0; q < G; ++q) w[q] = ao[q] < kLight ? arc_out[ob + ao[q]].x : v;
#pragma unroll
            for (int q = 0; q < G; ++q) {
                sw[q] = ao[q] < kLight ? sigma[w[q]] : 1.0;
                dw[q] = ao[q] < kLight ? delta[w[q]] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < G; ++q)
                if (ao[q] < kLight) acc = __dadd_rn(acc, __dmul_rn(__ddiv_rn(sv, sw[q]), __dadd_rn(1.0, dw[q])));
        }
        delta[v] = v == s ? 0.0 : acc;   // the source's own dependency is not counted
    };
    while (waves > 0) {
        begin = __ldcg(&wave[waves - 1]);
        if (end - begin <= kNarrow) {
            if (warp == 0) {
                // the last 32 vertices of the sequence a lane each, newest first:
                // all that does not hang on a dependency is read for all of their
                // waves together, then the waves follow one another
                bool heavy = false;
                while (waves > 0 && !heavy) {
                    const uint32_t first = lane < waves ? end - 1 - __ldcg(&wave[waves - 1 - lane]) : 32u;
                    // lanes that hold a wave's first vertex, up to the one with a long list
                    uint32_t firsts = __reduce_or_sync(kFull, first < 32 ? 1u << first : 0u);
                    const bool on = lane < end;
                    const uint32_t v = on ? __ldcg(&seq[end - 1 - lane]) : s, mark = on ? __ldcg(mark_at(v)) : kShort;
                    const uint32_t longs = __ballot_sync(kFull, !(mark & kShort));
                    if (longs) firsts &= (longs & (0u - longs)) - 1u;
                    heavy = longs && !firsts;
                    if (!firsts) break;
                    const uint32_t below = kFull >> __clz(firsts);   // lanes of whole waves
                    const uint64_t ob = off_out[v];
                    const double sv = sigma[v];
                    uint32_t om = below >> lane & 1u ? mark >> 16 & 0xFFu : 0u;
                    int at[2];
                    take(at, om);
                    uint32_t w[2];
                    double q[2];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        w[i] = at[i] < kLight ? arc_out[ob + at[i]].x : v;
                        q[i] = at[i] < kLight ? __ddiv_rn(sv, sigma[w[i]]) : 0.0;
                    }
                    uint32_t from = 0;
                    for (uint32_t f = firsts; f; f &= f - 1) {
                        const uint32_t to = (uint32_t)__ffs(f);   // lanes [from, to) are a wave
                        if (lane >= from && lane < to) {
                            double acc = 0.0;
#pragma unroll
                            for (int i = 0; i < 2; ++i)
                                if (at[i] < kLight) acc = __dadd_rn(acc, __dmul_rn(q[i], __dadd_rn(1.0, delta[w[i]])));
                            for (uint32_t m = om; m; m &= m - 1) {
                                const uint32_t x = arc_out[ob + __ffs(m) - 1].x;
                                acc = __dadd_rn(acc, __dmul_rn(__ddiv_rn(sv, sigma[x]), __dadd_rn(1.0, delta[x])));
                            }
                            delta[v] = v == s ? 0.0 : acc;
                        }
                        __syncwarp();
                        from = to;
                    }
                    end -= from;
                    waves -= (uint32_t)__popc(firsts);
                }
                if (lane == 0) {
                    sh.b = end;
                    sh.c = waves;
                    sh.heavy = heavy ? 1u : 0u;
                }
            }
            __syncthreads();
            end = sh.b;
            waves = sh.c;
            const bool heavy = sh.heavy != 0;
            __syncthreads();   // the state is read before it changes
            if (!heavy) continue;
            begin = __ldcg(&wave[waves - 1]);
        }
        --waves;
        if (tid == 0) sh.heavy = 0;
        __syncthreads();
        for (uint32_t i = begin + tid; i < end; i += kOrdThreads) {
            const uint32_t v = __ldcg(&seq[i]), mark = __ldcg(mark_at(v));
            if (mark & kShort) depend(v, mark);
            else sh.heavy = 1;
        }
        __syncthreads();
        if (sh.heavy) {
            for_heavy(seq + begin, end - begin, is_long, [&](uint32_t v) {
                const uint64_t oe = off_out[v + 1];
                const uint32_t dv = dist_at(v);
                const double sv = sigma[v];
                double acc = 0.0;
                for (uint64_t a = off_out[v]; a < oe; a += 32) {
                    bool on = false;
                    double t = 0.0;
                    if (a + lane < oe) {
                        const uint2 hl = arc_out[a + lane];
                        const uint32_t d = dist_at(hl.x);
                        on = d != kInfD && dv + hl.y == d;
                        if (on) t = __dmul_rn(__ddiv_rn(sv, sigma[hl.x]), __dadd_rn(1.0, delta[hl.x]));
                    }
                    for (uint32_t m = __ballot_sync(kFull, on); m; m &= m - 1)
                        acc = __dadd_rn(acc, __shfl_sync(kFull, t, __ffs(m) - 1));
                }
                if (lane == 0) delta[v] = v == s ? 0.0 : acc;
            });
        }
        __syncthreads();
        end = begin;
    }
}

__global__ void bc_sum(uint32_t n, uint32_t count, const double *deltas, double *bc) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        double acc = 0.0;
        for (uint32_t j = 0; j < count; ++j) acc = __dadd_rn(acc, deltas[(size_t)j * n + v]);
        bc[v] = acc;
    }
}

struct Buf {   // temporary of one call, on the null stream
    void *p = nullptr;
    size_t bytes = 0;
    Buf() = default;
    Buf(const Buf &) = delete;
    Buf &operator=(const Buf &) = delete;
    ~Buf() { tmp_free(p, bytes, 0); }
    template <typename T>
    T *as() const { return (T *)p; }
};

int alloc(Buf &b, size_t bytes) {
    b.bytes = bytes ? bytes : 1;
    return tmp_alloc(&b.p, b.bytes, 0);
}

// Sort vertices by (primary descending, tie ascending); `primary` fills key
// from the tie-sorted vertex list.
template <typename F>
int order_by(uint32_t n, uint64_t seed, F primary, int primary_bits, uint32_t *order_h) {
    Buf k0, k1, v0, v1, tmp, cnt;
    int rc;
    if ((rc = alloc(k0, (size_t)n * 8)) || (rc = alloc(k1, (size_t)n * 8)) || (rc = alloc(v0, (size_t)n * 4)) ||
        (rc = alloc(v1, (size_t)n * 4)) || (rc = alloc(tmp, radix_tmp_bytes())) || (rc = alloc(cnt, 8)))
        return rc;
    const uint64_t n64 = n;
    CHL_CUDA(cudaMemcpy(cnt.p, &n64, 8, cudaMemcpyHostToDevice));
    const int grid = device_sms() * 4;
    tie_keys<<<grid, 256>>>(n, seed, k0.as<uint64_t>(), v0.as<uint32_t>());
    int par = 0;
    if ((rc = radix_sort_pairs(k0.as<uint64_t>(), v0.as<uint32_t>(), k1.as<uint64_t>(), v1.as<uint32_t>(),
                               cnt.as<uint64_t>(), n, 64, tmp.p, radix_tmp_bytes(), 0, &par)))
        return rc;
    uint64_t *ka = par ? k1.as<uint64_t>() : k0.as<uint64_t>();
    uint32_t *va = par ? v1.as<uint32_t>() : v0.as<uint32_t>();
    uint64_t *kb = par ? k0.as<uint64_t>() : k1.as<uint64_t>();
    uint32_t *vb = par ? v0.as<uint32_t>() : v1.as<uint32_t>();
    primary(va, ka);
    int par2 = 0;
    if ((rc = radix_sort_pairs(ka, va, kb, vb, cnt.as<uint64_t>(), n, primary_bits, tmp.p,
                               radix_tmp_bytes(), 0, &par2)))
        return rc;
    CHL_CUDA(cudaMemcpy(order_h, par2 ? vb : va, (size_t)n * 4, cudaMemcpyDeviceToHost));
    return CHL_OK;
}

// float score descending: order-preserving map of the IEEE bits, then complemented
__global__ void score_keys(uint32_t n, const float *score, const uint32_t *vals, uint64_t *key) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t b = __float_as_uint(score[vals[i]]);
        b = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
        key[i] = (uint64_t)(~b);
    }
}

}  // namespace

int order_by_score(uint32_t n, uint64_t seed, const float *d_score, uint32_t *order_h) {
    if (n == 0) return CHL_OK;
    const int grid = device_sms() * 4;
    return order_by(
        n, seed, [&](const uint32_t *vals, uint64_t *key) { score_keys<<<grid, 256>>>(n, d_score, vals, key); }, 32,
        order_h);
}

}  // namespace chl

using namespace chl;

extern "C" int chl_order_degree(const chl_graph *g, uint64_t seed, uint32_t *order) {
    if (!g || !order) return CHL_ERR_INVALID;
    if (g->n == 0) return CHL_OK;
    Buf off_out, off_in;
    int rc;
    if ((rc = alloc(off_out, ((size_t)g->n + 1) * 8)) || (rc = alloc(off_in, ((size_t)g->n + 1) * 8))) return rc;
    CHL_CUDA(cudaMemcpy(off_out.p, g->off[1].data(), ((size_t)g->n + 1) * 8, cudaMemcpyHostToDevice));
    CHL_CUDA(cudaMemcpy(off_in.p, g->off[0].data(), ((size_t)g->n + 1) * 8, cudaMemcpyHostToDevice));
    const int grid = device_sms() * 4;
    const uint32_t n = g->n;
    return order_by(
        n, seed,
        [&](const uint32_t *vals, uint64_t *key) {
            degree_keys<<<grid, 256>>>(n, off_out.as<uint64_t>(), off_in.as<uint64_t>(), vals, key);
        },
        64, order);
}

extern "C" int chl_order_betweenness(const chl_graph *g, uint32_t sources, uint64_t seed,
                                     uint32_t *order) {
    if (!g || !order || g->min_len < 1) return CHL_ERR_INVALID;
    const uint32_t n = g->n;
    if (n == 0) return CHL_OK;
    if (sources > n) sources = n;
    if (sources == 0) sources = 1;
    // sources: mix64(seed + j) % n, skipping repeats (host; O(sources))
    std::vector<uint32_t> src;
    {
        std::vector<uint8_t> seen(n, 0);
        for (uint64_t j = 0; src.size() < sources; ++j) {
            uint32_t s = (uint32_t)(mix64(seed + j) % n);
            if (seen[s]) continue;
            seen[s] = 1;
            src.push_back(s);
        }
    }
    Buf off_out, off_in, arc_out, arc_in, dsrc, deltas, bc;
    int rc;
    const uint64_t mo = g->off[1][n], mi = g->off[0][n];
    if ((rc = alloc(off_out, ((size_t)n + 1) * 8)) || (rc = alloc(off_in, ((size_t)n + 1) * 8)) ||
        (rc = alloc(arc_out, mo * 8)) || (rc = alloc(arc_in, mi * 8)) ||
        (rc = alloc(dsrc, (size_t)sources * 4)) || (rc = alloc(deltas, (size_t)sources * n * 8)) ||
        (rc = alloc(bc, (size_t)n * 8)))
        return rc;
    CHL_CUDA(cudaMemcpy(off_out.p, g->off[1].data(), ((size_t)n + 1) * 8, cudaMemcpyHostToDevice));
    CHL_CUDA(cudaMemcpy(off_in.p, g->off[0].data(), ((size_t)n + 1) * 8, cudaMemcpyHostToDevice));
    CHL_CUDA(cudaMemcpy(dsrc.p, src.data(), (size_t)sources * 4, cudaMemcpyHostToDevice));
    const int grid = device_sms() * 4;
    {
        Buf head, len;
        const uint64_t most = std::max(mo, mi);
        if ((rc = alloc(head, most * 4)) || (rc = alloc(len, most * 4))) return rc;
        for (int f = 1; f >= 0; --f) {
            const uint64_t m = f ? mo : mi;
            if (m == 0) continue;
            CHL_CUDA(cudaMemcpy(head.p, g->head[f].data(), m * 4, cudaMemcpyHostToDevice));
            CHL_CUDA(cudaMemcpy(len.p, g->len[f].data(), m * 4, cudaMemcpyHostToDevice));
            pack_arcs<<<grid, 256>>>(m, head.as<uint32_t>(), len.as<int32_t>(), (f ? arc_out : arc_in).as<uint2>());
            CHL_CUDA(cudaGetLastError());
        }
        CHL_CUDA(cudaDeviceSynchronize());
    }
    // one block per source
    Buf ww, wl, wsg;
    if ((rc = alloc(ww, (size_t)sources * n * 8)) || (rc = alloc(wl, (size_t)sources * n * 8)) || (rc = alloc(wsg, (size_t)sources * n * 8)))
        return rc;
    brandes_kernel<<<sources, kOrdThreads>>>(n, off_out.as<uint64_t>(), arc_out.as<uint2>(), off_in.as<uint64_t>(),
                                             arc_in.as<uint2>(), dsrc.as<uint32_t>(),
                                             ww.as<unsigned long long>(), wl.as<uint32_t>(), wsg.as<double>(),
                                             deltas.as<double>());
    CHL_CUDA(cudaGetLastError());
    bc_sum<<<device_sms() * 4, 256>>>(n, sources, deltas.as<double>(), bc.as<double>());
    CHL_CUDA(cudaGetLastError());
    return order_by(
        n, seed,
        [&](const uint32_t *vals, uint64_t *key) { bc_keys<<<grid, 256>>>(n, bc.as<double>(), vals, key); },
        64, order);
}
