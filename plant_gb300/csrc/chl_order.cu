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
// operations (no contraction), matching the CPU restatement bit for bit.  On
// the 256-square grid the kernel takes 8.2 ms, one lane per source with a
// binary heap took 308.
// A vertex of up to kLight arcs belongs to one thread, half of its arcs in
// flight at a time; others to one warp.
constexpr int kOrdThreads = 512;
constexpr uint32_t kOrdWarps = kOrdThreads / 32;
constexpr int kLight = 8;
constexpr int kGroup = kLight / 2;
constexpr uint32_t kWindow = 4096;

constexpr uint32_t kFarMark = 0xFFFFFFFFu;   // above every pass

struct OrdShared {
    uint32_t nn, npile, nkeep, heavy, lo, kmin, kmax;
};

__global__ void __launch_bounds__(kOrdThreads) brandes_kernel(uint32_t n, const uint64_t *off_out, const uint2 *arc_out,
                                                              const uint64_t *off_in, const uint2 *arc_in,
                                                              const uint32_t *src, unsigned long long *ws_word,
                                                              uint32_t *ws_list, double *ws_sigma, double *deltas) {
    __shared__ OrdShared sh;
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    const uint32_t j = blockIdx.x;
    // word of a vertex: distance in the high half; in the low one the last pass
    // it was queued in (phase 1), the predecessors not yet counted (phase 2)
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
    // run body(v) by whole warps for the listed vertices with more than kLight arcs
    auto for_heavy = [&](const uint32_t *list, uint32_t cnt, const uint64_t *off, auto body) {
        for (uint32_t i0 = warp * 32; i0 < cnt; i0 += kOrdThreads) {
            uint32_t v = 0;
            bool h = false;
            if (i0 + lane < cnt) {
                v = __ldcg(&list[i0 + lane]);
                h = off[v + 1] - off[v] > kLight;
            }
            for (uint32_t m = __ballot_sync(kFull, h); m; m &= m - 1) body(__shfl_sync(kFull, v, __ffs(m) - 1));
        }
    };

    // ---- phase 1: distances
    uint32_t nf = 1, thr = 1, width = 0, pass = 0, members = 0;
    while (true) {
        // passes over the window until no distance below thr falls
        while (nf) {
            ++pass;
            if (tid == 0) {
                sh.nn = 0;
                sh.heavy = 0;
            }
            __syncthreads();
            uint32_t lo = kInfD;   // smallest distance at or past thr this thread has set
            auto relax = [&](uint32_t w, uint32_t dd, uint32_t seen) {
                // distances only fall: a read no larger than dd proves the atomic idle
                if (dd >= seen) return;
                // one minimum over distance and mark: the smaller distance wins
                // and brings its mark
                const uint32_t stamp = dd < thr ? pass : kFarMark;
                const unsigned long long was = atomicMin(&word[w], (unsigned long long)dd << 32 | stamp);
                const uint32_t old = (uint32_t)(was >> 32), mark = (uint32_t)was;
                if (dd > old || (dd == old && stamp >= mark)) return;
                if (dd < thr) {
                    // a vertex of the far pile whose distance falls below thr
                    // leaves a stale entry there; an equal distance only takes
                    // the mark of a vertex the sweep queued: queued again
                    if (mark != pass) __stcg(&fnext[atomicAdd(&sh.nn, 1u)], w);
                } else {
                    lo = min(lo, dd);
                    if (old == kInfD) __stcg(&pile[atomicAdd(&sh.npile, 1u)], w);
                }
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
                for_heavy(front, nf, off_out, [&](uint32_t v) {
                    const uint32_t dv = dist_at(v);
                    for (uint64_t a = off_out[v] + lane; a < off_out[v + 1]; a += 32) {
                        const uint2 hl = arc_out[a];
                        relax(hl.x, dv + hl.y, dist_at(hl.x));
                    }
                    __syncwarp();
                });
            }
            lo = __reduce_min_sync(kFull, lo);
            if (lane == 0 && lo != kInfD) atomicMin(&sh.lo, lo);
            __syncthreads();
            members += nf;
            nf = sh.nn;
            uint32_t *t = front;
            front = fnext;
            fnext = t;
            __syncthreads();   // the counters are read before the next pass clears them
        }
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

    // ---- phase 2: tight in-arcs of every reached vertex, then the waves
    for (uint32_t v0 = warp * 32; v0 < n; v0 += kOrdThreads) {
        const uint32_t v = v0 + lane;
        bool h = false;
        if (v < n) {
            const uint32_t dv = dist_at(v);
            const uint64_t ib = off_in[v], ie = off_in[v + 1];
            uint32_t c = 0;
            h = dv != kInfD && ie - ib > kLight;
            if (dv != kInfD && !h) {
#pragma unroll
                for (int g = 0; g < kLight; g += kGroup) {
                    if (ib + g >= ie) break;
                    uint2 hl[kGroup];
#pragma unroll
                    for (int q = 0; q < kGroup; ++q) hl[q] = ib + g + q < ie ? arc_in[ib + g + q] : make_uint2(v, 1u);
#pragma unroll
                    for (int q = 0; q < kGroup; ++q) c += dist_at(hl[q].x) + hl[q].y == dv ? 1u : 0u;
                }
            }
            if (!h) __stcg(mark_at(v), c);
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
    while (begin < end) {
        if (tid == 0) {
            __stcg(&wave[waves], begin);
            sh.nn = 0;
            sh.heavy = 0;
        }
        __syncthreads();
        auto count_down = [&](uint32_t w, uint32_t dd, uint32_t dw) {
            if (dd == dw && dw != kInfD && atomicSub(mark_at(w), 1u) == 1u) __stcg(&seq[end + atomicAdd(&sh.nn, 1u)], w);
        };
        for (uint32_t i = begin + tid; i < end; i += kOrdThreads) {
            const uint32_t v = __ldcg(&seq[i]);
            const uint64_t ib = off_in[v], ie = off_in[v + 1], ob = off_out[v], oe = off_out[v + 1];
            const uint32_t dv = dist_at(v);
            if (ie - ib > kLight || oe - ob > kLight) sh.heavy = 1;
            if (ie - ib <= kLight) {
                double acc = 0.0;
#pragma unroll
                for (int h = 0; h < kLight; h += kGroup) {
                    if (ib + h >= ie) break;
                    uint2 hl[kGroup];
                    double sp[kGroup];
#pragma unroll
                    for (int q = 0; q < kGroup; ++q)
                        hl[q] = ib + h + q < ie ? arc_in[ib + h + q] : make_uint2(v, 1u);   // d(v) + 1 != d(v)
#pragma unroll
                    for (int q = 0; q < kGroup; ++q)
                        sp[q] = dist_at(hl[q].x) + hl[q].y == dv ? __ldcg(&sigma[hl[q].x]) : 0.0;
#pragma unroll
                    for (int q = 0; q < kGroup; ++q) acc = __dadd_rn(acc, sp[q]);
                }
                __stcg(&sigma[v], v == s ? 1.0 : acc);
            }
            if (oe - ob <= kLight) {
#pragma unroll
                for (int h = 0; h < kLight; h += kGroup) {
                    if (ob + h >= oe) break;
                    uint2 hl[kGroup];
                    uint32_t dw[kGroup];
#pragma unroll
                    for (int q = 0; q < kGroup; ++q)
                        hl[q] = ob + h + q < oe ? arc_out[ob + h + q] : make_uint2(v, 1u);
#pragma unroll
                    for (int q = 0; q < kGroup; ++q) dw[q] = dist_at(hl[q].x);
#pragma unroll
                    for (int q = 0; q < kGroup; ++q) count_down(hl[q].x, dv + hl[q].y, dw[q]);
                }
            }
        }
        __syncthreads();
        if (sh.heavy) {
            for_heavy(seq + begin, end - begin, off_in, [&](uint32_t v) {
                const uint32_t dv = dist_at(v);
                const uint64_t ie = off_in[v + 1];
                double acc = 0.0;
                for (uint64_t a = off_in[v]; a < ie; a += 32) {
                    double sp = 0.0;
                    if (a + lane < ie) {
                        const uint2 hl = arc_in[a + lane];
                        if (dist_at(hl.x) + hl.y == dv) sp = __ldcg(&sigma[hl.x]);
                    }
                    for (uint32_t m = __ballot_sync(kFull, sp != 0.0); m; m &= m - 1)
                        acc = __dadd_rn(acc, __shfl_sync(kFull, sp, __ffs(m) - 1));
                }
                if (lane == 0) __stcg(&sigma[v], v == s ? 1.0 : acc);
            });
            for_heavy(seq + begin, end - begin, off_out, [&](uint32_t v) {
                const uint32_t dv = dist_at(v);
                for (uint64_t a = off_out[v] + lane; a < off_out[v + 1]; a += 32) {
                    const uint2 hl = arc_out[a];
                    count_down(hl.x, dv + hl.y, dist_at(hl.x));
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
    while (waves-- > 0) {
        begin = __ldcg(&wave[waves]);
        if (tid == 0) sh.heavy = 0;
        __syncthreads();
        for (uint32_t i = begin + tid; i < end; i += kOrdThreads) {
            const uint32_t v = __ldcg(&seq[i]);
            const uint64_t ob = off_out[v], oe = off_out[v + 1];
            if (oe - ob > kLight) {
                sh.heavy = 1;
                continue;
            }
            const uint32_t dv = dist_at(v);
            const double sv = __ldcg(&sigma[v]);
            double acc = 0.0;
#pragma unroll
            for (int h = 0; h < kLight; h += kGroup) {
                if (ob + h >= oe) break;
                uint2 hl[kGroup];
                bool on[kGroup];
                double sw[kGroup], dw[kGroup];
#pragma unroll
                for (int q = 0; q < kGroup; ++q) hl[q] = ob + h + q < oe ? arc_out[ob + h + q] : make_uint2(v, 1u);
#pragma unroll
                for (int q = 0; q < kGroup; ++q) {
                    const uint32_t d = dist_at(hl[q].x);
                    on[q] = d != kInfD && dv + hl[q].y == d;
                }
#pragma unroll
                for (int q = 0; q < kGroup; ++q) {
                    sw[q] = on[q] ? __ldcg(&sigma[hl[q].x]) : 1.0;
                    dw[q] = on[q] ? __ldcg(&delta[hl[q].x]) : 0.0;
                }
#pragma unroll
                for (int q = 0; q < kGroup; ++q)
                    if (on[q]) acc = __dadd_rn(acc, __dmul_rn(__ddiv_rn(sv, sw[q]), __dadd_rn(1.0, dw[q])));
            }
            __stcg(&delta[v], v == s ? 0.0 : acc);   // the source's own dependency is not counted
        }
        __syncthreads();
        if (sh.heavy) {
            for_heavy(seq + begin, end - begin, off_out, [&](uint32_t v) {
                const uint64_t oe = off_out[v + 1];
                const uint32_t dv = dist_at(v);
                const double sv = __ldcg(&sigma[v]);
                double acc = 0.0;
                for (uint64_t a = off_out[v]; a < oe; a += 32) {
                    bool on = false;
                    double t = 0.0;
                    if (a + lane < oe) {
                        const uint2 hl = arc_out[a + lane];
                        const uint32_t d = dist_at(hl.x);
                        on = d != kInfD && dv + hl.y == d;
                        if (on)
                            t = __dmul_rn(__ddiv_rn(sv, __ldcg(&sigma[hl.x])), __dadd_rn(1.0, __ldcg(&delta[hl.x])));
                    }
                    for (uint32_t m = __ballot_sync(kFull, on); m; m &= m - 1)
                        acc = __dadd_rn(acc, __shfl_sync(kFull, t, __ffs(m) - 1));
                }
                if (lane == 0) __stcg(&delta[v], v == s ? 0.0 : acc);
            });
        }
        __syncthreads();
        end = begin;
    }
}

// bc[v] = sum over sources j (in list order) of delta_j[v]
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
