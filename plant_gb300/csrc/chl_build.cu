// Canonical hub label construction on one GPU.
//
// Reference path being replaced:
//   hl::run_paraPLL            shared_memory/akiba.hpp:132-217  (GLL supersteps)
//   hl::Akiba::iteration_gll   shared_memory/akiba.hpp:65-125   (pruned Dijkstra)
//   hl::Akiba::plant           distributed_memory/akiba.hpp:52-104 (PLaNT tree)
//   BasicDijkstra::update_wo_prune distributed_memory/dijkstra.hpp:56-78
//   hl::run (hybrid switch)    distributed_memory/akiba.hpp:290-336, 479-480
//   Labeling::sort / clean_cover shared_memory/labeling.hpp:222-256, 78-88
//
// Design (one process, one GPU):
//  * Roots are taken in rank order in supersteps.  A persistent kernel runs
//    one tree per block or warp, or 1,024 at once (below); its blocks pull
//    roots from a device counter until the superstep's label budget (sf * n,
//    the reference's label_limit) is spent.
//  * Every tree prunes only against labels committed by EARLIER supersteps
//    (read-only during the kernel), so a superstep's output does not depend
//    on warp scheduling.
//  * PLaNT trees track the "via a higher-ranked vertex" flag exactly as
//    update_wo_prune does and emit canonical labels directly; GLL trees skip
//    higher-ranked vertices and emit a superset that the clean kernel
//    filters with the reference's clean_cover rule.
//  * New labels are sorted by (vertex, side, hub) with a stable radix sort
//    and merged into the committed CSR (double-buffered) in one pass; a
//    second copy of every list, ordered by (distance, hub), is merged too.
//  * Large trees are searched by a block each (team_kernel), label-correcting
//    in distance windows; on road-like graphs without prune tests and mostly
//    in one superstep.
//  * Unit-length heavy-tailed graphs grow 32 trees per 32-bit word of a vertex,
//    level by level and all roots at once (bit_level), up to where their trees
//    are small.
//  * Small pruned trees are built by a warp each (batch_kernel): vertices
//    settle in batches by the IN criterion from a near/far queue and are
//    pruned with one 16-entry item of the distance-ordered lists per lane
//    against a shared-memory hash of the root's label.
#include "chl_dev.cuh"

#include <algorithm>
#include <chrono>
#include <type_traits>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <memory>
#include <vector>

namespace chl {

namespace {

constexpr uint32_t kInf = 0xFFFFFFFFu;
constexpr int kWarpsPerBlock = 4;
#ifndef CHL_PHASE_TIMING
#define CHL_PHASE_TIMING 0              // 1: per-phase clock64 counters (diagnostic builds)
#endif
constexpr bool kPhaseTiming = CHL_PHASE_TIMING != 0;
// batched settle code-shape switches (for A/B measurements)
#ifndef CHL_SCAN_CHUNKS
#define CHL_SCAN_CHUNKS 4    // 32-entry frontier chunks per scan step
#endif
#ifndef CHL_SMEM_CAP_KB
#define CHL_SMEM_CAP_KB 112  // dynamic shared memory per block, at most (2 blocks per SM)
#endif
#ifndef CHL_BATCH_MIN_BLOCKS
#define CHL_BATCH_MIN_BLOCKS 0   // batched settle launch bound (0: compiler's choice;
                                 // 1 measured slower: more registers, fewer warps)
#endif
#ifndef CHL_RELAX_PRECHECK
#define CHL_RELAX_PRECHECK 1   // read a key before its atomicMin; skip the atomic when it cannot lower it
#endif
#ifndef CHL_RELAX_CHUNKS
#define CHL_RELAX_CHUNKS 3   // 32-arc chunks per relax step
#endif

struct BuildCtl {
    unsigned long long next_root;   // root fetch counter (absolute rank)
    unsigned long long nlab;        // labels emitted this superstep
    unsigned long long visits;
    unsigned long long label_reads;
    unsigned long long arcs;
    unsigned long long n_keep;      // labels surviving the clean pass
    unsigned int overflow;
    unsigned int err;               // 1: distance overflow, 2: workspace bound
    unsigned int max_dist;          // largest distance of a label emitted this superstep
    unsigned int ratio_stop;        // the superstep ended by TreeArgs::visit_ratio
    unsigned long long max_ratio_num;  // (tree, labels) of the worst root
    unsigned long long max_ratio_den;
    unsigned long long running;     // trees of the nominal root range in progress
    unsigned long long close_at;    // first root refused after the extension closed
    unsigned long long cyc[10];     // per-phase SM cycles summed over warps (diagnostics; [8]: prune
                                    // item selection, part of [2]; [9]: selection passes, a count)
    unsigned long long cnt[4];      // frontier entries scanned, rounds, settle calls, far pile entries read
};

struct TreeArgs {
    uint32_t n;
    int sides;                      // 1: symmetric graph, one label side stored
    const uint64_t *g_off[2];       // [f]: arcs traversed by trees of side f
    const uint4 *g_farc[2];         // (head, length, rank[head], win[head]) per arc
    const uint2 *g_fhead[2];        // (head, rank[head]) per arc, unit lengths
    const uint4 *g_row[2];          // weighted unpruned trees: kRowArcs records per vertex, see arc_rows
    const uint32_t *order;
    const uint32_t *newid, *orig;   // team kernel without prune tests: the graph's numbering there (null: the caller's)
    const uint32_t *rank;
    const uint64_t *l_off;          // committed labels, index lidx(v, side)
    const uint2 *l_ent;             // entries ordered by hub
    const uint2 *l_dent;            // the same entries ordered by (distance, hub)
    uint32_t r0, r_end;
    uint32_t r_hard;                // roots past r_end taken while nominal trees run
    unsigned long long budget;
    int hub_bits;
    uint64_t *out_key;
    uint32_t *out_val;
    unsigned long long out_cap;
    uint32_t *tree_size;            // per root (index r - r0), sides summed
    uint32_t *tree_labels;
    uint32_t *ws_key;               // per warp slot, n keys each (64-bit on weighted graphs)
    uint32_t *ws_vis;
    uint32_t *ws_front;             // per warp slot: queue, next queue, far pile
    uint32_t *ws_win;               // team kernel: 6 n words per tree (block)
    BuildCtl *ctl;
    uint32_t hash_slots;            // root hash table slots (a power of two)
    uint32_t hash_shift;            // 32 - log2(hash_slots)
    uint32_t near_on;               // queue size that starts the near/far split (0: never)
    uint32_t near_target;           // near entries aimed at per refill
    uint32_t visit_ratio;           // no new tree once more than this many vertices per
                                    // label were settled (0: no limit)
    unsigned long long visit_base;  // settled vertices the ratio lets pass at first
};

// Phase-timing clock: with CHL_PHASE_TIMING it is also a compiler memory
// barrier, so loads and stores are not moved across phase boundaries (a
// stall is charged to the phase that uses the value); otherwise 0.
__device__ __forceinline__ long long phase_clock() {
    if (!kPhaseTiming) return 0;
    long long t;
    asm volatile("mov.u64 %0, %%clock64;" : "=l"(t)::"memory");
    return t;
}

__device__ __forceinline__ uint32_t lidx(uint32_t v, int side, int sides) {
    return sides == 1 ? v : 2 * v + (uint32_t)side;
}

// ------------------------------------------------------ batch tree kernel
//
// One tree per warp, settled in batches.  A queued vertex v is final (its
// distance AND its via flag) once d(v) < dmin + win(v), where dmin is the
// smallest queued distance and win(v) the shortest arc into v: every
// predecessor p on a shortest path then has d(p) <= d(v) - win(v) < dmin and
// is already settled (the IN criterion of Crauser et al.).  All qualifying
// vertices are settled together:
//   * the queue is an unordered array scanned by the whole warp; a long
//     queue is split at a distance threshold into a near part, scanned
//     every round, and a far pile, read only when the near part runs out;
//   * prune tests are flattened to (vertex, 16-entry chunk) items taken
//     chunk-major, one per lane (default; 32- and 64-entry items in lane
//     groups, and one lane group per vertex, are options); with the
//     distance-ordered lists a vertex's remaining items are dropped once a
//     chunk passes d(r, u);
//   * the arcs of the batch are flattened over the lanes and relaxed with
//     atomicMin on the packed (distance, via) key.
// With unit lengths a batch is exactly one BFS level.  Relaxations from a
// batch cannot improve a batch vertex, so batch order never matters.
#ifndef CHL_KBATCH
#define CHL_KBATCH 256
#endif
constexpr int kBatch = CHL_KBATCH;   // settled vertices buffered per warp (<= 256: item packing)

constexpr int kEmit = 64;   // labels staged per warp before an append

__host__ __device__ constexpr size_t batch_smem_per_warp(uint32_t hash_slots) {
    return ((size_t)8 * kBatch + (size_t)8 * hash_slots + (size_t)4 * (8 * kBatch + 1) + 8 +
            (size_t)12 * kEmit + 15) &
           ~(size_t)15;
}

// The root's committed label as an open-addressing hash table in shared
// memory (linear probing, load <= 1/2), so the up to 8 lookups of a lane are
// independent instead of a chain of dependent binary-search probes.  Entries
// beyond the table's half capacity (the highest hubs) stay in the global
// sorted list and are searched there.  Slot = hub << 32 | dist; ~0 = empty
// (hub 0xFFFFFFFF never occurs: hubs are ranks < n < 2^32).
constexpr uint64_t kSlotEmpty = ~0ull;

__device__ __forceinline__ uint32_t slot_of(uint32_t h, uint32_t shift) { return (h * 0x9E3779B1u) >> shift; }

struct RootHash {
    const uint64_t *tab;
    uint32_t mask;      // table slots - 1
    uint32_t Th;        // entries hashed (the first Th of the list)
    uint32_t hlast;     // hub of entry Th - 1 (0 if Th == 0)
    const uint2 *g;     // whole list in global memory
    uint32_t R;
    // lookup of h; *dist set when found
    __device__ __forceinline__ bool find_tail(uint32_t h, uint32_t &dist) const {
        uint32_t lo = Th, hi = R;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(&g[mid].x) < h) lo = mid + 1;
            else hi = mid;
        }
        if (lo < R) {
            const uint2 e = __ldg(&g[lo]);
            if (e.x == h) {
                dist = e.y;
                return true;
            }
        }
        return false;
    }
};

// Work-conserving supersteps.  A superstep's nominal roots are [r0, r_end);
// while any nominal tree is still running, idle warps take further roots up
// to r_hard instead of waiting (a superstep is as long as its largest tree,
// which one warp builds).  The processed roots stay one contiguous range:
// the warp that ends the last running nominal tree sets kClosed in the fetch
// counter with one atomicOr, and every fetch returning a value with kClosed
// set is refused; close_at records the first refused rank.  Any consecutive
// root range per superstep gives the same labels: trees prune only against
// the labels of earlier supersteps.
constexpr unsigned long long kClosed = 1ull << 62;

__device__ __forceinline__ uint32_t sat_add(uint32_t x, uint32_t y) {
    const uint32_t z = x + y;
    return z < x ? 0xFFFFFFFFu : z;
}

__device__ __forceinline__ uint32_t fetch_root(const TreeArgs &a, bool &nominal) {
    nominal = false;
    const unsigned long long used = *(volatile unsigned long long *)&a.ctl->nlab;
    // no new tree once the budget is spent, or once the label buffer is full
    // (the superstep's range is then re-run with a larger buffer)
    if (used >= a.budget || used >= a.out_cap) return kInf;
    if (a.visit_ratio &&
        *(volatile unsigned long long *)&a.ctl->visits > a.visit_base + used * (unsigned long long)a.visit_ratio) {
        a.ctl->ratio_stop = 1;
        return kInf;
    }
    const unsigned long long t = atomicAdd(&a.ctl->next_root, 1ull);
    if (t & kClosed) return kInf;
    if (t < a.r_end) {
        atomicAdd(&a.ctl->running, 1ull);
        nominal = true;
        return (uint32_t)t;
    }
    return t < a.r_hard ? (uint32_t)t : kInf;
}

__device__ __forceinline__ void finish_root(const TreeArgs &a, bool nominal) {
    if (!nominal || a.r_hard <= a.r_end) return;
    if (atomicAdd(&a.ctl->running, ~0ull) == 1ull &&
        (*(volatile unsigned long long *)&a.ctl->next_root & ~kClosed) >= a.r_end) {
        const unsigned long long old = atomicOr(&a.ctl->next_root, kClosed);
        if (!(old & kClosed)) a.ctl->close_at = old;
    }
}

template <bool UNIT, bool PLANT>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, CHL_BATCH_MIN_BLOCKS)
batch_kernel(TreeArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t lane = lane_id(), wib = threadIdx.x >> 5;
    const uint32_t slot = blockIdx.x * kWarpsPerBlock + wib;
    unsigned char *base = smem + wib * batch_smem_per_warp(a.hash_slots);
    uint64_t *s_ba = (uint64_t *)base;                 // arc begin of batch vertex
    uint64_t *s_tab = s_ba + kBatch;                   // root label hash table
    uint32_t *s_bv = (uint32_t *)(s_tab + a.hash_slots);   // batch vertex
    uint32_t *s_bk = s_bv + kBatch;                    // batch key
    uint32_t *s_bp = s_bk + kBatch;                    // 1: pruned or skipped
    uint32_t *s_bx = s_bp + kBatch;                    // arc prefix (kBatch + 1)
    uint32_t *s_tl = s_bx + kBatch + 1;                // batch indices still to test
    uint32_t *s_bl = s_tl + kBatch;                    // label list length
    uint32_t *s_nch = s_bl + kBatch;                   // label list chunks
    uint32_t *s_as = s_nch + kBatch;                   // next chunk to test, per batch vertex
    uint64_t *s_ek = (uint64_t *)(((uintptr_t)(s_as + kBatch) + 7) & ~(uintptr_t)7);   // staged label keys
    uint32_t *s_ev = (uint32_t *)(s_ek + kEmit);       // staged label distances

    // A vertex's key (distance * 2 + not-via).  On weighted graphs it shares
    // a 64-bit word with win(v), the shortest arc into v (key in the high
    // half, so atomicMin orders by key): the frontier scan gets both with
    // one load.  Unit lengths have win(v) = 1 and 32-bit keys.
    using KeyW = typename std::conditional<UNIT, uint32_t, unsigned long long>::type;
    KeyW *key = (KeyW *)a.ws_key + (size_t)slot * a.n;
    constexpr KeyW kKeyNone = (KeyW)~(KeyW)0;
    uint32_t *vis = a.ws_vis + (size_t)slot * a.n;
    // queue as two arrays: a round reads `front` and writes the vertices it
    // keeps, and those its relaxations add, to `fnext`; then they swap
    uint32_t *front = a.ws_front + (size_t)slot * 3 * a.n;
    uint32_t *fnext = front + a.n;
    // far pile of the near/far queue (see the round loop)
    uint32_t *pile = fnext + a.n;
    unsigned long long c_vis = 0, c_reads = 0, c_arcs = 0;
    long long cyc[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};   // phase cycles (diagnostics)
    unsigned long long dcnt[4] = {0, 0, 0, 0};      // scanned, rounds, settles, far pile entries
    const long long k_start = phase_clock();

    // emitted labels are staged in shared memory and appended to the new
    // label arrays kEmit at a time (one atomic per flush instead of one
    // per settle round)
    uint32_t n_emit = 0;
    uint32_t d_hi = 0;   // largest distance this lane has written
    auto flush_labels = [&]() {
        __syncwarp();
        if (n_emit) {
            unsigned long long b = 0;
            if (lane == 0) b = atomicAdd(&a.ctl->nlab, (unsigned long long)n_emit);
            b = __shfl_sync(kFull, b, 0);
            for (uint32_t k = lane; k < n_emit; k += 32) {
                const unsigned long long p = b + k;
                d_hi = max(d_hi, s_ev[k]);
                if (p < a.out_cap) {
                    a.out_key[p] = s_ek[k];
                    a.out_val[p] = s_ev[k];
                } else {
                    a.ctl->overflow = 1;
                }
            }
        }
        n_emit = 0;
        __syncwarp();
    };
    for (uint32_t k = lane; k < a.hash_slots; k += 32) s_tab[k] = kSlotEmpty;
    __syncwarp();
    while (true) {
        uint32_t r = kInf;
        bool r_nominal = false;
        if (lane == 0) r = fetch_root(a, r_nominal);
        r = __shfl_sync(kFull, r, 0);
        r_nominal = __shfl_sync(kFull, r_nominal ? 1u : 0u, 0) != 0;
        if (r == kInf) break;
        uint32_t t_size = 0, t_lab = 0;
        const uint32_t v = a.order[r];
        for (int sd = 0; sd < a.sides; ++sd) {
            const long long tr0 = phase_clock();
            const int f = (a.sides == 1) ? 1 : sd;
            const uint64_t *goff = a.g_off[f];
            const uint4 *farc = a.g_farc[f];
            const uint2 *fhead = a.g_fhead[f];
            // label entries the prune tests scan: the distance-ordered copy
            const uint2 *lscan = a.l_dent;
            const uint32_t ridx = lidx(v, f, a.sides);
            const uint64_t rb = a.l_off[ridx], re = a.l_off[ridx + 1];
            const uint32_t R = (uint32_t)(re - rb);
            RootHash rhash;
            rhash.tab = s_tab;
            rhash.mask = a.hash_slots - 1;
            rhash.g = a.l_ent + rb;
            rhash.R = R;
            rhash.hlast = 0;
            rhash.Th = min(R, a.hash_slots / 2);
            for (uint32_t k = lane; k < rhash.Th; k += 32) {
                const uint2 e = a.l_ent[rb + k];
                const uint64_t val = ((uint64_t)e.x << 32) | e.y;
                uint32_t sl = slot_of(e.x, a.hash_shift);
                while (atomicCAS((unsigned long long *)&s_tab[sl], (unsigned long long)kSlotEmpty,
                                 (unsigned long long)val) != (unsigned long long)kSlotEmpty)
                    sl = (sl + 1) & rhash.mask;
            }
            if (rhash.Th) rhash.hlast = a.l_ent[rb + rhash.Th - 1].x;
            // Prune test of one lane's 16 consecutive entries of the
            // distance-ordered L(u) against the hashed root label.  vm marks the entries that belong to the list;
            // an entry beyond d(r, u) witnesses nothing and, the list being
            // in distance order, marks the list exhausted.
            auto test16d = [&](const uint4 (&q)[8], uint32_t vm, uint32_t gdj, bool &exhausted) -> bool {
                bool hit = false;
                uint64_t v[16];
                uint32_t sl[16];
                uint32_t pend = 0;
#pragma unroll
                for (int t = 0; t < 16; ++t) {
                    const uint32_t hh = (t & 1) ? q[t >> 1].z : q[t >> 1].x;
                    const uint32_t dd = (t & 1) ? q[t >> 1].w : q[t >> 1].y;
                    const bool in = (vm >> t) & 1u;
                    v[t] = kSlotEmpty;
                    sl[t] = 0;
                    if (in && dd > gdj) exhausted = true;
                    if (in && dd <= gdj && rhash.Th && hh <= rhash.hlast) {
                        sl[t] = slot_of(hh, a.hash_shift);
                        v[t] = s_tab[sl[t]];
                        pend |= 1u << t;
                    }
                }
                if (rhash.Th < R) {
                    // hubs past the hashed prefix: binary search of the rest
#pragma unroll
                    for (int t = 0; t < 16; ++t) {
                        const uint32_t hh = (t & 1) ? q[t >> 1].z : q[t >> 1].x;
                        const uint32_t dd = (t & 1) ? q[t >> 1].w : q[t >> 1].y;
                        if (((vm >> t) & 1u) && dd <= gdj && !(rhash.Th && hh <= rhash.hlast)) {
                            uint32_t dr;
                            if (rhash.find_tail(hh, dr) && dr + dd <= gdj) hit = true;
                        }
                    }
                }
#pragma unroll
                for (int t = 0; t < 16; ++t) {
                    if (!(pend >> t & 1u)) continue;
                    const uint32_t hh = (t & 1) ? q[t >> 1].z : q[t >> 1].x;
                    const uint32_t dd = (t & 1) ? q[t >> 1].w : q[t >> 1].y;
                    uint64_t w = v[t];
                    uint32_t z = sl[t];
                    while (w != kSlotEmpty && (uint32_t)(w >> 32) != hh) {
                        z = (z + 1) & rhash.mask;
                        w = s_tab[z];
                    }
                    if (w != kSlotEmpty && (uint32_t)w + dd <= gdj) hit = true;
                }
                return hit;
            };
            if (lane == 0) {
                __stcg(&key[v], UNIT ? (KeyW)1u : (KeyW)((1ull << 32) | 1u));   // win 1 admits the root
                vis[0] = v;
                front[0] = v;
            }
            __syncwarp();
            cyc[5] += phase_clock() - tr0;
            uint32_t nvis = 1, nf = 1, nn = 0;   // queue sizes in front and fnext
            // Near/far queue.  A large queue is split at a threshold thr:
            // keys below it are queued in front/fnext and scanned every
            // round, the rest in the far pile, read only when the near
            // vertices run out.  thr == kInf: no split (all queued near).
            uint32_t npile = 0;         // far pile entries (stale ones included)
            uint32_t thr = kInf;
            uint32_t pmin = kInf;       // per lane: lower bound of the live far keys
            uint32_t delta = 0;         // threshold step (0: choose at the next refill)
            int ql = 1;
            uint32_t dmin = 0;          // smallest queued distance (exact, see below)
            bool stop = false;
            uint32_t nb = 0;            // vertices in the smem batch

            // Settle the batch held in smem: prune tests, labels, relaxations.
            // New vertices are appended to fnext; every key decrease of
            // a queued vertex lowers dnext, so dnext is the exact minimum of
            // the queue after the round.
            uint32_t dnext = kInf;
            auto settle = [&]() {
                long long tc0 = phase_clock();
                if (kPhaseTiming) dcnt[2]++;
                t_size += nb;
                int nv_batch = 0;
                for (uint32_t j = lane; j < nb; j += 32) {
                    const uint32_t kx = s_bk[j];
                    const uint32_t rx = __ldg(&a.rank[s_bv[j]]);   // batch vertices only, not every scanned one
                    uint32_t skip;
                    if (PLANT) {
                        nv_batch += (int)(kx & 1u);
                        // a committed vertex (rank < r0) always has a committed
                        // witness: pruned without reading its labels
                        skip = rx < a.r0 ? 1u : 0u;
                    } else {
                        skip = rx < r ? 1u : 0u;   // iteration_gll :92
                    }
                    s_bp[j] = skip;
                }
                if (PLANT) ql -= __reduce_add_sync(kFull, nv_batch);
                __syncwarp();
                long long tc1 = phase_clock();
                cyc[1] += tc1 - tc0;
                if (R > 0) {
                    // Prune tests as (vertex, 16-entry chunk) items, one per
                    // lane and step.  The vertices still under test wait in a
                    // circular queue (s_tl, kBatch entries): a step takes up
                    // to 32 from its front -- with fewer than 32, each gets
                    // several consecutive chunks -- and puts back at the end
                    // those with no witness yet whose list has not passed
                    // d(r, u).  Each vertex gets about one chunk per trip
                    // through the queue (chunk-major order), and no step
                    // looks at a vertex that is already decided.
                    uint32_t nq = 0;
                    for (uint32_t j0 = 0; j0 < nb; j0 += 32) {
                        const uint32_t j = j0 + lane;
                        const bool t = j < nb && s_bp[j] == 0;
                        const uint32_t m = __ballot_sync(kFull, t);
                        if (t) {
                            s_tl[nq + __popc(m & lanemask_lt())] = j;
                            const uint32_t xu = lidx(s_bv[j], 1 - f, a.sides);
                            const uint64_t lb = a.l_off[xu], le = a.l_off[xu + 1];
                            s_ba[j] = lb;
                            s_bl[j] = (uint32_t)(le - lb);
                            s_nch[j] = (uint32_t)((le - (lb & ~1ull) + 15) >> 4);
                            s_as[j] = 0;   // next chunk to test
                        }
                        nq += __popc(m);
                    }
                    __syncwarp();
                    uint32_t qh = 0, nread = 0;
                    while (nq > 0) {
                        const long long tsel = phase_clock();
                        if (kPhaseTiming) cyc[9]++;
                        const uint32_t t = min(nq, 32u);
                        // lane -> (vertex of the queue front, chunk)
                        const uint32_t vi = lane % t;
                        const uint32_t lj = s_tl[(qh + vi) % (uint32_t)kBatch];
                        const uint32_t c = s_as[lj] + lane / t;
                        const bool act = c < s_nch[lj];
                        cyc[8] += phase_clock() - tsel;
                        // one 16-entry item per lane (8 loads of one 128-byte
                        // line in flight per lane)
                        bool hit = false, exhausted = false;
                        if (act) {
                            const uint64_t glb = s_ba[lj];
                            const uint64_t gle = glb + s_bl[lj];
                            const uint32_t gdj = s_bk[lj] >> 1;
                            const uint64_t e0 = (glb & ~1ull) + 16ull * c;
                            // entries [lo, hi) of the 16 belong to the list: lo
                            // is 1 only in chunk 0 of an odd start, and an
                            // active item has e0 < gle
                            const uint32_t lo = (uint32_t)(glb - min(glb, e0));
                            const uint64_t span = gle - e0;
                            const uint32_t hi = span < 16 ? (uint32_t)span : 16u;
                            const uint32_t vm = ((1u << hi) - 1u) & ~((1u << lo) - 1u);
                            uint4 q[8];
#pragma unroll
                            for (int u = 0; u < 8; ++u) {
                                q[u] = make_uint4(0, 0, 0, 0);
                                if ((vm >> (2 * u)) & 3u) q[u] = *(const uint4 *)(lscan + e0 + 2 * u);
                            }
                            hit = test16d(q, vm, gdj, exhausted);
                            nread += 16;
                        }
                        if (hit) s_bp[lj] = 1;
                        else if (exhausted) atomicOr(&s_bp[lj], 2u);
                        __syncwarp();
                        // the front t vertices leave the queue; those still
                        // undecided with chunks left go back at the end
                        bool back = false;
                        uint32_t bj = 0;
                        if (lane < t) {
                            bj = lj;   // vi == lane here
                            const uint32_t taken = 32u / t + (lane < 32u % t ? 1u : 0u);
                            const uint32_t nc = s_as[bj] + taken;
                            s_as[bj] = nc;
                            back = s_bp[bj] == 0 && nc < s_nch[bj];
                        }
                        const uint32_t bm = __ballot_sync(kFull, back);
                        qh = (qh + t) % (uint32_t)kBatch;
                        nq -= t;
                        if (back) s_tl[(qh + nq + __popc(bm & lanemask_lt())) % (uint32_t)kBatch] = bj;
                        nq += __popc(bm);
                        __syncwarp();
                    }
                    c_reads += nread;
                    __syncwarp();
                }
                long long tc2 = phase_clock();
                cyc[2] += tc2 - tc1;
                for (uint32_t j0 = 0; j0 < nb; j0 += 32) {
                    const uint32_t j = j0 + lane;
                    bool emit = false;
                    uint32_t xu = 0, dj = 0;
                    if (j < nb && (s_bp[j] & 1u) == 0) {
                        const uint32_t kx = s_bk[j];
                        emit = !PLANT || (kx & 1u);
                        xu = lidx(s_bv[j], 1 - f, a.sides);
                        dj = kx >> 1;
                    }
                    const uint32_t em = __ballot_sync(kFull, emit);
                    if (em) {
                        // labels go through the warp's shared staging buffer
                        if (n_emit + 32 > (uint32_t)kEmit) flush_labels();
                        if (emit) {
                            const uint32_t at = n_emit + __popc(em & lanemask_lt());
                            s_ek[at] = ((uint64_t)xu << a.hub_bits) | (uint64_t)(r - a.r0);
                            s_ev[at] = dj;
                        }
                        n_emit += __popc(em);
                        t_lab += __popc(em);
                    }
                }
                long long tc3 = phase_clock();
                cyc[3] += tc3 - tc2;
                // arcs of the batch flattened over the lanes: the vertices
                // with arcs are compacted (s_tl[k] = batch index, s_bx[k] =
                // first flattened arc), so the owner of arc t0 + lane is the
                // window's first owner plus the vertex starts inside the
                // window below the lane (one OR-reduction, no search)
                uint32_t total = 0, ncomp = 0;
                for (uint32_t j0 = 0; j0 < nb; j0 += 32) {
                    const uint32_t j = j0 + lane;
                    uint32_t deg = 0;
                    if (j < nb && (s_bp[j] & 1u) == 0) {
                        const uint32_t x = s_bv[j];
                        const uint64_t ab = goff[x];
                        deg = (uint32_t)(goff[x + 1] - ab);
                        s_ba[j] = ab;
                    }
                    uint32_t incl = deg;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t y = __shfl_up_sync(kFull, incl, o);
                        if (lane >= (uint32_t)o) incl += y;
                    }
                    const uint32_t nem = __ballot_sync(kFull, deg > 0);
                    if (deg > 0) {
                        const uint32_t k = ncomp + __popc(nem & lanemask_lt());
                        s_tl[k] = j;
                        s_bx[k] = total + incl - deg;
                    }
                    total += __shfl_sync(kFull, incl, 31);
                    ncomp += __popc(nem);
                }
                if (lane == 0) s_bx[ncomp] = total;
                __syncwarp();
                c_arcs += total;
                uint32_t cur = 0;   // compacted owner of arc t0
                // owner (compacted index) of arc t0 + lane
                auto owner = [&](uint32_t t0) -> uint32_t {
                    if (cur + 1 < ncomp && s_bx[cur + 1] <= t0) ++cur;
                    uint32_t bit = 0;
                    const uint32_t kk = cur + 1 + lane;
                    if (kk < ncomp) {
                        const uint32_t st = s_bx[kk];
                        if (st < t0 + 32) bit = 1u << (st - t0);
                    }
                    const uint32_t starts = __reduce_or_sync(kFull, bit);
                    const uint32_t upto = lane == 31 ? kFull : ((2u << lane) - 1u);
                    const uint32_t own = cur + (uint32_t)__popc(starts & upto);
                    cur += (uint32_t)__popc(starts);
                    return own;
                };
                // CHL_RELAX_CHUNKS 32-arc chunks per step: their arc loads and
                // atomics are issued together (three measured best on the
                // 1024-square grid and RMAT-20: 3.43 -> 3.31 s and 2.06 ->
                // 1.90 s against two)
                constexpr int RC = CHL_RELAX_CHUNKS;
                int dql = 0;   // this lane's change of the queued not-via count
                for (uint32_t t0 = 0; t0 < total; t0 += 32 * RC) {
                    uint32_t w[RC], nk[RC], old[RC], kxs[RC], len[RC], rk[RC], wn[RC];
                    bool act[RC], upd[RC];
#pragma unroll
                    for (int c = 0; c < RC; ++c) {
                        w[c] = 0;
                        nk[c] = 0;
                        old[c] = kInf;
                        kxs[c] = 0;
                        len[c] = 0;
                        rk[c] = 0;
                        wn[c] = 1;
                        act[c] = false;
                        upd[c] = false;
                    }
#pragma unroll
                    for (int c = 0; c < RC; ++c) {
                        const uint32_t tc = t0 + 32u * c;
                        const uint32_t own = tc < total ? owner(tc) : 0u;
                        const uint32_t t = tc + lane;
                        if (t < total) {
                            const uint32_t lo = s_tl[own];
                            const uint64_t e = s_ba[lo] + (t - s_bx[own]);
                            if (UNIT) {
                                const uint2 hr = fhead[e];
                                w[c] = hr.x;
                                rk[c] = hr.y;
                                len[c] = 1;
                            } else {
                                const uint4 hl = farc[e];
                                w[c] = hl.x;
                                len[c] = hl.y;
                                rk[c] = hl.z;
                                wn[c] = hl.w;
                            }
                            kxs[c] = s_bk[lo];
                            act[c] = true;
                        }
                    }
                    uint32_t nv[RC];
                    KeyW pre[RC];   // the key word before the atomic (keys only decrease)
#pragma unroll
                    for (int c = 0; c < RC; ++c) {
                        nv[c] = (!PLANT || ((kxs[c] & 1u) && rk[c] >= r)) ? 1u : 0u;
                        pre[c] = (CHL_RELAX_PRECHECK && act[c]) ? __ldcg(&key[w[c]]) : kKeyNone;
                    }
#pragma unroll
                    for (int c = 0; c < RC; ++c) {
                        if (!act[c]) continue;
                        const uint64_t dd64 = (uint64_t)(kxs[c] >> 1) + len[c];
                        if (dd64 < 0x7FFFFFFFull) {
                            nk[c] = (uint32_t)dd64 * 2u + nv[c];
                            const uint32_t pk = UNIT ? (uint32_t)pre[c] : (uint32_t)((unsigned long long)pre[c] >> 32);
                            if (pk <= nk[c]) {
                                old[c] = pk;   // no decrease: no atomic
                            } else if (UNIT) {
                                old[c] = (uint32_t)atomicMin(&key[w[c]], (KeyW)nk[c]);
                            } else {
                                const unsigned long long o64 =
                                    atomicMin(&key[w[c]], (KeyW)(((unsigned long long)nk[c] << 32) | wn[c]));
                                old[c] = (uint32_t)(o64 >> 32);
                            }
                            upd[c] = nk[c] < old[c];
                            if (upd[c]) dnext = min(dnext, nk[c] >> 1);
                        } else {
                            a.ctl->err = 1;   // the reference asserts dd < infty
                        }
                    }
#pragma unroll
                    for (int c = 0; c < RC; ++c) {
                        const bool fresh = upd[c] && old[c] == kInf;
                        // queued near: a new key below thr, or a far vertex
                        // whose key drops below it (its far entry goes stale)
                        const uint32_t dk = nk[c] >> 1;
                        const bool to_near = upd[c] && dk < thr && (old[c] == kInf || (old[c] >> 1) >= thr);
                        const uint32_t fm = __ballot_sync(kFull, to_near);
                        if (to_near) {
                            const uint32_t o = __popc(fm & lanemask_lt());
                            if (nn + o < a.n) fnext[nn + o] = w[c];
                            else a.ctl->err = 2;
                        }
                        nn = min(nn + __popc(fm), a.n);
                        const uint32_t vm = thr == kInf ? fm : __ballot_sync(kFull, fresh);
                        if (fresh) {
                            const uint32_t o = __popc(vm & lanemask_lt());
                            if (nvis + o < a.n) vis[nvis + o] = w[c];
                            else a.ctl->err = 2;
                        }
                        nvis = min(nvis + __popc(vm), a.n);
                        if (thr != kInf) {
                            if (upd[c] && dk >= thr) pmin = min(pmin, dk);
                            const bool to_far = fresh && dk >= thr;
                            const uint32_t pm = __ballot_sync(kFull, to_far);
                            if (to_far) {
                                const uint32_t o = __popc(pm & lanemask_lt());
                                if (npile + o < a.n) pile[npile + o] = w[c];
                                else a.ctl->err = 2;
                            }
                            npile = min(npile + __popc(pm), a.n);
                        }
                        if (PLANT && upd[c]) dql += (int)(nk[c] & 1u) - (old[c] == kInf ? 0 : (int)(old[c] & 1u));
                    }
                }
                if (PLANT) ql += __reduce_add_sync(kFull, dql);
                __syncwarp();
                nb = 0;
                if (PLANT && ql == 0) stop = true;   // plant :95 early exit
                cyc[4] += phase_clock() - tc3;
            };

            // Refill the (empty) near queue from the far pile: entries whose
            // key is below the old threshold are stale (their vertex was
            // queued near and is settled), entries below the new threshold
            // thr = (their minimum) + delta move near, the rest stay,
            // compacted in place.  From the second pass on the minimum is
            // exact, so a refill takes at most two passes.
            auto refill = [&]() {
                const long long tf0 = phase_clock();
                uint32_t lo = __reduce_min_sync(kFull, pmin);
                if (delta == 0) {
                    // first refill of the split: delta for about near_target
                    // entries, taking the keys as spread evenly over [min, max]
                    uint32_t mn = kInf, mx = 0;
                    for (uint32_t i = lane; i < npile; i += 32) {
                        const uint32_t k = (uint32_t)(__ldcg(&key[pile[i]]) >> (UNIT ? 1 : 33));
                        mn = min(mn, k);
                        mx = max(mx, k);
                    }
                    mn = __reduce_min_sync(kFull, mn);
                    mx = __reduce_max_sync(kFull, mx);
                    lo = mn;
                    uint64_t d = (uint64_t)(mx - min(mn, mx)) * a.near_target / max(npile, 1u);
                    if (d < 1) d = 1;
                    if (d > 0x7FFFFFFFull) d = 0x7FFFFFFFull;
                    delta = (uint32_t)d;
                    if (kPhaseTiming) dcnt[3] += npile;
                }
                for (int pass = 0; pass < 4 && nf == 0 && npile > 0; ++pass) {
                    const uint32_t t_old = thr;
                    thr = sat_add(lo, delta);
                    uint32_t keep = 0, moved = 0, kmin = kInf, nmin = kInf;
                    if (kPhaseTiming) dcnt[3] += npile;
                    for (uint32_t b0 = 0; b0 < npile; b0 += 32) {
                        const uint32_t i = b0 + lane;
                        const bool valid = i < npile;
                        const uint32_t x = valid ? pile[i] : 0u;
                        const uint32_t k = valid ? (uint32_t)(__ldcg(&key[x]) >> (UNIT ? 1 : 33)) : kInf;
                        const bool live = valid && k >= t_old;
                        const bool nr = live && k < thr;
                        const bool kp = live && !nr;
                        const uint32_t nm = __ballot_sync(kFull, nr);
                        const uint32_t km = __ballot_sync(kFull, kp);
                        // every lane has read its entry (ballots above), and
                        // a kept entry moves only to a lower index
                        if (nr) {
                            front[moved + __popc(nm & lanemask_lt())] = x;
                            nmin = min(nmin, k);
                        }
                        if (kp) {
                            pile[keep + __popc(km & lanemask_lt())] = x;
                            kmin = min(kmin, k);
                        }
                        moved += __popc(nm);
                        keep += __popc(km);
                    }
                    __syncwarp();
                    npile = keep;
                    nf = moved;
                    lo = __reduce_min_sync(kFull, kmin);
                    dmin = __reduce_min_sync(kFull, nmin);   // far keys are >= thr
                    pmin = lane == 0 ? lo : kInf;
                    if (moved < a.near_target / 4) delta = delta < 0x40000000u ? 2u * delta : 0x7FFFFFFFu;
                    else if (moved > 4 * a.near_target) delta = max(delta / 2, 1u);
                }
                if (nf == 0 && npile > 0) a.ctl->err = 2;   // not reached: see above
                cyc[0] += phase_clock() - tf0;
            };

            while ((nf > 0 || npile > 0) && !stop) {
                if (nf == 0) {
                    refill();
                    if (nf == 0) break;
                }
                // One round: walk the queue once.  Vertices with
                // d < dmin + win are final and go to the batch (settled
                // whenever it fills); the rest go to fnext, where the
                // round's relaxations add new vertices (which cannot
                // qualify in this round: their d >= dmin + win).
                const uint32_t nf0 = nf;
                nn = 0;
                dnext = kInf;
                if (kPhaseTiming) {
                    dcnt[0] += nf0;
                    dcnt[1]++;
                }
                // several 32-entry chunks per step: their loads are issued
                // together
                auto classify = [&](bool valid, uint32_t x, uint32_t kx, uint32_t wx) {
                    const bool take = valid && (uint64_t)(kx >> 1) < (uint64_t)dmin + wx;
                    const uint32_t tm = __ballot_sync(kFull, take);
                    if (take) {
                        const uint32_t at = nb + __popc(tm & lanemask_lt());
                        s_bv[at] = x;
                        s_bk[at] = kx;
                    }
                    nb += __popc(tm);
                    const bool kp = valid && !take;
                    const uint32_t km = __ballot_sync(kFull, kp);
                    if (kp) {
                        fnext[nn + __popc(km & lanemask_lt())] = x;
                        dnext = min(dnext, kx >> 1);
                    }
                    nn += __popc(km);
                };
                for (uint32_t b0 = 0; b0 < nf0 && !stop; b0 += 32 * CHL_SCAN_CHUNKS) {
                    if (nb > (uint32_t)kBatch - 32 * CHL_SCAN_CHUNKS) settle();
                    if (stop) break;
                    const long long ts0 = phase_clock();
                    bool vv[CHL_SCAN_CHUNKS];
                    uint32_t xx[CHL_SCAN_CHUNKS], kk[CHL_SCAN_CHUNKS], ww[CHL_SCAN_CHUNKS];
#pragma unroll
                    for (int c = 0; c < CHL_SCAN_CHUNKS; ++c) {
                        const uint32_t i = b0 + 32 * c + lane;
                        vv[c] = i < nf0;
                        xx[c] = vv[c] ? front[i] : 0u;
                    }
#pragma unroll
                    for (int c = 0; c < CHL_SCAN_CHUNKS; ++c) {
                        const KeyW k = vv[c] ? __ldcg(&key[xx[c]]) : kKeyNone;
                        kk[c] = UNIT ? (uint32_t)k : (uint32_t)((unsigned long long)k >> 32);
                        // unit lengths: every queued vertex but the root has an
                        // in-arc of length 1, and 1 also admits the root
                        ww[c] = UNIT ? 1u : (uint32_t)k;
                    }
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < CHL_SCAN_CHUNKS; ++c) classify(vv[c], xx[c], kk[c], ww[c]);
                    __syncwarp();
                    cyc[0] += phase_clock() - ts0;
                }
                if (nb && !stop) settle();
                if (stop) break;
                __syncwarp();
                {
                    uint32_t *t = front;
                    front = fnext;
                    fnext = t;
                }
                nf = nn;
                dmin = __reduce_min_sync(kFull, dnext);
                if (thr == kInf && nf > a.near_on && a.near_on) {
                    // the queue grew large: all of it goes to the far pile,
                    // and the next refill splits it
                    uint32_t *t = pile;
                    pile = front;
                    front = t;
                    npile = nf;
                    nf = 0;
                    thr = 0;
                    delta = 0;
                }
            }
            c_vis += t_size;
            const long long tz0 = phase_clock();
            for (uint32_t k = lane; k < nvis; k += 32) __stcg(&key[vis[k]], kKeyNone);
            for (uint32_t k = lane; k < a.hash_slots; k += 32) s_tab[k] = kSlotEmpty;
            cyc[6] += phase_clock() - tz0;
            __syncwarp();
        }
        flush_labels();
        if (lane == 0) {
            a.tree_size[r - a.r0] = t_size;
            a.tree_labels[r - a.r0] = t_lab;
            finish_root(a, r_nominal);
        }
    }
    d_hi = __reduce_max_sync(kFull, d_hi);
    if (lane == 0) {
        atomicAdd(&a.ctl->visits, c_vis);
        atomicAdd(&a.ctl->arcs, c_arcs);
        if (d_hi) atomicMax(&a.ctl->max_dist, d_hi);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c_reads += __shfl_xor_sync(kFull, c_reads, o);
    if (lane == 0) {
        atomicAdd(&a.ctl->label_reads, c_reads);
        if (kPhaseTiming) {
            cyc[7] = phase_clock() - k_start;   // whole residency of the warp
#pragma unroll
            for (int i = 0; i < 10; ++i) atomicAdd(&a.ctl->cyc[i], (unsigned long long)cyc[i]);
#pragma unroll
            for (int i = 0; i < 4; ++i) atomicAdd(&a.ctl->cnt[i], dcnt[i]);
        }
    }
}

// ------------------------------------------------------ team kernel
//
// One tree per block of T threads, searched label-correcting in distance
// windows [.., thr): every vertex whose key drops below thr is relaxed (again)
// in the next pass until a pass drops none.  Then every key below thr is final
// -- it is the minimum over all paths, and every other queued key is at least
// thr -- so the window's labels are emitted from the final keys, and the next
// window, [thr, lo + width), is taken from the far pile (lo its smallest live
// key).  Keys carry PLaNT's via flag (distance * 2 + not-via), and a flag
// change is a key decrease, so relaxing again on every decrease keeps the
// flags exact; PLaNT's early exit (distributed_memory/akiba.hpp:95) is tested
// at window ends, where the count of queued not-via keys is exact.
//
// Pruning with committed labels stays exact under tentative distances: a
// vertex is tested at the distance d' it is relaxed with.  A witness h with
// d(r, h) + d(h, v) <= d also holds at any d' >= d, so a pruned vertex is
// never expanded, and one that is unpruned at its final d was tested with it
// last.  A vertex ranked above every root of the superstep (rank < r0) always
// has a committed witness, and GLL trees skip every vertex ranked above the
// root (iteration_gll, shared_memory/akiba.hpp:92): neither is queued at all.
//
// Bound by the latency of a pass's chain (entry, key word, arcs, atomic), so
// key and pass mark fall in one 64-bit minimum (the 512-square grid's trees
// 86.5 -> 77.6 ms against two atomics), short lists do without a read of the
// key first (77.1; long lists keep it: on heavy tails 98% of the atomics would
// change nothing), a pass holds only the vertices that changed, a thread
// walks one vertex's arcs with four in flight (weighted trees without prune
// tests: four lanes take a vertex's row, see arc_rows), and one barrier ends a
// pass.  Warps whose vertices have more than kTeamLight arcs, or more than
// their row holds, flatten them over the lanes instead.  Windows are as wide as to hold about near_target vertices.
// Per tree, in the workspace (6 n words): key and pass mark of each vertex in
// one 64-bit word, the vertices that joined a window, and three lists that
// change roles (queue, next queue, far pile).
constexpr int kTeamLight = 8;
constexpr int kTeamArcs = 4;      // arcs in flight per thread
constexpr int kRowArcs = 4;       // arc records per row: one per lane of a group
constexpr int kRowSteps = 3;      // steps of 8 vertices in flight per warp (512-square trees 90.4, 86.8, 85.9, 95.5 ms with 1 to 4)
constexpr int kItem = 8;          // label entries per lane and step of a prune test
// Register budget, as resident warps per SM.  The chains leave a scheduler
// idle most of the time, so more warps pay even at the cost of registers:
// trees of a 512-square grid 159 ms with 20 unpruned warps, 117 with 32, 95
// with 48; pruned ones (1024-square grid, label budget 1024 n) 1.32 s with 20,
// 1.27 with 28, 1.33 with 32.  The budget costs spills: unpruned trees of 2 to
// 8 warps have 40 registers and spill up to 16 bytes, 32 to 80 where they read
// rows; pruned ones have 72 or 80 and spill 48 to 140.
constexpr int team_warps_per_sm(bool prune) { return prune ? 28 : 48; }

struct TeamShared {
    uint32_t root, nominal;
    uint32_t nn[3];     // next queue's length, one counter per pass in turn
    uint32_t nm;        // vertices that joined a window
    uint32_t npile;     // far pile entries (stale ones included)
    uint32_t nkeep;     // entries a refill keeps
    uint32_t lo;        // lower bound of the live far keys' distances
    uint32_t kmin, kmax;
    int ql;             // queued not-via keys (PLaNT)
    uint32_t dnv;       // largest distance of a not-via member so far (PLaNT)
    uint32_t t_size, t_lab;
    uint32_t big;       // a tentative distance reached INT_MAX
    uint32_t err;
};

__host__ __device__ constexpr size_t team_head() { return (sizeof(TeamShared) + 15) & ~(size_t)15; }
__host__ __device__ constexpr size_t team_smem_per_warp() { return (size_t)12 * kEmit + 32 * 4; }
__host__ __device__ constexpr size_t team_smem(int t, uint32_t hash_slots) {
    return team_head() + (size_t)8 * hash_slots + (size_t)(t / 32) * team_smem_per_warp();
}

template <bool UNIT, bool PLANT, bool PRUNE, bool ROWS, int T>
__global__ void __launch_bounds__(T, team_warps_per_sm(PRUNE) * 32 / T) team_kernel(TreeArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    TeamShared &sh = *(TeamShared *)smem;
    uint64_t *s_tab = (uint64_t *)(smem + team_head());   // root label hash table
    const uint32_t tid = threadIdx.x, lane = lane_id(), wib = tid >> 5;
    unsigned char *base = smem + team_head() + (size_t)8 * a.hash_slots + wib * team_smem_per_warp();
    uint64_t *s_ek = (uint64_t *)base;           // staged label keys
    uint32_t *s_ev = (uint32_t *)(s_ek + kEmit); // staged label distances
    uint32_t *s_ow = s_ev + kEmit;               // lanes with arcs, compacted

    // word of a vertex: key in the high half, (pass << 1 | not pruned) in the low
    unsigned long long *kw = (unsigned long long *)(a.ws_win + (size_t)blockIdx.x * 6 * a.n);
    uint32_t *memb = (uint32_t *)(kw + a.n);
    uint32_t *list0 = memb + a.n;
    const uint32_t n = a.n;
    static_assert(!ROWS || (!UNIT && !PRUNE), "rows hold lengths and are not tested");
    auto key_at = [&](uint32_t v) -> const uint32_t * { return (const uint32_t *)(kw + v) + 1; };   // read only
    unsigned long long c_arcs = 0, c_reads = 0;

    uint32_t n_emit = 0;
    uint32_t d_hi = 0;   // largest distance this lane has written
    auto flush_labels = [&]() {
        __syncwarp();
        if (n_emit) {
            unsigned long long b = 0;
            if (lane == 0) b = atomicAdd(&a.ctl->nlab, (unsigned long long)n_emit);
            b = __shfl_sync(kFull, b, 0);
            for (uint32_t k = lane; k < n_emit; k += 32) {
                const unsigned long long p = b + k;
                d_hi = max(d_hi, s_ev[k]);
                if (p < a.out_cap) {
                    a.out_key[p] = s_ek[k];
                    a.out_val[p] = s_ev[k];
                } else {
                    a.ctl->overflow = 1;
                }
            }
        }
        n_emit = 0;
        __syncwarp();
    };
    // warp-wide append of x by the lanes with `take` to a list of at most n
    auto append = [&](bool take, uint32_t x, uint32_t *list, uint32_t *counter) {
        const uint32_t m = __ballot_sync(kFull, take);
        if (!m) return;
        uint32_t b = 0;
        if (lane == 0) b = atomicAdd(counter, (uint32_t)__popc(m));
        b = __shfl_sync(kFull, b, 0) + __popc(m & lanemask_lt());
        if (take) {
            if (b < n) list[b] = x;
            else sh.err = 2;
        }
    };

    if (PRUNE)
        for (uint32_t k = tid; k < a.hash_slots; k += T) s_tab[k] = kSlotEmpty;
    while (true) {
        if (tid == 0) {
            bool nom = false;
            sh.root = fetch_root(a, nom);
            sh.nominal = nom ? 1u : 0u;
            sh.t_size = 0;
            sh.t_lab = 0;
        }
        __syncthreads();
        const uint32_t r = sh.root;
        if (r == kInf) break;
        const uint32_t v_root = !PRUNE && a.newid ? a.newid[a.order[r]] : a.order[r];
        for (int sd = 0; sd < a.sides; ++sd) {
            const int f = (a.sides == 1) ? 1 : sd;
            const uint64_t *goff = a.g_off[f];
            const uint4 *farc = a.g_farc[f];
            const uint2 *fhead = a.g_fhead[f];
            const uint4 *row = a.g_row[f];
            const uint2 *lscan = a.l_dent;
            // heads ranked above this are never queued; without prune tests
            // PLaNT trees need them all: their paths set the via flags
            const uint32_t rskip = PLANT ? (PRUNE ? a.r0 : 0u) : r;
            RootHash rhash;
            uint32_t R = 0;
            if (PRUNE) {
                const uint32_t ridx = lidx(v_root, f, a.sides);
                const uint64_t rb = a.l_off[ridx], re = a.l_off[ridx + 1];
                R = (uint32_t)(re - rb);
                rhash.tab = s_tab;
                rhash.mask = a.hash_slots - 1;
                rhash.g = a.l_ent + rb;
                rhash.R = R;
                rhash.hlast = 0;
                rhash.Th = min(R, a.hash_slots / 2);
                for (uint32_t k = tid; k < rhash.Th; k += T) {
                    const uint2 e = a.l_ent[rb + k];
                    const uint64_t val = ((uint64_t)e.x << 32) | e.y;
                    uint32_t sl = slot_of(e.x, a.hash_shift);
                    while (atomicCAS((unsigned long long *)&s_tab[sl], (unsigned long long)kSlotEmpty,
                                     (unsigned long long)val) != (unsigned long long)kSlotEmpty)
                        sl = (sl + 1) & rhash.mask;
                }
                if (rhash.Th) rhash.hlast = a.l_ent[rb + rhash.Th - 1].x;
            }
            uint32_t *front = list0, *fnext = list0 + n, *pile = list0 + 2 * (size_t)n;
            if (tid == 0) {
                __stcg(&kw[v_root], (1ull << 32) | 1ull);
                memb[0] = v_root;
                front[0] = v_root;
                sh.nn[0] = sh.nn[1] = sh.nn[2] = 0;
                sh.nm = 1;
                sh.npile = 0;
                sh.lo = kInf;
                sh.ql = 1;
                sh.dnv = 0;
                sh.big = 0;
                sh.err = 0;
            }
            __syncthreads();
            uint32_t thr = 1;         // the first window holds the root alone
            uint32_t width = 0;       // 0: choose at the first refill
            uint32_t pass = 1;        // stamps of this tree: 2 * pass, never the reset value
            uint32_t nf = 1, wbegin = 0;
            uint32_t lo = kInf;       // per lane: smallest far distance set since the last refill
            int dql = 0;              // per lane: change of the queued not-via count

            // one relaxed arc per lane: key decrease, and the lists its head joins
            auto relax = [&](bool act, uint32_t k, uint32_t w, uint32_t len, uint32_t rk, uint32_t pre) {
                const uint32_t dd = (k >> 1) + len;   // both below 2^31
                const uint32_t nk = dd * 2u + ((!PLANT || ((k & 1u) && rk >= r)) ? 1u : 0u);
                if (act && dd >= 0x7FFFFFFFu) {
                    sh.big = 1;
                    act = false;
                }
                // keys only decrease: a read no larger than nk proves the atomic idle
                act = act && rk >= rskip && nk < pre;
                const bool near = dd < thr;
                const uint32_t stamp = near ? pass << 1 | 1u : kInf;
                uint32_t old = 0, mark = 0;
                if (act) {
                    // one minimum over key and mark: the smaller key wins, and
                    // brings its mark
                    const unsigned long long was = atomicMin(kw + w, (unsigned long long)nk << 32 | stamp);
                    old = (uint32_t)(was >> 32);
                    mark = (uint32_t)was;
                    act = nk < old || (nk == old && stamp < mark);
                }
                if (!__any_sync(kFull, act)) return;
                bool join = false, next = false, far = false;
                if (act) {
                    if (PLANT && nk < old) dql += (int)(nk & 1u) - (old == kInf ? 0 : (int)(old & 1u));
                    if (near) {
                        // a far vertex whose key drops into the window leaves a stale far entry
                        join = old == kInf || (old >> 1) >= thr;
                        // (an equal key only takes the mark of a vertex the refill
                        // queued: queued again, so that the mark stays true)
                        next = (mark | 1u) != stamp;
                    } else {
                        lo = min(lo, dd);
                        far = old == kInf;
                    }
                }
                append(next, w, fnext, &sh.nn[pass % 3]);
                append(join, w, memb, &sh.nm);
                append(far, w, pile, &sh.npile);
            };

            // arcs flattened over the lanes: lane i owns deg arcs from ab on of a
            // vertex with key k
            auto relax_flat = [&](uint32_t deg, uint64_t ab, uint32_t k) {
                // owner of arc t0 + lane from the list starts inside the 32-arc
                // group (one OR-reduction)
                uint32_t incl = deg;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(kFull, incl, o);
                    if (lane >= (uint32_t)o) incl += y;
                }
                const uint32_t start = incl - deg, total = __shfl_sync(kFull, incl, 31);
                const uint32_t nem = __ballot_sync(kFull, deg > 0);
                if (deg > 0) s_ow[__popc(nem & lanemask_lt())] = lane;
                __syncwarp();
                uint32_t before = 0;   // lists that start before the group
                constexpr int RC = CHL_RELAX_CHUNKS;
                for (uint32_t t0 = 0; t0 < total; t0 += 32 * RC) {
                    uint32_t w[RC], len[RC], rk[RC], pre[RC], kk[RC];
#pragma unroll
                    for (int c = 0; c < RC; ++c) {
                        const uint32_t tc = t0 + 32u * c;
                        const uint32_t bit = deg > 0 && start >= tc && start < tc + 32 ? 1u << (start - tc) : 0u;
                        const uint32_t starts = __reduce_or_sync(kFull, bit);
                        const uint32_t upto = lane == 31 ? kFull : ((2u << lane) - 1u);
                        const uint32_t own = before + (uint32_t)__popc(starts & upto);
                        before += (uint32_t)__popc(starts);
                        const uint32_t ol = s_ow[own ? own - 1 : 0];
                        const uint64_t oab = __shfl_sync(kFull, ab, ol);
                        const uint32_t ost = __shfl_sync(kFull, start, ol);
                        kk[c] = __shfl_sync(kFull, k, ol);
                        w[c] = 0;
                        len[c] = 1;
                        rk[c] = 0;
                        if (tc + lane < total) {
                            const uint64_t e = oab + (tc + lane - ost);
                            if (UNIT) {
                                const uint2 x = fhead[e];
                                w[c] = x.x;
                                rk[c] = x.y;
                            } else {
                                const uint4 x = farc[e];
                                w[c] = x.x;
                                len[c] = x.y;
                                rk[c] = x.z;
                            }
                        }
                    }
#pragma unroll
                    for (int c = 0; c < RC; ++c)
                        pre[c] = t0 + 32u * c + lane < total && rk[c] >= rskip ? __ldcg(key_at(w[c])) : 0u;
#pragma unroll
                    for (int c = 0; c < RC; ++c)
                        relax(t0 + 32u * c + lane < total, kk[c], w[c], len[c], rk[c], pre[c]);
                }
                __syncwarp();
            };

            // one pass over rows: four lanes per vertex, so that a row is one
            // access, eight vertices per step and up to kRowSteps steps in flight
            auto pass_rows = [&]() {
                const uint32_t steps = min((nf + T / 4 - 1) / (T / 4), (uint32_t)kRowSteps);
                const uint32_t g = lane / kRowArcs, slot = lane % kRowArcs;
                for (uint32_t i0 = wib * 8 * steps; i0 < nf; i0 += 8 * steps * (T / 32)) {
                    uint32_t v[kRowSteps], k[kRowSteps];
                    uint4 x[kRowSteps];
#pragma unroll
                    for (int u = 0; u < kRowSteps; ++u) {
                        const uint32_t i = i0 + 8 * u + g;
                        v[u] = (uint32_t)u < steps && i < nf ? __ldcg(&front[i]) : kInf;
                    }
#pragma unroll
                    for (int u = 0; u < kRowSteps; ++u) {
                        k[u] = 0;
                        x[u] = make_uint4(0, 0, 0, 0);
                        if (v[u] != kInf) {
                            x[u] = row[(size_t)v[u] * kRowArcs + slot];
                            k[u] = __ldcg(key_at(v[u]));
                        }
                    }
                    // the vertex of step u is owned by its group's lane u from here on
                    uint32_t deg = 0, own_k = 0;
#pragma unroll
                    for (int u = 0; u < kRowSteps; ++u) {
                        v[u] = __shfl_sync(kFull, x[u].w, lane & ~(kRowArcs - 1));   // the degree
                        if (slot == (uint32_t)u) {
                            deg = v[u];
                            own_k = k[u];
                        }
                    }
                    c_arcs += deg;
                    const bool heavy = __any_sync(kFull, deg > (uint32_t)kTeamLight);
                    uint64_t ab = 0;
                    if (__any_sync(kFull, deg > (uint32_t)kRowArcs)) {
#pragma unroll
                        for (int u = 0; u < kRowSteps; ++u) {
                            const uint32_t lo_w = __shfl_sync(kFull, x[u].w, (lane & ~(kRowArcs - 1)) | 1);
                            const uint32_t hi_w = __shfl_sync(kFull, x[u].w, (lane & ~(kRowArcs - 1)) | 2);
                            if (slot == (uint32_t)u) ab = lo_w | (uint64_t)hi_w << 32;
                        }
                    }
#pragma unroll
                    for (int u = 0; u < kRowSteps; ++u) {
                        if ((uint32_t)u >= steps) break;
                        const bool on = slot < v[u];
                        const uint32_t pre = heavy && on && x[u].z >= rskip ? __ldcg(key_at(x[u].x)) : kInf;
                        relax(on, k[u], x[u].x, x[u].y, x[u].z, pre);   // no read first unless heavy, see above
                    }
                    if (__any_sync(kFull, deg > (uint32_t)kRowArcs))
                        relax_flat(deg > (uint32_t)kRowArcs ? deg - kRowArcs : 0u, ab + kRowArcs, own_k);
                }
            };

            while (true) {
                // passes over the window until no key below thr drops
                while (nf) {
                    if (tid == 0) sh.nn[(pass + 1) % 3] = 0;   // last read two barriers ago
                    if (ROWS) pass_rows();
                    for (uint32_t i0 = wib * 32; !ROWS && i0 < nf; i0 += T) {
                        const bool valid = i0 + lane < nf;
                        uint32_t v = 0, k = 0, deg = 0;
                        uint64_t ab = 0;
                        unsigned long long word = 0;
                        bool test = false;
                        uint64_t lb = 0;
                        uint32_t ln = 0;
                        if (valid) {
                            v = __ldcg(&front[i0 + lane]);
                            word = __ldcg(&kw[v]);
                            ab = goff[v];
                            deg = (uint32_t)(goff[v + 1] - ab);
                            k = (uint32_t)(word >> 32);
                            if (PRUNE && R > 0) {
                                const uint32_t xu = lidx(v, 1 - f, a.sides);
                                lb = a.l_off[xu];
                                ln = (uint32_t)(a.l_off[xu + 1] - lb);
                                test = ln > 0;
                            }
                        }
                        if (PRUNE && R > 0) {
                            // Prune tests: every lane owns a vertex; the lanes take
                            // (vertex, kItem-entry chunk) items of the vertices still
                            // under test, several consecutive chunks of each once
                            // fewer than 32 are left.  Lists are in distance order,
                            // so one is done at its first entry beyond d(r, u).
                            bool hit = false;
                            uint32_t ch = 0;                                  // next chunk of the own vertex
                            const uint32_t nch = (uint32_t)(((lb & 1ull) + ln + kItem - 1) / kItem);
                            uint32_t live = __ballot_sync(kFull, test);
                            while (live) {
                                const uint32_t t = (uint32_t)__popc(live);
                                // lane -> (owner, chunk offset)
                                const uint32_t vi = lane % t, co = lane / t;
                                if (live >> lane & 1u) s_ow[__popc(live & lanemask_lt())] = lane;
                                __syncwarp();
                                const uint32_t ow = s_ow[vi];
                                const uint64_t glb = __shfl_sync(kFull, lb, ow);
                                const uint32_t gln = __shfl_sync(kFull, ln, ow);
                                const uint32_t gd = __shfl_sync(kFull, k, ow) >> 1;
                                const uint32_t c = __shfl_sync(kFull, ch, ow) + co;
                                const uint32_t gnc = __shfl_sync(kFull, nch, ow);
                                bool h = false, done = false;
                                if (c < gnc) {
                                    const uint64_t e0 = (glb & ~1ull) + (uint64_t)kItem * c;
                                    const uint32_t first = e0 < glb ? 1u : 0u;   // odd start: entry 0 is the list before
                                    const uint64_t span = glb + gln - e0;
                                    const uint32_t last = span < kItem ? (uint32_t)span : (uint32_t)kItem;
                                    uint4 q[kItem / 2];
#pragma unroll
                                    for (int u = 0; u < kItem / 2; ++u) {
                                        q[u] = make_uint4(0, 0xFFFFFFFFu, 0, 0xFFFFFFFFu);
                                        if (2u * u < last) q[u] = *(const uint4 *)(lscan + e0 + 2 * u);
                                    }
                                    c_reads += kItem;
                                    uint64_t w[kItem];
                                    uint32_t sl[kItem];
                                    uint32_t pend = 0;
#pragma unroll
                                    for (int u = 0; u < kItem; ++u) {
                                        const uint32_t hh = (u & 1) ? q[u >> 1].z : q[u >> 1].x;
                                        const uint32_t dd = (u & 1) ? q[u >> 1].w : q[u >> 1].y;
                                        const bool in = (uint32_t)u >= first && (uint32_t)u < last;
                                        w[u] = kSlotEmpty;
                                        sl[u] = 0;
                                        if (in && dd > gd) done = true;
                                        if (in && dd <= gd) {
                                            if (hh <= rhash.hlast) {
                                                sl[u] = slot_of(hh, a.hash_shift);
                                                w[u] = s_tab[sl[u]];
                                                pend |= 1u << u;
                                            } else if (rhash.Th < R) {
                                                // hubs past the hashed prefix
                                                uint32_t dr;
                                                if (rhash.find_tail(hh, dr) && dr + dd <= gd) h = true;
                                            }
                                        }
                                    }
#pragma unroll
                                    for (int u = 0; u < kItem; ++u) {
                                        if (!(pend >> u & 1u)) continue;
                                        const uint32_t hh = (u & 1) ? q[u >> 1].z : q[u >> 1].x;
                                        const uint32_t dd = (u & 1) ? q[u >> 1].w : q[u >> 1].y;
                                        uint64_t x = w[u];
                                        uint32_t z = sl[u];
                                        while (x != kSlotEmpty && (uint32_t)(x >> 32) != hh) {
                                            z = (z + 1) & rhash.mask;
                                            x = s_tab[z];
                                        }
                                        if (x != kSlotEmpty && (uint32_t)x + dd <= gd) h = true;
                                    }
                                }
                                const uint32_t hm = __ballot_sync(kFull, h), dm = __ballot_sync(kFull, h || done);
                                if (live >> lane & 1u) {
                                    // this owner's items are lanes vi0, vi0 + t, ...
                                    uint32_t pat = 0;
                                    for (uint32_t x = __popc(live & lanemask_lt()); x < 32; x += t) pat |= 1u << x;
                                    hit = (hm & pat) != 0;
                                    ch += __popc(pat);
                                    test = !(dm & pat) && ch < nch;
                                }
                                live = __ballot_sync(kFull, test);
                            }
                            if (valid) {
                                // 64 bits wide like the minimum that other warps lower
                                // the word with: atomics of different widths on the
                                // same bytes are not atomic to each other
                                if (hit) {
                                    atomicAnd(kw + v, ~1ull);
                                    deg = 0;
                                } else if (!((uint32_t)word & 1u)) {
                                    atomicOr(kw + v, 1ull);   // was pruned at a larger distance
                                }
                            }
                        }
                        c_arcs += deg;
                        const uint32_t most = __reduce_max_sync(kFull, deg);
                        if (most <= (uint32_t)kTeamLight) {
                            for (uint32_t h = 0; h < most; h += kTeamArcs) {
                                uint32_t w[kTeamArcs], len[kTeamArcs], rk[kTeamArcs];
#pragma unroll
                                for (int q = 0; q < kTeamArcs; ++q) {
                                    w[q] = v;
                                    len[q] = 1;
                                    rk[q] = 0;
                                    if (h + q < deg) {
                                        if (UNIT) {
                                            const uint2 x = fhead[ab + h + q];
                                            w[q] = x.x;
                                            rk[q] = x.y;
                                        } else {
                                            const uint4 x = farc[ab + h + q];
                                            w[q] = x.x;
                                            len[q] = x.y;
                                            rk[q] = x.z;
                                        }
                                    }
                                }
#pragma unroll
                                for (int q = 0; q < kTeamArcs; ++q)
                                    relax(h + q < deg, k, w[q], len[q], rk[q], kInf);   // no read first, see above
                            }
                        } else {
                            relax_flat(deg, ab, k);
                        }
                    }
                    __syncthreads();
                    nf = min(sh.nn[pass % 3], n);
                    ++pass;
                    uint32_t *t = front;
                    front = fnext;
                    fnext = t;
                }
                // the window is final: its labels, from the final keys
                const uint32_t nm = min(sh.nm, n);
                const bool big = sh.big != 0;
                int nv_final = 0;
                uint32_t lab = 0, dnv = 0;
                for (uint32_t b0 = wbegin + wib * 32; b0 < nm; b0 += T) {
                    const uint32_t i = b0 + lane;
                    bool emit = false;
                    uint32_t x = 0, k = 0;
                    if (i < nm) {
                        x = __ldcg(&memb[i]);
                        const unsigned long long word = __ldcg(&kw[x]);
                        k = (uint32_t)(word >> 32);
                        const bool unpruned = !PRUNE || R == 0 || ((uint32_t)word & 1u);
                        if (PLANT) {
                            nv_final += (int)(k & 1u);
                            if (k & 1u) dnv = max(dnv, k >> 1);
                        }
                        emit = unpruned && (!PLANT || (k & 1u));
                        if (big && unpruned)
                            for (uint64_t e = goff[x]; e < goff[x + 1]; ++e)
                                if ((uint64_t)(k >> 1) + (UNIT ? 1u : farc[e].y) >= 0x7FFFFFFFull)
                                    a.ctl->err = 1;   // the reference asserts dd < infty
                    }
                    const uint32_t em = __ballot_sync(kFull, emit);
                    if (em) {
                        if (n_emit + 32 > (uint32_t)kEmit) flush_labels();
                        if (emit) {
                            const uint32_t at = n_emit + __popc(em & lanemask_lt());
                            const uint32_t o = !PRUNE && a.orig ? a.orig[x] : x;
                            s_ek[at] = ((uint64_t)lidx(o, 1 - f, a.sides) << a.hub_bits) | (uint64_t)(r - a.r0);
                            s_ev[at] = k >> 1;
                        }
                        n_emit += __popc(em);
                        lab += __popc(em);
                    }
                }
                if (PLANT) {
                    nv_final = __reduce_add_sync(kFull, nv_final - dql);
                    dnv = __reduce_max_sync(kFull, dnv);
                    dql = 0;
                }
                lo = __reduce_min_sync(kFull, lo);
                if (lane == 0) {
                    if (PLANT && nv_final) atomicSub(&sh.ql, nv_final);
                    if (PLANT && dnv) atomicMax(&sh.dnv, dnv);
                    if (lab) atomicAdd(&sh.t_lab, lab);
                    if (lo != kInf) atomicMin(&sh.lo, lo);
                }
                lo = kInf;
                __syncthreads();
                if (PLANT && sh.ql == 0) break;   // plant :95 early exit (all queued keys are via)
                uint32_t np = min(sh.npile, n), low = sh.lo;
                if (np == 0 || sh.err) {
                    if (tid == 0) sh.t_size += nm - wbegin;
                    wbegin = nm;
                    break;
                }
                __syncthreads();   // the window's state is read
                if (tid == 0) {
                    sh.t_size += nm - wbegin;
                    sh.kmin = kInf;
                    sh.kmax = 0;
                }
                if (width == 0) {
                    // the first width: the spread of the root's neighbours' distances
                    __syncthreads();
                    uint32_t mn = kInf, mx = 0;
                    for (uint32_t i = tid; i < np; i += T) {
                        const uint32_t d = __ldcg(key_at(__ldcg(&pile[i]))) >> 1;
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
                    low = sh.kmin;
                    width = max(sh.kmax - min(sh.kmin, sh.kmax), 1u);
                } else if (nm - wbegin > 2 * a.near_target) {
                    width = max(width / 2, 1u);
                } else if (nm - wbegin < a.near_target / 2) {
                    width = width < 0x40000000u ? 2 * width : 0x7FFFFFFFu;
                }
                wbegin = nm;
                // next window from the far pile: entries below the old thr are
                // stale (they joined a window), entries below the new one join,
                // the rest stay.  low is exact from the second sweep on.
                while (nf == 0 && np > 0) {
                    const uint32_t t_old = thr;
                    thr = sat_add(low, width);
                    __syncthreads();
                    if (tid == 0) {
                        sh.nn[0] = 0;
                        sh.nkeep = 0;
                        sh.lo = kInf;
                    }
                    __syncthreads();
                    for (uint32_t i0 = wib * 32; i0 < np; i0 += T) {
                        const uint32_t i = i0 + lane;
                        const uint32_t x = i < np ? __ldcg(&pile[i]) : 0u;
                        const uint32_t d = i < np ? __ldcg(key_at(x)) >> 1 : 0u;
                        const bool live = i < np && d >= t_old;
                        append(live && d < thr, x, front, &sh.nn[0]);
                        append(live && d >= thr, x, fnext, &sh.nkeep);
                        if (live && d >= thr) lo = min(lo, d);
                    }
                    lo = __reduce_min_sync(kFull, lo);
                    if (lane == 0 && lo != kInf) atomicMin(&sh.lo, lo);
                    lo = kInf;
                    __syncthreads();
                    nf = sh.nn[0];
                    np = sh.nkeep;
                    low = sh.lo;
                    uint32_t *t = pile;   // the kept entries are the pile now
                    pile = fnext;
                    fnext = t;
                }
                for (uint32_t i = tid; i < nf; i += T) memb[nm + i] = front[i];
                __syncthreads();
                if (tid == 0) {
                    sh.nm = nm + nf;
                    sh.npile = np;
                    sh.nn[0] = sh.nn[1] = sh.nn[2] = 0;
                }
                __syncthreads();
                if (nf == 0) break;   // only stale entries were left
            }
            __syncthreads();
            if (sh.err && tid == 0) a.ctl->err = 2;
            const uint32_t nm = min(sh.nm, n), np = min(sh.npile, n);
            if (PLANT && wbegin < nm) {
                // the early exit ended the tree inside this window: count its
                // members no farther than the last not-via vertex, the ones
                // the reference's Dijkstra pops before it stops
                // (distributed_memory/akiba.hpp:69-95)
                const uint32_t dl = sh.dnv;
                uint32_t c = 0;
                for (uint32_t i = wbegin + tid; i < nm; i += T) c += (__ldcg(key_at(__ldcg(&memb[i]))) >> 1) <= dl ? 1u : 0u;
                c = __reduce_add_sync(kFull, c);
                if (lane == 0 && c) atomicAdd(&sh.t_size, c);
                __syncthreads();
            }
            for (uint32_t i = tid; i < nm; i += T) __stcg(&kw[__ldcg(&memb[i])], ~0ull);
            for (uint32_t i = tid; i < np; i += T) __stcg(&kw[__ldcg(&pile[i])], ~0ull);
            if (PRUNE)
                for (uint32_t k = tid; k < a.hash_slots; k += T) s_tab[k] = kSlotEmpty;
            __syncthreads();
        }
        flush_labels();
        if (tid == 0) {
            atomicAdd(&a.ctl->visits, (unsigned long long)sh.t_size);   // fetch_root reads it
            a.tree_size[r - a.r0] = sh.t_size;
            a.tree_labels[r - a.r0] = sh.t_lab;
            finish_root(a, sh.nominal != 0);
        }
        __syncthreads();
    }
    d_hi = __reduce_max_sync(kFull, d_hi);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c_arcs += __shfl_xor_sync(kFull, c_arcs, o);
        c_reads += __shfl_xor_sync(kFull, c_reads, o);
    }
    if (lane == 0) {
        atomicAdd(&a.ctl->arcs, c_arcs);
        atomicAdd(&a.ctl->label_reads, c_reads);
        if (d_hi) atomicMax(&a.ctl->max_dist, d_hi);
    }
}

using TreeKernel = void (*)(TreeArgs);

template <bool UNIT, bool PLANT, bool PRUNE, bool ROWS>
TreeKernel team_kernel_tw(uint32_t tw) {
    if constexpr (!PRUNE)   // pruned trees never take 32 warps
        if (tw == 32) return team_kernel<UNIT, PLANT, PRUNE, ROWS, 1024>;
    switch (tw) {
    case 1: return team_kernel<UNIT, PLANT, PRUNE, ROWS, 32>;
    case 2: return team_kernel<UNIT, PLANT, PRUNE, ROWS, 64>;
    case 8: return team_kernel<UNIT, PLANT, PRUNE, ROWS, 256>;
    default: return team_kernel<UNIT, PLANT, PRUNE, ROWS, 128>;
    }
}

template <bool UNIT, bool PLANT>
TreeKernel team_kernel_pr(bool prune, bool rows, uint32_t tw) {
    if (prune) return team_kernel_tw<UNIT, PLANT, true, false>(tw);
    return rows ? team_kernel_tw<UNIT, PLANT, false, !UNIT>(tw) : team_kernel_tw<UNIT, PLANT, false, false>(tw);
}

// rows: weighted graphs only
TreeKernel team_kernel_for(bool unit, bool plant, bool prune, bool rows, uint32_t tw) {
    if (unit) return plant ? team_kernel_pr<true, true>(prune, rows, tw) : team_kernel_pr<true, false>(prune, rows, tw);
    return plant ? team_kernel_pr<false, true>(prune, rows, tw) : team_kernel_pr<false, false>(prune, rows, tw);
}

// ------------------------------------------------------ bit-parallel trees
//
// Unit lengths: the trees of kBitRoots roots are searched together, a level
// at a time, one bit per root.  A vertex's row of kBitWords words holds the
// roots that reached it in the last level, and those of them by a via path.
// A level pulls: vertex w ORs its in-neighbours' rows, keeps the roots that
// have not seen w, marks as via those with a via predecessor or ranked below
// w (update_wo_prune's flag: every shortest-path predecessor is in the last
// level), drops those with a committed witness, and emits a label for each
// that is left and not via.  The witness test reads L(w) once for all roots:
// an entry (h, dh) prunes the roots within d - dh of h, one row of the table
// M[h][.] of the batch's own committed labels.  A root whose level has no
// not-via vertex is done (plant :95).
// Rows of 16 lanes x 16 bytes make every gather coalesced; a batch moves each
// arc's row once per level instead of once per root and level.  RMAT scale 17:
// the first 1,024 roots take 0.76 ms where their trees took 24, the next 2,048
// (pruned) 2.1 where theirs took 6.
constexpr int kBitWords = 16;
constexpr uint32_t kBitRoots = 64 * kBitWords;
constexpr uint32_t kBitHeavy = 512;       // longer lists are pulled by a block each
constexpr int kBitThreads = 256;
constexpr int kBitGroups = kBitThreads / kBitWords;
constexpr uint32_t kBitLevels = 64;       // more levels than this: the other kernels
constexpr uint32_t kBitDist = 32;         // largest committed distance the table takes, exclusive

struct BitArgs {
    uint32_t n;
    int sides, f;                   // trees of side f: rows are pulled over the reverse arcs
    const uint64_t *roff;
    const uint2 *rhead;
    const uint64_t *foff;           // lists of the arcs the trees follow (statistics)
    const uint32_t *order, *rank;
    const uint64_t *l_off;
    const uint2 *l_ent, *l_dent;
    uint32_t r0, rb, nb;            // superstep's first root, batch's first root and size
    uint32_t d;                     // level
    uint32_t K;                     // table distances 0 .. K - 1 (K - 1 the largest committed one)
    const ulonglong2 *cur;          // (reached, via) per vertex and word
    ulonglong2 *nxt;
    unsigned long long *seen;
    const uint8_t *act;             // rows of cur that are set
    uint8_t *act_out;
    const unsigned long long *live; // roots with a not-via vertex in the last level
    unsigned long long *live_out;
    unsigned long long *M;
    const uint32_t *heavy;          // heavy[0]: number of long lists, then their vertices
    int hub_bits;
    uint64_t *out_key;
    uint32_t *out_val;
    unsigned long long out_cap;
    BuildCtl *ctl;
};

__global__ void bit_heavy(uint32_t n, const uint64_t *off, uint32_t *heavy) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        if (off[v + 1] - off[v] > kBitHeavy) heavy[1 + atomicAdd(&heavy[0], 1u)] = v;
}

// labels of the bits of nv for vertex w, by 16 lanes (mask gm, lane's word wd)
__device__ __forceinline__ void bit_emit(const BitArgs &a, uint32_t gm, uint32_t wd, uint32_t w, unsigned long long nv) {
    const uint32_t c = (uint32_t)__popcll(nv);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < kBitWords; o <<= 1) {
        const uint32_t y = __shfl_up_sync(gm, incl, o, kBitWords);
        if (wd >= (uint32_t)o) incl += y;
    }
    const uint32_t total = __shfl_sync(gm, incl, kBitWords - 1, kBitWords);
    if (total == 0) return;
    unsigned long long b = 0;
    if (wd == 0) b = atomicAdd(&a.ctl->nlab, (unsigned long long)total);
    b = __shfl_sync(gm, b, 0, kBitWords) + (incl - c);
    const uint64_t list = (uint64_t)lidx(w, 1 - a.f, a.sides) << a.hub_bits;
    const uint32_t rel = a.rb - a.r0 + 64u * wd;
    for (; nv; nv &= nv - 1, ++b) {
        if (b < a.out_cap) {
            a.out_key[b] = list | (uint64_t)(rel + (uint32_t)__ffsll((long long)nv) - 1u);
            a.out_val[b] = a.d;
        } else {
            a.ctl->overflow = 1;
        }
    }
}

// the batch's roots at level 0, 16 lanes each
__global__ void bit_roots(BitArgs a) {
    const uint32_t wd = threadIdx.x % kBitWords, gm = 0xFFFFu << (threadIdx.x & 16u);
    const uint32_t i = blockIdx.x * kBitGroups + threadIdx.x / kBitWords;
    if (i >= a.nb) return;
    const uint32_t v = a.order[a.rb + i];
    const unsigned long long bit = wd == i / 64 ? 1ull << (i % 64) : 0ull;
    a.nxt[(size_t)v * kBitWords + wd] = make_ulonglong2(bit, 0ull);
    a.seen[(size_t)v * kBitWords + wd] = bit;
    if (bit) atomicOr(&a.live_out[wd], bit);
    if (wd == 0) {
        a.act_out[v] = 1;
        atomicAdd(&a.ctl->arcs, (unsigned long long)(a.foff[v + 1] - a.foff[v]));
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&a.ctl->visits, (unsigned long long)a.nb);
    bit_emit(a, gm, wd, v, bit);
}

// M[h][k] = roots of the batch within distance k of committed hub h; a warp per root
__global__ void bit_table(BitArgs a) {
    const uint32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (i >= a.nb) return;
    const uint32_t x = lidx(a.order[a.rb + i], a.f, a.sides);
    const unsigned long long bit = 1ull << (i % 64);
    for (uint64_t e = a.l_off[x] + lane_id(); e < a.l_off[x + 1]; e += 32) {
        const uint2 q = a.l_ent[e];
        for (uint32_t k = q.y; k < a.K; ++k) atomicOr(&a.M[((size_t)q.x * a.K + k) * kBitWords + i / 64], bit);
    }
}

// One level.  HEAVY: a block per long list, its 16 groups of 16 lanes taking
// every 16th arc group; otherwise 16 lanes per vertex.
template <bool HEAVY, bool PRUNE>
__global__ void __launch_bounds__(kBitThreads) bit_level(BitArgs a) {
    __shared__ unsigned long long s_acc[kBitGroups][kBitWords], s_via[kBitGroups][kBitWords];
    const uint32_t wd = threadIdx.x % kBitWords, grp = threadIdx.x / kBitWords;
    const uint32_t gm = 0xFFFFu << (threadIdx.x & 16u);
    const uint32_t items = HEAVY ? a.heavy[0] : a.n;
    const unsigned long long live = a.live[wd];
    const unsigned long long valid =
        a.nb >= 64u * wd + 64u ? ~0ull : (a.nb > 64u * wd ? (1ull << (a.nb - 64u * wd)) - 1ull : 0ull);
    unsigned long long c_new = 0, c_reads = 0, c_arcs = 0, nv_any = 0;
    const uint32_t step = HEAVY ? gridDim.x : gridDim.x * kBitGroups;
    for (uint32_t it = HEAVY ? blockIdx.x : blockIdx.x * kBitGroups + grp; it < items; it += step) {
        const uint32_t w = HEAVY ? a.heavy[1 + it] : it;
        const uint64_t b = a.roff[w], e = a.roff[w + 1];
        if (!HEAVY && e - b > kBitHeavy) continue;
        const uint32_t rw = a.rank[w];
        unsigned long long acc = 0, via = 0, seen = 0;
        // a vertex ranked above the superstep's roots always has a committed witness
        const bool skip = PRUNE && rw < a.r0;
        if (!skip) {
            seen = a.seen[(size_t)w * kBitWords + wd];
            // roots ranked below w reach it by a via path
            const int64_t t = (int64_t)rw - (int64_t)a.rb - 64ll * wd;
            via = t < 0 ? ~0ull : t >= 63 ? 0ull : ~0ull << (t + 1);
            const unsigned long long want = valid & ~seen & live;
            // heads and their flags 16 at a time, the set rows 4 at a time; done
            // once every wanted root has arrived by a via path
            const uint64_t first = b + (HEAVY ? (uint64_t)grp * kBitWords : 0), stride = HEAVY ? kBitThreads : kBitWords;
            if (__any_sync(gm, want != 0)) {
                uint32_t hn = first + wd < e ? a.rhead[first + wd].x : 0u;
                for (uint64_t q = first; q < e; q += stride) {
                    const uint32_t hd = hn;
                    const bool on = q + wd < e && a.act[hd];
                    hn = q + stride + wd < e ? a.rhead[q + stride + wd].x : 0u;
                    uint32_t m = __ballot_sync(gm, on) >> (threadIdx.x & 16u) & 0xFFFFu;
                    if (!m) continue;
                    while (m) {
                        ulonglong2 r[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            r[u] = make_ulonglong2(0ull, 0ull);
                            const uint32_t x = __shfl_sync(gm, hd, m ? __ffs(m) - 1 : 0, kBitWords);
                            if (m) r[u] = a.cur[(size_t)x * kBitWords + wd];
                            m &= m - 1;
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            acc |= r[u].x;
                            via |= r[u].y;
                        }
                    }
                    if (!__any_sync(gm, (want & ~(acc & via)) != 0)) break;
                }
            }
            acc &= want;
        }
        if (HEAVY) {
            s_acc[grp][wd] = acc;
            s_via[grp][wd] = via;
            __syncthreads();
            if (grp == 0) {
#pragma unroll
                for (int g = 1; g < kBitGroups; ++g) {
                    acc |= s_acc[g][wd];
                    via |= s_via[g][wd];
                }
            }
            __syncthreads();
        }
        if (!HEAVY || grp == 0) {
            unsigned long long left = acc;
            if (PRUNE && !skip && __any_sync(gm, left != 0)) {
                const uint32_t x = lidx(w, 1 - a.f, a.sides);
                const uint64_t le = a.l_off[x + 1];
                // entries 16 at a time (their list is in distance order), 4 table rows in flight
                for (uint64_t q = a.l_off[x]; q < le; q += kBitWords) {
                    const uint2 en = q + wd < le ? a.l_dent[q + wd] : make_uint2(0u, 0xFFFFFFFFu);
                    const uint32_t cnt = (uint32_t)__popc(__ballot_sync(gm, en.y <= a.d));
                    const size_t row = ((size_t)en.x * a.K + min(a.d - min(en.y, a.d), a.K - 1)) * kBitWords;
                    for (uint32_t j = 0; j < cnt; j += 4) {
                        unsigned long long p[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const size_t rr = __shfl_sync(gm, row, (j + u) & (kBitWords - 1), kBitWords);
                            p[u] = j + u < cnt ? a.M[rr + wd] : 0ull;
                        }
                        left &= ~(p[0] | p[1] | p[2] | p[3]);
                    }
                    if (wd == 0) c_reads += cnt;
                    if (cnt < kBitWords || !__any_sync(gm, left != 0)) break;
                }
            }
            c_new += (unsigned long long)__popcll(acc);
            const bool any = __any_sync(gm, left != 0);
            if (__any_sync(gm, acc != 0)) a.seen[(size_t)w * kBitWords + wd] = seen | acc;
            if (wd == 0) a.act_out[w] = any ? 1 : 0;
            if (any) {
                a.nxt[(size_t)w * kBitWords + wd] = make_ulonglong2(left, left & via);
                const unsigned long long nv = left & ~via;
                nv_any |= nv;
                c_arcs += (unsigned long long)__popcll(left) * (a.sides == 1 ? e - b : a.foff[w + 1] - a.foff[w]);
                bit_emit(a, gm, wd, w, nv);
            }
        }
    }
    // totals and the roots still live, one atomic per warp
    nv_any |= __shfl_xor_sync(kFull, nv_any, 16);
    if (lane_id() < kBitWords && (nv_any & ~*(volatile unsigned long long *)&a.live_out[wd])) atomicOr(&a.live_out[wd], nv_any);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c_new += __shfl_xor_sync(kFull, c_new, o);
        c_reads += __shfl_xor_sync(kFull, c_reads, o);
        c_arcs += __shfl_xor_sync(kFull, c_arcs, o);
    }
    if (lane_id() == 0) {
        if (c_arcs) atomicAdd(&a.ctl->arcs, c_arcs);
        if (c_new) atomicAdd(&a.ctl->visits, c_new);
        if (c_reads) atomicAdd(&a.ctl->label_reads, c_reads);
    }
}

__global__ void fat_arcs(uint64_t m, const uint2 *arc, const uint32_t *rank, const uint32_t *win, uint4 *out) {
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint2 a = arc[e];
        out[e] = make_uint4(a.x, a.y, rank[a.x], win[a.x]);
    }
}

__global__ void fat_heads(uint64_t m, const uint32_t *head, const uint32_t *rank, uint2 *out) {
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t h = head[e];
        out[e] = make_uint2(h, rank[h]);
    }
}

// Rows of the unpruned trees on weighted graphs of few arcs a vertex: its first
// kRowArcs arc records at a place known from its number alone, so they are read
// beside its key word instead of after its list's offset, and by four lanes in
// one access instead of one lane in four (a pass of few vertices takes fewer
// steps, and the L1, at 58% of its throughput, fewer lines).  What the records'
// last word holds otherwise (win) no unpruned tree reads: it is the degree,
// then the two halves of the list's offset, for lists that go on past the row.
// Trees of the 100-, 512- and 1024-square grids 1.66, 94.8, 895 ms -> 1.46,
// 85.9, 775; rows read a vertex per lane 1.63, 93.9, 836.  Unit lengths' 8-byte
// records gain nothing (62.8 and 538 against 63.3 and 536) and stay in their
// lists.
__global__ void arc_rows(uint32_t n, const uint64_t *off, const uint4 *farc, uint4 *row) {
    const uint64_t cnt = (uint64_t)n * kRowArcs;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < cnt; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = (uint32_t)(i / kRowArcs), q = (uint32_t)(i % kRowArcs);
        const uint64_t b = off[v], deg = off[v + 1] - b;
        uint4 t = make_uint4(0, 0, 0, 0);
        if (q < deg) t = farc[b + q];
        t.w = q == 0 ? (uint32_t)deg : q == 1 ? (uint32_t)b : q == 2 ? (uint32_t)(b >> 32) : 0u;
        row[i] = t;
    }
}

// -------------------------------------------------------------- numbering
//
// The unpruned trees of a large graph miss the L2 in their key words, so what
// they touch together should lie together: vertices are numbered by cells of
// about 16 (one 128-byte line of key words) inside cells of about 256.  Cells
// grow around hashed centres over the arcs, a hop per round.  Trees of the
// 1024-square grid 866 -> 699 ms, of the 512-square one 80 -> 73; with the
// caller's vertices numbered at random 1,817 -> 809 and 198 -> 78.
constexpr uint32_t kCellNone = 0xFFFFFFFFu;
constexpr int kCellSmall = 16, kCellLarge = 256;      // vertices per centre
constexpr int kGrowSmall = 8, kGrowLarge = 24;        // rounds: about twice the cells' radius
constexpr uint32_t kNumberedFrom = 1u << 16;          // vertices (below, the 0.3 ms it takes are not won back)

__global__ void cell_centres(uint32_t n, uint32_t *small, uint32_t *large) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        uint32_t h = v * 0x9E3779B1u;
        h ^= h >> 15;
        h *= 0x85EBCA77u;
        h ^= h >> 13;
        small[v] = h % kCellSmall == 0 ? v : kCellNone;
        large[v] = h % kCellLarge == 0 ? v : kCellNone;
    }
}

// one hop: a vertex without a cell joins a neighbour's (any: the numbering
// changes speed alone)
__global__ void cell_grow(uint32_t n, const uint64_t *off, const uint4 *farc, const uint2 *fhead, uint32_t *cell) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        if (cell[v] != kCellNone) continue;
        uint32_t c = kCellNone;
        for (uint64_t e = off[v]; e < off[v + 1]; ++e) c = min(c, __ldcg(&cell[farc ? farc[e].x : fhead[e].x]));
        if (c != kCellNone) __stcg(&cell[v], c);
    }
}

__global__ void cell_keys(uint32_t n, const uint32_t *small, const uint32_t *large, int bits, uint64_t *key,
                          uint32_t *val) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const uint32_t c = small[v] == kCellNone ? v : small[v];
        const uint32_t l = large[c] == kCellNone ? c : large[c];
        key[v] = ((uint64_t)l << bits) | c;
        val[v] = v;
    }
}

__global__ void invert(uint32_t n, const uint32_t *orig, uint32_t *newid) {
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < n; x += gridDim.x * blockDim.x) newid[orig[x]] = x;
}

__global__ void numbered_degrees(uint32_t n, const uint32_t *orig, const uint64_t *off, uint32_t *deg) {
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < n; x += gridDim.x * blockDim.x)
        deg[x] = (uint32_t)(off[orig[x] + 1] - off[orig[x]]);
}

// the arc records of the new numbering, 8 lanes per vertex
__global__ void numbered_arcs(uint32_t n, const uint32_t *orig, const uint32_t *newid, const uint64_t *off,
                              const uint64_t *off2, const uint4 *farc, const uint2 *fhead, uint4 *farc2, uint2 *fhead2) {
    const uint32_t groups = gridDim.x * (blockDim.x >> 3);
    for (uint32_t x = blockIdx.x * (blockDim.x >> 3) + (threadIdx.x >> 3); x < n; x += groups) {
        const uint64_t b = off[orig[x]], b2 = off2[x], m = off2[x + 1] - b2;
        for (uint64_t k = threadIdx.x & 7u; k < m; k += 8) {
            if (farc) {
                uint4 t = farc[b + k];
                t.x = newid[t.x];
                farc2[b2 + k] = t;
            } else {
                uint2 t = fhead[b + k];
                t.x = newid[t.x];
                fhead2[b2 + k] = t;
            }
        }
    }
}

// ---------------------------------------------------------- commit chain

// Count new labels per label list (sorted keys).
__global__ void count_keys(const uint64_t *keys, const unsigned long long *d_n,
                           unsigned long long cap, int hub_bits, uint32_t *cnt) {
    unsigned long long n = *d_n;
    if (n > cap) n = cap;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
         i < n; i += (unsigned long long)gridDim.x * blockDim.x)
        atomicAdd(&cnt[keys[i] >> hub_bits], 1u);
}

// GLL clean (shared_memory/akiba.hpp:197-208 with Labeling::clean_cover,
// shared_memory/labeling.hpp:78-88): a new label (h, d) of list (u, s) is
// dropped if some hub h' < h appears in both the new L(u, s) and the new
// L(order[h], !s) with d' + d'' <= d.  Only this superstep's labels take
// part; earlier labels were already used for pruning.
__global__ void clean_mark(const uint64_t *keys, const uint32_t *vals,
                           const unsigned long long *d_n, unsigned long long cap,
                           int hub_bits, uint32_t r0, const uint64_t *pre,
                           const uint32_t *order, const uint32_t *rank, int sides,
                           uint32_t *keep) {
    unsigned long long n = *d_n;
    if (n > cap) n = cap;
    const uint64_t mask = (1ull << hub_bits) - 1;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
         i < n; i += (unsigned long long)gridDim.x * blockDim.x) {
        const uint64_t k = keys[i];
        const uint32_t x = (uint32_t)(k >> hub_bits);
        const uint32_t hrel = (uint32_t)(k & mask);
        const uint32_t d = vals[i];
        const uint32_t hv = order[r0 + hrel];
        uint32_t y;
        if (sides == 1) {
            y = hv;
        } else {
            const uint32_t s = x & 1u;
            y = 2 * hv + (1u - s);
        }
        uint64_t a = pre[x], ae = pre[x + 1];
        uint64_t b = pre[y], be = pre[y + 1];
        bool covered = false;
        while (a < ae && b < be) {
            const uint32_t ha = (uint32_t)(keys[a] & mask), hb = (uint32_t)(keys[b] & mask);
            if (ha >= hrel || hb >= hrel) break;
            if (ha == hb) {
                if (vals[a] + vals[b] <= d) {
                    covered = true;
                    break;
                }
                ++a;
                ++b;
            } else if (ha < hb) {
                ++a;
            } else {
                ++b;
            }
        }
        keep[i] = covered ? 0u : 1u;
    }
}

__global__ void compact_kept(const uint64_t *kin, const uint32_t *vin, const uint32_t *keep,
                             const uint64_t *kpre, const unsigned long long *d_n,
                             unsigned long long cap, uint64_t *kout, uint32_t *vout,
                             unsigned long long *d_nkeep) {
    unsigned long long n = *d_n;
    if (n > cap) n = cap;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
         i < n; i += (unsigned long long)gridDim.x * blockDim.x) {
        if (keep[i]) {
            const uint64_t p = kpre[i];
            kout[p] = kin[i];
            vout[p] = vin[i];
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *d_nkeep = kpre[cap];
}

// new_off[x] = old_off[x] + pre[x]  (pre = exclusive scan of new counts)
__global__ void merge_offsets(const uint64_t *old_off, const uint64_t *pre, uint64_t *new_off,
                              uint32_t nl) {
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x <= nl; x += gridDim.x * blockDim.x)
        new_off[x] = old_off[x] + pre[x];
}

// Copy every committed list to its new position (one warp per list).
__global__ void copy_old_lists(const uint64_t *old_off, const uint2 *old_ent,
                               const uint64_t *new_off, uint2 *new_ent, uint32_t nl) {
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t x = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); x < nl; x += warps) {
        const uint64_t b = old_off[x], e = old_off[x + 1], nb = new_off[x];
        for (uint64_t k = b + lane_id(); k < e; k += 32) new_ent[nb + (k - b)] = old_ent[k];
    }
}

// Append the sorted new labels behind each list's committed part.
__global__ void place_new(const uint64_t *keys, const uint32_t *vals,
                          const unsigned long long *d_n, unsigned long long cap, int hub_bits,
                          uint32_t r0, const uint64_t *pre, const uint64_t *old_off,
                          const uint64_t *new_off, uint2 *new_ent) {
    unsigned long long n = *d_n;
    if (n > cap) n = cap;
    const uint64_t mask = (1ull << hub_bits) - 1;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
         i < n; i += (unsigned long long)gridDim.x * blockDim.x) {
        const uint64_t k = keys[i];
        const uint32_t x = (uint32_t)(k >> hub_bits);
        const uint64_t dst = new_off[x] + (old_off[x + 1] - old_off[x]) + (i - pre[x]);
        new_ent[dst] = make_uint2(r0 + (uint32_t)(k & mask), vals[i]);
    }
}

// ---- distance-ordered copy of the committed labels (prune tests only)
// Lists in the same CSR offsets, entries ordered by (distance, hub): an
// entry (h, dd) of L(u) can only witness d(r, u) if dd <= d(r, u), so a
// prune test stops at the first chunk whose entries all exceed d(r, u).

__device__ __forceinline__ bool ent_less(uint2 a, uint2 b) { return a.y < b.y || (a.y == b.y && a.x < b.x); }

// new labels sorted by (list, hub) -> keys (list << 32 | dist), values hub
__global__ void dist_keys(const uint64_t *keys, const uint32_t *vals, const unsigned long long *d_n,
                          unsigned long long cap, int hub_bits, int dist_bits, uint32_t r0, uint64_t *k2,
                          uint32_t *v2) {
    unsigned long long n = *d_n;
    if (n > cap) n = cap;
    const uint64_t mask = (1ull << hub_bits) - 1;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const uint64_t k = keys[i];
        k2[i] = ((k >> hub_bits) << dist_bits) | vals[i];
        v2[i] = r0 + (uint32_t)(k & mask);
    }
}

// Merge, per list, the committed distance-ordered entries with the new ones
// (sorted by (list, dist) in k2/v2, the distance in k2's low dist_bits bits,
// the list's run at [pre[x], pre[x+1])).
// One warp per list; every entry's final slot is its rank in the other run
// (binary search) plus its own index.  Ties in distance order by hub.
__global__ void merge_dist_lists(const uint64_t *old_off, const uint2 *old_ent, const uint64_t *new_off,
                                 const uint64_t *pre, const uint64_t *k2, const uint32_t *v2, uint2 *out,
                                 uint32_t nl, int dist_bits) {
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint64_t dmask = (1ull << dist_bits) - 1;
    for (uint32_t x = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); x < nl; x += warps) {
        const uint64_t ob = old_off[x], oe = old_off[x + 1], nb = new_off[x];
        const uint64_t pb = pre[x], pe = pre[x + 1];
        const uint64_t no = oe - ob, nn = pe - pb;
        for (uint64_t i = lane_id(); i < no; i += 32) {
            const uint2 e = old_ent[ob + i];
            uint64_t lo = 0, hi = nn;   // new entries before e
            while (lo < hi) {
                const uint64_t mid = (lo + hi) >> 1;
                const uint2 m = make_uint2(v2[pb + mid], (uint32_t)(k2[pb + mid] & dmask));
                if (ent_less(m, e)) lo = mid + 1;
                else hi = mid;
            }
            out[nb + i + lo] = e;
        }
        for (uint64_t t = lane_id(); t < nn; t += 32) {
            const uint2 e = make_uint2(v2[pb + t], (uint32_t)(k2[pb + t] & dmask));
            uint64_t lo = 0, hi = no;   // old entries before e
            while (lo < hi) {
                const uint64_t mid = (lo + hi) >> 1;
                if (ent_less(old_ent[ob + mid], e)) lo = mid + 1;
                else hi = mid;
            }
            out[nb + t + lo] = e;
        }
    }
}

// Largest tree/label ratio over the superstep's roots (hybrid switch rule,
// distributed_memory/akiba.hpp:297-303), kept as an exact fraction.
__global__ void ratio_max(const uint32_t *tsize, const uint32_t *tlab, const unsigned long long *next_root,
                          uint32_t r0, uint32_t r_end, BuildCtl *ctl) {
    unsigned long long r1 = *next_root;
    if (r1 > r_end) r1 = r_end;
    const uint32_t cnt = (uint32_t)(r1 - r0);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
        // pack ratio as a double's bits (positive doubles order like integers)
        const double ratio = tlab[i] ? (double)tsize[i] / (double)tlab[i] : 1e300;
        atomicMax(&ctl->max_ratio_num, (unsigned long long)__double_as_longlong(ratio));
    }
}

// Longest label list (sizes the root-label staging of the next superstep).
__global__ void max_list_len(const uint64_t *off, uint32_t nl, unsigned long long *out) {
    unsigned long long mx = 0;
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < nl; x += gridDim.x * blockDim.x)
        mx = max(mx, (unsigned long long)(off[x + 1] - off[x]));
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(kFull, mx, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, mx);
}

// max and sum of per-root tree sizes of a superstep (diagnostics)
__global__ void tree_stats(const uint32_t *tsize, uint32_t cnt, unsigned long long *out2) {
    unsigned long long mx = 0, sm = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
        mx = max(mx, (unsigned long long)tsize[i]);
        sm += tsize[i];
    }
    for (int o = 16; o > 0; o >>= 1) {
        mx = max(mx, __shfl_xor_sync(kFull, mx, o));
        sm += __shfl_xor_sync(kFull, sm, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&out2[0], mx);
        atomicAdd(&out2[1], sm);
    }
}

inline int bits_for(uint64_t x) {   // bits needed to represent values < x
    int b = 0;
    while (b < 64 && (1ull << b) < x) ++b;
    return b < 1 ? 1 : b;
}

template <typename T>
int dalloc(T **p, size_t count) {
    *p = nullptr;
    if (count == 0) count = 1;
    cudaError_t e = long_malloc((void **)p, count * sizeof(T));
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error(std::string("device allocation failed: ") + cudaGetErrorString(e));
        return CHL_ERR_OOM;
    }
    return CHL_OK;
}

struct DevGraph {
    uint64_t *off[2] = {nullptr, nullptr};
    uint2 *arc[2] = {nullptr, nullptr};
    uint32_t *head[2] = {nullptr, nullptr};
    uint32_t *win[2] = {nullptr, nullptr};   // shortest arc into v, per direction
    void release() {
        // side 1 may alias side 0 (symmetric graphs): free each buffer once
        if (off[1] != off[0]) cudaFree(off[1]);
        if (arc[1] != arc[0]) cudaFree(arc[1]);
        if (head[1] != head[0]) cudaFree(head[1]);
        if (win[1] != win[0]) cudaFree(win[1]);
        cudaFree(off[0]);
        cudaFree(arc[0]);
        cudaFree(head[0]);
        cudaFree(win[0]);
        for (int s = 0; s < 2; ++s) {
            off[s] = nullptr;
            arc[s] = nullptr;
            head[s] = nullptr;
            win[s] = nullptr;
        }
    }
};

int upload_graph(const chl_graph *g, DevGraph &dg, cudaStream_t st) {
    const int nsides = g->symmetric ? 1 : 2;
    for (int s = 0; s < nsides; ++s) {
        const int src = g->symmetric ? 1 : s;
        const uint64_t m = g->off[src][g->n];
        int rc = dalloc(&dg.off[s], (size_t)g->n + 1);
        if (rc) return rc;
        CHL_CUDA(cudaMemcpyAsync(dg.off[s], g->off[src].data(), ((size_t)g->n + 1) * 8,
                                 cudaMemcpyHostToDevice, st));
        if (g->unit) {
            rc = dalloc(&dg.head[s], m);
            if (rc) return rc;
            CHL_CUDA(cudaMemcpyAsync(dg.head[s], g->head[src].data(), m * 4,
                                     cudaMemcpyHostToDevice, st));
        } else {
            std::vector<uint2> pk(m);
            for (uint64_t i = 0; i < m; ++i)
                pk[i] = make_uint2(g->head[src][i], (uint32_t)g->len[src][i]);
            rc = dalloc(&dg.arc[s], m);
            if (rc) return rc;
            CHL_CUDA(cudaMemcpy(dg.arc[s], pk.data(), m * 8, cudaMemcpyHostToDevice));
        }
    }
    for (int s = 0; s < nsides; ++s) {
        const int src = g->symmetric ? 1 : s;
        std::vector<uint32_t> w(g->n, 0x7FFFFFFFu);
        const uint64_t m = g->off[src][g->n];
        for (uint64_t i = 0; i < m; ++i) {
            const uint32_t h = g->head[src][i];
            w[h] = std::min<uint32_t>(w[h], (uint32_t)g->len[src][i]);
        }
        int rc = dalloc(&dg.win[s], (size_t)g->n);
        if (rc) return rc;
        CHL_CUDA(cudaMemcpy(dg.win[s], w.data(), (size_t)g->n * 4, cudaMemcpyHostToDevice));
    }
    if (nsides == 1) {
        dg.off[1] = dg.off[0];
        dg.arc[1] = dg.arc[0];
        dg.head[1] = dg.head[0];
        dg.win[1] = dg.win[0];
    }
    return CHL_OK;
}

}  // namespace

void graph_release_device(chl_graph *g) {
    if (g && g->dev) {
        DevGraph *d = (DevGraph *)g->dev;
        d->release();
        delete d;
        g->dev = nullptr;
    }
}

namespace {

struct Build {
    // sizes
    uint32_t n = 0;
    int sides = 1;
    uint32_t nl = 0;       // number of label lists on the device
    int hub_bits = 0;
    int key_bits = 0;
    // device buffers
    DevGraph own;                   // graph uploaded for this build only
    const DevGraph *dg = nullptr;
    uint32_t *order = nullptr, *rank = nullptr;
    uint64_t *off_a = nullptr, *off_b = nullptr;
    uint2 *ent_a = nullptr, *ent_b = nullptr;
    uint64_t ent_cap_a = 0, ent_cap_b = 0;
    uint2 *dent_a = nullptr, *dent_b = nullptr;   // (distance, hub)-ordered copies
    uint64_t dent_cap_a = 0, dent_cap_b = 0;
    std::unique_ptr<TmpSet> mem;   // every buffer below but the committed CSR, which becomes the labels'
    uint64_t *nk0 = nullptr, *nk1 = nullptr;   // new labels as the trees emit them, and the sort's other half
    uint32_t *nv0 = nullptr, *nv1 = nullptr;
    uint64_t new_cap = 0, sort_cap = 0, keep_cap = 0;
    uint32_t *cnt = nullptr;
    uint64_t *pre = nullptr;
    uint32_t *keep = nullptr;
    uint64_t *kpre = nullptr;
    uint32_t *tsize = nullptr, *tlab = nullptr;
    uint32_t *ws_all = nullptr;   // tree workspace (both kernels' layouts)
    uint32_t *ws_key = nullptr, *ws_vis = nullptr, *ws_front = nullptr;   // batch_kernel views
    uint32_t win_trees = 0, win_tw = 4;   // team_kernel: trees (blocks) and warps per tree
    int ws_layout = 0;   // 1: batch_kernel keys all INF, 2: team_kernel keys all INF
    BuildCtl *ctl = nullptr;
    void *tmp = nullptr;
    size_t tmp_bytes = 0;
    cudaStream_t st = nullptr;
    uint32_t warps = 0;   // warps the schedule is sized for
    uint32_t slots = 0;   // warp slots launched by batch_kernel
    uint32_t hash_max = 2048;                // largest root hash table (slots)
    uint4 *farc[2] = {nullptr, nullptr};     // (head, length, rank[head], win[head]) per arc
    uint2 *fhead[2] = {nullptr, nullptr};    // (head, rank[head]) per arc, unit lengths
    uint32_t *newid = nullptr, *orig = nullptr;   // numbering of the unpruned trees, and the graph in it
    uint64_t *off_n[2] = {nullptr, nullptr};
    uint4 *farc_n[2] = {nullptr, nullptr};
    uint4 *row[2] = {nullptr, nullptr};    // arc_rows of the numbering that row_numbered says
    bool row_numbered = false;
    uint2 *fhead_n[2] = {nullptr, nullptr};
    cudaGraphExec_t commit_exec = nullptr;   // captured commit chain
    uint64_t graph_launches = 0;

    ~Build() {
        if (commit_exec) cudaGraphExecDestroy(commit_exec);
        mem.reset();
        own.release();
        cudaFree(off_a);
        cudaFree(off_b);
        cudaFree(ent_a);
        cudaFree(ent_b);
        cudaFree(dent_a);
        cudaFree(dent_b);
        if (st) cudaStreamDestroy(st);
    }
};

// New-label buffers with room for `need` entries (their contents are dead
// between supersteps).  An overflowed superstep counts every label it tried
// to append, so its re-run needs exactly that many: no doubling.
int grow_new(Build &b, uint64_t need) {
    if (need <= b.new_cap) return CHL_OK;
    b.mem->put(b.nk0);
    b.mem->put(b.nv0);
    b.new_cap = 0;
    int rc;
    if ((rc = b.mem->get(&b.nk0, need)) || (rc = b.mem->get(&b.nv0, need))) return rc;
    b.new_cap = need;
    return CHL_OK;
}

// The rest of the commit's buffers, for the m labels a superstep has emitted:
// the sort's other half, the scans' temporaries and, for a clean, its flags
// and their prefix.
int grow_sort(Build &b, uint64_t m, bool clean) {
    int rc;
    if (m > b.sort_cap || !b.nk1) {
        b.mem->put(b.nk1);
        b.mem->put(b.nv1);
        b.sort_cap = 0;
        if ((rc = b.mem->get(&b.nk1, m)) || (rc = b.mem->get(&b.nv1, m))) return rc;
        b.sort_cap = m;
    }
    if (clean && (m > b.keep_cap || !b.keep)) {
        b.mem->put(b.keep);
        b.mem->put(b.kpre);
        b.keep_cap = 0;
        if ((rc = b.mem->get(&b.keep, m)) || (rc = b.mem->get(&b.kpre, m + 1))) return rc;
        b.keep_cap = m;
    }
    const size_t need_tmp = std::max(radix_tmp_bytes(), scan_tmp_bytes(std::max<uint64_t>(m, b.nl)));
    if (need_tmp > b.tmp_bytes) {
        char *t = (char *)b.tmp;
        b.mem->put(t);
        b.tmp = nullptr;
        b.tmp_bytes = 0;
        if ((rc = b.mem->get(&t, need_tmp))) return rc;
        b.tmp = t;
        b.tmp_bytes = need_tmp;
    }
    return CHL_OK;
}

// newid, orig and the graph's arcs in that numbering (see cell_grow)
int number_by_cells(Build &b, const chl_graph *g, int sms, unsigned long long &kernels) {
    const uint32_t n = b.n;
    const int grid = sms * 8;
    const int bits = b.hub_bits;
    int rc;
    TmpSet t(b.st);
    uint32_t *small, *large, *v0, *v1, *deg;
    uint64_t *k0, *k1, *d_n;
    char *tmp;
    const size_t tmp_bytes = std::max(radix_tmp_bytes(), scan_tmp_bytes(n));
    if ((rc = t.get(&small, n)) || (rc = t.get(&large, n)) || (rc = t.get(&v0, n)) || (rc = t.get(&v1, n)) ||
        (rc = t.get(&deg, n)) || (rc = t.get(&k0, n)) || (rc = t.get(&k1, n)) || (rc = t.get(&d_n, 1)) ||
        (rc = t.get(&tmp, tmp_bytes)) || (rc = b.mem->get(&b.newid, n)) || (rc = b.mem->get(&b.orig, n)))
        return rc;
    const uint64_t n64 = n;
    CHL_CUDA(cudaMemcpyAsync(d_n, &n64, 8, cudaMemcpyHostToDevice, b.st));
    cell_centres<<<grid, 256, 0, b.st>>>(n, small, large);
    for (int i = 0; i < kGrowSmall; ++i) cell_grow<<<grid, 256, 0, b.st>>>(n, b.dg->off[1], b.farc[1], b.fhead[1], small);
    for (int i = 0; i < kGrowLarge; ++i) cell_grow<<<grid, 256, 0, b.st>>>(n, b.dg->off[1], b.farc[1], b.fhead[1], large);
    cell_keys<<<grid, 256, 0, b.st>>>(n, small, large, bits, k0, v0);
    int par = 0;
    if ((rc = radix_sort_pairs(k0, v0, k1, v1, d_n, n, 2 * bits, tmp, tmp_bytes, b.st, &par))) return rc;
    CHL_CUDA(cudaMemcpyAsync(b.orig, par ? v1 : v0, (size_t)n * 4, cudaMemcpyDeviceToDevice, b.st));
    invert<<<grid, 256, 0, b.st>>>(n, b.orig, b.newid);
    const int sides = g->symmetric ? 1 : 2;
    for (int s = 0; s < sides; ++s) {
        const uint64_t m = g->off[g->symmetric ? 1 : s][n];
        if ((rc = b.mem->get(&b.off_n[s], (uint64_t)n + 1))) return rc;
        if (g->unit ? (rc = b.mem->get(&b.fhead_n[s], m)) : (rc = b.mem->get(&b.farc_n[s], m))) return rc;
        numbered_degrees<<<grid, 256, 0, b.st>>>(n, b.orig, b.dg->off[s], deg);
        if ((rc = scan_u32_excl(deg, b.off_n[s], n, nullptr, tmp, tmp_bytes, b.st))) return rc;
        numbered_arcs<<<grid, 256, 0, b.st>>>(n, b.orig, b.newid, b.dg->off[s], b.off_n[s], b.farc[s], b.fhead[s],
                                              b.farc_n[s], b.fhead_n[s]);
    }
    if (sides == 1) {
        b.off_n[1] = b.off_n[0];
        b.farc_n[1] = b.farc_n[0];
        b.fhead_n[1] = b.fhead_n[0];
    }
    CHL_CUDA(cudaGetLastError());
    kernels += 3 + kGrowSmall + kGrowLarge + 3 * ((2 * bits + 7) / 8) + 5 * sides;
    return CHL_OK;
}

// the rows of the numbering a launch uses (arc_rows)
int fill_rows(Build &b, TreeArgs &ta, int sms, unsigned long long &kernels) {
    const bool numbered = ta.newid != nullptr;
    const int sides = ta.g_off[0] == ta.g_off[1] ? 1 : 2;
    if (!b.row[0] || b.row_numbered != numbered) {
        int rc;
        for (int s = 0; s < sides; ++s) {
            if (!b.row[s] && (rc = b.mem->get(&b.row[s], (uint64_t)b.n * kRowArcs))) return rc;
            arc_rows<<<sms * 8, 256, 0, b.st>>>(b.n, ta.g_off[s], ta.g_farc[s], b.row[s]);
        }
        CHL_CUDA(cudaGetLastError());
        b.row_numbered = numbered;
        kernels += sides;
    }
    ta.g_row[0] = b.row[0];
    ta.g_row[1] = b.row[sides - 1];
    return CHL_OK;
}

// Gives back the copies of the graph that are there for speed alone: the
// numbering (its arcs in it) and the rows.  False if there were none.
bool drop_copies(Build &b) {
    if (!b.newid && !b.row[0]) return false;
    b.mem->put(b.newid);
    b.mem->put(b.orig);
    for (int s = 0; s < 2; ++s) {   // side 1 may be side 0's: put knows what is held
        b.mem->put(b.off_n[s]);
        b.mem->put(b.farc_n[s]);
        b.mem->put(b.fhead_n[s]);
        b.mem->put(b.row[s]);
    }
    return true;
}

// What get() allocates, without those copies if there is no room beside them.
template <typename Get>
int with_room(Build &b, Get get) {
    int rc = get();
    if (rc == CHL_ERR_OOM && drop_copies(b)) rc = get();
    return rc;
}

int ensure_ent(uint2 **p, uint64_t *cap, uint64_t need) {
    if (need <= *cap) return CHL_OK;
    uint64_t c = std::max<uint64_t>(need, *cap + *cap / 2);
    cudaFree(*p);
    *p = nullptr;
    // 4 spare entries: the prune test reads 16-byte pairs of entries
    int rc = dalloc(p, c + 4);
    if (rc) return rc;
    *cap = c;
    return CHL_OK;
}

}  // namespace

// Host orchestration of one build.
int build_labels(const chl_graph *g, const uint32_t *order_h, uint32_t n,
                 const chl_build_opts *opts_in, chl_labels **out) {
    chl_build_opts opts;
    if (opts_in) opts = *opts_in;
    else chl_build_opts_default(&opts);
    if (g && opts.autotune) apply_tuned_schedule(g, opts);
    if (!g || !order_h || !out || n != g->n) {
        set_error("order size must equal the number of graph vertices");
        return CHL_ERR_INVALID;
    }
    if (g->min_len < 1) {
        set_error("arc lengths must be positive (the reference asserts dd > d)");
        return CHL_ERR_INVALID;
    }
    // order must be a permutation
    std::vector<uint32_t> rank_h(n, kInf);
    for (uint32_t i = 0; i < n; ++i) {
        if (order_h[i] >= n || rank_h[order_h[i]] != kInf) {
            set_error("order is not a permutation of the vertex ids");
            return CHL_ERR_INVALID;
        }
        rank_h[order_h[i]] = i;
    }
    auto t_wall0 = std::chrono::steady_clock::now();
    Build b;
    b.n = n;
    b.sides = g->symmetric ? 1 : 2;
    b.nl = g->symmetric ? n : 2 * n;
    b.hub_bits = bits_for(std::max<uint64_t>(n, 2));
    b.key_bits = b.hub_bits + bits_for((uint64_t)b.nl + 1);
    if (b.key_bits > 64) return CHL_ERR_INVALID;
    CHL_CUDA(cudaStreamCreateWithFlags(&b.st, cudaStreamNonBlocking));
    b.mem.reset(new TmpSet(b.st));
    cudaEvent_t ev0, ev1, ev_a, ev_b, ev_up;
    CHL_CUDA(cudaEventCreate(&ev_up));
    CHL_CUDA(cudaEventCreate(&ev0));
    CHL_CUDA(cudaEventCreate(&ev1));
    CHL_CUDA(cudaEventCreate(&ev_a));
    CHL_CUDA(cudaEventCreate(&ev_b));
    struct EvGuard {
        cudaEvent_t e[5];
        ~EvGuard() {
            for (auto x : e) cudaEventDestroy(x);
        }
    } evg{{ev0, ev1, ev_a, ev_b, ev_up}};

    CHL_CUDA(cudaEventRecord(ev0, b.st));
    int rc;
    if (g->dev) {
        b.dg = (const DevGraph *)g->dev;
    } else {
        if ((rc = upload_graph(g, b.own, b.st))) return rc;
        b.dg = &b.own;
    }
    if ((rc = b.mem->get(&b.order, n)) || (rc = b.mem->get(&b.rank, n))) return rc;
    CHL_CUDA(cudaMemcpyAsync(b.order, order_h, (size_t)n * 4, cudaMemcpyHostToDevice, b.st));
    CHL_CUDA(cudaMemcpyAsync(b.rank, rank_h.data(), (size_t)n * 4, cudaMemcpyHostToDevice, b.st));
    CHL_CUDA(cudaEventRecord(ev_up, b.st));

    // committed label CSR (double buffered)
    if ((rc = dalloc(&b.off_a, (size_t)b.nl + 1)) || (rc = dalloc(&b.off_b, (size_t)b.nl + 1)))
        return rc;
    CHL_CUDA(cudaMemsetAsync(b.off_a, 0, ((size_t)b.nl + 1) * 8, b.st));
    if ((rc = b.mem->get(&b.cnt, (size_t)b.nl + 1)) || (rc = b.mem->get(&b.pre, (size_t)b.nl + 2))) return rc;
    CHL_CUDA(cudaMemsetAsync(b.cnt, 0, ((size_t)b.nl + 1) * 4, b.st));
    if ((rc = b.mem->get(&b.tsize, n)) || (rc = b.mem->get(&b.tlab, n))) return rc;
    if ((rc = b.mem->get(&b.ctl, 1))) return rc;
    if (opts.label_cap && (rc = grow_new(b, opts.label_cap))) return rc;

    // heavy-tailed degree distribution: the largest out-degree above 32
    // times the mean (scale-free graphs); bounded-degree (road-like)
    // otherwise.  Several schedule defaults below depend on it.
    bool heavy_tail = false;
    {
        uint64_t maxdeg = 0;
        for (uint32_t v = 0; v < n; ++v) maxdeg = std::max<uint64_t>(maxdeg, g->off[1][v + 1] - g->off[1][v]);
        const double avgdeg = n ? (double)g->off[1][n] / n : 0.0;
        heavy_tail = maxdeg > 32.0 * std::max(1.0, avgdeg);
    }
    // Rows of arcs (arc_rows) where at most an eighth of the lists go on past
    // theirs.  Grids gain 7 to 13% of their trees' time; random graphs of mean
    // degree 4 to 10, a third of whose lists and more do, lose 4 to 14 (20,000
    // vertices, degree 6: 33.9 and 38.8 ms).
    bool rows = !g->unit;
    for (int s = g->symmetric ? 1 : 0; s < 2 && rows; ++s) {
        uint64_t past = 0;
        for (uint32_t v = 0; v < n; ++v) past += g->off[s][v + 1] - g->off[s][v] > (uint64_t)kRowArcs;
        rows = past <= n / 8;
    }
    // vertices per distance window of the team kernel (1: settle rounds by the
    // IN criterion instead).  Larger graphs' trees are better with wider
    // windows: tree ms of grids of 400 to 900 squared with 512, 1,024 and 2,048
    //   160,000 vertices  36.0  36.2  39.1      462,000  221.0  207.1  208.2
    //   202,500           56.7  54.8  58.1      524,000  263.3  245.5  245.7
    //   262,000           85.7  83.2  86.7      590,000  334.3  308.4  305.5
    //   360,000          142.1 135.2 138.4      810,000  566.1  514.4  500.7
    // so the lines lie at 3 * 2^16 and 2^19
    const uint32_t win_target = opts.window_target ? opts.window_target
                                : heavy_tail       ? 1024u
                                : n < (3u << 16)   ? 512u
                                : n < (1u << 19)   ? 1024u
                                                   : 2048u;
    // Road-like graphs build whole: PLaNT trees without prune tests are exact
    // by their via flags alone, and cost 0.14 ns a settled vertex where a
    // pruned one costs 1 to 2 (its list and the root's).  They settle 3.5 to
    // 8 vertices per label on grids, pruned ones 1.3 to 2.5, so supersteps
    // with prune tests only pay where trees stay large: on heavy-tailed
    // graphs, and once kFreeVisits vertices per label were settled (fetch_root
    // ends the superstep).  The 1024-square grid: trees 0.81 s in one unpruned
    // superstep, 1.09 to 1.32 s with a label budget of 1024 n (0.70 in one
    // since the trees have a numbering of their own, see number_by_cells).
    const bool whole = !heavy_tail && win_target > 1 && opts.mode != CHL_MODE_GLL && opts.first_superstep == 0;
    constexpr uint32_t kFreeVisits = 16;
    // pruned trees of at least this many settled vertices (by the last
    // superstep's mean) are built by the team kernel, smaller ones a warp each
    // (the 1024-square grid within 1% between 300 and 3,000)
    constexpr double kTeamVisits = 1000;
    // workspace: one slot per resident warp
    const int sms = device_sms();
    const bool unit = g->unit;
    size_t free_b = 0, total_b = 0;
    CHL_CUDA(cudaMemGetInfo(&free_b, &total_b));
    unsigned long long prep_kernels = 0;
    {
        // arcs with their head's rank for this order
        const int nsides_g = g->symmetric ? 1 : 2;
        for (int s = 0; s < nsides_g; ++s) {
            const int src = g->symmetric ? 1 : s;
            const uint64_t m = g->off[src][n];
            const int grid = std::max(1, sms * 8);
            if (unit) {
                if ((rc = b.mem->get(&b.fhead[s], m))) return rc;
                fat_heads<<<grid, 256, 0, b.st>>>(m, b.dg->head[s], b.rank, b.fhead[s]);
            } else {
                if ((rc = b.mem->get(&b.farc[s], m))) return rc;
                fat_arcs<<<grid, 256, 0, b.st>>>(m, b.dg->arc[s], b.rank, b.dg->win[s], b.farc[s]);
            }
            CHL_CUDA(cudaGetLastError());
            ++prep_kernels;
        }
        if (nsides_g == 1) {
            b.farc[1] = b.farc[0];
            b.fhead[1] = b.fhead[0];
        }
    }
    // (the numbering and the rows are for speed alone: without room the trees
    // walk the caller's lists, and what is needed later takes their place)
    if (whole && n >= kNumberedFrom && (rc = number_by_cells(b, g, sms, prep_kernels))) {
        if (rc != CHL_ERR_OOM) return rc;
        drop_copies(b);
    }
    // key, vis and three queue arrays per warp slot (the 32-bit-key size
    // sets the schedule's warp count; the slots below use the real one)
    const size_t per_slot = (size_t)n * 20;
    uint32_t want = (uint32_t)sms * 48;   // 12 blocks of 4 warps per SM at most
    if (opts.max_warps) want = std::min<uint32_t>(want, opts.max_warps);
    const size_t ws_budget = free_b / 3;
    uint32_t fit = (uint32_t)std::max<size_t>(1, ws_budget / std::max<size_t>(per_slot, 1));
    b.warps = std::max<uint32_t>(kWarpsPerBlock, std::min(want, fit));
    b.warps = (b.warps / kWarpsPerBlock) * kWarpsPerBlock;
    // Only the blocks resident from the start build trees: a block leaves
    // when no root is left for the superstep, and every refusal of a root is
    // final for it.  The grid and the workspace cover those alone (b.warps
    // still sets the first superstep's size).
    int nbo = 0;
    CHL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &nbo, unit ? batch_kernel<true, true> : batch_kernel<false, true>, kWarpsPerBlock * 32, 0));
    nbo = std::max(nbo, 1);
    b.slots = std::min(b.warps, (uint32_t)nbo * (uint32_t)sms * kWarpsPerBlock);
    {
        // weighted graphs hold 64-bit keys: 24 bytes per vertex and slot
        const size_t slot_bytes = (size_t)n * (unit ? 20 : 24);
        const uint32_t fit_slots = (uint32_t)std::max<size_t>(kWarpsPerBlock, ws_budget / std::max<size_t>(slot_bytes, 1));
        b.slots = std::max<uint32_t>(kWarpsPerBlock, (std::min(b.slots, fit_slots) / kWarpsPerBlock) * kWarpsPerBlock);
    }
    // team kernel: one tree per block of win_tw warps (auto: 8 on heavy-tailed
    // graphs, 4 otherwise), as many trees as are resident, 6 n words each
    b.win_tw = opts.window_warps ? opts.window_warps : (heavy_tail ? 8 : 4);
    if (b.win_tw != 1 && b.win_tw != 2 && b.win_tw != 4 && b.win_tw != 8) {
        set_error("window_warps must be 0, 1, 2, 4 or 8");
        return CHL_ERR_INVALID;
    }
    // Warps per tree of a superstep: where at most two roots per SM start
    // (unpruned first supersteps), as many as a block holds; a tree of 29,000
    // vertices on a directed skewed graph of 2^15 is one of 152 then (build
    // 14.6 ms with 8 warps, 8.6 with 32; weighted RMAT scale 17 in GLL mode
    // 62 and 43).  Pruned trees keep win_tw (38.5 there with 8, 43 with 32).
    auto team_warps = [&](bool prune, uint32_t roots) -> uint32_t {
        return opts.window_warps == 0 && !prune && roots <= 2u * sms ? 32u : b.win_tw;
    };
    // root hash slots: at most 2048 per warp-built tree within CHL_SMEM_CAP_KB
    // of shared memory per block, and 4096 per block-built one
    int max_smem = 0;
    CHL_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, 0));
    // A kernel's limit of dynamic shared memory belongs to the process: it is
    // always raised to the same value, so that builds of other threads never
    // find it below what they launch with.  (The occupancy query counts a
    // block's dynamic shared memory only up to that limit, 48 KB by default.)
    auto allow_smem = [&](TreeKernel k) -> int {
        CHL_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
        return CHL_OK;
    };
    auto team_blocks = [&](bool plant, bool prune, uint32_t tw, uint32_t hash_slots, int *blocks) -> int {
        TreeKernel k = team_kernel_for(unit, plant, prune, rows, tw);
        const int sm = (int)team_smem((int)tw * 32, hash_slots);
        if ((rc = allow_smem(k))) return rc;
        CHL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k, tw * 32, sm));
        *blocks = std::max(*blocks, 1) * sms;
        return CHL_OK;
    };
    {
        int blocks = 0;
        if ((rc = team_blocks(true, false, b.win_tw, 0, &blocks))) return rc;
        const uint64_t fit_trees = std::max<uint64_t>(1, ws_budget / std::max<uint64_t>(24ull * n, 1));
        b.win_trees = (uint32_t)std::min<uint64_t>((uint64_t)blocks, fit_trees);
        if (opts.max_warps) b.win_trees = std::min(b.win_trees, opts.max_warps);   // the cap on concurrent trees
    }
    // one workspace for both layouts: batch_kernel's key (two words on
    // weighted graphs), vis and queue arrays per warp slot (5 or 6 n words),
    // team_kernel's 6 n words per tree
    const size_t key_words = unit ? 1 : 2;
    const size_t ws_words = std::max((size_t)b.slots * (4 + key_words) * n, (size_t)b.win_trees * 6 * n);
    if ((rc = with_room(b, [&] { return b.mem->get(&b.ws_all, ws_words); }))) return rc;
    b.ws_key = b.ws_all;
    b.ws_vis = b.ws_all + (size_t)b.slots * key_words * n;
    b.ws_front = b.ws_vis + (size_t)b.slots * n;
    b.ws_layout = 0;   // set before each tree launch
    {
        // root hash slots: at most 2048, and within CHL_SMEM_CAP_KB of shared
        // memory per block (measured on the 1024-square grid: 2048 slots at 2
        // resident blocks per SM beat 1024 slots at 3 by 1.3x -- entries past
        // half the table are searched in global memory)
        const size_t smem_cap = std::min<size_t>((size_t)max_smem, CHL_SMEM_CAP_KB * 1024);
        uint32_t t = 64;
        while (2 * t <= 2048 && kWarpsPerBlock * batch_smem_per_warp(2 * t) <= smem_cap) t *= 2;
        b.hash_max = t;
    }

    // bit-parallel first supersteps: unit lengths and few levels (see
    // bit_level); rows of cur, nxt and seen and two flags per vertex, in the
    // trees' workspace
    const size_t bit_row = (size_t)n * kBitWords;
    bool bits_ok = unit && heavy_tail && win_target > 1 && opts.max_warps == 0 &&
                   ws_words * 4 >= bit_row * (2 * sizeof(ulonglong2) + 8) + 2 * (size_t)n;
    // superstep loop
    // label budget per superstep (the reference's sf * N); auto: 32 on
    // heavy-tailed graphs, 1024 on road-like ones.  On road-like graphs a
    // superstep lasts as long as its largest tree, so fewer, larger
    // supersteps pay off once the near/far queue and the distance cutoff
    // keep the less-pruned trees cheap; from 1024 on the growth schedule,
    // not the budget, sets their size (measured on the 512/1024-square
    // grids: 1024 and unbounded within 1%, 128 1.27x slower; RMAT scale
    // 20: 16-64 within 3%)
    // (bit-parallel supersteps have no largest tree to wait for and pay for
    // every commit: RMAT scale 20 342 ms with 128, 309 with 512)
    // label_limit = sf * N counts both sides' labels (shared_memory/hhl.cpp:65);
    // a symmetric build stores one side.
    auto label_budget = [&]() -> unsigned long long {
        const double sf = opts.sf > 0 ? opts.sf : bits_ok ? 512.0 : heavy_tail ? 32.0 : 1024.0;
        return (unsigned long long)std::max(1.0, sf * (double)n / (b.sides == 1 ? 2.0 : 1.0));
    };
    unsigned long long budget_base = label_budget();
    // Supersteps of unpruned trees (whole) end at the label buffer, which has
    // room for lists of 1.7 sqrt(n) (grids have 0.7 to 1.5 sqrt(n)) within a
    // quarter of the free memory; a seventh of it is left to the trees still
    // running when the budget is spent.
    const bool whole_budget = whole && opts.sf <= 0 && opts.label_cap == 0;
    if (whole_budget) {
        size_t fr = 0, tot = 0;
        CHL_CUDA(cudaMemGetInfo(&fr, &tot));
        const uint64_t want = (uint64_t)(2.0 * std::sqrt((double)n) * n * b.sides) + (1u << 20);
        if ((rc = with_room(b, [&] { return grow_new(b, std::min<uint64_t>(want, fr / 4 / 36)); }))) return rc;
        budget_base = b.new_cap - b.new_cap / 7;
    }
    if (opts.label_cap == 0 && !whole_budget) {
        // Room for every new label of a superstep: the budget plus what the
        // trees still running when it is spent can add (at most sides * n
        // each), so that a superstep does not overflow and run twice.  At
        // most a quarter of the free memory (36 bytes per entry: two key and
        // two value arrays for the sort, the clean's flags and prefix);
        // beyond that an overflow re-runs the superstep's root range.
        size_t fr = 0, tot = 0;
        CHL_CUDA(cudaMemGetInfo(&fr, &tot));
        // Bit-parallel batches end a superstep exactly; the trees after them
        // label a few vertices each, so room for 64 whole ones is kept.
        const uint64_t running = bits_ok ? 64u : std::max(b.slots, b.win_trees);
        const uint64_t want = (uint64_t)budget_base + running * b.sides * n;
        const uint64_t fit = (uint64_t)(fr / 4 / 36);
        const uint64_t cap = std::max<uint64_t>(std::min(want, fit), std::max<uint64_t>(4ull * n, 1u << 20));
        if ((rc = with_room(b, [&] { return grow_new(b, cap); }))) return rc;
    }
    uint32_t *bit_long[2] = {nullptr, nullptr};   // long lists of each direction
    unsigned long long *bit_live = nullptr;       // kBitLevels + 1 rows
    uint32_t dist_hi = 0;                         // largest committed distance
    uint32_t bit_hi = 0;                          // and of the superstep's labels
    uint32_t bit_steps = 0;                       // supersteps built bit-parallel
    double bit_mean = 0;                          // vertices a root of the last batch reached
    constexpr double kBitShare = 10, kBitShareNext = 7;
    bool do_plant = opts.mode != CHL_MODE_GLL;
    bool switch_open = opts.mode == CHL_MODE_HYBRID;
    uint32_t r0 = 0;
    uint64_t committed = 0;
    uint32_t supersteps = 0, plant_roots = 0;
    unsigned long long visits = 0, reads = 0, arcs = 0, launches = 0, kernels = prep_kernels;
    double tree_ms = 0, sort_ms = 0, commit_ms = 0;
    uint32_t max_list = 0;   // longest committed list
    float step_tree_ms = 0;
    uint32_t step_slots = 0;   // warp slots of the last tree launch
    double mean_visits = 0;    // settled vertices per tree of the last superstep
    bool ratio_stopped = false;
    // Superstep schedule: superstep k covers roots [r0, r0 + size) with
    // size = clamp(growth * r0, first, n) -- small while the top hubs are not
    // yet committed (their labels prune everything later), geometric after.
    // The label budget sf * n (the reference's label_limit) also ends a
    // superstep early.
    // Bit-parallel graphs start with two batches and treble (RMAT scale 17
    // doubling 14.2 ms, trebling 13.2; scale 20 315 and 307).  Other
    // heavy-tailed degree distributions start with one root per SM and grow
    // eightfold: their commits cost more than the pruning of small trees
    // saves (a directed skewed graph of 2^15 vertices 10.0 ms growing twofold,
    // 8.9 eightfold; weighted RMAT scale 17 74 and 70).  GLL trees emit a
    // superset that grows with the unpruned superstep, so road-like graphs in
    // GLL mode start with one root per SM as well and treble, without
    // extending (the 256-square grid 67 ms; 217 with 14,592 roots, of which
    // the clean took 176).  Bounded-degree graphs with an option that keeps
    // them from the whole rule start with two roots per warp of the schedule
    // and grow by half of the committed prefix.
    const bool gll_auto = !heavy_tail && opts.mode == CHL_MODE_GLL && win_target > 1 && opts.first_superstep == 0;
    // (a build that leaves the bit-parallel kernel goes on by the schedule of
    // the others: step_end and label_budget are asked again)
    auto step_end = [&](uint32_t from) -> uint32_t {
        const uint32_t auto_first = bits_ok ? 2 * kBitRoots
                                    : win_target > 1 && (heavy_tail || gll_auto) ? std::max<uint32_t>(64u, sms)
                                    : heavy_tail ? 1024u
                                                 : std::max<uint32_t>(64u, 2 * b.warps);
        const double auto_growth = bits_ok ? 3.0 : heavy_tail ? 8.0 : gll_auto ? 2.0 : 0.5;
        const uint32_t first = opts.first_superstep ? opts.first_superstep : auto_first;
        const double growth = opts.growth > 0 ? opts.growth : auto_growth;
        const uint64_t size = std::max<uint64_t>(first, (uint64_t)(growth * (double)from));
        const uint32_t end = (uint32_t)std::min<uint64_t>(n, (uint64_t)from + size);
        return opts.root_limit ? std::min<uint32_t>(end, opts.root_limit) : end;
    };
    // phase switch ratio (the reference's -ps, default 1024): auto 8 on
    // heavy-tailed graphs (RMAT scale 20: pruned GLL supersteps after the
    // first are faster than PLaNT trees there)
    const double ps = opts.ps > 0 ? opts.ps : (heavy_tail ? 8.0 : 1024.0);
    // The roots [r0, r_end) by bit_level, a batch at a time until the label
    // budget is spent; *done: the first root not taken, *off: gave up, at
    // kBitLevels or for want of room for the table (up to 4 KB per committed
    // root).  The host reads the live roots after each level.
    auto bit_superstep = [&](unsigned long long budget, uint32_t r_end, uint32_t *done, bool *off) -> int {
        if (!bit_live) {
            if ((rc = b.mem->get(&bit_live, (uint64_t)(kBitLevels + 1) * kBitWords))) return rc;
            for (int f = 0; f < b.sides; ++f) {
                const int rev = b.sides == 1 ? 1 : 1 - f;
                const uint64_t m = g->off[g->symmetric ? 1 : rev][n];
                if ((rc = b.mem->get(&bit_long[f], m / kBitHeavy + 1))) return rc;
                CHL_CUDA(cudaMemsetAsync(bit_long[f], 0, 4, b.st));
                bit_heavy<<<sms, 256, 0, b.st>>>(n, b.dg->off[rev], bit_long[f]);
                CHL_CUDA(cudaGetLastError());
                ++kernels;
            }
        }
        b.ws_layout = 0;
        ulonglong2 *rows[2] = {(ulonglong2 *)b.ws_all, (ulonglong2 *)b.ws_all + bit_row};
        unsigned long long *seen = (unsigned long long *)(rows[1] + bit_row);
        uint8_t *act[2] = {(uint8_t *)(seen + bit_row), (uint8_t *)(seen + bit_row) + n};
        const uint32_t K = dist_hi + 1;
        unsigned long long *M = nullptr;
        if (r0 && (rc = b.mem->get(&M, (uint64_t)r0 * K * kBitWords))) {
            *off = rc == CHL_ERR_OOM;
            return *off ? CHL_OK : rc;
        }
        CHL_CUDA(cudaMemsetAsync(b.tsize + 0, 0, (size_t)(r_end - r0) * 4, b.st));
        CHL_CUDA(cudaMemsetAsync(b.tlab + 0, 0, (size_t)(r_end - r0) * 4, b.st));
        uint32_t rb = r0;
        unsigned long long used = 0, visited = 0;
        bit_mean = (double)n;
        // (a re-run takes the same roots whatever they reach)
        for (; rb < r_end && used < budget && (bit_mean * kBitShare >= n || budget == ~0ull); rb += kBitRoots) {
            const uint32_t nb = std::min(kBitRoots, r_end - rb);
            uint32_t last_level = 0;
            for (int sd = 0; sd < b.sides; ++sd) {
                const int f = b.sides == 1 ? 1 : sd, rev = b.sides == 1 ? 1 : 1 - f;
                BitArgs a;
                a.n = n;
                a.sides = b.sides;
                a.f = f;
                a.roff = b.dg->off[rev];
                a.rhead = b.fhead[rev];
                a.foff = b.dg->off[f];
                a.order = b.order;
                a.rank = b.rank;
                a.l_off = b.off_a;
                a.l_ent = b.ent_a;
                a.l_dent = b.dent_a;
                a.r0 = r0;
                a.rb = rb;
                a.nb = nb;
                a.d = 0;
                a.K = K;
                a.seen = seen;
                a.M = M;
                a.heavy = bit_long[b.sides == 1 ? 0 : f];
                a.hub_bits = b.hub_bits;
                a.out_key = b.nk0;
                a.out_val = b.nv0;
                a.out_cap = b.new_cap;
                a.ctl = b.ctl;
                CHL_CUDA(cudaMemsetAsync(seen, 0, bit_row * 8, b.st));
                CHL_CUDA(cudaMemsetAsync(act[0], 0, n, b.st));
                CHL_CUDA(cudaMemsetAsync(bit_live, 0, (size_t)(kBitLevels + 1) * kBitWords * 8, b.st));
                a.cur = rows[1];
                a.nxt = rows[0];
                a.act = act[1];
                a.act_out = act[0];
                a.live = bit_live;
                a.live_out = bit_live;
                bit_roots<<<(nb + kBitGroups - 1) / kBitGroups, kBitThreads, 0, b.st>>>(a);
                if (r0) {
                    CHL_CUDA(cudaMemsetAsync(M, 0, (size_t)r0 * K * kBitWords * 8, b.st));
                    bit_table<<<(nb + 7) / 8, 256, 0, b.st>>>(a);
                }
                CHL_CUDA(cudaGetLastError());
                kernels += r0 ? 2 : 1;
                launches += r0 ? 2 : 1;
                for (uint32_t d = 1;; ++d) {
                    if (d > kBitLevels) {
                        *off = true;
                        b.mem->put(M);
                        return CHL_OK;
                    }
                    a.d = d;
                    a.cur = rows[(d - 1) & 1];
                    a.nxt = rows[d & 1];
                    a.act = act[(d - 1) & 1];
                    a.act_out = act[d & 1];
                    a.live = bit_live + (size_t)(d - 1) * kBitWords;
                    a.live_out = bit_live + (size_t)d * kBitWords;
                    if (r0) {
                        bit_level<true, true><<<sms * 4, kBitThreads, 0, b.st>>>(a);
                        bit_level<false, true><<<sms * 8, kBitThreads, 0, b.st>>>(a);
                    } else {
                        bit_level<true, false><<<sms * 4, kBitThreads, 0, b.st>>>(a);
                        bit_level<false, false><<<sms * 8, kBitThreads, 0, b.st>>>(a);
                    }
                    CHL_CUDA(cudaGetLastError());
                    kernels += 2;
                    launches += 2;
                    unsigned long long live[kBitWords], any = 0;
                    CHL_CUDA(cudaMemcpyAsync(live, a.live_out, sizeof(live), cudaMemcpyDeviceToHost, b.st));
                    CHL_CUDA(cudaStreamSynchronize(b.st));
                    for (unsigned long long x : live) any |= x;
                    last_level = std::max(last_level, any ? d : d - 1);
                    if (!any) break;
                }
            }
            // labels reach the last level with a not-via vertex
            unsigned long long tot[2] = {0, 0};
            static_assert(offsetof(BuildCtl, visits) == offsetof(BuildCtl, nlab) + 8, "read together");
            CHL_CUDA(cudaMemcpyAsync(tot, &b.ctl->nlab, 16, cudaMemcpyDeviceToHost, b.st));
            CHL_CUDA(cudaStreamSynchronize(b.st));
            used = tot[0];
            bit_mean = (double)(tot[1] - visited) / nb;
            visited = tot[1];
            bit_hi = std::max(bit_hi, last_level);
            CHL_CUDA(cudaMemcpyAsync(&b.ctl->max_dist, &bit_hi, 4, cudaMemcpyHostToDevice, b.st));
        }
        *done = std::min(rb, r_end);
        b.mem->put(M);
        return CHL_OK;
    };
    while (r0 < n && (opts.root_limit == 0 || r0 < opts.root_limit)) {
        const uint32_t r_begin = r0;
        bit_hi = 0;
        const bool plant_now = do_plant;
        unsigned long long budget = budget_base;
        // trees without prune tests, over all roots that are left
        const bool unpruned = whole && plant_now && !ratio_stopped;
        uint32_t r_end = step_end(r0);
        if (unpruned) r_end = opts.root_limit ? std::min<uint32_t>(n, opts.root_limit) : n;
        BuildCtl hc;
        bool rerun = false;
        uint32_t step_reruns = 0;
        // root hash table: a power of two at least twice the longest committed
        // list, within the occupancy-preserving size (entries beyond half the
        // table are searched in the global list)
        uint32_t hash_slots = 64;
        while (hash_slots < 2 * std::max<uint32_t>(max_list, 32) && 2 * hash_slots <= b.hash_max) hash_slots *= 2;
        const size_t smem = kWarpsPerBlock * batch_smem_per_warp(hash_slots);
        // A batch costs its sweeps over all rows however few vertices its
        // roots still reach, so a superstep ends with the first batch whose
        // roots reach less than a tenth of the graph, and the next one is
        // built by trees unless the last batch reached a seventh (more
        // committed labels: RMAT scale 17 12% in roots 1,024-3,071, 1% in the
        // next superstep, where batches would take twice the trees' 2.9 ms;
        // scale 20 20% and then 7%, 68 ms for 6,144 roots in batches against
        // 146 in trees)
        bool bits_now = bits_ok && dist_hi < kBitDist && (r0 == 0 || (bit_steps == supersteps && bit_mean * kBitShareNext >= n));
        while (true) {
            std::memset(&hc, 0, sizeof(hc));
            hc.next_root = r0;
            CHL_CUDA(cudaMemcpyAsync(b.ctl, &hc, sizeof(hc), cudaMemcpyHostToDevice, b.st));
            if (bits_now) {
                uint32_t done = r0;
                bool off = false;
                CHL_CUDA(cudaEventRecord(ev_a, b.st));
                if ((rc = bit_superstep(rerun ? ~0ull : budget, r_end, &done, &off))) return rc;
                CHL_CUDA(cudaEventRecord(ev_b, b.st));
                CHL_CUDA(cudaMemcpyAsync(&hc, b.ctl, sizeof(hc), cudaMemcpyDeviceToHost, b.st));
                CHL_CUDA(cudaStreamSynchronize(b.st));
                float ms = 0;
                CHL_CUDA(cudaEventElapsedTime(&ms, ev_a, ev_b));
                tree_ms += ms;
                step_tree_ms = ms;
                if (off) {   // these roots by the other kernels
                    bits_ok = bits_now = false;
                    if (rerun) continue;   // over the same range
                    r_end = step_end(r0);
                    budget = budget_base = label_budget();
                    continue;
                }
                if (hc.overflow || hc.nlab > b.new_cap) {
                    ++step_reruns;
                    if ((rc = with_room(b, [&] { return grow_new(b, hc.nlab + hc.nlab / 4 + 1024); }))) return rc;
                    r_end = done;
                    rerun = true;
                    continue;
                }
                r_end = done;
                break;
            }
            TreeArgs ta;
            ta.n = n;
            ta.sides = b.sides;
            for (int s = 0; s < 2; ++s) {
                ta.g_off[s] = b.dg->off[s];
                ta.g_farc[s] = b.farc[s];
                ta.g_fhead[s] = b.fhead[s];
            }
            ta.order = b.order;
            ta.g_row[0] = ta.g_row[1] = nullptr;
            ta.newid = ta.orig = nullptr;
            ta.rank = b.rank;
            ta.l_off = b.off_a;
            ta.l_ent = b.ent_a;
            ta.l_dent = b.dent_a;
            ta.r0 = r0;
            ta.r_end = r_end;
            // work-conserving extension: up to ext x the nominal size while
            // nominal trees run; none on a rerun
            uint32_t ext = opts.superstep_extend == 0 ? (heavy_tail || gll_auto ? 1u : 4u)
                                                      : (uint32_t)std::max(1, opts.superstep_extend);
            if (rerun) ext = 1;
            ta.r_hard = (uint32_t)std::min<uint64_t>(n, (uint64_t)r0 + (uint64_t)ext * (r_end - r0));
            if (opts.root_limit) ta.r_hard = std::min<uint32_t>(ta.r_hard, std::max(opts.root_limit, r_end));
            ta.budget = rerun ? ~0ull : budget;
            ta.hub_bits = b.hub_bits;
            ta.out_key = b.nk0;
            ta.out_val = b.nv0;
            ta.out_cap = b.new_cap;
            ta.tree_size = b.tsize;
            ta.tree_labels = b.tlab;
            ta.ws_key = b.ws_key;
            ta.ws_vis = b.ws_vis;
            ta.ws_front = b.ws_front;
            ta.ctl = b.ctl;
            ta.hash_slots = hash_slots;
            ta.hash_shift = 32;
            for (uint32_t t = hash_slots; t > 1; t >>= 1) --ta.hash_shift;
            const int blocks = (int)(b.slots / kWarpsPerBlock);
            // near/far queue.  Auto: split above 1024 queued vertices on
            // road-like graphs, whose queues are long rings of close keys
            // (1.25x faster builds of the 512/1024-square grids); off on
            // heavy-tailed ones, whose few-level queues gain nothing (RMAT
            // scale 20: 4% slower with it)
            ta.near_on = 0;
            ta.near_target = 1;
            const int qs = opts.queue_split ? opts.queue_split : (heavy_tail ? 1 : 1024);
            if (qs > 1) {
                ta.near_on = (uint32_t)qs;
                ta.near_target = std::max<uint32_t>(1, ta.near_on / 4);
            }
            void (*kern)(TreeArgs);
            size_t smem_launch = smem;
            int grid = blocks, block = kWarpsPerBlock * 32;
            const bool windowed = win_target > 1 && (committed == 0 || unpruned || mean_visits >= kTeamVisits);
            ta.visit_ratio = unpruned && !rerun ? kFreeVisits : 0;
            ta.visit_base = 64ull * n;
            if (windowed) {
                const bool prune = committed > 0 && !unpruned;
                uint32_t slots = prune ? 64 : 0;   // no committed labels: no root label to hash
                while (prune && slots < 2 * max_list && slots < 4096) slots *= 2;
                ta.hash_slots = slots;
                ta.hash_shift = 32;
                for (uint32_t t = slots; t > 1; t >>= 1) --ta.hash_shift;
                ta.near_target = win_target;
                ta.ws_win = b.ws_all;
                if (unpruned && b.newid) {
                    ta.newid = b.newid;
                    ta.orig = b.orig;
                    for (int s = 0; s < 2; ++s) {
                        ta.g_off[s] = b.off_n[s];
                        ta.g_farc[s] = b.farc_n[s];
                        ta.g_fhead[s] = b.fhead_n[s];
                    }
                }
                if (rows && !prune && (rc = fill_rows(b, ta, sms, kernels))) {
                    if (rc != CHL_ERR_OOM) return rc;
                    for (auto &r : b.row) b.mem->put(r);
                    rows = false;
                }
                int fit = 0;
                const uint32_t tw = team_warps(prune, r_end - r0);
                if ((rc = team_blocks(plant_now, prune, tw, slots, &fit))) return rc;
                grid = (int)std::min<uint32_t>((uint32_t)fit, b.win_trees);
                block = (int)tw * 32;
                smem_launch = team_smem(block, slots);
                kern = team_kernel_for(unit, plant_now, prune, rows, tw);
            } else if (unit) {
                kern = plant_now ? batch_kernel<true, true> : batch_kernel<true, false>;
            } else {
                kern = plant_now ? batch_kernel<false, true> : batch_kernel<false, false>;
            }
            // the two layouts share the workspace: every key the next kernel
            // reads is INF (each tree resets its own keys when it ends)
            const int layout = windowed ? 2 : 1;
            if (b.ws_layout != layout) {
                if (windowed)
                    CHL_CUDA(cudaMemset2DAsync(b.ws_all, (size_t)n * 24, 0xFF, (size_t)n * 8, b.win_trees, b.st));
                else
                    CHL_CUDA(cudaMemsetAsync(b.ws_all, 0xFF, (size_t)b.slots * key_words * n * 4, b.st));
                b.ws_layout = layout;
            }
            if ((rc = allow_smem(kern))) return rc;
            CHL_CUDA(cudaEventRecord(ev_a, b.st));
            kern<<<grid, block, smem_launch, b.st>>>(ta);
            step_slots = (uint32_t)grid * (uint32_t)block / 32;
            CHL_CUDA(cudaGetLastError());
            CHL_CUDA(cudaEventRecord(ev_b, b.st));
            ++launches;
            ++kernels;
            CHL_CUDA(cudaMemcpyAsync(&hc, b.ctl, sizeof(hc), cudaMemcpyDeviceToHost, b.st));
            CHL_CUDA(cudaStreamSynchronize(b.st));
            float ms = 0;
            CHL_CUDA(cudaEventElapsedTime(&ms, ev_a, ev_b));
            tree_ms += ms;
            step_tree_ms = ms;
            const unsigned long long fetched = (hc.next_root & kClosed) ? hc.close_at : hc.next_root;
            uint32_t r1 = (uint32_t)std::min<unsigned long long>(fetched, std::max(ta.r_hard, r_end));
            if (hc.err) {
                set_error(hc.err == 1 ? "a shortest-path distance reaches INT_MAX (the reference asserts dd < infty)"
                                      : "tree workspace bound exceeded");
                return CHL_ERR_INVALID;
            }
            if (hc.overflow || hc.nlab > b.new_cap) {
                ++step_reruns;
                // re-run the same root range with room for every label
                if ((rc = with_room(b, [&] { return grow_new(b, hc.nlab + hc.nlab / 4 + 1024); }))) return rc;
                r_end = r1;
                rerun = true;
                continue;
            }
            r_end = r1;
            break;
        }
        const uint32_t r1 = r_end;
        mean_visits = (double)hc.visits / std::max<uint32_t>(1, r1 - r0);
        ratio_stopped |= hc.ratio_stop != 0;
        dist_hi = std::max<uint32_t>(dist_hi, hc.max_dist);
        const bool last = r1 >= n || (opts.root_limit && r1 >= opts.root_limit);
        visits += hc.visits;
        reads += hc.label_reads;
        arcs += hc.arcs;
        if (plant_now) plant_roots += r1 - r0;
        unsigned long long M = hc.nlab;
        // hybrid switch (distributed_memory/akiba.hpp:297-303, 362-376)
        // (heavy-tailed graphs switch after their bit-parallel supersteps, which
        // measure no tree sizes: their first trees are 10 times their labels)
        bit_steps += bits_now ? 1 : 0;
        if (bits_now && switch_open && opts.ps <= 0) {
            do_plant = false;
            switch_open = false;
        } else if (plant_now && switch_open && !bits_now) {
            unsigned long long zero = 0;
            CHL_CUDA(cudaMemcpyAsync(&b.ctl->max_ratio_num, &zero, 8, cudaMemcpyHostToDevice, b.st));
            ratio_max<<<std::max(1, sms), 256, 0, b.st>>>(b.tsize, b.tlab, &b.ctl->next_root, r0, r1, b.ctl);
            ++kernels;
            unsigned long long bits = 0;
            CHL_CUDA(cudaMemcpyAsync(&bits, &b.ctl->max_ratio_num, 8, cudaMemcpyDeviceToHost, b.st));
            CHL_CUDA(cudaStreamSynchronize(b.st));
            double ratio;
            std::memcpy(&ratio, &bits, 8);
            if (ratio > ps) {
                do_plant = false;
                switch_open = false;
            }
        }
        // Sort, GLL clean and merge of the new labels, then the longest
        // committed list: one stream-ordered chain with no host round trip,
        // captured as a CUDA graph when opts.use_graphs is set.  The entry
        // array is sized for every new label before the chain (the clean
        // only removes labels).
        const bool clean_now = !plant_now && !bits_now && M > 0;   // bit-parallel labels are canonical
        auto commit_room = [&]() -> int {
            if ((rc = grow_sort(b, M, clean_now))) return rc;
            if ((rc = ensure_ent(&b.ent_b, &b.ent_cap_b, committed + M))) return rc;
            return last ? CHL_OK : ensure_ent(&b.dent_b, &b.dent_cap_b, committed + M);
        };
        if ((rc = with_room(b, commit_room))) return rc;
        // bits of the distance part of the (list, distance) sort key
        const int dist_bits = bits_for((uint64_t)hc.max_dist + 1);
        auto chain = [&]() -> int {
            int rc2;
            const uint64_t m_cap = M;   // the sort sees the count in device memory as well
            // --- sort the new labels by (list, hub)
            int parity = 0;
            if ((rc2 = radix_sort_pairs(b.nk0, b.nv0, b.nk1, b.nv1, (const uint64_t *)&b.ctl->nlab, m_cap,
                                        b.key_bits, b.tmp, b.tmp_bytes, b.st, &parity)))
                return rc2;
            uint64_t *sk = parity ? b.nk1 : b.nk0;
            uint32_t *sv = parity ? b.nv1 : b.nv0;
            uint64_t *ak = parity ? b.nk0 : b.nk1;
            uint32_t *av = parity ? b.nv0 : b.nv1;
            const int cgrid = sms * 8;
            const unsigned long long *d_count = &b.ctl->nlab;
            // --- GLL clean (drops labels covered through a higher-ranked hub)
            if (clean_now) {
                CHL_CUDA(cudaMemsetAsync(b.cnt, 0, ((size_t)b.nl + 1) * 4, b.st));
                count_keys<<<cgrid, 256, 0, b.st>>>(sk, d_count, m_cap, b.hub_bits, b.cnt);
                if ((rc2 = scan_u32_excl(b.cnt, b.pre, b.nl, nullptr, b.tmp, b.tmp_bytes, b.st))) return rc2;
                clean_mark<<<cgrid, 256, 0, b.st>>>(sk, sv, d_count, m_cap, b.hub_bits, r0, b.pre, b.order,
                                                    b.rank, b.sides, b.keep);
                if ((rc2 = scan_u32_excl(b.keep, b.kpre, m_cap, (const uint64_t *)d_count, b.tmp,
                                         b.tmp_bytes, b.st)))
                    return rc2;
                compact_kept<<<cgrid, 256, 0, b.st>>>(sk, sv, b.keep, b.kpre, d_count, m_cap, ak, av,
                                                      &b.ctl->n_keep);
                CHL_CUDA(cudaMemcpyAsync(&b.ctl->nlab, &b.ctl->n_keep, 8, cudaMemcpyDeviceToDevice, b.st));
                std::swap(sk, ak);
                std::swap(sv, av);
            }
            // --- commit: merge the sorted new labels into the committed CSR
            CHL_CUDA(cudaMemsetAsync(b.cnt, 0, ((size_t)b.nl + 1) * 4, b.st));
            count_keys<<<cgrid, 256, 0, b.st>>>(sk, d_count, m_cap, b.hub_bits, b.cnt);
            if ((rc2 = scan_u32_excl(b.cnt, b.pre, b.nl, nullptr, b.tmp, b.tmp_bytes, b.st))) return rc2;
            merge_offsets<<<cgrid, 256, 0, b.st>>>(b.off_a, b.pre, b.off_b, b.nl);
            copy_old_lists<<<cgrid, 256, 0, b.st>>>(b.off_a, b.ent_a, b.off_b, b.ent_b, b.nl);
            place_new<<<cgrid, 256, 0, b.st>>>(sk, sv, d_count, m_cap, b.hub_bits, r0, b.pre, b.off_a,
                                               b.off_b, b.ent_b);
            if (!last) {
                // the same labels by (list, distance, hub), merged into the
                // distance-ordered copy (the sort is stable: equal distances
                // keep hub order); the key holds the distance in the bits the
                // superstep's largest distance needs
                dist_keys<<<cgrid, 256, 0, b.st>>>(sk, sv, d_count, m_cap, b.hub_bits, dist_bits, r0, ak, av);
                int par2 = 0;
                if ((rc2 = radix_sort_pairs(ak, av, sk, sv, (const uint64_t *)d_count, m_cap,
                                            b.key_bits - b.hub_bits + dist_bits, b.tmp, b.tmp_bytes, b.st, &par2)))
                    return rc2;
                merge_dist_lists<<<cgrid, 256, 0, b.st>>>(b.off_a, b.dent_a, b.off_b, b.pre, par2 ? sk : ak,
                                                          par2 ? sv : av, b.dent_b, b.nl, dist_bits);
            }
            // longest committed list, for the next superstep's root staging
            CHL_CUDA(cudaMemsetAsync(&b.ctl->max_ratio_den, 0, 8, b.st));
            max_list_len<<<cgrid, 256, 0, b.st>>>(b.off_b, b.nl, &b.ctl->max_ratio_den);
            CHL_CUDA(cudaGetLastError());
            return CHL_OK;
        };
        kernels += 3 * ((b.key_bits + 7) / 8) + (clean_now ? 9 : 0) + 8;
        if (!last) kernels += 2 + 3 * ((b.key_bits - b.hub_bits + dist_bits + 7) / 8);
        CHL_CUDA(cudaEventRecord(ev_a, b.st));
        if (opts.use_graphs) {
            CHL_CUDA(cudaStreamBeginCapture(b.st, cudaStreamCaptureModeThreadLocal));
            const int crc = chain();
            cudaGraph_t cg = nullptr;
            const cudaError_t ce = cudaStreamEndCapture(b.st, &cg);
            if (crc) {
                if (cg) cudaGraphDestroy(cg);
                return crc;
            }
            CHL_CUDA(ce);
            // reuse the executable graph when only kernel arguments changed
            bool updated = false;
            if (b.commit_exec) {
                cudaGraphExecUpdateResultInfo info;
                updated = cudaGraphExecUpdate(b.commit_exec, cg, &info) == cudaSuccess;
                if (!updated) {
                    (void)cudaGetLastError();
                    cudaGraphExecDestroy(b.commit_exec);
                    b.commit_exec = nullptr;
                }
            }
            cudaError_t ie = cudaSuccess;
            if (!updated) ie = cudaGraphInstantiate(&b.commit_exec, cg, 0);
            cudaGraphDestroy(cg);
            CHL_CUDA(ie);
            CHL_CUDA(cudaGraphLaunch(b.commit_exec, b.st));
            ++b.graph_launches;
        } else if ((rc = chain())) {
            return rc;
        }
        CHL_CUDA(cudaEventRecord(ev_b, b.st));
        std::swap(b.off_a, b.off_b);
        std::swap(b.ent_a, b.ent_b);
        std::swap(b.ent_cap_a, b.ent_cap_b);
        std::swap(b.dent_a, b.dent_b);
        std::swap(b.dent_cap_a, b.dent_cap_b);
        CHL_CUDA(cudaMemcpyAsync(&hc, b.ctl, sizeof(hc), cudaMemcpyDeviceToHost, b.st));
        CHL_CUDA(cudaStreamSynchronize(b.st));
        M = hc.nlab;
        committed += M;
        max_list = (uint32_t)std::min<unsigned long long>(hc.max_ratio_den, 0xFFFFFFFFu);
        float ms1 = 0;
        CHL_CUDA(cudaEventElapsedTime(&ms1, ev_a, ev_b));
        commit_ms += ms1;
        ++supersteps;
        r0 = r1;
        unsigned long long tstat[2] = {0, 0};
        if (opts.verbose >= 2) {
            CHL_CUDA(cudaMemsetAsync(&b.ctl->max_ratio_num, 0, 16, b.st));
            tree_stats<<<sms, 256, 0, b.st>>>(b.tsize, r1 - r_begin, &b.ctl->max_ratio_num);
            CHL_CUDA(cudaMemcpyAsync(tstat, &b.ctl->max_ratio_num, 16, cudaMemcpyDeviceToHost, b.st));
            CHL_CUDA(cudaStreamSynchronize(b.st));
        }
        if (opts.verbose >= 2) {
            const double tot = (double)std::max<unsigned long long>(1, hc.cyc[7]);
            fprintf(stderr, "  warp cycles: scan %.1f%% flags %.1f%% prune %.1f%% emit %.1f%% relax %.1f%% "
                            "stage %.1f%% reset %.1f%% (sum of warp residencies %.3g cycles)\n",
                    100 * hc.cyc[0] / tot, 100 * hc.cyc[1] / tot, 100 * hc.cyc[2] / tot, 100 * hc.cyc[3] / tot,
                    100 * hc.cyc[4] / tot, 100 * hc.cyc[5] / tot, 100 * hc.cyc[6] / tot, tot);
            if (kPhaseTiming) {
                // warp slots busy: summed residencies over (slots x superstep time)
                int khz = 0;
                cudaDeviceGetAttribute(&khz, cudaDevAttrClockRate, 0);
                const double avail = (double)step_slots * step_tree_ms * 1e-3 * khz * 1e3;
                fprintf(stderr, "  warp slots busy %.1f%% (at the maximum SM clock)\n", 100 * tot / std::max(avail, 1.0));
            }
            fprintf(stderr, "  prune item selection %.1f%% of warp cycles, %llu passes (%.2f per visit)\n",
                    100 * hc.cyc[8] / tot, hc.cyc[9],
                    (double)hc.cyc[9] / std::max<unsigned long long>(1, hc.visits));
            fprintf(stderr, "  frontier entries scanned %llu rounds %llu settles %llu (per visit: scanned %.2f)\n",
                    hc.cnt[0], hc.cnt[1], hc.cnt[2], (double)hc.cnt[0] / std::max<unsigned long long>(1, hc.visits));
            fprintf(stderr, "  far pile entries read by refills: %llu (%.1f%% of the frontier entries scanned)\n",
                    hc.cnt[3], 100.0 * hc.cnt[3] / std::max<unsigned long long>(1, hc.cnt[0]));
        }
        if (opts.verbose >= 2)
            fprintf(stderr, "  tree size max %llu mean %.1f\n", tstat[0],
                    (double)tstat[1] / std::max<uint32_t>(1, r1 - r_begin));
        if (opts.verbose >= 2)
            fprintf(stderr,
                    "superstep %u: roots [%u,%u) %s tree_ms %.2f commit_ms %.2f labels %llu visits %llu reads %llu "
                    "arcs %llu committed %llu max_list %u label_cap %llu reruns %u\n",
                    supersteps, r_begin, r1, plant_now ? "plant" : "gll",
                    step_tree_ms, ms1, (unsigned long long)M, (unsigned long long)hc.visits,
                    (unsigned long long)hc.label_reads, (unsigned long long)hc.arcs, (unsigned long long)committed,
                    max_list, (unsigned long long)b.new_cap, step_reruns);
    }
    CHL_CUDA(cudaEventRecord(ev1, b.st));
    CHL_CUDA(cudaStreamSynchronize(b.st));
    float total_ms = 0, up_ms = 0;
    CHL_CUDA(cudaEventElapsedTime(&total_ms, ev_up, ev1));
    CHL_CUDA(cudaEventElapsedTime(&up_ms, ev0, ev_up));

    chl_labels *L = new (std::nothrow) chl_labels();
    if (!L) return CHL_ERR_OOM;
    L->n = n;
    L->sym = b.sides == 1;
    L->d_off = b.off_a;
    L->d_ent = (LabelEnt *)b.ent_a;
    L->total = committed;
    b.off_a = nullptr;
    b.ent_a = nullptr;
    chl_build_stats &S = L->stats;
    S.build_ms = total_ms;
    S.h2d_ms = up_ms;
    S.kernel_launches = kernels;
    S.tree_ms = tree_ms;
    S.sort_ms = sort_ms;
    S.commit_ms = commit_ms;
    S.labels = committed * (L->sym ? 2 : 1);
    S.visits = visits;
    S.label_reads = reads;
    S.arcs = arcs;
    S.supersteps = supersteps;
    S.plant_roots = plant_roots;
    S.tree_launches = launches;
    S.avg_label = n ? (double)S.labels / n / 2.0 : 0.0;
    (void)t_wall0;
    *out = L;
    if (opts.verbose) {
        // the reference's summary line (shared_memory/akiba.hpp:214)
        printf("Average label size after gll is %g, labeling time = %g, sorting time = %g, "
               "cleaning time = %g, total time = %g\n",
               S.avg_label, tree_ms / 1e3, sort_ms / 1e3, commit_ms / 1e3, total_ms / 1e3);
        printf("%g %g\n", S.avg_label, total_ms / 1e3);
    }
    return CHL_OK;
}

}  // namespace chl

extern "C" void chl_build_opts_default(chl_build_opts *o) {
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->mode = CHL_MODE_HYBRID;
    o->sf = 0.0;
    o->ps = 0.0;
    o->autotune = 1;
    o->use_graphs = 1;
    o->verbose = 0;
}

extern "C" int chl_build(const chl_graph *g, const uint32_t *order, uint32_t n,
                         const chl_build_opts *opts, chl_labels **out) {
    try {
        return chl::build_labels(g, order, n, opts, out);
    } catch (...) {
        chl::set_error("host allocation failed during build");
        return CHL_ERR_OOM;
    }
}

extern "C" int chl_graph_to_device(chl_graph *g) {
    if (!g) return CHL_ERR_INVALID;
    if (g->dev) return CHL_OK;
    chl::DevGraph *d = new (std::nothrow) chl::DevGraph();
    if (!d) return CHL_ERR_OOM;
    int rc = chl::upload_graph(g, *d, 0);
    if (rc == CHL_OK) {
        cudaError_t e = cudaDeviceSynchronize();
        if (e != cudaSuccess) rc = chl::cuda_status(e, "graph upload", __FILE__, __LINE__);
    }
    if (rc != CHL_OK) {
        d->release();
        delete d;
        return rc;
    }
    g->dev = d;
    return CHL_OK;
}

extern "C" int chl_graph_release_device(chl_graph *g) {
    if (!g) return CHL_ERR_INVALID;
    chl::graph_release_device(g);
    chl::tmp_trim();
    return CHL_OK;
}

extern "C" int chl_build_get_stats(const chl_labels *l, chl_build_stats *s) {
    if (!l || !s) return CHL_ERR_INVALID;
    *s = l->stats;
    return CHL_OK;
}
