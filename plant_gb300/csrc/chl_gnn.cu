// Learned vertex ranking: a small message-passing network that proposes the
// CHL order (no reference counterpart; the reference takes its order from
// outside tools, README.md:24).
//
// Network (hidden width H = 64, L = 3 message-passing layers):
//   x_v   = standardised [log1p deg(v), log1p sum_{u in N(v)} deg(u), cc(v)]
//   h0    = relu(x W0 + b0)                          (fp32 math, K = 3)
//   m_l   = mean_{u in N(v)} h_{l-1}(u)              (0 without neighbours)
//   h_l   = relu([h_{l-1}, m_l] W_l + b_l)           (BF16 tensor-core GEMM, K = 128)
//   s_v   = h_L . w_out + b_out                      (fp32)
// h_l and m_l are stored in BF16; GEMM operands are BF16 with FP32
// accumulation (mma.sync m16n8k16); master weights and Adam state are FP32.
// Loss: mean squared error to a per-graph target (standardised log1p hub
// frequency).  deg(v) = Graph::get_degree (out + in arcs); N(v) = out-arcs;
// cc(v) = fraction of 16 seeded neighbour pairs (a, b) with b among the
// first 256 out-arcs of a.
//
// The GEMMs are [n x 128] x [128 x 64]: far below the tensor-core ridge,
// bound by reading the activations (HBM), like every other kernel here.
#include "chl_dev.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

namespace chl {
namespace {

constexpr int H = 64;          // hidden width
constexpr int K2 = 2 * H;      // concatenated [h, m]
constexpr int NF = 3;          // input features
constexpr int kClusterSamples = 16;
constexpr int kClusterScan = 256;

__device__ __forceinline__ uint64_t gmix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// raw features: log1p deg, log1p 2-hop degree sum, sampled clustering.
// A warp takes vpw vertices (32 once there are enough to fill the GPU so,
// down to 2: a warp's vertices are walked one pair after the other).  Degree sums: a lane each while lists are short,
// the whole warp where a list has more than kFeatLight arcs (whole numbers:
// the sum is the same in any order).  Clustering: 16 lanes, one sample each,
// on two vertices at a time.  The logarithms are double and the GPU's slow
// unit, so all 32 lanes take them together.  One thread per vertex took
// 2.61 ms on a 2^15-vertex RMAT graph (its hubs; 0.85 with them split off, the
// others' neighbours being hubs), 16 lanes per vertex for everything 0.55 ms
// on a 512-square grid (two lanes' logarithms at a time).
constexpr uint32_t kFeatLight = 32;
constexpr int kFeatLoads = 8;
static_assert(kClusterSamples == 16, "two vertices' samples fill a warp");

// whether c is among the first kClusterScan out-arcs of a
__device__ __forceinline__ bool has_arc(const uint64_t *off, const uint32_t *head, uint32_t a, uint32_t c) {
    const uint64_t ab = off[a], ae = min(off[a + 1], ab + kClusterScan);
    for (uint64_t q = ab; q < ae; q += 2 * kFeatLoads) {
        bool hit = false;
#pragma unroll
        for (int t = 0; t < 2 * kFeatLoads; ++t) hit |= q + t < ae && head[q + t] == c;
        if (hit) return true;
    }
    return false;
}

// clustering sample k of v, whose d >= 2 arcs start at b
__device__ __forceinline__ bool closed_pair(const uint64_t *off, const uint32_t *head, uint64_t seed, uint32_t v, int k,
                                            uint64_t b, uint32_t d) {
    const uint64_t h = gmix(seed ^ ((uint64_t)v * 0x100000001B3ull + (uint64_t)k));
    const uint64_t i = h % d;
    uint64_t j = (h >> 32) % (d - 1);
    if (j >= i) ++j;
    return has_arc(off, head, head[b + i], head[b + j]);
}

__global__ void feat_raw(uint32_t n, const uint64_t *off_out, const uint32_t *head_out, const uint64_t *off_in,
                         uint64_t seed, uint32_t vpw, float *x) {
    const uint32_t lane = lane_id();
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint64_t v0 = (uint64_t)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * vpw; v0 < n;
         v0 += (uint64_t)warps * vpw) {
        const uint32_t v = (uint32_t)v0 + lane;
        uint64_t b = 0, sum = 0;
        uint32_t d = 0, hits = 0, deg_in = 0;
        const bool mine = lane < vpw && v < n;
        if (mine) {
            b = off_out[v];
            d = (uint32_t)(off_out[v + 1] - b);
            deg_in = (uint32_t)(off_in[v + 1] - off_in[v]);
        }
        auto degree = [&](uint32_t u) { return (off_out[u + 1] - off_out[u]) + (off_in[u + 1] - off_in[u]); };
        if (d <= kFeatLight) {
            for (uint32_t a = 0; a < d; a += kFeatLoads) {
                uint32_t u[kFeatLoads];
#pragma unroll
                for (int q = 0; q < kFeatLoads; ++q) u[q] = a + q < d ? head_out[b + a + q] : 0u;
#pragma unroll
                for (int q = 0; q < kFeatLoads; ++q)
                    if (a + q < d) sum += degree(u[q]);
            }
        }
        __syncwarp();
        for (uint32_t m = __ballot_sync(kFull, d > kFeatLight); m; m &= m - 1) {
            const int o = __ffs(m) - 1;
            const uint64_t ob = __shfl_sync(kFull, b, o);
            const uint32_t od = __shfl_sync(kFull, d, o);
            uint64_t s = 0;
            for (uint32_t a = lane; a < od; a += 32 * kFeatLoads) {
                uint32_t u[kFeatLoads];
#pragma unroll
                for (int q = 0; q < kFeatLoads; ++q) u[q] = a + 32 * q < od ? head_out[ob + a + 32 * q] : 0u;
#pragma unroll
                for (int q = 0; q < kFeatLoads; ++q)
                    if (a + 32 * q < od) s += degree(u[q]);
            }
#pragma unroll
            for (int w = 16; w > 0; w >>= 1) s += __shfl_xor_sync(kFull, s, w);
            if (lane == (uint32_t)o) sum = s;
        }
        for (uint32_t j = 0; j < vpw; j += 2) {
            const uint32_t o = j + (lane >> 4);
            const uint64_t ob = __shfl_sync(kFull, b, o);
            const uint32_t od = __shfl_sync(kFull, d, o);
            const bool hit = od >= 2 && closed_pair(off_out, head_out, seed, (uint32_t)v0 + o, (int)(lane & 15), ob, od);
            const uint32_t c = __ballot_sync(kFull, hit);
            if ((lane & ~1u) == j) hits = __popc(lane & 1u ? c >> 16 : c & 0xFFFFu);
        }
        if (mine) {
            x[(size_t)v * NF + 0] = (float)log1p((double)d + (double)deg_in);
            x[(size_t)v * NF + 1] = (float)log1p((double)sum);
            x[(size_t)v * NF + 2] = (float)hits / (float)kClusterSamples;
        }
    }
}

// vertices per warp of feat_raw's launch
uint32_t feat_vpw(uint32_t n, int sms) {
    uint32_t v = 2;
    while (v < 32 && (uint64_t)v * sms * 4 * 8 < n) v *= 2;
    return v;
}

// Standardised feature columns, (x - mean) / population sd in double: column
// sums, then squared deviations, each as one partial per block summed in
// block order (the same result for the same graph), then the columns in
// place.  On the host the same three passes and the two copies were 1.6 ms of
// a 2.6 ms prediction for 2^18 vertices.
constexpr int kStatThreads = 256;
constexpr int kStatBlocks = 128;   // at most

__device__ void col_totals(const double *part, int blocks, double *tot) {
    // every thread calls; tot (shared) holds NF totals afterwards
    // (a fixed tree, so every block and every run finds the same totals)
    __shared__ double ws[kStatBlocks / 32][NF];
    __syncthreads();
    if (threadIdx.x < kStatBlocks) {
#pragma unroll
        for (int k = 0; k < NF; ++k) {
            double t = (int)threadIdx.x < blocks ? part[threadIdx.x * NF + k] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
            if (lane_id() == 0) ws[threadIdx.x >> 5][k] = t;
        }
    }
    __syncthreads();
    if (threadIdx.x < NF) {
        double t = 0.0;
        for (int w = 0; w < kStatBlocks / 32; ++w) t += ws[w][threadIdx.x];
        tot[threadIdx.x] = t;
    }
    __syncthreads();
}

// part[block][k] = sum over the block's vertices of x (sums == null), or of
// (x - mean)^2 with the means of the column sums `sums`
__global__ void __launch_bounds__(kStatThreads) feat_stats(uint32_t n, const float *x, const double *sums,
                                                           double *part) {
    __shared__ double tot[NF];
    __shared__ double wsum[kStatThreads / 32][NF];
    double mean[NF] = {0.0, 0.0, 0.0}, acc[NF] = {0.0, 0.0, 0.0};
    if (sums) {
        col_totals(sums, gridDim.x, tot);
        for (int k = 0; k < NF; ++k) mean[k] = tot[k] / n;
    }
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
#pragma unroll
        for (int k = 0; k < NF; ++k) {
            const double d = (double)x[(size_t)v * NF + k] - mean[k];
            acc[k] += sums ? d * d : d;
        }
    }
#pragma unroll
    for (int k = 0; k < NF; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(kFull, acc[k], o);
        if (lane_id() == 0) wsum[threadIdx.x >> 5][k] = acc[k];
    }
    __syncthreads();
    if (threadIdx.x < NF) {
        double t = 0.0;
        for (int w = 0; w < kStatThreads / 32; ++w) t += wsum[w][threadIdx.x];
        part[blockIdx.x * NF + threadIdx.x] = t;
    }
}

__global__ void __launch_bounds__(kStatThreads) feat_scale(uint32_t n, const double *sums, const double *squares,
                                                           int blocks, float *x) {
    __shared__ double tot[NF], tot2[NF];
    col_totals(sums, blocks, tot);
    col_totals(squares, blocks, tot2);
    double mean[NF], inv[NF];
    for (int k = 0; k < NF; ++k) {
        mean[k] = tot[k] / n;
        const double sd = n > 1 ? sqrt(tot2[k] / n) : 0.0;
        inv[k] = sd > 1e-12 ? 1.0 / sd : 0.0;
    }
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        for (int k = 0; k < NF; ++k)
            x[(size_t)v * NF + k] = (float)(((double)x[(size_t)v * NF + k] - mean[k]) * inv[k]);
}

// h0 = relu(x W0 + b0), one thread per (vertex, channel)
__global__ void layer0_fwd(uint32_t n, const float *x, const float *W0, const float *b0, __nv_bfloat16 *h0) {
    const size_t tot = (size_t)n * H;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < tot; i += (size_t)gridDim.x * blockDim.x) {
        const size_t v = i / H;
        const int c = (int)(i % H);
        float z = b0[c];
#pragma unroll
        for (int k = 0; k < NF; ++k) z = fmaf(x[v * NF + k], W0[k * H + c], z);
        h0[i] = __float2bfloat16_rn(fmaxf(z, 0.f));
    }
}

// Vertices whose list is longer than kHubArcs are summed by a block each
// (hub_sum below), the others by a warp each.
constexpr uint32_t kHubArcs = 256;

// the hubs of one direction: hubs[0] = their number, hubs[1..] the vertices
__global__ void find_hubs(uint32_t n, const uint64_t *off, uint32_t *hubs) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        if (off[v + 1] - off[v] > kHubArcs) hubs[1 + atomicAdd(&hubs[0], 1u)] = v;
}

// Ordered sum of a hub's rows by one block: kHubRows rows at a time are
// gathered into shared memory by all threads (the next ones while these are
// added), and one thread per channel adds them in arc order -- the same
// additions, in the same order, as one warp walking the list, whose time is
// the latency of its row loads (a 2^15-vertex RMAT graph's hubs: 160 us a
// layer forward with 32 rows in flight, 680 us backward with 16).
// row(u, c): channel c of vertex u's row as a float2 pair of channels c, c + 1;
// scale(u): the factor of its row; init(c), done(c, sum).
constexpr int kHubThreads = 512;
constexpr int kHubRows = 128;
constexpr int kHubPairs = kHubRows * (H / 2) / kHubThreads;   // channel pairs per thread and step

template <bool SCALED, typename Row, typename Scale>
__device__ __forceinline__ float hub_sum(uint64_t b, uint64_t e, const uint32_t *head, float2 (*buf)[H / 2], float *fac,
                                         uint32_t *idx, float sum, Row row, Scale scale) {
    const uint32_t tid = threadIdx.x;
    float2 t[kHubPairs];
    float f = 0.f;
    // heads of a step are read one step ahead of its rows
    uint32_t hn = tid < kHubRows && b + tid < e ? head[b + tid] : 0u;
    auto fetch = [&](uint64_t a) {
        // idx holds the heads of rows [a, a + kHubRows)
#pragma unroll
        for (int q = 0; q < kHubPairs; ++q) {
            const uint32_t r = (q * kHubThreads + tid) / (H / 2), c = (q * kHubThreads + tid) % (H / 2);
            t[q] = a + r < e ? row(idx[r], 2 * c) : make_float2(0.f, 0.f);
        }
        if (SCALED && tid < kHubRows) f = a + tid < e ? scale(idx[tid]) : 0.f;
    };
    if (tid < kHubRows) idx[tid] = hn;
    hn = tid < kHubRows && b + kHubRows + tid < e ? head[b + kHubRows + tid] : 0u;
    __syncthreads();
    fetch(b);
    for (uint64_t a = b; a < e; a += kHubRows) {
        __syncthreads();   // the rows before are added, idx is read
#pragma unroll
        for (int q = 0; q < kHubPairs; ++q) (&buf[0][0])[q * kHubThreads + tid] = t[q];
        if (SCALED && tid < kHubRows) fac[tid] = f;
        if (tid < kHubRows) idx[tid] = hn;
        hn = tid < kHubRows && a + 2 * kHubRows + tid < e ? head[a + 2 * kHubRows + tid] : 0u;
        __syncthreads();
        if (a + kHubRows < e) fetch(a + kHubRows);
        if (tid < H) {
            const uint32_t cnt = e - a < kHubRows ? (uint32_t)(e - a) : (uint32_t)kHubRows;
            const float *col = (const float *)&buf[0][0] + tid;
#pragma unroll 16
            for (uint32_t r = 0; r < cnt; ++r) {
                if (SCALED) sum = __fmaf_rn(col[(size_t)r * H], fac[r], sum);
                else sum = __fadd_rn(sum, col[(size_t)r * H]);
            }
        }
    }
    __syncthreads();
    return sum;
}

// m(v) = mean over out-neighbours of h(u) of the hubs
__global__ void __launch_bounds__(kHubThreads) hub_mean(const uint32_t *hubs, const uint64_t *off, const uint32_t *head,
                                                        const __nv_bfloat16 *h, __nv_bfloat16 *m) {
    __shared__ float2 buf[kHubRows][H / 2];
    __shared__ uint32_t idx[kHubRows];
    const uint32_t cnt = hubs[0];
    for (uint32_t i = blockIdx.x; i < cnt; i += gridDim.x) {
        const uint32_t v = hubs[1 + i];
        const uint64_t b = off[v], e = off[v + 1];
        const float s = hub_sum<false>(
            b, e, head, buf, nullptr, idx, 0.f,
            [&](uint32_t u, uint32_t c) {
                const __nv_bfloat162 t = *(const __nv_bfloat162 *)(h + (size_t)u * H + c);
                return make_float2(__bfloat162float(t.x), __bfloat162float(t.y));
            },
            [](uint32_t) { return 1.f; });
        if (threadIdx.x < H) m[(size_t)v * H + threadIdx.x] = __float2bfloat16_rn(s * (1.f / (float)(e - b)));
    }
}

// m(v) = mean over out-neighbours of h(u), hubs left out; 8 lanes per vertex,
// 8 channels (16 bytes) each, so a warp has four vertices' rows on their way
// and up to kRows of each.  Rows are added in arc order.  (A warp per vertex
// with 4 bytes per lane: 89 us a layer on a 512-square grid, bound by the
// chain offsets, heads, rows of one vertex after the other.)
constexpr int kRows = 8;

__global__ void aggregate_mean(uint32_t n, const uint64_t *off, const uint32_t *head, const __nv_bfloat16 *h,
                               __nv_bfloat16 *m) {
    const uint32_t sub = threadIdx.x & 7u, gm = 0xFFu << (threadIdx.x & 24u);
    const uint32_t groups = gridDim.x * (blockDim.x >> 3);
    for (uint32_t v = blockIdx.x * (blockDim.x >> 3) + (threadIdx.x >> 3); v < n; v += groups) {
        const uint64_t b = off[v], e = off[v + 1];
        if (e - b > kHubArcs) continue;
        float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        uint32_t next = b + sub < e ? head[b + sub] : 0u;
        for (uint64_t a = b; a < e; a += kRows) {
            const uint32_t cnt = e - a < kRows ? (uint32_t)(e - a) : (uint32_t)kRows;
            const uint32_t hd = next;
            next = a + kRows + sub < e ? head[a + kRows + sub] : 0u;
            uint4 t[kRows];
#pragma unroll
            for (uint32_t q = 0; q < kRows; ++q) {
                const uint32_t u = __shfl_sync(gm, hd, q, 8);
                if (q < cnt) t[q] = *(const uint4 *)(h + (size_t)u * H + 8 * sub);
            }
#pragma unroll
            for (uint32_t q = 0; q < kRows; ++q) {
                if (q < cnt) {
                    const uint32_t w[4] = {t[q].x, t[q].y, t[q].z, t[q].w};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {   // a BF16 is the high half of its FP32
                        s[2 * c] += __uint_as_float(w[c] << 16);
                        s[2 * c + 1] += __uint_as_float(w[c] & 0xFFFF0000u);
                    }
                }
            }
        }
        const float inv = e > b ? 1.f / (float)(e - b) : 0.f;
        uint32_t o[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const __nv_bfloat162 t = __floats2bfloat162_rn(s[2 * c] * inv, s[2 * c + 1] * inv);
            o[c] = *(const uint32_t *)&t;
        }
        *(uint4 *)(m + (size_t)v * H + 8 * sub) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// mma.sync m16n8k16, BF16 inputs, FP32 accumulators
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Y[n x 64] = A[n x K] B[K x 64] (+ bias, relu) where A's columns are the
// concatenation of two [n x 64] BF16 arrays A0 | A1 (K = 128) or one (K = 64).
// Each warp computes 16 rows at a time.  B is staged in shared memory as
// BF16, transposed (column-major, rows padded to K + 8 elements: 16-byte
// aligned rows whose eight-row groups fall in distinct banks) and read with
// ldmatrix; A fragments are read straight from global memory as BF16 pairs.
// mode 0: Y = relu(AB + bias) -> BF16 out_bf;  mode 1: Y = AB -> FP32 out_f.
template <int K>
__global__ void __launch_bounds__(128) gemm_rows(uint32_t n, const __nv_bfloat16 *A0, const __nv_bfloat16 *A1,
                                                 const float *B, const float *bias, int mode,
                                                 __nv_bfloat16 *out_bf, float *out_f, int ldo) {
    constexpr int KP = K + 8;
    __shared__ __align__(16) __nv_bfloat16 sBt[H * KP];
    for (int i = threadIdx.x; i < K * H; i += blockDim.x) sBt[(i % H) * KP + i / H] = __float2bfloat16_rn(B[i]);
    __syncthreads();
    const uint32_t lane = lane_id(), gid = lane >> 2, tig = lane & 3;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t tiles = (n + 15) / 16;
    for (uint32_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < tiles; t += warps) {
        const uint32_t r0 = t * 16 + gid, r1 = r0 + 8;
        float acc[8][4];
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[j][q] = 0.f;
        // two BF16 at (row, col), col even: one 4-byte load (0 past the end)
        auto ld2 = [&](const __nv_bfloat16 *src, uint32_t row, int col) -> uint32_t {
            return row < n ? __ldg((const unsigned int *)(src + (size_t)row * H + col)) : 0u;
        };
        uint32_t af[K / 16][4];
#pragma unroll
        for (int ks = 0; ks < K / 16; ++ks) {
            const __nv_bfloat16 *src = (ks * 16 < H) ? A0 : A1;
            const int kc = (ks * 16) % H + 2 * (int)tig;
            af[ks][0] = ld2(src, r0, kc);
            af[ks][1] = ld2(src, r1, kc);
            af[ks][2] = ld2(src, r0, kc + 8);
            af[ks][3] = ld2(src, r1, kc + 8);
        }
#pragma unroll
        for (int ks = 0; ks < K / 16; ++ks) {
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                // one ldmatrix.x4: the B fragments of column tiles j and j + 1
                // (8x8 matrices: rows = columns of B, 8 consecutive k each;
                // lane l addresses row l % 8 of matrix l / 8)
                const uint32_t mtx = lane >> 3;
                const __nv_bfloat16 *rowp =
                    sBt + ((j + (mtx >> 1)) * 8 + (lane & 7)) * KP + ks * 16 + (mtx & 1) * 8;
                uint32_t b[4];
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                             : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                             : "r"((uint32_t)__cvta_generic_to_shared(rowp)));
                const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
                mma_bf16(acc[j], af[ks], b0);
                mma_bf16(acc[j + 1], af[ks], b1);
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = j * 8 + 2 * tig;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const uint32_t row = half ? r1 : r0;
                if (row >= n) continue;
                float y0 = acc[j][2 * half], y1 = acc[j][2 * half + 1];
                if (mode == 0) {
                    y0 = fmaxf(y0 + bias[c], 0.f);
                    y1 = fmaxf(y1 + bias[c + 1], 0.f);
                    __nv_bfloat162 o;
                    o.x = __float2bfloat16_rn(y0);
                    o.y = __float2bfloat16_rn(y1);
                    *(__nv_bfloat162 *)(out_bf + (size_t)row * H + c) = o;
                } else {
                    *(float2 *)(out_f + (size_t)row * ldo + c) = make_float2(y0, y1);
                }
            }
        }
    }
}

// blocks of gemm_rows<K> that fill the GPU (resident blocks per SM x SMs)
template <int K>
int gemm_grid(int sms) {
    static int per_sm = 0;
    if (!per_sm) {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, gemm_rows<K>, 128, 0) != cudaSuccess || b < 1) {
            (void)cudaGetLastError();
            b = 4;
        }
        per_sm = b;
    }
    return per_sm * sms;
}

// s = h w_out + b_out; loss terms; ds = 2 (s - y) / n
__global__ void head_fwd_bwd(uint32_t n, const __nv_bfloat16 *h, const float *wout, const float *bout,
                             const float *y, float *s, float *ds, double *loss_acc) {
    const uint32_t lane = lane_id();
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    double lsum = 0.0;
    for (uint32_t v = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); v < n; v += warps) {
        const __nv_bfloat162 t = *(const __nv_bfloat162 *)(h + (size_t)v * H + 2 * lane);
        float p = __bfloat162float(t.x) * wout[2 * lane] + __bfloat162float(t.y) * wout[2 * lane + 1];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(kFull, p, o);
        const float sv = p + bout[0];
        if (lane == 0) {
            s[v] = sv;
            if (y) {
                const float r = sv - y[v];
                ds[v] = 2.f * r / (float)n;
                lsum += (double)r * r;
            }
        }
    }
    if (loss_acc && lane == 0 && lsum != 0.0) atomicAdd(loss_acc, lsum / (double)n);
}

// dW[k][c] += sum_v A[v][k] dz[v][c] (A = [h | m], BF16; dz in BF16) on the
// tensor cores: warp w of a block owns rows k in [16w, 16w+16) of dW and
// walks the block's slice of vertices 16 at a time (the reduction axis);
// partial tiles are added to dW atomically.  db[c] += sum_v dz[v][c].
// 32 vertices' rows are staged in shared memory with 16-byte loads, the next
// 32 on their way in registers, and both operands are read transposed with
// ldmatrix (rows padded to fall in distinct banks).  Bound by latency at
// training sizes: two-byte loads straight from global memory took 41 us a
// layer on 2^15 vertices.
constexpr int kGwRows = 32;
constexpr int kGwThreads = 256;   // 8 warps: 128 rows of dW
constexpr int kGwA = K2 + 8, kGwD = H + 8;   // padded rows

__device__ __forceinline__ void ldmatrix_t4(uint32_t (&r)[4], const __nv_bfloat16 *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

__global__ void __launch_bounds__(kGwThreads) grad_w_mma(uint32_t n, const __nv_bfloat16 *A0, const __nv_bfloat16 *A1,
                                                         const __nv_bfloat16 *dzb, const float *dz, float *dW,
                                                         float *db) {
    __shared__ __align__(16) __nv_bfloat16 sA[kGwRows * kGwA];
    __shared__ __align__(16) __nv_bfloat16 sD[kGwRows * kGwD];
    __shared__ float sb[kGwThreads];
    const uint32_t tid = threadIdx.x, lane = lane_id(), gid = lane >> 2, tig = lane & 3;
    const uint32_t warp = tid >> 5;
    const uint32_t per = ((n + gridDim.x - 1) / gridDim.x + 15) & ~15u;
    const uint32_t v0 = min(n, blockIdx.x * per), v1 = min(n, v0 + per);
    const int krow = (int)warp * 16;
    float acc[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[j][q] = 0.f;
    // a row is 8 pieces of 16 bytes in each of A0, A1 and dz: thread t holds
    // piece t % 8 of row t / 8 of all three (32 rows)
    const uint32_t row = tid >> 3, piece = (tid & 7) * 8;
    uint4 p0, p1, p2;
    auto fetch = [&](uint32_t vb) {
        p0 = p1 = p2 = make_uint4(0, 0, 0, 0);
        if (vb + row < v1) {
            const size_t at = (size_t)(vb + row) * H + piece;
            p0 = *(const uint4 *)(A0 + at);
            p1 = *(const uint4 *)(A1 + at);
            p2 = *(const uint4 *)(dzb + at);
        }
    };
    fetch(v0);
    for (uint32_t vb = v0; vb < v1; vb += kGwRows) {
        *(uint4 *)(sA + row * kGwA + piece) = p0;
        *(uint4 *)(sA + row * kGwA + H + piece) = p1;
        *(uint4 *)(sD + row * kGwD + piece) = p2;
        __syncthreads();
        if (vb + kGwRows < v1) fetch(vb + kGwRows);
        const uint32_t mtx = lane >> 3, mr = lane & 7;
#pragma unroll
        for (int s = 0; s < kGwRows; s += 16) {
            // A fragment: row = channel of A, column = vertex; matrices
            // (channels 0-7 | 8-15) x (vertices 0-7 | 8-15)
            uint32_t a[4];
            ldmatrix_t4(a, sA + (s + (mtx >> 1) * 8 + mr) * kGwA + krow + (mtx & 1) * 8);
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                // B fragments of column tiles j and j + 1: vertices 0-7 | 8-15
                uint32_t b[4];
                ldmatrix_t4(b, sD + (s + (mtx & 1) * 8 + mr) * kGwD + (j + (mtx >> 1)) * 8);
                const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
                mma_bf16(acc[j], a, b0);
                mma_bf16(acc[j + 1], a, b1);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = j * 8 + 2 * tig;
        atomicAdd(&dW[(size_t)(krow + gid) * H + c], acc[j][0]);
        atomicAdd(&dW[(size_t)(krow + gid) * H + c + 1], acc[j][1]);
        atomicAdd(&dW[(size_t)(krow + gid + 8) * H + c], acc[j][2]);
        atomicAdd(&dW[(size_t)(krow + gid + 8) * H + c + 1], acc[j][3]);
    }
    // bias gradient (fp32) from the same slice, four rows at a time
    float s = 0.f;
    for (uint32_t v = v0 + tid / H; v < v1; v += kGwThreads / H) s += dz[(size_t)v * H + tid % H];
    sb[tid] = s;
    __syncthreads();
    if (tid < H) atomicAdd(&db[tid], (sb[tid] + sb[tid + H]) + (sb[tid + 2 * H] + sb[tid + 3 * H]));
}

// Wt0[c][k] = W[k][c], Wt1[c][k] = W[H + k][c]  (W is [2H x H] row-major)
__global__ void transpose_w(const float *W, float *Wt0, float *Wt1) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < H * H; i += gridDim.x * blockDim.x) {
        const int c = i / H, k = i % H;
        Wt0[i] = W[(size_t)k * H + c];
        Wt1[i] = W[(size_t)(H + k) * H + c];
    }
}

// dz = dh * [h > 0] (relu derivative from the stored activation), written by
// the kernel that forms dh in FP32 and, for the GEMMs, in BF16
__device__ __forceinline__ void store_dz(size_t at, float d0, float d1, const __nv_bfloat16 *h, float *dz,
                                         __nv_bfloat16 *dzb) {
    const __nv_bfloat162 t = *(const __nv_bfloat162 *)(h + at);
    const float z0 = __bfloat162float(t.x) > 0.f ? d0 : 0.f, z1 = __bfloat162float(t.y) > 0.f ? d1 : 0.f;
    *(float2 *)(dz + at) = make_float2(z0, z1);
    __nv_bfloat162 o;
    o.x = __float2bfloat16_rn(z0);
    o.y = __float2bfloat16_rn(z1);
    *(__nv_bfloat162 *)(dzb + at) = o;
}

// dh_L = ds * w_out -> dz_L; dw_out += sum ds h_L; db_out += sum ds
__global__ void head_bwd(uint32_t n, const float *ds, const __nv_bfloat16 *h, const float *wout, float *dz,
                         __nv_bfloat16 *dzb, float *dwout, float *dbout) {
    __shared__ float acc[H + 1];
    for (int i = threadIdx.x; i <= H; i += blockDim.x) acc[i] = 0.f;
    __syncthreads();
    float a0 = 0.f, a1 = 0.f, ad = 0.f;
    const uint32_t lane = lane_id();
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const float w0 = wout[2 * lane], w1 = wout[2 * lane + 1];
    for (uint32_t v = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); v < n; v += warps) {
        const float d = ds[v];
        const size_t at = (size_t)v * H + 2 * lane;
        const __nv_bfloat162 t = *(const __nv_bfloat162 *)(h + at);
        a0 += d * __bfloat162float(t.x);
        a1 += d * __bfloat162float(t.y);
        if (lane == 0) ad += d;
        store_dz(at, d * w0, d * w1, h, dz, dzb);
    }
    atomicAdd(&acc[2 * lane], a0);
    atomicAdd(&acc[2 * lane + 1], a1);
    if (lane == 0) atomicAdd(&acc[H], ad);
    __syncthreads();
    for (int i = threadIdx.x; i < H; i += blockDim.x) atomicAdd(&dwout[i], acc[i]);
    if (threadIdx.x == 0) atomicAdd(dbout, acc[H]);
}

// 1 / out-degree (0 without out-arcs)
__global__ void inv_degree(uint32_t n, const uint64_t *off, float *inv) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const uint64_t d = off[v + 1] - off[v];
        inv[v] = d ? 1.f / (float)d : 0.f;
    }
}

// dh_prev(u) = dA[u, :64] + sum_{v: u in N(v)} dA[v, 64:] / deg(v), gathered
// over u's in-arcs (the reverse of the out-neighbour mean) in arc order, and
// dz_prev from it; hubs by hub_scatter.  16 lanes per vertex, 4 channels (16
// bytes) each, 8 rows in flight.
constexpr int kBwdRows = 8;

__global__ void __launch_bounds__(kHubThreads) hub_scatter(const uint32_t *hubs, const float *dA, const uint64_t *off_in,
                                                           const uint32_t *head_in, const float *inv_deg,
                                                           const __nv_bfloat16 *h, float *dz, __nv_bfloat16 *dzb) {
    __shared__ float2 buf[kHubRows][H / 2];
    __shared__ float fac[kHubRows];
    __shared__ uint32_t idx[kHubRows];
    const uint32_t cnt = hubs[0];
    for (uint32_t i = blockIdx.x; i < cnt; i += gridDim.x) {
        const uint32_t u = hubs[1 + i], c = threadIdx.x;
        const float own = c < H ? dA[(size_t)u * K2 + c] : 0.f;
        const float s = hub_sum<true>(
            off_in[u], off_in[u + 1], head_in, buf, fac, idx, own,
            [&](uint32_t v, uint32_t k) { return *(const float2 *)(dA + (size_t)v * K2 + H + k); },
            [&](uint32_t v) { return inv_deg[v]; });
        if (c < H) {
            const size_t at = (size_t)u * H + c;
            const float z = __bfloat162float(h[at]) > 0.f ? s : 0.f;
            dz[at] = z;
            dzb[at] = __float2bfloat16_rn(z);
        }
    }
}

__global__ void scatter_mean_bwd(uint32_t n, const float *dA, const uint64_t *off_in, const uint32_t *head_in,
                                 const float *inv_deg, const __nv_bfloat16 *h, float *dz, __nv_bfloat16 *dzb) {
    const uint32_t sub = threadIdx.x & 15u, gm = 0xFFFFu << (threadIdx.x & 16u);
    const uint32_t groups = gridDim.x * (blockDim.x >> 4);
    for (uint32_t u = blockIdx.x * (blockDim.x >> 4) + (threadIdx.x >> 4); u < n; u += groups) {
        const uint64_t b = off_in[u], e = off_in[u + 1];
        if (e - b > kHubArcs) continue;
        float4 s = *(const float4 *)(dA + (size_t)u * K2 + 4 * sub);
        // each lane of the group reads one of the next 16 heads and its factor
        uint32_t next = b + sub < e ? head_in[b + sub] : 0u;
        float inext = b + sub < e ? inv_deg[next] : 0.f;
        for (uint64_t a = b; a < e; a += 16) {
            const uint32_t cnt = e - a < 16 ? (uint32_t)(e - a) : 16u;
            const uint32_t hd = next;
            const float iv = inext;
            next = a + 16 + sub < e ? head_in[a + 16 + sub] : 0u;
            inext = a + 16 + sub < e ? inv_deg[next] : 0.f;
            for (uint32_t j = 0; j < cnt; j += kBwdRows) {
                float4 t[kBwdRows];
#pragma unroll
                for (uint32_t q = 0; q < kBwdRows; ++q) {
                    const uint32_t v = __shfl_sync(gm, hd, j + q, 16);
                    if (j + q < cnt) t[q] = *(const float4 *)(dA + (size_t)v * K2 + H + 4 * sub);
                }
#pragma unroll
                for (uint32_t q = 0; q < kBwdRows; ++q) {
                    const float w = __shfl_sync(gm, iv, j + q, 16);
                    if (j + q < cnt) {
                        s.x = __fmaf_rn(t[q].x, w, s.x);
                        s.y = __fmaf_rn(t[q].y, w, s.y);
                        s.z = __fmaf_rn(t[q].z, w, s.z);
                        s.w = __fmaf_rn(t[q].w, w, s.w);
                    }
                }
            }
        }
        const size_t at = (size_t)u * H + 4 * sub;
        store_dz(at, s.x, s.y, h, dz, dzb);
        store_dz(at + 2, s.z, s.w, h, dz, dzb);
    }
}

// part[block][k][c]: x^T dz0 (k < NF) and sum dz0 (k = NF) over the block's
// vertices, in double.  A block's warps walk its vertices (2 channels per
// lane) and are added up in order, as grad_w0_out adds up the blocks: the same
// graph gives the same bits.  One thread per (k, c) walking all vertices took
// 5.5 ms for 2^15 of them.
constexpr int kGw0Threads = 256;
constexpr int kGw0Rows = 64;         // vertices per block, at least
constexpr int kGw0 = (NF + 1) * H;   // sums
constexpr int kGw0Parts = 32;        // threads per sum of grad_w0_out, 32 sums a block

__global__ void __launch_bounds__(kGw0Threads) grad_w0(uint32_t n, const float *x, const float *dz, double *part) {
    __shared__ double sum[kGw0Threads / 32][kGw0];
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    double a[NF + 1][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
    for (uint32_t v = blockIdx.x * (blockDim.x >> 5) + warp; v < n; v += warps) {
        const float2 d = *(const float2 *)(dz + (size_t)v * H + 2 * lane);
#pragma unroll
        for (int k = 0; k <= NF; ++k) {
            const double f = k < NF ? (double)x[(size_t)v * NF + k] : 1.0;
            a[k][0] += f * d.x;
            a[k][1] += f * d.y;
        }
    }
#pragma unroll
    for (int k = 0; k <= NF; ++k) {
        sum[warp][k * H + 2 * lane] = a[k][0];
        sum[warp][k * H + 2 * lane + 1] = a[k][1];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kGw0; i += blockDim.x) {
        double t = 0.0;
        for (int w = 0; w < kGw0Threads / 32; ++w) t += sum[w][i];
        part[(size_t)blockIdx.x * kGw0 + i] = t;
    }
}

__global__ void __launch_bounds__(32 * kGw0Parts) grad_w0_out(const double *part, int blocks, float *dW0, float *db0) {
    __shared__ double sum[kGw0Parts][32];
    const int i = blockIdx.x * 32 + lane_id(), q = threadIdx.x >> 5;
    double t = 0.0;
    for (int j = q; j < blocks; j += kGw0Parts) t += part[(size_t)j * kGw0 + i];
    sum[q][lane_id()] = t;
    for (int w = kGw0Parts / 2; w > 0; w >>= 1) {
        __syncthreads();
        if (q < w) sum[q][lane_id()] += sum[q + w][lane_id()];
    }
    if (q) return;
    if (i < NF * H) dW0[i] += (float)sum[0][lane_id()];
    else db0[i - NF * H] += (float)sum[0][lane_id()];
}

__global__ void adam_step(size_t np, float *p, const float *g, float *m, float *vv, float lr, float b1, float b2,
                          float eps, float c1, float c2) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < np; i += (size_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        m[i] = b1 * m[i] + (1.f - b1) * gi;
        vv[i] = b2 * vv[i] + (1.f - b2) * gi * gi;
        p[i] -= lr * (m[i] / c1) / (sqrtf(vv[i] / c2) + eps);
    }
}

// parameter layout (fp32): W0[3*H] b0[H] | per layer: W[2H*H] b[H] | wout[H] bout[1]
constexpr size_t kP0 = (size_t)NF * H + H;
constexpr size_t kPL = (size_t)K2 * H + H;

struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
    ~DevBuf() { cudaFree(p); }
    int ensure(size_t b) {
        if (b <= bytes) return CHL_OK;
        cudaFree(p);
        p = nullptr;
        bytes = 0;
        cudaError_t e = long_malloc(&p, b ? b : 1);
        if (e != cudaSuccess) return cuda_status(e, "cudaMalloc", __FILE__, __LINE__);
        bytes = b;
        return CHL_OK;
    }
    template <typename T>
    T *as() const { return (T *)p; }
};

}  // namespace
}  // namespace chl

using namespace chl;

struct chl_gnn {
    uint32_t layers = 3;
    size_t np = 0;
    std::vector<float> host;       // parameter mirror
    DevBuf p, g, m, v;             // params, grads, Adam moments
    uint64_t step = 0;
    // per-graph scratch (grown on demand)
    DevBuf x, hb, mb, dz, dA, s, ds, y, loss, wt, inv, acc;
};

namespace {

// the column sums and squared deviations
constexpr size_t kAccBytes = sizeof(double) * 2 * kStatBlocks * NF;

size_t param_count(uint32_t layers) { return kP0 + (size_t)layers * kPL + H + 1; }

// a graph's arc lists for one call (symmetric graphs: one copy for both directions)
struct GraphDev {
    TmpSet tmp;
    uint64_t *off_out = nullptr, *off_in = nullptr;
    uint32_t *head_out = nullptr, *head_in = nullptr;
    uint32_t *hubs_out = nullptr, *hubs_in = nullptr;   // find_hubs of each direction
    uint32_t n = 0;
    // Hubs keep a few blocks busy for as long as all other vertices take
    // together, so their kernel runs beside the others' (a 2^15-vertex RMAT
    // graph's gradient 1.41 -> 1.33 ms).  Graphs of few arcs per vertex
    // hardly have any: one stream.
    cudaStream_t side = nullptr;
    cudaEvent_t ready = nullptr, done = nullptr;
    GraphDev() = default;
    GraphDev(const GraphDev &) = delete;
    GraphDev &operator=(const GraphDev &) = delete;
    ~GraphDev() {
        if (side) {
            cudaStreamSynchronize(side);
            cudaStreamDestroy(side);
        }
        if (ready) cudaEventDestroy(ready);
        if (done) cudaEventDestroy(done);
    }
    // side waits for what the null stream holds; then join() makes the null
    // stream wait for side
    int fork() {
        if (!side) return CHL_OK;
        CHL_CUDA(cudaEventRecord(ready, 0));
        CHL_CUDA(cudaStreamWaitEvent(side, ready, 0));
        return CHL_OK;
    }
    int join() {
        if (!side) return CHL_OK;
        CHL_CUDA(cudaEventRecord(done, side));
        CHL_CUDA(cudaStreamWaitEvent(0, done, 0));
        return CHL_OK;
    }
};

int upload_csr(const chl_graph *g, GraphDev &d) {
    const uint32_t n = g->n;
    d.n = n;
    int rc;
    if (g->off[1][n] >= 8ull * n) {
        CHL_CUDA(cudaStreamCreateWithFlags(&d.side, cudaStreamNonBlocking));
        CHL_CUDA(cudaEventCreateWithFlags(&d.ready, cudaEventDisableTiming));
        CHL_CUDA(cudaEventCreateWithFlags(&d.done, cudaEventDisableTiming));
    }
    auto put = [&](int f, uint64_t **off, uint32_t **head, uint32_t **hubs) -> int {
        const uint64_t m = g->off[f][n];
        if ((rc = d.tmp.get(off, (uint64_t)n + 1)) || (rc = d.tmp.get(head, m))) return rc;
        CHL_CUDA(cudaMemcpy(*off, g->off[f].data(), ((size_t)n + 1) * 8, cudaMemcpyHostToDevice));
        if (m) CHL_CUDA(cudaMemcpy(*head, g->head[f].data(), m * 4, cudaMemcpyHostToDevice));
        // at most m / kHubArcs lists are longer than kHubArcs
        if ((rc = d.tmp.get(hubs, m / kHubArcs + 1))) return rc;
        CHL_CUDA(cudaMemset(*hubs, 0, 4));
        find_hubs<<<device_sms(), 256>>>(n, *off, *hubs);
        CHL_CUDA(cudaGetLastError());
        return CHL_OK;
    };
    if ((rc = put(1, &d.off_out, &d.head_out, &d.hubs_out))) return rc;
    if (g->symmetric) {
        d.off_in = d.off_out;
        d.head_in = d.head_out;
        d.hubs_in = d.hubs_out;
        return CHL_OK;
    }
    return put(0, &d.off_in, &d.head_in, &d.hubs_in);
}

// standardise the feature columns of M->x in place; M->acc holds the partials
int standardise(chl_gnn *M, uint32_t n) {
    if (n == 0) return CHL_OK;
    const int blocks = (int)std::min<uint32_t>(kStatBlocks, (n + kStatThreads - 1) / kStatThreads);
    int rc = M->acc.ensure(kAccBytes);
    if (rc) return rc;
    double *sums = M->acc.as<double>(), *squares = sums + (size_t)kStatBlocks * NF;
    feat_stats<<<blocks, kStatThreads>>>(n, M->x.as<float>(), nullptr, sums);
    feat_stats<<<blocks, kStatThreads>>>(n, M->x.as<float>(), sums, squares);
    feat_scale<<<std::min(device_sms() * 4, (int)((n + kStatThreads - 1) / kStatThreads)), kStatThreads>>>(
        n, sums, squares, blocks, M->x.as<float>());
    CHL_CUDA(cudaGetLastError());
    return CHL_OK;
}

int ensure_scratch(chl_gnn *M, uint32_t n) {
    const uint32_t L = M->layers;
    int rc;
    if ((rc = M->x.ensure((size_t)n * NF * 4)) || (rc = M->hb.ensure((size_t)(L + 1) * n * H * 2)) ||
        (rc = M->mb.ensure((size_t)(L + 1) * n * H * 2)) || (rc = M->dz.ensure((size_t)n * H * 4)) ||
        (rc = M->inv.ensure((size_t)n * 4)) || (rc = M->dA.ensure(std::max((size_t)n * K2 * 4, kGw0 * sizeof(double)))) ||
        (rc = M->s.ensure((size_t)n * 4)) || (rc = M->ds.ensure((size_t)n * 4)) || (rc = M->y.ensure((size_t)n * 4)) ||
        (rc = M->loss.ensure(8)) || (rc = M->acc.ensure(kAccBytes)) || (rc = M->wt.ensure((size_t)2 * H * H * 4)))
        return rc;
    return CHL_OK;
}

// forward pass; leaves h_l, m_l in scratch and the scores in M->s
int forward(chl_gnn *M, GraphDev &G, uint64_t seed) {
    const uint32_t n = G.n;
    const int sms = device_sms();
    feat_raw<<<sms * 4, 256>>>(n, G.off_out, G.head_out, G.off_in,
                               seed, feat_vpw(n, sms), M->x.as<float>());
    CHL_CUDA(cudaGetLastError());
    int rc = standardise(M, n);
    if (rc) return rc;
    const float *P = M->p.as<float>();
    __nv_bfloat16 *hb = M->hb.as<__nv_bfloat16>(), *mb = M->mb.as<__nv_bfloat16>();
    layer0_fwd<<<sms * 8, 256>>>(n, M->x.as<float>(), P, P + NF * H, hb);
    for (uint32_t l = 1; l <= M->layers; ++l) {
        const float *W = P + kP0 + (size_t)(l - 1) * kPL;
        const __nv_bfloat16 *hp = hb + (size_t)(l - 1) * n * H;
        __nv_bfloat16 *ml = mb + (size_t)l * n * H;
        if ((rc = G.fork())) return rc;
        hub_mean<<<sms * 2, kHubThreads, 0, G.side>>>(G.hubs_out, G.off_out, G.head_out, hp, ml);
        aggregate_mean<<<sms * 8, 256>>>(n, G.off_out, G.head_out, hp, ml);
        if ((rc = G.join())) return rc;
        gemm_rows<K2><<<gemm_grid<K2>(sms), 128>>>(n, hp, ml, W, W + (size_t)K2 * H, 0, hb + (size_t)l * n * H, nullptr, 0);
    }
    const float *wout = P + kP0 + (size_t)M->layers * kPL;
    head_fwd_bwd<<<sms * 8, 256>>>(n, hb + (size_t)M->layers * n * H, wout, wout + H, nullptr, M->s.as<float>(),
                                   nullptr, nullptr);
    CHL_CUDA(cudaGetLastError());
    return CHL_OK;
}

// loss and gradients (into M->g) for target y (device)
int backward(chl_gnn *M, GraphDev &G, double *loss) {
    const uint32_t n = G.n;
    const int sms = device_sms();
    int rc;
    const uint32_t L = M->layers;
    const float *P = M->p.as<float>();
    float *Gp = M->g.as<float>();
    __nv_bfloat16 *hb = M->hb.as<__nv_bfloat16>(), *mb = M->mb.as<__nv_bfloat16>();
    CHL_CUDA(cudaMemset(M->g.p, 0, M->np * 4));
    CHL_CUDA(cudaMemset(M->loss.p, 0, 8));
    const float *wout = P + kP0 + (size_t)L * kPL;
    float *gwout = Gp + kP0 + (size_t)L * kPL;
    head_fwd_bwd<<<sms * 8, 256>>>(n, hb + (size_t)L * n * H, wout, wout + H, M->y.as<float>(), M->s.as<float>(),
                                   M->ds.as<float>(), M->loss.as<double>());
    // dz in BF16 goes to m_0's slot (unused after the forward pass)
    float *dz = M->dz.as<float>();
    head_bwd<<<sms * 4, 256>>>(n, M->ds.as<float>(), hb + (size_t)L * n * H, wout, dz, mb, gwout, gwout + H);
    inv_degree<<<sms, 256>>>(n, G.off_out, M->inv.as<float>());
    for (uint32_t l = L; l >= 1; --l) {
        const float *W = P + kP0 + (size_t)(l - 1) * kPL;
        float *gW = Gp + kP0 + (size_t)(l - 1) * kPL;
        const __nv_bfloat16 *hp = hb + (size_t)(l - 1) * n * H;
        const __nv_bfloat16 *ml = mb + (size_t)l * n * H;
        const uint32_t gblocks = std::max<uint32_t>(1, std::min<uint32_t>((uint32_t)sms * 2, (n + 255) / 256));
        grad_w_mma<<<gblocks, kGwThreads>>>(n, hp, ml, mb, dz, gW, gW + (size_t)K2 * H);
        // dA = dz W^T as two K = 64 GEMMs into the two column halves of dA
        transpose_w<<<16, 256>>>(W, M->wt.as<float>(), M->wt.as<float>() + H * H);
        gemm_rows<H><<<gemm_grid<H>(sms), 128>>>(n, mb, mb, M->wt.as<float>(), nullptr, 1, nullptr, M->dA.as<float>(), K2);
        gemm_rows<H><<<gemm_grid<H>(sms), 128>>>(n, mb, mb, M->wt.as<float>() + H * H, nullptr, 1, nullptr,
                                       M->dA.as<float>() + H, K2);
        if ((rc = G.fork())) return rc;
        hub_scatter<<<sms * 2, kHubThreads, 0, G.side>>>(G.hubs_in, M->dA.as<float>(), G.off_in, G.head_in,
                                                         M->inv.as<float>(), hp, dz, mb);
        scatter_mean_bwd<<<sms * 8, 256>>>(n, M->dA.as<float>(), G.off_in, G.head_in, M->inv.as<float>(), hp, dz, mb);
        if ((rc = G.join())) return rc;
    }
    // the parts go to dA, which is done with: 512 bytes per vertex (2 KB at
    // least, one part) against 2 KB per kGw0Rows vertices
    const int blocks = std::max(1, std::min(sms, (int)((n + kGw0Rows - 1) / kGw0Rows)));
    grad_w0<<<blocks, kGw0Threads>>>(n, M->x.as<float>(), dz, M->dA.as<double>());
    grad_w0_out<<<kGw0 / 32, 32 * kGw0Parts>>>(M->dA.as<double>(), blocks, Gp, Gp + NF * H);
    CHL_CUDA(cudaGetLastError());
    CHL_CUDA(cudaMemcpy(loss, M->loss.p, 8, cudaMemcpyDeviceToHost));
    return CHL_OK;
}

}  // namespace

extern "C" int chl_gnn_create(uint32_t layers, uint64_t seed, chl_gnn **out) {
    if (!out || layers == 0 || layers > 8) return CHL_ERR_INVALID;
    chl_gnn *M = new (std::nothrow) chl_gnn();
    if (!M) return CHL_ERR_OOM;
    M->layers = layers;
    M->np = param_count(layers);
    M->host.assign(M->np, 0.f);
    // Glorot-uniform weights from the seeded stream, zero biases
    Rng rng(seed);
    auto fill = [&](float *w, int fan_in, int fan_out, size_t cnt) {
        const double lim = std::sqrt(6.0 / (fan_in + fan_out));
        for (size_t i = 0; i < cnt; ++i) w[i] = (float)((2.0 * rng.unit() - 1.0) * lim);
    };
    float *p = M->host.data();
    fill(p, NF, H, (size_t)NF * H);
    for (uint32_t l = 0; l < layers; ++l) fill(p + kP0 + l * kPL, K2, H, (size_t)K2 * H);
    fill(p + kP0 + layers * kPL, H, 1, H);
    int rc;
    if ((rc = M->p.ensure(M->np * 4)) || (rc = M->g.ensure(M->np * 4)) || (rc = M->m.ensure(M->np * 4)) ||
        (rc = M->v.ensure(M->np * 4))) {
        delete M;
        return rc;
    }
    cudaMemcpy(M->p.p, M->host.data(), M->np * 4, cudaMemcpyHostToDevice);
    cudaMemset(M->m.p, 0, M->np * 4);
    cudaMemset(M->v.p, 0, M->np * 4);
    *out = M;
    return CHL_OK;
}

extern "C" size_t chl_gnn_param_count(const chl_gnn *m) { return m ? m->np : 0; }

extern "C" int chl_gnn_get_params(const chl_gnn *m, float *out) {
    if (!m || !out) return CHL_ERR_INVALID;
    CHL_CUDA(cudaMemcpy(out, m->p.p, m->np * 4, cudaMemcpyDeviceToHost));
    return CHL_OK;
}

extern "C" int chl_gnn_set_params(chl_gnn *m, const float *in) {
    if (!m || !in) return CHL_ERR_INVALID;
    CHL_CUDA(cudaMemcpy(m->p.p, in, m->np * 4, cudaMemcpyHostToDevice));
    return CHL_OK;
}

extern "C" int chl_gnn_features(const chl_graph *g, uint64_t seed, float *x) {
    if (!g || !x) return CHL_ERR_INVALID;
    chl_gnn tmp;
    GraphDev G;
    int rc;
    if ((rc = upload_csr(g, G)) || (rc = tmp.x.ensure((size_t)g->n * NF * 4))) return rc;
    feat_raw<<<device_sms() * 4, 256>>>(g->n, G.off_out, G.head_out,
                                        G.off_in, seed, feat_vpw(g->n, device_sms()), tmp.x.as<float>());
    CHL_CUDA(cudaGetLastError());
    if ((rc = standardise(&tmp, g->n))) return rc;
    CHL_CUDA(cudaMemcpy(x, tmp.x.p, (size_t)g->n * NF * 4, cudaMemcpyDeviceToHost));
    return CHL_OK;
}

extern "C" int chl_gnn_predict(chl_gnn *m, const chl_graph *g, uint64_t seed, float *score) {
    if (!m || !g || !score) return CHL_ERR_INVALID;
    GraphDev G;
    int rc;
    if ((rc = upload_csr(g, G)) || (rc = ensure_scratch(m, g->n)) || (rc = forward(m, G, seed))) return rc;
    CHL_CUDA(cudaMemcpy(score, m->s.p, (size_t)g->n * 4, cudaMemcpyDeviceToHost));
    return CHL_OK;
}

extern "C" int chl_gnn_grad(chl_gnn *m, const chl_graph *g, uint64_t seed, const float *target, double *loss,
                            float *grads) {
    if (!m || !g || !target || !loss) return CHL_ERR_INVALID;
    GraphDev G;
    int rc;
    if ((rc = upload_csr(g, G)) || (rc = ensure_scratch(m, g->n)) || (rc = forward(m, G, seed))) return rc;
    CHL_CUDA(cudaMemcpy(m->y.p, target, (size_t)g->n * 4, cudaMemcpyHostToDevice));
    if ((rc = backward(m, G, loss))) return rc;
    if (grads) CHL_CUDA(cudaMemcpy(grads, m->g.p, m->np * 4, cudaMemcpyDeviceToHost));
    return CHL_OK;
}

extern "C" int chl_gnn_train_step(chl_gnn *m, const chl_graph *g, uint64_t seed, const float *target, float lr,
                                  double *loss) {
    double l = 0;
    int rc = chl_gnn_grad(m, g, seed, target, &l, nullptr);
    if (rc) return rc;
    m->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - (float)std::pow((double)b1, (double)m->step);
    const float c2 = 1.f - (float)std::pow((double)b2, (double)m->step);
    adam_step<<<64, 256>>>(m->np, m->p.as<float>(), m->g.as<float>(), m->m.as<float>(), m->v.as<float>(), lr, b1, b2,
                           1e-8f, c1, c2);
    CHL_CUDA(cudaGetLastError());
    if (loss) *loss = l;
    return CHL_OK;
}

extern "C" int chl_gnn_order(chl_gnn *m, const chl_graph *g, uint64_t seed, uint32_t *order) {
    if (!m || !g || !order) return CHL_ERR_INVALID;
    const uint32_t n = g->n;
    if (n == 0) return CHL_OK;
    GraphDev G;
    int rc;
    if ((rc = upload_csr(g, G)) || (rc = ensure_scratch(m, n)) || (rc = forward(m, G, seed))) return rc;
    return order_by_score(n, seed, m->s.as<float>(), order);
}

extern "C" void chl_gnn_free(chl_gnn *m) { delete m; }
