// Device-side helpers shared by the CUDA translation units.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>

#include "chl_internal.h"

namespace chl {

constexpr uint32_t kFull = 0xFFFFFFFFu;

// Record a CUDA failure as the thread's last error and map it to a status.
int cuda_status(cudaError_t e, const char *what, const char *file, int line);

#define CHL_CUDA(call)                                                        \
    do {                                                                      \
        cudaError_t _e = (call);                                              \
        if (_e != cudaSuccess) return ::chl::cuda_status(_e, #call, __FILE__, __LINE__); \
    } while (0)

// Number of SMs of the current device (cached).
int device_sms();

// Temporary device memory of one call, ordered on stream s.  Blocks of up to
// kTmpMost bytes come from a pool of the library's own that keeps at most
// kTmpKeep bytes between calls (a cudaMalloc and cudaFree pair costs 60 us and
// a synchronisation, and a small call makes a dozen); larger ones are plain
// allocations (mapping them through a pool costs more: 16 GB 35 ms against
// 7.7).  What outlives a call (labels, graphs, networks) is never taken from
// here.  The pool is stream-ordered, so calls on any threads and streams may
// share it; it is emptied when an allocation fails (a tmp_alloc or a
// long_malloc) and when a graph's device copy is released.
constexpr size_t kTmpMost = (size_t)512 << 20;
constexpr size_t kTmpKeep = (size_t)1 << 30;
int tmp_alloc(void **p, size_t bytes, cudaStream_t s);
void tmp_free(void *p, size_t bytes, cudaStream_t s);
void tmp_trim();
// cudaMalloc for what outlives a call: once more without the pool's idle
// memory if there is no room.
cudaError_t long_malloc(void **p, size_t bytes);
template <typename T>
cudaError_t long_malloc(T **p, size_t bytes) {
    return long_malloc((void **)p, bytes);
}

// The temporaries of one call, freed together (or one by one) on their stream.
class TmpSet {
  public:
    explicit TmpSet(cudaStream_t s = 0) : st(s) {}
    TmpSet(const TmpSet &) = delete;
    TmpSet &operator=(const TmpSet &) = delete;
    ~TmpSet() {
        for (const auto &x : held) tmp_free(x.first, x.second, st);
    }
    template <typename T>
    int get(T **p, uint64_t count) {
        const size_t bytes = (size_t)(count ? count : 1) * sizeof(T);
        *p = nullptr;
        try {
            held.emplace_back(nullptr, bytes);
        } catch (...) {   // callers are C entries
            return CHL_ERR_OOM;
        }
        const int rc = tmp_alloc(&held.back().first, bytes, st);
        *p = (T *)held.back().first;
        if (rc) held.pop_back();
        return rc;
    }
    template <typename T>
    void put(T *&p) {
        for (size_t i = 0; i < held.size(); ++i)
            if (held[i].first == (void *)p) {
                tmp_free(held[i].first, held[i].second, st);
                held.erase(held.begin() + i);
                break;
            }
        p = nullptr;
    }
    cudaStream_t st;

  private:
    std::vector<std::pair<void *, size_t>> held;
};

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// ---------------------------------------------------------------- scans
// Exclusive prefix sum of n u32 values into u64 outputs; out[n] = total.
// With d_n, only the first *d_n entries are read and only their prefixes and
// out[n] are written, so the launch shape depends only on the host bound n.
int scan_u32_excl(const uint32_t *in, uint64_t *out, uint64_t n,
                  const uint64_t *d_n, void *tmp, size_t tmp_bytes,
                  cudaStream_t s);
size_t scan_tmp_bytes(uint64_t n);

// ---------------------------------------------------------------- sort
// Stable LSD radix sort of (key, value) pairs on the low `bits` key bits.
// The item count is read from device memory (*d_n <= cap); the result ends
// in (k0, v0) if the returned parity is 0, else in (k1, v1).
int radix_sort_pairs(uint64_t *k0, uint32_t *v0, uint64_t *k1, uint32_t *v1,
                     const uint64_t *d_n, uint64_t cap, int bits, void *tmp,
                     size_t tmp_bytes, cudaStream_t s, int *parity);
size_t radix_tmp_bytes();

// Vertices by device score descending, ties by the seeded tie key (the same
// rule as the degree order); writes the host order array (rank -> vertex).
int order_by_score(uint32_t n, uint64_t seed, const float *d_score, uint32_t *order_h);

}  // namespace chl
