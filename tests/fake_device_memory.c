/* A device of as many bytes as fake_device_set says, for tests of what the
 * library does when an allocation finds no room: preloaded before the CUDA
 * runtime, it answers cudaErrorMemoryAllocation on the host, and passes every
 * other call on.  Nothing is filled up on the GPU. */
#include <dlfcn.h>
#include <pthread.h>
#include <stddef.h>

typedef int cudaError_t;   /* cudaSuccess 0, cudaErrorMemoryAllocation 2 */

#define SLOTS 4096
static struct {
    void *p;
    size_t bytes;
} held[SLOTS];
static size_t limit = (size_t)-1, live;
static pthread_mutex_t mu = PTHREAD_MUTEX_INITIALIZER;

/* the runtime is loaded beside the library, out of RTLD_NEXT's sight */
static void *real_call(const char *name) {
    static void *rt;
    if (!rt) rt = dlopen("libcudart.so.13", RTLD_NOW);
    if (!rt) rt = dlopen("libcudart.so", RTLD_NOW);
    return rt ? dlsym(rt, name) : NULL;
}

void fake_device_set(size_t bytes) { limit = bytes; }
size_t fake_device_live(void) { return live; }

static int room(size_t bytes) {
    pthread_mutex_lock(&mu);
    const int ok = bytes <= limit && live <= limit - bytes;
    pthread_mutex_unlock(&mu);
    return ok;
}

static void note(void *p, size_t bytes) {
    pthread_mutex_lock(&mu);
    for (int i = 0; i < SLOTS; ++i)
        if (!held[i].p) {
            held[i].p = p;
            held[i].bytes = bytes;
            live += bytes;
            break;
        }
    pthread_mutex_unlock(&mu);
}

static void drop(void *p) {
    if (!p) return;
    pthread_mutex_lock(&mu);
    for (int i = 0; i < SLOTS; ++i)
        if (held[i].p == p) {
            live -= held[i].bytes;
            held[i].p = NULL;
            break;
        }
    pthread_mutex_unlock(&mu);
}

cudaError_t cudaMalloc(void **p, size_t bytes) {
    cudaError_t (*real)(void **, size_t) = real_call("cudaMalloc");
    if (!room(bytes)) return 2;
    const cudaError_t e = real(p, bytes);
    if (e == 0) note(*p, bytes);
    return e;
}

cudaError_t cudaMallocFromPoolAsync(void **p, size_t bytes, void *pool, void *stream) {
    cudaError_t (*real)(void **, size_t, void *, void *) = real_call("cudaMallocFromPoolAsync");
    if (!room(bytes)) return 2;
    const cudaError_t e = real(p, bytes, pool, stream);
    if (e == 0) note(*p, bytes);
    return e;
}

cudaError_t cudaFree(void *p) {
    cudaError_t (*real)(void *) = real_call("cudaFree");
    drop(p);
    return real(p);
}

cudaError_t cudaFreeAsync(void *p, void *stream) {
    cudaError_t (*real)(void *, void *) = real_call("cudaFreeAsync");
    drop(p);
    return real(p, stream);
}

cudaError_t cudaMemGetInfo(size_t *free_bytes, size_t *total) {
    cudaError_t (*real)(size_t *, size_t *) = real_call("cudaMemGetInfo");
    const cudaError_t e = real(free_bytes, total);
    if (e == 0 && limit != (size_t)-1) {
        *total = limit;
        *free_bytes = live < limit ? limit - live : 0;
    }
    return e;
}
