// HostCopy over fakes of the CUDA runtime's and the C library's calls, with one kind of call made to fail.
//   host_copy event N      the N-th cudaEventCreateWithFlags fails
//   host_copy ring         cudaHostAlloc fails
//   host_copy thread N     pthread_create fails from the N-th call on
//   host_copy resident     nothing was prepared: no copy may allocate
// Every copy has to end, with the right bytes, and what a failed start has made has to be given back.
#include "../../aspen_b200/csrc/hostcopy.h"

#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <cstdio>
#include <cstdlib>
#include <string>

static int g_event_fails = -1, g_thread_fails = -1, g_events = 0, g_threads = 0, g_live_events = 0, g_live_blocks = 0, g_allocs = 0;
static bool g_ring_fails = false;

extern "C" {
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    if (g_ring_fails && n > HostCopy::SMALL) return cudaErrorMemoryAllocation;
    g_live_blocks++;
    g_allocs++;
    return (*p = malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeHost(void *p) { g_live_blocks--; free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    if (++g_events == g_event_fails) return cudaErrorMemoryAllocation;
    g_live_events++;
    *e = (cudaEvent_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { g_live_events--; free((void *)e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return e ? cudaSuccess : cudaErrorInvalidResourceHandle; }
cudaError_t cudaEventQuery(cudaEvent_t e) { return e ? cudaSuccess : cudaErrorInvalidResourceHandle; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }

int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
    if (g_thread_fails >= 0 && ++g_threads >= g_thread_fails) return EAGAIN;
    static auto real = (int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *))dlsym(RTLD_NEXT, "pthread_create");
    return real(t, a, f, arg);
}
}

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    const int n = argc > 2 ? atoi(argv[2]) : 0;
    if (what == "event") g_event_fails = n;
    else if (what == "ring") g_ring_fails = true;
    else if (what == "thread") g_thread_fails = n;
    int bad = 0;
    {
        HostCopy copy;
        for (size_t bytes : {(size_t)1000, HostCopy::SMALL + 4, HostCopy::MIN_BYTES, 40 * HostCopy::PIECE + 12, 3 * HostCopy::PIECE}) {
            std::vector<char> src(bytes), dst(bytes);
            if (what != "resident") copy.prepare(bytes);
            const int allocs = g_allocs;
            for (size_t i = 0; i < bytes; i++) src[i] = (char)(i * 2654435761u >> 13);
            if (copy.down(dst.data(), src.data(), bytes, nullptr) != cudaSuccess || src != dst) { printf("copy of %zu bytes is wrong\n", bytes); bad = 1; }
            if (g_allocs != allocs) { printf("copy of %zu bytes allocates pinned memory\n", bytes); bad = 1; }
        }
    }
    if (g_live_events || g_live_blocks) { printf("%d events and %d blocks are left\n", g_live_events, g_live_blocks); bad = 1; }
    return bad;
}
