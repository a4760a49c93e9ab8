/* A host-only stand-in for the few CUDA runtime calls of the library's memory code, so that its bounds
   and failure paths run on a machine without a GPU: four devices whose pools are plain accounts
   (reserved and used bytes), streams that only order releases, and switches that make the next call of
   a kind fail. */
#pragma once
#include <cstdint>
#include <cstdlib>
#include <map>
#include <mutex>
#include <set>
#include <vector>

#define __host__
#define __device__
#define __forceinline__ inline

enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorInvalidDevice = 101,
                   cudaErrorStreamCaptureUnsupported = 900 };
inline const char *cudaGetErrorString(cudaError_t) { return "fake"; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }

namespace fake {

struct Stream { int dev; };
struct Block { size_t bytes; int state; Stream *on; };        /* state: 0 free, 1 used, 2 freed in on's order */
struct Pool {
    int dev = 0;
    unsigned long long threshold = 0, reserved = 0;
    std::map<char *, Block> blocks;
};

inline std::recursive_mutex mu;
inline thread_local int device = 0;
inline unsigned long long capacity = 1ull << 62;  /* bytes a device can reserve */
inline std::vector<Pool *> pools;
inline std::vector<int> synced;                   /* devices waited for, in order */
inline int maps = 0;                              /* reservations made */
inline int host_allocs = 0, host_frees = 0;
inline int refuse_device_sync = 0;                /* device waits to refuse */
inline int fail_host_allocs = 0;                  /* page-locked allocations to fail */
inline std::set<void *> host;
inline char *next_address = (char *) 0x10000000;

inline void trim(Pool *p, unsigned long long keep) {
    for (auto it = p->blocks.begin(); it != p->blocks.end() && p->reserved > keep;)
        if (it->second.state == 0) { p->reserved -= it->second.bytes; it = p->blocks.erase(it); }
        else ++it;
}
inline void complete(int dev, Stream *only) {
    for (Pool *p : pools) {
        if (p->dev != dev) continue;
        for (auto &b : p->blocks)
            if (b.second.state == 2 && (!only || b.second.on == only)) b.second.state = 0;
        trim(p, p->threshold);
    }
}

}  // namespace fake

typedef fake::Stream *cudaStream_t;
typedef fake::Pool *cudaMemPool_t;
enum { cudaMemAllocationTypePinned = 1, cudaMemLocationTypeDevice = 1, cudaStreamNonBlocking = 1 };
struct cudaMemPoolProps { int allocType; struct { int type, id; } location; };
enum cudaMemPoolAttr { cudaMemPoolReuseAllowInternalDependencies, cudaMemPoolAttrReleaseThreshold,
                       cudaMemPoolAttrReservedMemCurrent };

inline cudaError_t cudaGetDevice(int *d) { *d = fake::device; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d > 3) return cudaErrorInvalidDevice;
    fake::device = d;
    return cudaSuccess;
}
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, int) { *s = new fake::Stream{fake::device}; return cudaSuccess; }
inline cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *props) {
    std::lock_guard<std::recursive_mutex> l(fake::mu);
    *p = new fake::Pool();
    (*p)->dev = props->location.id;
    fake::pools.push_back(*p);
    return cudaSuccess;
}
inline cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
inline cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void *v) {
    std::lock_guard<std::recursive_mutex> l(fake::mu);
    if (a == cudaMemPoolAttrReleaseThreshold) p->threshold = *(unsigned long long *) v;
    return cudaSuccess;
}
inline cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void *v) {
    std::lock_guard<std::recursive_mutex> l(fake::mu);
    if (a == cudaMemPoolAttrReservedMemCurrent) *(unsigned long long *) v = p->reserved;
    return cudaSuccess;
}
inline cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep) {
    std::lock_guard<std::recursive_mutex> l(fake::mu);
    fake::trim(p, keep);
    return cudaSuccess;
}
inline cudaError_t cudaMallocFromPoolAsync(void **out, size_t bytes, cudaMemPool_t p, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> l(fake::mu);
    for (auto &b : p->blocks)                     /* the first free block of that size, or freed on the same stream */
        if (b.second.bytes == bytes && (b.second.state == 0 || (b.second.state == 2 && b.second.on == st))) {
            b.second.state = 1;
            *out = b.first;
            return cudaSuccess;
        }
    if (p->reserved + bytes > fake::capacity) return cudaErrorMemoryAllocation;
    p->reserved += bytes;
    fake::maps++;
    p->blocks[fake::next_address] = {bytes, 1, nullptr};
    *out = fake::next_address;
    fake::next_address += bytes + 512;
    return cudaSuccess;
}
inline cudaError_t cudaFreeAsync(void *ptr, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> l(fake::mu);
    for (fake::Pool *p : fake::pools) {
        auto it = p->blocks.find((char *) ptr);
        if (it != p->blocks.end()) { it->second.state = 2; it->second.on = st; }
    }
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> l(fake::mu);
    fake::complete(s->dev, s);
    return cudaSuccess;
}
inline cudaError_t cudaDeviceSynchronize() {
    std::lock_guard<std::recursive_mutex> l(fake::mu);
    if (fake::refuse_device_sync > 0) { fake::refuse_device_sync--; return cudaErrorStreamCaptureUnsupported; }
    fake::synced.push_back(fake::device);
    fake::complete(fake::device, nullptr);
    return cudaSuccess;
}
inline cudaError_t cudaMallocHost(void **p, size_t bytes) {
    std::lock_guard<std::recursive_mutex> l(fake::mu);
    if (fake::fail_host_allocs > 0) { fake::fail_host_allocs--; *p = nullptr; return cudaErrorMemoryAllocation; }
    fake::host_allocs++;
    *p = malloc(bytes < 64 ? bytes : 64);         /* never written */
    fake::host.insert(*p);
    return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void *p) {
    std::lock_guard<std::recursive_mutex> l(fake::mu);
    fake::host_frees++;
    fake::host.erase(p);
    free(p);
    return cudaSuccess;
}
