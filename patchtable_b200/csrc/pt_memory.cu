/* Device and page-locked host memory of the library.

   Builds take about sixty device buffers and give most of them back, and a cudaMalloc or cudaFree
   costs 0.1 ms and up (with the mapping of large blocks, 18 of the 31 ms of a 240 x 320 build; a
   cudaFree also waits for the whole device).  Buffers therefore come from one CUDA memory pool per
   device.  Scratch buffers (DevBuf given a stream) are freed in that stream's order; all others may
   have been used on any stream, so their release waits for the device first, as cudaFree did; while
   that wait is refused (another thread's stream capture forbids it) they are held back from reuse.
   Reuse across streams that would make one stream wait for another is switched off: the steps of a
   build run beside each other.

   What the pool keeps for reuse is bounded: at most PT_POOL_KEEP bytes per device stay reserved
   beside the live buffers; a device whose allocation fails gets all its free memory back before it
   is tried once more, and pt_release_memory() gives everything back.  CUDA's release threshold counts every reserved byte, live ones
   too, so it follows them (set_keep): with a constant one a program with more than that live would
   give all its free memory back at the next wait and map it again in every build (a 1080p build beside
   7 GiB of live buffers: 75 ms with 4 GiB, 46 ms so, 46 ms with nothing live).  Page-locked blocks are kept the same way, at most
   PT_PINNED_KEEP bytes per process, and given back before a failed allocation's second try.  Both are safe with any number of threads and streams. */
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "patchtable_b200.h"
#include "pt_internal.h"

namespace {

constexpr unsigned long long PT_POOL_KEEP = 4ull << 30;
constexpr size_t PT_PINNED_KEEP = 256u << 20;
constexpr int MAX_DEVICES = 64;

struct Block { void *p; size_t bytes; };

struct DevicePool {
    std::mutex mu;
    cudaMemPool_t pool = nullptr;
    cudaStream_t st = nullptr;            /* order of the buffers that belong to no stream */
    unsigned long long live = 0;          /* bytes of the buffers in use */
    std::vector<Block> held;              /* released, but their device could not be waited for */
};
DevicePool g_pool[MAX_DEVICES];

std::mutex g_pinned_mu;
std::vector<Block> g_pinned;             /* free page-locked blocks */
size_t g_pinned_bytes = 0;

/* The current device's pool, created on first use. */
cudaError_t device_pool(DevicePool **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    DevicePool &d = g_pool[dev];
    std::lock_guard<std::mutex> lock(d.mu);
    if (!d.pool) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        if ((e = cudaMemPoolCreate(&pool, &props)) != cudaSuccess) return e;
        int off = 0;
        cudaStream_t st = nullptr;
        if ((e = cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &off)) != cudaSuccess ||
            (e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)) != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            return e;
        }
        d.st = st;
        d.pool = pool;
    }
    *out = &d;
    return cudaSuccess;
}

/* What a device's pool has reserved and may keep reserved, beside its live bytes. */
struct Reserve {
    unsigned long long reserved, keep, live;
    bool over() const { return reserved > keep; }
};

/* Adds to the device's live bytes and moves the pool's release threshold with them.  Under a cap
   (pt_set_device_alloc_limit) what is kept for reuse stays within it too; a release still counts as
   live there. */
Reserve set_keep(DevicePool &d, long long bytes) {
    const long long room = pt_alloc_room();
    std::lock_guard<std::mutex> lock(d.mu);
    d.live += bytes;
    unsigned long long spare = PT_POOL_KEEP, reserved = 0;
    if (room >= 0) spare = std::min(spare, (unsigned long long) (room + (bytes < 0 ? -bytes : 0)));
    unsigned long long keep = d.live + spare;
    cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (bytes <= 0 || room >= 0) cudaMemPoolGetAttribute(d.pool, cudaMemPoolAttrReservedMemCurrent, &reserved);
    return {reserved, keep, d.live};
}

/* Waits for the current device (d's) and gives b and the blocks held back before to the pool; holds
   them all back when the wait is refused. */
void wait_and_free(DevicePool &d, Block b) {
    std::vector<Block> blocks;
    {
        std::lock_guard<std::mutex> lock(d.mu);
        blocks.swap(d.held);
    }
    if (b.p) blocks.push_back(b);
    if (cudaDeviceSynchronize() != cudaSuccess) {
        cudaGetLastError();
        std::lock_guard<std::mutex> lock(d.mu);
        d.held.insert(d.held.end(), blocks.begin(), blocks.end());
        return;
    }
    long long bytes = 0;
    for (const Block &x : blocks) {
        cudaFreeAsync(x.p, d.st);
        bytes += (long long) x.bytes;
    }
    /* the threshold takes effect at a wait; the last of many frees may have none after it */
    if (bytes && set_keep(d, -bytes).over()) cudaStreamSynchronize(d.st);
}

/* Makes a device current for a scope. */
struct OnDevice {
    int cur;
    explicit OnDevice(int dev) : cur(dev) {
        cudaGetDevice(&cur);
        if (cur != dev) cudaSetDevice(dev);
        else cur = -1;
    }
    ~OnDevice() { if (cur >= 0) cudaSetDevice(cur); }
};

/* Frees the page-locked blocks kept for reuse; returns whether there were any. */
bool drop_pinned() {
    std::vector<Block> held;
    {
        std::lock_guard<std::mutex> lock(g_pinned_mu);
        held.swap(g_pinned);
        g_pinned_bytes = 0;
    }
    for (const Block &b : held) cudaFreeHost(b.p);
    return !held.empty();
}

}  // namespace

cudaError_t pt_dev_alloc(void **p, size_t bytes, cudaStream_t st, bool scratch) {
    DevicePool *d = nullptr;
    cudaError_t e = device_pool(&d);
    if (e != cudaSuccess) return e;
    if (!scratch) st = d->st;
    const bool capped = pt_alloc_room() >= 0;
    Reserve r = set_keep(*d, (long long) bytes);
    if (capped && r.reserved < r.live && r.reserved + bytes > r.keep) {      /* needs new memory, beyond the cap */
        wait_and_free(*d, {});
        cudaMemPoolTrimTo(d->pool, r.keep - bytes);
    }
    e = cudaMallocFromPoolAsync(p, bytes, d->pool, st);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        wait_and_free(*d, {});
        cudaMemPoolTrimTo(d->pool, 0);
        e = cudaMallocFromPoolAsync(p, bytes, d->pool, st);
        if (e != cudaSuccess) cudaGetLastError();
    }
    if (capped && e == cudaSuccess && (r = set_keep(*d, 0)).over()) {        /* no free block was large enough */
        wait_and_free(*d, {});
        cudaMemPoolTrimTo(d->pool, r.keep);
    }
    /* a buffer of no stream must be usable on every stream when this returns */
    if (e == cudaSuccess && !scratch && (e = cudaStreamSynchronize(st)) != cudaSuccess) cudaFreeAsync(*p, st);
    if (e != cudaSuccess) set_keep(*d, -(long long) bytes);
    return e;
}

void pt_dev_free(void *p, size_t bytes, int dev, cudaStream_t st, bool scratch) {
    const OnDevice on(dev);
    DevicePool &d = g_pool[dev];
    if (!scratch) {
        wait_and_free(d, {p, bytes});
        return;
    }
    cudaFreeAsync(p, st);
    set_keep(d, -(long long) bytes);
}

cudaError_t pt_pinned_alloc(void **p, size_t bytes, size_t *got) {
    {
        std::lock_guard<std::mutex> lock(g_pinned_mu);
        int best = -1;
        for (int i = 0; i < (int) g_pinned.size(); i++)
            if (g_pinned[i].bytes >= bytes && g_pinned[i].bytes <= 2 * bytes &&
                (best < 0 || g_pinned[i].bytes < g_pinned[best].bytes))
                best = i;
        if (best >= 0) {
            *p = g_pinned[best].p;
            *got = g_pinned[best].bytes;
            g_pinned_bytes -= *got;
            g_pinned.erase(g_pinned.begin() + best);
            return cudaSuccess;
        }
    }
    *got = bytes;
    cudaError_t e = cudaMallocHost(p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        if (drop_pinned()) e = cudaMallocHost(p, bytes);
        if (e != cudaSuccess) cudaGetLastError();
    }
    return e;
}

void pt_pinned_free(void *p, size_t bytes, int dev) {
    const OnDevice on(dev);
    /* no copy of a failed call may still use a block that is kept */
    if (cudaDeviceSynchronize() == cudaSuccess) {
        std::lock_guard<std::mutex> lock(g_pinned_mu);
        if (g_pinned_bytes + bytes <= PT_PINNED_KEEP) {
            g_pinned.push_back({p, bytes});
            g_pinned_bytes += bytes;
            return;
        }
    } else {
        cudaGetLastError();
    }
    cudaFreeHost(p);
}

void pt_dev_cap_changed() {
    for (DevicePool &d : g_pool) {
        {
            std::lock_guard<std::mutex> lock(d.mu);
            if (!d.pool) continue;
        }
        if (set_keep(d, 0).over()) cudaStreamSynchronize(d.st);
    }
}

extern "C" pt_status pt_release_memory(void) {
    for (int dev = 0; dev < MAX_DEVICES; dev++) {
        DevicePool &d = g_pool[dev];
        bool held;
        {
            std::lock_guard<std::mutex> lock(d.mu);
            if (!d.pool) continue;
            held = !d.held.empty();
        }
        if (held) {
            const OnDevice on(dev);
            wait_and_free(d, {});
        }
        cudaStreamSynchronize(d.st);
        PT_CUDA(cudaMemPoolTrimTo(d.pool, 0));
    }
    drop_pinned();
    return PT_OK;
}
