/* Checks of the library's memory code (pt_memory.cu and the buffers of pt_internal.h) over a stand-in
   for the CUDA runtime.  Usage: memory_pool CHECK; prints what failed and returns 1. */
#include <cstdio>
#include <cstring>
#include <memory>

#include "pt_memory.cu"

#include <atomic>

pt_status pt_fail(pt_status s, const char *, ...) { return s; }
static long long limit = -1, live = 0;
bool pt_alloc_admit(size_t n) {
    if (limit >= 0 && live + (long long) n > limit) return false;
    live += n;
    return true;
}
void pt_alloc_release(size_t n) { live -= n; }
long long pt_alloc_room() { return limit < 0 ? -1 : limit < live ? 0 : limit - live; }

#define EXPECT(c) do { if (!(c)) { printf("%s:%d: %s\n", __FILE__, __LINE__, #c); return 1; } } while (0)

static const size_t GiB = 1ull << 30;
static fake::Pool &pool(int dev = 0) {
    for (fake::Pool *p : fake::pools) if (p->dev == dev) return *p;
    abort();
}

/* A build's scratch, freed in its stream's order, with a wait at the end as every build has. */
static void build(cudaStream_t st) {
    DevBuf<char> a(st), b(st), c(st);
    a.reserve(GiB); b.reserve(GiB); c.reserve(GiB / 2);
    a.release(); b.release(); c.release();
    cudaStreamSynchronize(st);
}

/* What is kept for reuse does not depend on how much is live. */
static int reuse_beside_live() {
    cudaStream_t st;
    cudaStreamCreateWithFlags(&st, 0);
    DevBuf<char> tables[6];
    for (auto &t : tables) EXPECT(t.reserve(GiB) == cudaSuccess);
    build(st);
    const int maps = fake::maps;
    for (int i = 0; i < 3; i++) build(st);
    EXPECT(fake::maps == maps);
    EXPECT(pool().reserved == 6 * GiB + 2 * GiB + GiB / 2);
    return 0;
}

/* At most 4 GiB stay beside the live buffers, whatever is freed last. */
static int bound() {
    {
        DevBuf<char> big[3], small;
        for (auto &t : big) EXPECT(t.reserve(3 * GiB) == cudaSuccess);
        EXPECT(small.reserve(GiB) == cudaSuccess);
        big[0].release();
        big[1].release();
        EXPECT(pool().reserved <= 4 * GiB + 4 * GiB);
    }
    EXPECT(pool().reserved <= 4 * GiB);
    {
        DevBuf<char> one;
        EXPECT(one.reserve(9 * GiB) == cudaSuccess);
    }
    EXPECT(pool().reserved <= 4 * GiB);
    EXPECT(pt_release_memory() == PT_OK && pool().reserved == 0);
    return 0;
}

/* An allocation that does not fit beside what is kept for reuse is made in its place; one that does not
   fit at all fails, and leaves the accounts as they were. */
static int retry() {
    fake::capacity = 5 * GiB;
    { DevBuf<char> a; EXPECT(a.reserve(3 * GiB) == cudaSuccess); }
    EXPECT(pool().reserved == 3 * GiB);
    DevBuf<char> b, c;
    EXPECT(b.reserve(4 * GiB) == cudaSuccess && b.p);
    EXPECT(c.reserve(2 * GiB) == cudaErrorMemoryAllocation && !c.p);
    EXPECT(pool().threshold == 8 * GiB);
    b.release();
    EXPECT(pt_release_memory() == PT_OK && pool().reserved == 0 && pool().threshold == 4 * GiB);
    return 0;
}

/* A page-locked allocation that fails is tried again without the blocks kept for reuse, of which at most
   256 MiB are. */
static int pinned() {
    const size_t MiB = 1u << 20;
    {
        PinnedBuf<char> b[4];
        for (auto &x : b) EXPECT(x.reserve(100 * MiB) == cudaSuccess);
    }
    EXPECT(fake::host.size() == 2);                       /* 200 of 400 MiB kept */
    fake::fail_host_allocs = 1;
    PinnedBuf<char> c, d;
    EXPECT(c.reserve(500 * MiB) == cudaSuccess && c.p && fake::host.size() == 1);
    fake::fail_host_allocs = 1;                           /* nothing left to give back */
    EXPECT(d.reserve(500 * MiB) == cudaErrorMemoryAllocation && !d.p);
    return 0;
}

/* Memory of one device released while another is current: its own device is waited for, and goes back to
   its own pool. */
static int other_device() {
    cudaSetDevice(2);
    PinnedBuf<char> h;
    DevBuf<char> b;
    EXPECT(h.reserve(1000) == cudaSuccess && b.reserve(1000) == cudaSuccess);
    cudaSetDevice(0);
    h.release();
    EXPECT(fake::synced.size() == 1 && fake::synced[0] == 2 && fake::device == 0);
    b.release();
    EXPECT(fake::synced.size() == 2 && fake::synced[1] == 2 && fake::device == 0);
    EXPECT(pt_release_memory() == PT_OK && pool(2).reserved == 0 && fake::device == 0);
    return 0;
}

/* A block whose device could not be waited for is not used again before a wait succeeds. */
static int refused_wait() {
    char *b0;
    {
        PinnedBuf<char> h;
        DevBuf<char> b;
        EXPECT(h.reserve(1000) == cudaSuccess && b.reserve(1000) == cudaSuccess);
        b0 = b.p;
        fake::refuse_device_sync = 2;
    }
    EXPECT(fake::host.empty());                           /* not kept */
    DevBuf<char> c, d;
    EXPECT(c.reserve(1000) == cudaSuccess && c.p != b0);
    EXPECT(pool().threshold == 4 * GiB + 2000);
    c.release();                                          /* waits, and frees b's block too */
    EXPECT(pool().threshold == 4 * GiB);
    EXPECT(d.reserve(1000) == cudaSuccess && (d.p == b0 || pool().blocks.size() == 2));
    d.release();
    {
        DevBuf<char> e;
        EXPECT(e.reserve(1000) == cudaSuccess);
        fake::refuse_device_sync = 1;
    }
    EXPECT(pt_release_memory() == PT_OK && pool().reserved == 0);
    return 0;
}

/* A worker thread's buffers come from the device that its caller works on. */
static int worker_device() {
    cudaSetDevice(3);
    DevBuf<char> b;
    int dev = -1;
    pt_device_thread([&] {
        cudaGetDevice(&dev);
        b.reserve(1000);
    }).join();
    EXPECT(dev == 3 && b.p && pool(3).reserved == 1000 && fake::pools.size() == 1);
    return 0;
}

/* Under a cap, live buffers and what is kept for reuse stay within it together. */
static int cap() {
    cudaStream_t st;
    cudaStreamCreateWithFlags(&st, 0);
    DevBuf<char> table;
    EXPECT(table.reserve(GiB) == cudaSuccess);
    build(st);
    EXPECT(pool().reserved == 3 * GiB + GiB / 2);
    limit = 2 * GiB;
    pt_dev_cap_changed();
    EXPECT(pool().reserved <= 2 * GiB);
    {
        DevBuf<char> a(st), b;
        EXPECT(a.reserve(GiB - 1) == cudaSuccess && pool().reserved <= 2 * GiB);
        EXPECT(b.reserve(2) == cudaErrorMemoryAllocation);
        a.release();
        EXPECT(b.reserve(GiB - 2) == cudaSuccess && pool().reserved <= 2 * GiB);
    }
    EXPECT(pool().reserved <= 2 * GiB);
    const int maps = fake::maps;
    { DevBuf<char> a; EXPECT(a.reserve(GiB - 2) == cudaSuccess); }      /* kept, and used again */
    EXPECT(fake::maps == maps);
    limit = -1;
    pt_dev_cap_changed();
    EXPECT(pool().threshold == GiB + 4 * GiB);
    return 0;
}

int main(int argc, char **argv) {
    const struct { const char *name; int (*run)(); } checks[] = {
        {"reuse_beside_live", reuse_beside_live}, {"bound", bound}, {"retry", retry}, {"pinned", pinned}, {"other_device", other_device},
        {"refused_wait", refused_wait}, {"worker_device", worker_device}, {"cap", cap},
    };
    for (const auto &c : checks)
        if (argc == 2 && !strcmp(argv[1], c.name)) return c.run();
    printf("unknown check\n");
    return 2;
}
