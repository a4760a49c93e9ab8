/* Batched queries: the choose and the pull of many images in one persistent launch each. */
#include "k_query.cuh"

namespace {

/* ---- batched queries: many images, one launch per phase over a flattened tile list ---- */

/* Index of the image that owns flattened tile s (segs[i] = first tile of image i). */
__device__ __forceinline__ int owner(const PtBatchImage *__restrict__ imgs, int n, long long s, int twi) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&imgs[mid].seg_off[twi]) <= s) lo = mid; else hi = mid - 1;
    }
    return lo;
}

/* Runs body(s) for the tiles this CTA takes from the launch's work counter (zeroed before
   the launch): tiles go out in order, one at a time, to whichever CTA is free, so uneven
   tile costs cannot leave some CTAs with a longer share.  A CTA claims its next tile when it
   starts the current one and reads the claim only after it, so the counter's round trip overlaps
   the work. */
template<class Body>
__device__ __forceinline__ void for_each_tile(unsigned long long *work, long long nseg, Body &&body) {
    __shared__ long long s_next;
    if (threadIdx.x == 0) s_next = (long long) atomicAdd(work, 1ull);
    __syncthreads();
    long long s = s_next;
    while (s < nseg) {
        long long claim = 0;
        if (threadIdx.x == 0) claim = (long long) atomicAdd(work, 1ull);
        body(s);
        __syncthreads();                       /* every thread is done with s_next and the staged tile */
        if (threadIdx.x == 0) s_next = claim;
        __syncthreads();
        s = s_next;
    }
}

/* Persistent choose over every tile of every image, handed out by a work counter. */
template<int TP, bool LEAN = false>
__global__ void __launch_bounds__(TP, min_ctas(LEAN ? CHOOSE_LEAN_LANES : CHOOSE_LANES, TP))
k_choose_batch(const QPlan base, const PtBatchImage *__restrict__ imgs, int n, long long nseg, int twi,
               const float *__restrict__ a, const int *cur_pos,
               const float *cur_d, const int *tcand, const int2 *__restrict__ kcoh, int do_table,
               int *ch_pos, float *ch_d, int *kc_done, int use_done, unsigned long long *work) {
    extern __shared__ float at[];
    LearnedArgs none;
    none.cand = nullptr; none.conf = nullptr; none.threshold = 0.f; none.kcoh_confident = 0; none.counters = nullptr;
    for_each_tile(work, nseg, [&](long long s) {
        const int i = owner(imgs, n, s, twi);
        const PtBatchImage &g = imgs[i];
        const int ls = (int) (s - g.seg_off[twi]);
        const int spr = (g.ew + tile_w(TP) - 1) / tile_w(TP);
        QPlan q = base;
        q.aw = g.w; q.ah = g.h; q.ew = g.ew; q.eh = g.eh;
        const long long o = g.patch_off;
        choose_tile<TP, false, LEAN>(q, at, a + 3 * g.pix_off, cur_pos ? cur_pos + o : nullptr,
                                            cur_d ? cur_d + o : nullptr, tcand + o, kcoh, do_table, ch_pos + o, ch_d + o,
                                            kc_done + o, use_done, nullptr, none, (ls % spr) * tile_w(TP),
                                            (ls / spr) * tile_h(TP), g.eh);
    });
}

template<int TP, int R, bool ONE = false, bool NX = false>
__global__ void __launch_bounds__(TP, min_ctas(ONE ? PULL_ONE_LANES : PULL_LANES, TP))
k_pull_batch(const QPlan base, const PtBatchImage *__restrict__ imgs, int n, long long nseg, int twi,
             const float *__restrict__ a, const int *cur_pos,
             const float *cur_d, const int *ch_pos, const float *ch_d,
             int *nxt_pos, float *nxt_d, unsigned long long *work) {
    extern __shared__ float at[];
    for_each_tile(work, nseg, [&](long long s) {
        const int i = owner(imgs, n, s, twi);
        const PtBatchImage &g = imgs[i];
        const int ls = (int) (s - g.seg_off[twi]);
        const int spr = (g.ew + tile_w(TP) - 1) / tile_w(TP);
        QPlan q = base;
        q.aw = g.w; q.ah = g.h; q.ew = g.ew; q.eh = g.eh;
        const long long o = g.patch_off;
        if (base.ann) q.ann = base.ann + 3 * o;        /* last pass: this image's NNF records */
        if (base.nx.ch_pos) { q.nx.ch_pos += o; q.nx.ch_d += o; q.nx.kc_done += o; }
        pull_tile<TP, R, false, ONE, NX>(q, at, a + 3 * g.pix_off, cur_pos ? cur_pos + o : nullptr,
                                     cur_d ? cur_d + o : nullptr, ch_pos + o, ch_d + o, nxt_pos + o, nxt_d + o, nullptr,
                                     (ls % spr) * tile_w(TP), (ls / spr) * tile_h(TP), g.eh);
    });
}

}  // namespace

/* ---- batched launchers ---- */

namespace {

constexpr int BATCH_TW[PT_BATCH_NTW] = {32, 64, 128, 256};

template<class K>
int persistent_grid(K kernel, int threads, size_t smem, long long work) {
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem) != cudaSuccess || per < 1) per = 1;
    const long long g = (long long) per * sm_count();
    return (int) (work < g ? work : g);
}

}  // namespace

int pt_batch_tw(int twi) { return (twi >= 0 && twi < PT_BATCH_NTW) ? BATCH_TW[twi] : 0; }

long long pt_batch_tiles(int twi, int ew, int eh) {
    const int tp = pt_batch_tw(twi);
    return (long long) ((ew + tile_w(tp) - 1) / tile_w(tp)) * ((eh + tile_h(tp) - 1) / tile_h(tp));
}

pt_status pt_launch_choose_batch(const QuerySetup &s, const PtBatchImage *imgs, int n, long long nseg, int twi,
                                 const float *a, const int *cur_pos, const float *cur_d,
                                 const int *tcand, const int2 *kcoh, int do_table, int *ch_pos, float *ch_d, int *kc_done,
                                 int use_done, unsigned long long *work, cudaStream_t st) {
    QPlan q;
    PT_TRY(make_qplan(s, q));
    if (nseg <= 0) return PT_OK;
    PT_CUDA(cudaMemsetAsync(work, 0, sizeof(unsigned long long), st));
#define PT_CHOOSE_B(T) { const size_t sm = atile_bytes(T); \
        if (lean) { const int g = persistent_grid(k_choose_batch<T, true>, T, sm, nseg); \
            k_choose_batch<T, true><<<g, T, sm, st>>>(q, imgs, n, nseg, twi, a, cur_pos, cur_d, tcand, kcoh, do_table, \
                                                      ch_pos, ch_d, kc_done, use_done, work); } \
        else { const int g = persistent_grid(k_choose_batch<T>, T, sm, nseg); \
            k_choose_batch<T><<<g, T, sm, st>>>(q, imgs, n, nseg, twi, a, cur_pos, cur_d, tcand, kcoh, do_table, ch_pos, \
                                                ch_d, kc_done, use_done, work); } }
    const bool lean = lean_choose(q);
    switch (BATCH_TW[twi]) {
        case 32: PT_CHOOSE_B(32) break;
        case 64: PT_CHOOSE_B(64) break;
        case 128: PT_CHOOSE_B(128) break;
        default: PT_CHOOSE_B(256) break;
    }
#undef PT_CHOOSE_B
    PT_LAUNCHED();
    return PT_OK;
}

pt_status pt_launch_pull_batch(const QuerySetup &s, const PtBatchImage *imgs, int n, long long nseg, int twi,
                               const float *a, const int *cur_pos, const float *cur_d, const int *ch_pos,
                               const float *ch_d, int *nxt_pos, float *nxt_d, unsigned long long *work,
                               cudaStream_t st) {
    QPlan q;
    PT_TRY(make_qplan(s, q));
    if (nseg <= 0) return PT_OK;
    PT_CUDA(cudaMemsetAsync(work, 0, sizeof(unsigned long long), st));
#define PT_PULL_B(T, RR) { const size_t sm = atile_bytes(T); \
        if (one) { const int g = persistent_grid(k_pull_batch<T, RR, true>, T, sm, nseg); \
            k_pull_batch<T, RR, true><<<g, T, sm, st>>>(q, imgs, n, nseg, twi, a, cur_pos, cur_d, ch_pos, ch_d, nxt_pos, \
                                                        nxt_d, work); } \
        else if (q.nx.ch_pos) { const int g = persistent_grid(k_pull_batch<T, RR, false, true>, T, sm, nseg); \
            k_pull_batch<T, RR, false, true><<<g, T, sm, st>>>(q, imgs, n, nseg, twi, a, cur_pos, cur_d, ch_pos, ch_d, \
                                                               nxt_pos, nxt_d, work); } \
        else { const int g = persistent_grid(k_pull_batch<T, RR>, T, sm, nseg); \
            k_pull_batch<T, RR><<<g, T, sm, st>>>(q, imgs, n, nseg, twi, a, cur_pos, cur_d, ch_pos, ch_d, nxt_pos, nxt_d, \
                                                  work); } }
    const bool one = one_pull(q) && !q.nx.ch_pos;
    const bool r1 = q.radius <= 1;
    switch (BATCH_TW[twi]) {
        case 32: if (r1) PT_PULL_B(32, 1) else PT_PULL_B(32, 2) break;
        case 64: if (r1) PT_PULL_B(64, 1) else PT_PULL_B(64, 2) break;
        case 128: if (r1) PT_PULL_B(128, 1) else PT_PULL_B(128, 2) break;
        default: if (r1) PT_PULL_B(256, 1) else PT_PULL_B(256, 2) break;
    }
#undef PT_PULL_B
    PT_LAUNCHED();
    return PT_OK;
}
