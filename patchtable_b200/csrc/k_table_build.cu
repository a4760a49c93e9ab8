/* The table's cells in one cooperative launch: fill, populate, resolve, seed, the propagation
   distance transform and fill_zeros.

   References (patchtable/patchtable.h):
     populate (fast, random order)  :3121-3159
     do_dt_prop                     :2081-2165  (edge labels PropEdge :1435-1447)
     fill_zeros                     :2063-2079

   Every CTA of the grid is resident at once (cudaLaunchCooperativeKernel), and the phases are
   separated by grid barriers whose waits are bounded: a CTA that polls longer than the process's
   spin limit (pt_set_spin_limit) records PT_TIMEOUT, and every CTA leaves at its next barrier, so
   the launch always ends and the host reports the status.

   Phases (one grid barrier after each):
     fill      every cell empty;
     populate  each allowed patch's cell takes the smallest shuffle rank that reaches it (the first
               visitor of the reference's random_shuffle order wins);
     resolve   ranks become packed positions; each CTA counts the seeded cells of its contiguous
               range of cells;
     seed      the seeded cells, in increasing cell order, become the first frontier (label 0):
               each CTA writes its range at the prefix of the counts before it;
     levels    the reference's breadth-first fill, level-synchronously: every frontier element
               claims the empty neighbours its label allows with an atomicMin on (element, edge),
               and the bits of the claims it holds are kept in its edge mask: an element toggles the
               bits it claims, and the bit of the holder it takes a cell from, so that after the
               phase the masks hold the winners (toggles commute).  Each CTA counts the bits of its
               contiguous range of elements; winners fill their cells and append (cell, label) to
               the next frontier at the scanned offsets, i.e. in (element, edge) order, which is the
               order of the reference's next frontier list.
   A filled cell holds its packed position (below 2^30), an empty one 0xffffffff, and a claimed one
   the claim's key, 2^30 + (element, edge), which its winner overwrites: the claims need no array of
   their own while every key fits, and a neighbour's one read says whether it is empty and
   whether an earlier element already holds it.
   The filled table is therefore bit-identical to the reference's.  Data written by other CTAs in
   an earlier phase is read with L2-only loads (ld.global.cg), never from a CTA's own L1. */
#include <cuda_runtime.h>
#include <cub/block/block_reduce.cuh>
#include <cub/block/block_scan.cuh>

#include <atomic>

#include "pt_bins.cuh"
#include "pt_internal.h"
#include "pt_kernels.h"

namespace {

constexpr int NT = 256;
constexpr int STAGE = 2048;                     /* new cells staged in shared memory at a time */
constexpr unsigned EMPTY = 0xffffffffu;
constexpr unsigned KEY_BASE = 1u << 30;         /* smallest claim key: packed positions lie below */
constexpr long long KEY_ELEMENTS = 1ll << 27;   /* separate claims: key = element << 5 | edge */

struct CellBuild {
    int G;
    float min_val[PT_DESC_MAX], range[PT_DESC_MAX];
    long long stride[PT_DESC_MAX];
    int nslices[PT_DESC_MAX];
    const float *desc;
    int ds;
    int ew;
    long long np;                /* entries of order_xy */
    const int *to_bin;
    const int *order_xy;         /* packed position of each shuffle rank */
    unsigned *table;
    long long ncells;
    unsigned *claim;             /* the table itself while the keys fit, or one key per cell */
    unsigned key_base;
    int ebits;                   /* edge bits of a key */
    unsigned div_mul[PT_DESC_MAX];   /* division by nslices: floor(x / n) = umulhi(x, mul) >> shift for x < 2^31 */
    int div_shift[PT_DESC_MAX];
    int *fidx[2];
    unsigned char *flab[2];
    unsigned *emask[2];          /* per frontier element: the edges whose claims it holds */
    long long *ctot;             /* per-CTA totals */
    unsigned *bar;               /* [0] arrivals, [1] generation */
    int *status;                 /* [0] pt_status of the launch, [1] levels, [2] phase that failed */
    long long *seeded;
    int run_dt, dt_iters, fill_zeros, vfill;
    long long spin_limit;
};

/* Grid barrier with a bounded wait.  Returns false once any CTA has recorded an error. */
__device__ __forceinline__ bool grid_barrier(const CellBuild &a, int phase) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned *vgen = a.bar + 1;
        volatile int *vstatus = a.status;
        int ok = 1;
        const unsigned gen = *vgen;            /* read before arriving: it cannot move until we do */
        __threadfence();
        if (atomicAdd(a.bar, 1u) == gridDim.x - 1) {
            atomicExch(a.bar, 0u);
            __threadfence();
            atomicAdd(a.bar + 1, 1u);
        } else {
            long long polls = 0;
            while (*vgen == gen) {
                if (*vstatus != 0) { ok = 0; break; }
                if (++polls > a.spin_limit) {
                    if (atomicCAS(a.status, 0, (int) PT_TIMEOUT) == 0) a.status[2] = phase;
                    ok = 0;
                    break;
                }
                __nanosleep(128);
            }
        }
        __threadfence();
        if (*vstatus != 0) ok = 0;
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

typedef cub::BlockReduce<long long, NT> Reduce;
typedef cub::BlockScan<int, NT> Scan;

union Shared {
    typename Reduce::TempStorage reduce;
    typename Scan::TempStorage scan;
};

/* Sum of a value over the CTA (every thread receives it). */
__device__ __forceinline__ long long cta_sum(Shared &sh, long long v) {
    __shared__ long long s_sum;
    __syncthreads();
    const long long t = Reduce(sh.reduce).Sum(v);
    if (threadIdx.x == 0) s_sum = t;
    __syncthreads();
    return s_sum;
}

/* Prefix of the per-CTA totals before this CTA, and their sum. */
__device__ __forceinline__ void cta_prefix(Shared &sh, const CellBuild &a, long long &before, long long &total) {
    long long b = 0, t = 0;
    for (int k = threadIdx.x; k < (int) gridDim.x; k += NT) {
        const long long v = __ldcg(a.ctot + k);
        t += v;
        if (k < (int) blockIdx.x) b += v;
    }
    before = cta_sum(sh, b);
    total = cta_sum(sh, t);
}

/* Edge e of label lab (patchtable.h:2101-2120): label 0 -> (i, -1), (i, +1) for every dimension i;
   label 2i + 1 + (dir + 1) / 2 -> (i, dir), then (j, -1), (j, +1) for every j > i.  The label the
   filled cell receives is that of the edge's own (dimension, direction). */
__device__ __forceinline__ void edge_of(int lab, int e, int &dim, int &dir) {
    if (lab == 0) { dim = e >> 1; dir = (e & 1) ? 1 : -1; return; }
    const int i = (lab - 1) >> 1;
    if (e == 0) { dim = i; dir = ((lab - 1) & 1) ? 1 : -1; return; }
    dim = i + 1 + ((e - 1) >> 1);
    dir = ((e - 1) & 1) ? 1 : -1;
}

/* x / nslices[d] for x < 2^31. */
__device__ __forceinline__ unsigned div_slices(const CellBuild &a, int d, unsigned x) {
    return a.div_mul[d] ? __umulhi(x, a.div_mul[d]) >> a.div_shift[d] : x;
}

/* The claims of frontier element i (cell g, label lab): all its neighbours are read before the first
   claim, so an element waits for memory twice, not once per edge. */
template<int MAXG>
__device__ __forceinline__ void claim_neighbours(const CellBuild &a, unsigned *emask, unsigned i, unsigned g, int lab) {
    const int li = lab == 0 ? -1 : (lab - 1) >> 1, lp = (lab - 1) & 1;
    unsigned v[2 * MAXG];
    unsigned r = g;
#pragma unroll
    for (int d = MAXG - 1; d >= 0; d--) {
        v[2 * d] = v[2 * d + 1] = 0;
        if (d < a.G) {
            const unsigned q = div_slices(a, d, r), dig = r - q * (unsigned) a.nslices[d], st = (unsigned) a.stride[d];
            r = q;
            if (dig > 0 && (d > li || (d == li && !lp))) v[2 * d] = __ldcg(a.table + (g - st));
            if (dig + 1 < (unsigned) a.nslices[d] && (d > li || (d == li && lp))) v[2 * d + 1] = __ldcg(a.table + (g + st));
        }
    }
    const unsigned key0 = a.key_base + (i << a.ebits);
    unsigned old[2 * MAXG];
#pragma unroll
    for (int k = 0; k < 2 * MAXG; k++) {
        const int d = k >> 1;
        const unsigned e = lab == 0 ? k : d == li ? 0 : 2 * (d - li) - 1 + (k & 1);
        old[k] = 0;
        if (v[k] >= KEY_BASE && (a.claim != a.table || key0 + e < v[k]))
            old[k] = atomicMin(a.claim + ((k & 1) ? g + (unsigned) a.stride[d] : g - (unsigned) a.stride[d]), key0 + e);
    }
    unsigned won = 0;
#pragma unroll
    for (int k = 0; k < 2 * MAXG; k++) {
        const int d = k >> 1;
        const unsigned e = lab == 0 ? k : d == li ? 0 : 2 * (d - li) - 1 + (k & 1);
        if (old[k] > key0 + e) {
            won |= 1u << e;
            if (old[k] != EMPTY) {
                const unsigned o = old[k] - a.key_base;
                atomicXor(emask + (o >> a.ebits), 1u << (o & ((1u << a.ebits) - 1)));
            }
        }
    }
    if (won) atomicXor(emask + i, won);
}

/* Bound: the latency of the levels' random accesses (98 M elements over 25 levels in a 1920x1080
   table).  6.4 ms there, of which claims 2.9, counts 0.16, emission 2.8 and the rest 0.5 ms; 14.8 ms
   (6.5, 4.2, 3.2, 0.9) with claims in an array of their own, one dependent read per edge with 64-bit
   divisions, a count phase that read every claim again and lists written a thread's run at a time.
   Claims unrolled over 8 dimensions instead of 6 take 3.2 ms; a register cap of 5 CTAs per SM (3 fit
   as compiled, 80 registers) changes nothing, one of 6 makes the whole build 7.3. */
template<int MAXG>
__global__ void __launch_bounds__(NT) k_table_build(const CellBuild a) {
    __shared__ Shared sh;
    __shared__ int st_cell[STAGE];
    __shared__ unsigned st_val[STAGE];
    __shared__ unsigned char st_lab[STAGE];
    const long long nthr = (long long) gridDim.x * NT;
    const long long tid = (long long) blockIdx.x * NT + threadIdx.x;

    /* fill */
    for (long long i = tid; i < a.ncells; i += nthr) {
        a.table[i] = EMPTY;
        if (a.run_dt && a.claim != a.table) a.claim[i] = EMPTY;
    }
    if (!grid_barrier(a, 0)) return;

    /* populate: first visitor in shuffled order wins (patchtable.h:3142-3154) */
    for (long long r = tid; r < a.np; r += nthr) {
        const int xy = __ldg(a.order_xy + r);
        const long long p = (long long) (pt_y(xy) - 7) * a.ew + (pt_x(xy) - 7);
        const float *v = a.desc + p * a.ds;
        long long cell = 0;
        for (int d = 0; d < a.G; d++)
            cell += (long long) pt_get_bin(a.min_val[d], a.range[d], a.to_bin + d * PT_NMAP, __ldg(v + d)) * a.stride[d];
        atomicMin(a.table + cell, (unsigned) r);
    }
    if (!grid_barrier(a, 1)) return;

    /* resolve: ranks -> packed positions; seeded cells of this CTA's range */
    const long long chunk = ((a.ncells + gridDim.x - 1) / gridDim.x + 3) & ~3ll;
    const long long c0 = min(a.ncells, (long long) blockIdx.x * chunk), c1 = min(a.ncells, c0 + chunk);
    {
        long long local = 0;
        for (long long j = c0 + threadIdx.x; j < c1; j += NT) {
            const unsigned v = __ldcg(a.table + j);
            if (v != EMPTY) { a.table[j] = (unsigned) __ldg(a.order_xy + v); local++; }
        }
        const long long s = cta_sum(sh, local);
        if (threadIdx.x == 0) a.ctot[blockIdx.x] = s;
    }
    if (!grid_barrier(a, 2)) return;

    long long before, n;
    cta_prefix(sh, a, before, n);
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.seeded = n;
    int levels = 0;
    if (a.run_dt) {
        /* seed: the first frontier in increasing cell order, label 0 (patchtable.h:2087-2093) */
        long long o = before;
        for (long long j0 = c0; j0 < c1; j0 += 4 * NT) {
            const long long j = j0 + 4 * threadIdx.x;
            unsigned f = 0;
            if (j < c1) {
                const uint4 v = __ldcg(reinterpret_cast<const uint4 *>(a.table + j));
                f = (v.x != EMPTY ? 1u : 0u) | (v.y != EMPTY ? 2u : 0u) | (v.z != EMPTY ? 4u : 0u) | (v.w != EMPTY ? 8u : 0u);
                if (j + 4 > c1) f &= (1u << (c1 - j)) - 1;
            }
            int off, tot;
            __syncthreads();
            Scan(sh.scan).ExclusiveSum(__popc(f), off, tot);
            long long w = o + off;
            while (f) {
                const int k = __ffs(f) - 1;
                f &= f - 1;
                a.fidx[0][w] = (int) (j + k);
                a.flab[0][w] = 0;
                a.emask[0][w] = 0;
                w++;
            }
            o += tot;
        }
        if (!grid_barrier(a, 3)) return;
        int cur = 0;
        for (int iter = 0;; iter++) {
            if (a.dt_iters > 0 && iter > a.dt_iters) break;
            if (n == 0) break;
            if (a.claim != a.table && n >= KEY_ELEMENTS) {
                if (blockIdx.x == 0 && threadIdx.x == 0 && atomicCAS(a.status, 0, (int) PT_UNSUPPORTED) == 0) a.status[2] = 4;
                return;
            }
            const int *fi = a.fidx[cur];
            const unsigned char *fl = a.flab[cur];
            unsigned *em = a.emask[cur];
            /* claim: the smallest (element, edge) key wins each empty neighbour (:2131-2156) */
            for (long long i = tid; i < n; i += nthr)
                claim_neighbours<MAXG>(a, em, (unsigned) i, (unsigned) __ldcg(fi + i), __ldcg(fl + i));
            if (!grid_barrier(a, 5)) return;
            /* count the claims won in this CTA's range of elements */
            const long long ech = ((n + gridDim.x - 1) / gridDim.x + 3) & ~3ll;
            const long long e0 = min(n, (long long) blockIdx.x * ech), e1 = min(n, e0 + ech);
            {
                long long local = 0;
                for (long long i = e0 + 4 * threadIdx.x; i < e1; i += 4 * NT) {
                    const uint4 w = __ldcg(reinterpret_cast<const uint4 *>(em + i));
                    local += __popc(w.x) + (i + 1 < e1 ? __popc(w.y) : 0) + (i + 2 < e1 ? __popc(w.z) : 0) +
                             (i + 3 < e1 ? __popc(w.w) : 0);
                }
                const long long s = cta_sum(sh, local);
                if (threadIdx.x == 0) a.ctot[blockIdx.x] = s;
            }
            if (!grid_barrier(a, 6)) return;
            long long base, next;
            cta_prefix(sh, a, base, next);
            /* emit: winners fill their cells and append to the next frontier in (element, edge)
               order, four consecutive elements per thread */
            int *nfi = a.fidx[1 - cur];
            unsigned char *nfl = a.flab[1 - cur];
            unsigned *nem = a.emask[1 - cur];
            long long o2 = base;
            for (long long t0 = e0; t0 < e1; t0 += 4 * NT) {
                const long long i = t0 + 4 * threadIdx.x;
                unsigned won[4] = {0, 0, 0, 0};
                int g[4] = {0, 0, 0, 0}, lab[4] = {0, 0, 0, 0};
                unsigned val[4] = {0, 0, 0, 0};
                if (i < e1) {
                    const uint4 w = __ldcg(reinterpret_cast<const uint4 *>(em + i));
                    const int4 gi = __ldcg(reinterpret_cast<const int4 *>(fi + i));
                    const uchar4 li = __ldcg(reinterpret_cast<const uchar4 *>(fl + i));
                    won[0] = w.x; won[1] = w.y; won[2] = w.z; won[3] = w.w;
                    g[0] = gi.x; g[1] = gi.y; g[2] = gi.z; g[3] = gi.w;
                    lab[0] = li.x; lab[1] = li.y; lab[2] = li.z; lab[3] = li.w;
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        if (i + k >= e1) won[k] = 0;
                        if (won[k]) val[k] = __ldcg(a.table + g[k]);
                    }
                }
                int off, tot;
                __syncthreads();
                Scan(sh.scan).ExclusiveSum(__popc(won[0]) + __popc(won[1]) + __popc(won[2]) + __popc(won[3]), off, tot);
                /* the tile's new cells in order, through shared memory, so that the lists are written
                   in whole lines */
                for (int r0 = 0; r0 < tot; r0 += STAGE) {
                    int w = off - r0;
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        unsigned m = won[k];
                        while (m) {
                            const int e = __ffs(m) - 1;
                            m &= m - 1;
                            if (w >= 0 && w < STAGE) {
                                int dim, dir;
                                edge_of(lab[k], e, dim, dir);
                                st_cell[w] = g[k] + dir * (int) a.stride[dim];
                                st_val[w] = val[k];
                                st_lab[w] = (unsigned char) (2 * dim + 1 + (dir + 1) / 2);
                            }
                            w++;
                        }
                    }
                    __syncthreads();
                    const int cnt = min(STAGE, tot - r0);
                    for (int j = threadIdx.x; j < cnt; j += NT) {
                        const long long o = o2 + r0 + j;
                        const int gp = st_cell[j];
                        a.table[gp] = st_val[j];
                        nfi[o] = gp;
                        nfl[o] = st_lab[j];
                        nem[o] = 0;
                    }
                    __syncthreads();
                }
                o2 += tot;
            }
            n = next;
            cur = 1 - cur;
            levels++;
            if (!grid_barrier(a, 7)) return;
        }
    }
    /* cells no patch reached: fill_zeros' value (patchtable.h:2063-2079) or TABLE_UNUSED */
    const unsigned rest = a.fill_zeros ? (unsigned) a.vfill : (unsigned) PT_UNUSED;
    for (long long i = tid; i < a.ncells; i += nthr)
        if (__ldcg(a.table + i) == EMPTY) a.table[i] = rest;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.status[1] = levels;
}

std::atomic<long long> g_spin_limit{1ll << 24};

}  // namespace

long long pt_spin_limit() { return g_spin_limit.load(); }

extern "C" int64_t pt_set_spin_limit(int64_t polls) {
    if (polls < 0) polls = 1ll << 24;
    return g_spin_limit.exchange(polls);
}

pt_status pt_build_cells(const PtBins &bins, const int *nslices, const float *desc, int ds, int ew, long long np,
                         const int *to_bin, const int *order_xy, int *table, long long ncells, int run_dt, int dt_iters,
                         int fill_zeros, int vfill, long long *seeded, int *levels, cudaStream_t st) {
    if (ncells >= (1ll << 31)) return pt_fail(PT_UNSUPPORTED, "tables above 2^31 cells are not supported");
    if (bins.G < 1 || bins.G > PT_DESC_MAX) return pt_fail(PT_UNSUPPORTED, "grid dims %d", bins.G);
    int dev = 0, coop = 0, nsm = 0, per = 0;
    PT_CUDA(cudaGetDevice(&dev));
    PT_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) return pt_fail(PT_UNSUPPORTED, "the table build needs cooperative launches");
    PT_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const void *kernel = bins.G <= 6 ? (const void *) k_table_build<6>
                         : bins.G <= 8 ? (const void *) k_table_build<8> : (const void *) k_table_build<PT_DESC_MAX>;
    PT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, NT, 0));
    if (per < 1) return pt_fail(PT_CUDA_ERR, "the table build kernel cannot be resident");
    const int grid = nsm * per;

    CellBuild a;
    memset(&a, 0, sizeof(a));
    a.G = bins.G;
    for (int d = 0; d < bins.G; d++) {
        a.min_val[d] = bins.min_val[d];
        a.range[d] = bins.range[d];
        a.stride[d] = bins.stride[d];
        a.nslices[d] = nslices[d];
    }
    a.desc = desc; a.ds = ds; a.ew = ew; a.np = np; a.to_bin = to_bin; a.order_xy = order_xy;
    a.table = reinterpret_cast<unsigned *>(table); a.ncells = ncells;
    for (int d = 0; d < bins.G; d++) {
        /* ceil(2^(31 + l) / n) with 2^(l-1) < n <= 2^l: exact for dividends below 2^31 */
        int l = 1;
        while ((1ll << l) < nslices[d]) l++;
        a.div_mul[d] = nslices[d] > 1 ? (unsigned) (((1ull << (31 + l)) + nslices[d] - 1) / nslices[d]) : 0;
        a.div_shift[d] = l - 1;
    }
    /* claim keys share the table's words while 2^30 + (element, edge) stays below 2^32 for every
       possible element; otherwise they get an array of their own */
    a.ebits = bins.G <= 8 ? 4 : 5;
    const bool fused = ncells <= (long long) ((EMPTY - KEY_BASE) >> a.ebits);
    a.key_base = fused ? KEY_BASE : 0;
    if (!fused) a.ebits = 5;
    a.run_dt = run_dt; a.dt_iters = dt_iters; a.fill_zeros = fill_zeros; a.vfill = vfill;
    a.spin_limit = pt_spin_limit();
    /* Scratch: two frontiers of at most one element per cell, and the claim keys that do not share the
       table's words. */
    DevBuf<unsigned> claim(st);
    DevBuf<int> fidx0(st), fidx1(st), status(st);
    DevBuf<unsigned char> flab0(st), flab1(st);
    DevBuf<unsigned> emask0(st), emask1(st);
    DevBuf<long long> ctot(st), seed_n(st);
    DevBuf<unsigned> bar(st);
    if (run_dt) {
        if (!fused) PT_CUDA(claim.reserve(ncells));
        PT_CUDA(fidx0.reserve(ncells + 4)); PT_CUDA(fidx1.reserve(ncells + 4));
        PT_CUDA(flab0.reserve(ncells + 4)); PT_CUDA(flab1.reserve(ncells + 4));
        PT_CUDA(emask0.reserve(ncells + 4)); PT_CUDA(emask1.reserve(ncells + 4));
    }
    PT_CUDA(ctot.reserve(grid));
    PT_CUDA(seed_n.reserve(1));
    PT_CUDA(bar.reserve(2));
    PT_CUDA(status.reserve(4));
    PT_CUDA(cudaMemsetAsync(bar.p, 0, 2 * sizeof(unsigned), st));
    PT_CUDA(cudaMemsetAsync(status.p, 0, 4 * sizeof(int), st));
    a.claim = fused ? a.table : claim.p;
    a.fidx[0] = fidx0.p; a.fidx[1] = fidx1.p;
    a.flab[0] = flab0.p; a.flab[1] = flab1.p;
    a.emask[0] = emask0.p; a.emask[1] = emask1.p;
    a.ctot = ctot.p;
    a.bar = bar.p;
    a.status = status.p;
    a.seeded = seed_n.p;
    void *args[] = {&a};
    PT_CUDA(cudaLaunchCooperativeKernel(kernel, grid, NT, args, 0, st));
    PT_LAUNCHED();
    int hs[4] = {0, 0, 0, 0};
    long long hn = 0;
    PT_CUDA(cudaMemcpyAsync(hs, status.p, sizeof(hs), cudaMemcpyDeviceToHost, st));
    PT_CUDA(cudaMemcpyAsync(&hn, seed_n.p, sizeof(hn), cudaMemcpyDeviceToHost, st));
    PT_CUDA(cudaStreamSynchronize(st));
    if (hs[0] == PT_TIMEOUT)
        return pt_fail(PT_TIMEOUT, "table build: a grid barrier wait gave up after %lld polls (phase %d)", a.spin_limit, hs[2]);
    if (hs[0] != 0) return pt_fail((pt_status) hs[0], "table build: a DT frontier reached 2^27 elements");
    if (seeded) *seeded = hn;
    if (levels) *levels = hs[1];
    return PT_OK;
}
