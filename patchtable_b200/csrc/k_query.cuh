/* Query kernels: nearest-neighbour field from image a to the table image b.

   Replaces lookup_templated<0,0> (patchtable/patchtable.h:3468-4217).  The reference sweeps the
   patches in scanline order (reversed on odd iterations); at each patch it
     1. starts from the stored match with its distance scaled by prop_scale = 1/(1+coherence_spatial),
     2. tries the table cell of the patch's descriptor on the first iteration (:3641-3709),
     3. tries the k-coherence neighbours of the current best, stopping once the stored
        distance of a neighbour reaches triangle_factor * best (:3750-3851),
     4. pushes the chosen offset to the 3x3 neighbourhood, replacing a neighbour's match when the
        pushed patch is closer (summed-area-table propagation, :3908-4145).
   Here every patch runs steps 1-3 at once ("choose"), then every patch takes the best of the
   offsets its neighbours chose ("pull", the mirror image of the push), and the pair of phases
   repeats for a fixed number of passes.  All distances are the reference's patch_dist_exact
   (patchtable.h:330-373) evaluated in the same float order, so every returned NNF_DIST is that
   function's value for the returned match; a candidate's sum stops early once its partial sum
   already reaches the value it must beat (the partial sum can only grow). */
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstring>

#include "pt_internal.h"
#include "pt_descdist.cuh"
#include "pt_kernels.h"

/* This header holds what the query kernels share.  They are compiled in four files, so that a program
   loads the code it runs: k_query.cu (single images at the default width), k_query_tiles.cu (the other
   widths, learned proposals), k_query_desc.cu (descriptor mode) and k_query_batch.cu.  Code is loaded when
   its first kernel is launched: the first build and lookup of a process (60 x 80) take 21 ms, and 46 with
   all of them in one file. */

/* SMs of the current device, asked once. */
inline int sm_count() {
    static std::atomic<int> n{0};
    int v = n.load(std::memory_order_relaxed);
    if (!v) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v < 1) v = 148;
        n.store(v, std::memory_order_relaxed);
    }
    return v;
}

bool pt_lean_kernels();                   /* pt_set_lean_kernels */

namespace {

constexpr int NT = 256;

/* The next pass's choose, done by the pull for the match it has just found (ch_pos NULL: none). */
struct NextChoose {
    const int2 *kcoh;
    int *kc_done;
    int use_done, do_kcoh, pass;
    int *ch_pos;
    float *ch_d;
};

struct QPlan {
    NextChoose nx;
    int aw, ah;              /* a image size (pixels) */
    int ew, eh;              /* a patches */
    int bw, bh;              /* b image size */
    int bew, beh;            /* b patches */
    double prop_scale;
    double triangle;
    int kc, ks;              /* kcoherence (entries per cell), kcoherence_step */
    int kc_try;              /* entries tried per patch (<= kc) */
    int radius;              /* query_step + prop_dist */
    int do_kcoh;
    int step;                /* neighbour spacing of this pull pass (jump flooding) */
    int pull_max;            /* most neighbour candidates scored per patch */
    int tile;                /* query patches per CTA (single-image launches) */
    int auto_tile;           /* no width was asked for */
    int row0, rows;          /* patch rows of a single-image launch */
    const float *brow;       /* row store of the table image (k_row_store) */
    int nline;               /* its lines per image row */
    const int *allowed;      /* b patches that may be matched (allowed[p] == allowed_index), or NULL */
    int allowed_index;
    const float4 *adesc;     /* descriptor mode: query descriptor store (ds4 float4 per patch), or NULL */
    const float4 *bdesc;     /* descriptor mode: table descriptor store */
    int ds4, nd;             /* float4 per store entry, descriptor dimensions */
    const int *tcand_more;   /* further tables' entries, [table][patch] (ntables > 1), or NULL */
    int ntc;
    int spatial, do_rs, pass; /* spatial search radius, random search, pass index (its seed) */
    double *ann;             /* last pull: the float64 NNF written directly, or NULL */
};

/* lowbias32 integer hash (C. Wellons' published constants): the random search's choice of
   neighbour for a patch in a pass, in place of the reference's sequential rand() stream. */
__device__ __forceinline__ unsigned mix32(unsigned x) {
    x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
    return x;
}

/* Programmatic dependent launch: a query's kernels let the next one start as soon as all their CTAs run
   (pdl_trigger), and wait for the ones before them to end (pdl_wait) before they read anything.  Every
   CTA waits, so a kernel never ends before its predecessors.  What a predecessor may still be writing
   when the kernel starts -- table entries, states and choices -- is not read-only for the kernel's
   life: those pointers carry no __restrict__, which would allow non-coherent loads. */
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ float finf() { return __int_as_float(0x7f800000); }

/* Adds per-thread counts to counters[0..1] with one atomic per warp (profiling only). */
__device__ __forceinline__ void count_work(unsigned long long *counters, unsigned cand, unsigned rows) {
    if (!counters) return;
    unsigned c = __reduce_add_sync(0xffffffffu, cand), r = __reduce_add_sync(0xffffffffu, rows);
    if ((threadIdx.x & 31) == 0) { atomicAdd(counters, (unsigned long long) c); atomicAdd(counters + 1, (unsigned long long) r); }
}

/* Threads per SM the register caps leave room for, and the rows a choose keeps in flight.  The kernels
   wait on gathers from L2: more resident warps pay until the row buffers spill.  Measured at 1080p,
   128 patches per CTA, in ms: lean choose at 16 / 18 / 20 / 22 x 64 threads per SM 0.152 / 0.154 / 0.150 /
   0.160, one-candidate pull at 14 / 16 / 18 / 20 0.195 / 0.182 / 0.182 / 0.191, the default schedule's
   four pulls at 10 / 12 / 14 / 16 2.83 / 2.78 / 2.87 / 2.83, its chooses at 8 / 10 / 12 / 14 0.80 / 0.85 /
   0.88 / 0.85, and 0.785 at 8 with two rows in flight. */
constexpr int CHOOSE_LANES = 8 * 64, CHOOSE_LEAN_LANES = 20 * 64, PULL_LANES = 12 * 64, PULL_ONE_LANES = 16 * 64;
constexpr int CHOOSE_D = 2;
/* Warps that share one 8 x 4 tile's candidate lists in the pull of a small image, and how many tiles
   per SM still are one (k_pull_tile's launcher). */
constexpr int SPLIT_W = 4, SPLIT_D = 4, SPLIT_TILES = 4;
constexpr int min_ctas(int lanes, int tp) { return lanes / tp < 32 ? lanes / tp : 32; }

/* A CTA covers TP query patches: warps of 8 x 4 patches (8 columns, 4 rows; lane l is the patch
   at column l / 4, row l % 4), side by side and stacked to the tile below.  A square-ish tile
   keeps the candidate rows that neighbouring patches share in the SM's L1, and four lanes that
   work on one patch find the patches of their four rounds in the same image columns. */
constexpr int WTW = 8, WTH = 4;           /* query patches per warp: columns, rows */
constexpr int TILE_DEFAULT = 128;         /* query patches per CTA when none is chosen */
constexpr int TILE_DESC = 64;             /* query patches per CTA in descriptor mode (of one row) */
__host__ __device__ constexpr int tile_w(int tp) { return tp <= 32 ? 8 : tp <= 128 ? 16 : 32; }
__host__ __device__ constexpr int tile_h(int tp) { return tp / tile_w(tp); }
__host__ __device__ constexpr int stage_pitch(int tp) { return 3 * (tile_w(tp) + 7); }
__host__ __device__ constexpr int stage_rows(int tp) { return tile_h(tp) + 7; }

/* Columns and rows of a CTA's tile in image mode, and in descriptor mode (a row segment). */
__host__ __device__ constexpr int cta_w(int tp, bool desc) { return desc ? tp : tile_w(tp); }
__host__ __device__ constexpr int cta_h(int tp, bool desc) { return desc ? 1 : tile_h(tp); }

/* Shared-memory bytes of a staged query tile of TP patches. */
constexpr size_t atile_bytes(int tp) { return sizeof(float) * stage_pitch(tp) * stage_rows(tp); }

/* Starts copying the pixels under a CTA's tile into shared memory as packed rows, 3 floats per pixel
   (zeros beyond the image): asynchronous 4-byte copies, any row is only 4-byte aligned.  The tile may
   be read after stage_wait and a __syncthreads; what does not need it goes in between. */
template<int TP, int THREADS = TP>
__device__ __forceinline__ void stage_a(float *at, const float *__restrict__ a, int aw, int ah, int x0, int y0) {
    constexpr int PITCH = stage_pitch(TP);
    const int left = 3 * (aw - x0);
    for (int i = threadIdx.x; i < PITCH * stage_rows(TP); i += THREADS) {
        const int r = i / PITCH, c = i - r * PITCH;
        const int gy = y0 + r;
        const bool in = gy < ah && c < left;
        const float *src = a + (in ? ((size_t) gy * aw + x0) * 3 + c : 0);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                     :: "r"((unsigned) __cvta_generic_to_shared(at + i)), "l"(src), "r"(in ? 4 : 0) : "memory");
    }
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

typedef unsigned long long f32x2;         /* two floats in a register pair (.f32x2 arithmetic) */
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
/* a - b, as b * -1 + a: one rounding, the subtraction's bits. */
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("{\n\t.reg .b64 m;\n\tmov.b64 m, 0xbf800000bf800000;\n\tfma.rn.f32x2 %0, %2, m, %1;\n\t}" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

/* One 32-byte read-only load. */
__device__ __forceinline__ void ld8(const float *p, float (&v)[8]) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(p));
}

/* Lane j of a quad holds the quad's partial sums of patch s in acc[s] (its SSE lane j); returns,
   to lane s, patch s's total in the reference's order ((l0 + l1) + l2) + l3: a 4 x 4 transpose in
   two exchange steps. */
__device__ __forceinline__ float quad_total(const float (&acc)[4]) {
    const unsigned FULL = 0xffffffffu;
    const bool b0 = threadIdx.x & 1, b1 = threadIdx.x & 2;
    const float r0 = __shfl_xor_sync(FULL, b0 ? acc[0] : acc[1], 1), r1 = __shfl_xor_sync(FULL, b0 ? acc[2] : acc[3], 1);
    const float t0 = b0 ? acc[1] : acc[0], t1 = b0 ? acc[3] : acc[2];
    const float k0 = b1 ? t1 : t0, k1 = b1 ? r1 : r0;
    const float g0 = __shfl_xor_sync(FULL, b1 ? t0 : t1, 2), g1 = __shfl_xor_sync(FULL, b1 ? r0 : r1, 2);
    const float lo0 = b1 ? g0 : k0, lo1 = b1 ? g1 : k1, h0 = b1 ? k0 : g0, h1 = b1 ? k1 : g1;
    return __fadd_rn(__fadd_rn(__fadd_rn(lo0, lo1), b0 ? h1 : h0), b0 ? h0 : h1);
}

/* patch_dist_exact (patchtable.h:330-373) of one candidate per lane, 32 of them per call: the
   whole warp takes part, lanes without a candidate pass valid = false.

   The reference keeps four SSE lane sums, the interleaved RGB float e of a patch row going to sum
   e & 3 in increasing e; a quad of lanes scores one patch, lane j holding sum j, so every sum is
   accumulated in exactly that order.  Each quad scores its four lanes' patches together, row by
   row.  A candidate row is one aligned 128-byte line of the table image's row store (k_row_store):
   lane j reads its 32 bytes with one load and picks its six floats by the column's parity.  The four
   patches of a quad lie in the same columns on consecutive rows: a staged query row is read from
   shared memory once for all of them (11 rows instead of 32).

   Bound: the L1 data pipe (128 bytes per clock: 256 wavefronts for 32 candidates' lines, 66 for the
   query rows, 24 for the exchanges) at 77-82 % of its peak in the general pulls, issue slots at 53-64 %.
   The gather this replaced -- each lane its own candidate's 8 pixels, four 32-byte loads from 32
   different lines, 24 shared loads per row -- spent one wavefront on every lane's load and ran at
   89 % of the same pipe: at 1080p the lean choose took 0.265 ms (now 0.150), the one-candidate pull
   0.257 (0.182), the default schedule's pulls 4.01 (2.78).

   D rows per candidate are in flight at a time: more registers, fewer waits.

   With EXIT a candidate is abandoned (+inf returned) once its partial total reaches `bound`, tested
   after rows 2, 4 and 6 (the total can only grow, so nothing that would be accepted is lost). */
template<int TP, bool EXIT, int D>
__device__ __forceinline__ float score32(const QPlan &q, const float *al, int cand, bool valid, float bound, unsigned &rows) {
    constexpr int PITCH = stage_pitch(TP);
    const unsigned FULL = 0xffffffffu;
    unsigned live = __ballot_sync(FULL, valid);
    if (!live) return finf();
    const int lane = threadIdx.x & 31, qb = lane & ~3, j = lane & 3;
    unsigned v = 0;                       /* line << 1 | odd column; lanes without a candidate read line 0 */
    if (valid) {
        const unsigned x = (unsigned) pt_x(cand);
        v = (((unsigned) pt_y(cand) * (unsigned) q.nline + (x >> 1)) << 1) | (x & 1);
    }
    const float *p[4];
    bool off[4];                          /* the lane's floats start at 1 instead of 0 of its 8 */
#pragma unroll
    for (int s = 0; s < 4; s++) {
        const unsigned vs = __shfl_sync(FULL, v, qb | s);
        const int i0 = 3 * (int) (vs & 1) + j;
        p[s] = q.brow + (size_t) (vs >> 1) * 32 + (i0 & 3) * 8;
        off[s] = i0 >= 4;
    }
    const size_t pitch = (size_t) q.nline * 32;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    f32x2 aw[4][3];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int n = 0; n < 3; n++) aw[r][n] = pack2(al[r * PITCH + 8 * n], al[r * PITCH + 8 * n + 4]);
    float u[D][4][8];                     /* the next D rows, on their way or arrived */
#pragma unroll
    for (int r = 0; r < D - 1; r++)
#pragma unroll
        for (int s = 0; s < 4; s++) { ld8(p[s], u[r][s]); p[s] += pitch; }
#pragma unroll
    for (int r = 0; r < 8; r++) {
#pragma unroll
        for (int n = 0; n < 3; n++) aw[(r + 3) & 3][n] = pack2(al[(r + 3) * PITCH + 8 * n], al[(r + 3) * PITCH + 8 * n + 4]);
        if (r + D - 1 < 8) {
#pragma unroll
            for (int s = 0; s < 4; s++) { ld8(p[s], u[(r + D - 1) % D][s]); p[s] += pitch; }
        }
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const float (&ur)[8] = u[r % D][s];
            float w[6];
#pragma unroll
            for (int n = 0; n < 6; n++) w[n] = off[s] ? ur[n + 1] : ur[n];
#pragma unroll
            for (int n = 0; n < 3; n++) {
                const f32x2 t = sub2(pack2(w[2 * n], w[2 * n + 1]), aw[(r + s) & 3][n]);
                float lo, hi;
                unpack2(mul2(t, t), lo, hi);
                acc[s] = __fadd_rn(__fadd_rn(acc[s], lo), hi);
            }
        }
        if (EXIT && (r == 1 || r == 3 || r == 5)) {
            const bool own = (live >> lane) & 1;
            if (own) rows += 2;
            const float part = quad_total(acc);
            live = __ballot_sync(FULL, own && !(part >= bound));
            if (!live) return finf();
#pragma unroll
            for (int s = 0; s < 4; s++)
                if (!((live >> (qb | s)) & 1)) p[s] = q.brow;      /* dead: all read one line */
        }
    }
    const float tot = quad_total(acc);
    const bool own = (live >> lane) & 1;
    if (own) rows += EXIT ? 2 : 8;
    return own ? tot : finf();
}

/* The first eight candidates of `mask` (bit l: lane l's, v its line << 1 | odd column), one per quad:
   the k-th goes to quad k, which reads the query rows of its lane's patch.  Returns its lane the total
   (+inf when abandoned at `bound` after row 4); other lanes get no meaningful value. */
template<int TP, bool EXIT>
__device__ __forceinline__ float score8(const QPlan &q, const float *al, unsigned mask, unsigned v, float bound) {
    constexpr int PITCH = stage_pitch(TP);
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, k = lane >> 2, j = lane & 3;
    unsigned m = mask;
#pragma unroll
    for (int i = 0; i < 7; i++)
        if (k > i) m &= m - 1;
    const bool on = m != 0;
    const int src = on ? __ffs(m) - 1 : __ffs(mask) - 1;
    const unsigned vs = __shfl_sync(FULL, v, src);
    const int i0 = 3 * (int) (vs & 1) + j;
    const bool off = i0 >= 4;
    const float *p = q.brow + (size_t) (vs >> 1) * 32 + (i0 & 3) * 8;
    const size_t pitch = (size_t) q.nline * 32;
    /* the address of patch src's first query float for SSE lane j, from this lane's own */
    const float *as = al + (src & 3) * PITCH + 3 * ((src >> 2) - k);
    float acc = 0.f, part = 0.f;
#pragma unroll
    for (int r0 = 0; r0 < 8; r0 += 4) {
        float u[4][8];
#pragma unroll
        for (int r = 0; r < 4; r++) { ld8(p, u[r]); p += pitch; }
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float *ar = as + (r0 + r) * PITCH;
#pragma unroll
            for (int n = 0; n < 3; n++) {
                const f32x2 w = pack2(off ? u[r][2 * n + 1] : u[r][2 * n], off ? u[r][2 * n + 2] : u[r][2 * n + 1]);
                const f32x2 t = sub2(w, pack2(ar[8 * n], ar[8 * n + 4]));
                float lo, hi;
                unpack2(mul2(t, t), lo, hi);
                acc = __fadd_rn(__fadd_rn(acc, lo), hi);
            }
        }
        const int qb = lane & ~3;
        const float l0 = __shfl_sync(FULL, acc, qb), l1 = __shfl_sync(FULL, acc, qb | 1), l2 = __shfl_sync(FULL, acc, qb | 2),
                    l3 = __shfl_sync(FULL, acc, qb | 3);
        part = __fadd_rn(__fadd_rn(__fadd_rn(l0, l1), l2), l3);
        if (EXIT && r0 == 0) {
            const float b = __shfl_sync(FULL, bound, src);
            if (!__any_sync(FULL, on && !(part >= b))) { part = finf(); break; }
        }
    }
    return __shfl_sync(FULL, part, 4 * (__popc(mask & ((1u << lane) - 1)) & 7));
}

/* One candidate's distance per lane, all 32 lanes of the warp together: in one round of 32, or, when
   at most 16 lanes have one (the ends of candidate lists, the later passes' few new neighbours), in
   rounds of eight, a candidate per quad: 280 instructions and 160 wavefronts each instead of 1,010 and
   346.  At 1080p the default schedule's pulls take 2.90 ms with the line at 16, 2.93 at 8 or 24 and
   3.03 with rounds of 32 only. */
template<int TP, bool EXIT, int D>
__device__ __forceinline__ float score_warp(const QPlan &q, const float *al, int cand, bool valid, float bound, unsigned &rows) {
    const unsigned FULL = 0xffffffffu;
    unsigned mask = __ballot_sync(FULL, valid);
    if (!mask) return finf();
    if (__popc(mask) > 16) return score32<TP, EXIT, D>(q, al, cand, valid, bound, rows);
    const int lane = threadIdx.x & 31;
    unsigned v = 0;
    if (valid) {
        const unsigned x = (unsigned) pt_x(cand);
        v = (((unsigned) pt_y(cand) * (unsigned) q.nline + (x >> 1)) << 1) | (x & 1);
        rows += 8;
    }
    float d = finf();
    while (mask) {
        const float e = score8<TP, EXIT>(q, al, mask, v, bound);
        unsigned rest = mask;
#pragma unroll
        for (int i = 0; i < 8; i++) rest &= rest - 1;
        if (((mask & ~rest) >> lane) & 1) d = e;
        mask = rest;
    }
    if (EXIT && valid && d == finf()) rows -= 4;      /* abandoned */
    return d;
}

/* The query patch a distance is taken from: its staged rows (image mode: the address of the lane's
   first float) or its descriptor in registers (descriptor mode). */
struct AQuery {
    const float *al;
    float4 v[4];
};

/* One candidate's distance per lane: patch_dist_exact for the whole warp at once (image mode), or
   patch_dist_approx of the descriptors (descriptor mode, always complete: a complete sum at or
   above the bound is rejected by the caller exactly as an abandoned one). */
template<int TP, bool DESC, bool EXIT, int D = 1>
__device__ __forceinline__ float dist32(const AQuery &aq, const QPlan &q, int cand, bool valid, float bound, unsigned &rows) {
    if constexpr (DESC) {
        if (!valid) return finf();
        rows++;
        return pt_desc_dist(aq.v, q.bdesc + ((size_t) pt_y(cand) * q.bew + pt_x(cand)) * q.ds4, q.nd);
    } else {
        return score_warp<TP, EXIT, D>(q, aq.al, cand, valid, bound, rows);
    }
}

/* This lane's patch of the tile with top-left patch (x0, y0), and its query. */
template<int TP, bool DESC, int WPT = 1>
__device__ __forceinline__ void tile_lane(const QPlan &q, const float *at, int x0, int y0, int &x, int &y, AQuery &aq) {
    const int wid = WPT > 1 ? 0 : threadIdx.x >> 5, lane = threadIdx.x & 31;
    if constexpr (DESC) {                 /* a row segment: nothing but the row order is shared */
        x = x0 + threadIdx.x;
        y = y0;
    } else {
        constexpr int WX = tile_w(TP) / WTW;
        const int cx = (wid % WX) * WTW + (lane >> 2), ry = (wid / WX) * WTH;
        x = x0 + cx;
        y = y0 + ry + (lane & 3);
        aq.al = at + ry * stage_pitch(TP) + 3 * cx + (lane & 3);
    }
}

/* The table entry v as a patch position, -1 when it lies outside b: a table built here only holds
   patches of b; the range test guards against a corrupt table file or entry array, which must not
   make a kernel read outside b. */
__device__ __forceinline__ int table_entry(const QPlan &q, int v) {
    const int xs = pt_x(v) - 7, ys = pt_y(v) - 7;
    return (xs >= 0 && ys >= 0 && xs < q.bew && ys < q.beh) ? pt_xy(xs, ys) : -1;
}

/* Random search (patchtable.h:3874-3903): one of the 8 neighbours of the best match, -1 when it lies
   outside b or is not allowed.  dx, dy + 1 for r = 0..7 are packed two bits each:
   {-1,0,1,-1,1,-1,0,1}, {-1,-1,-1,0,0,1,1,1}. */
__device__ __forceinline__ int random_neighbour(const QPlan &q, int pass, int p, int xb, int yb) {
    const unsigned r = mix32((unsigned) p * 2654435761u + (unsigned) pass * 0x9e3779b9u + 0x6a09e667u) & 7u;
    const int xs = xb + (int) ((37412u >> (2 * r)) & 3u) - 1, ys = yb + (int) ((43328u >> (2 * r)) & 3u) - 1;
    if (xs < 0 || xs >= q.bew || ys < 0 || ys >= q.beh) return -1;
    if (q.allowed && __ldg(q.allowed + (size_t) ys * q.bew + xs) != q.allowed_index) return -1;
    return pt_xy(xs, ys);
}

/* Proposals of the learned network for one patch (LEARNED instantiation of k_choose_tile). */
struct LearnedArgs {
    const int *cand;          /* n x 8 table entries, -1 = none; NULL on passes without proposals */
    const float *conf;        /* n: probability of the best proposed cell */
    float threshold;          /* patches below it keep the plain candidates */
    int kcoh_confident;       /* confident patches also try k-coherence */
    unsigned long long *counters;   /* [confident patches, proposals scored] or NULL */
};

/* A lane's walk through its patch's candidates in the reference's order: the table entries (TABLES),
   k-coherence neighbours, then spatial or random search (patchtable.h:3641-3903). */
template<bool TABLES>
struct Walk {
    enum { TABLE, ENTER, KCOH, WINDOW, RANDOM, DONE };
    int ph, it;
    int best;                             /* best match so far */
    float dbest, dch;                     /* the distance to beat, and the distance of the choice */
    int kc_src, kdx, kdy;
    bool repeat, accepted;
    const int2 *kp;
    int wx, wy, wx0, wx1, wy1, own;

    int prev;                             /* the previous table's entry */

    __device__ __forceinline__ void start(const QPlan &q, bool live, int pos, float dstore) {
        ph = live ? (TABLES ? TABLE : ENTER) : DONE;
        it = prev = 0;
        best = pos;
        dbest = (float) ((double) dstore * q.prop_scale);
        dch = dstore;
        repeat = accepted = false;
        kdx = kdy = 0;
    }
    __device__ __forceinline__ void offer(int c, float d) {
        if (d < dbest) {
            dbest = dch = d;
            best = c;
            if (ph == KCOH) accepted = true;
        }
    }
    __device__ __forceinline__ bool inside(const QPlan &q) const { return pt_x(best) < q.bew && pt_y(best) < q.beh; }

    /* The next candidate, or -1 when the walk has ended. */
    __device__ __forceinline__ int next(const QPlan &q, const int2 *__restrict__ kcoh, int *kc_done, int use_done,
                                        int do_kcoh, int pass, bool kc_here, int p, bool table = false,
                                        const int *tcand = nullptr) {
        int c = -1;
        while (c < 0 && ph != DONE) {
            if (TABLES && ph == TABLE) {
                /* the first table's entry, then the further tables' (patchtable.h:3711-3735): each is
                   scored unless it equals the best so far or the previous table's entry */
                if (!table || it > q.ntc) { ph = ENTER; continue; }
                const int v = it == 0 ? tcand[p] : q.tcand_more[(size_t) (it - 1) * q.ew * q.eh + p];
                const int e = table_entry(q, v);
                if (e >= 0 && e != best && (it == 0 || v != prev)) c = e;
                prev = v;
                it++;
            } else if (ph == ENTER) {
                ph = KCOH;
                kc_src = best;
                it = q.kc_try;            /* nothing to try, unless: */
                if (do_kcoh) {
                    repeat = use_done && kc_done[p] == kc_src;
                    if (kc_here && !repeat && inside(q)) {
                        const int ks = q.ks, xb = pt_x(best), yb = pt_y(best);
                        kp = kcoh + ((size_t) (yb / ks) * q.bew + (xb / ks)) * q.kc;
                        if (ks > 1) { kdx = xb % ks; kdy = yb % ks; }
                        it = 0;
                    }
                }
            } else if (ph == KCOH) {
                /* the reference tries the list in order and stops at the first neighbour whose
                   stored distance reaches triangle * best */
                int2 e = make_int2(0, 0);
                bool go = it < q.kc_try;
                if (go) {
                    e = kp[it++];
                    go = (double) __int_as_float(e.y) < q.triangle * (double) dbest;
                }
                if (go) {
                    c = pt_xy(min(pt_x(e.x) + kdx, q.bew - 1), min(pt_y(e.x) + kdy, q.beh - 1));
                    continue;
                }
                ph = DONE;
                if (do_kcoh) kc_done[p] = (repeat || !accepted) ? kc_src : -1;
                if (inside(q)) {
                    if (q.spatial > 0) {
                        /* Spatial search (patchtable.h:3855-3873): every other patch of the (2s+1)^2
                           window around the best match, rows then columns. */
                        const int S = q.spatial, xb = pt_x(best), yb = pt_y(best);
                        ph = WINDOW;
                        own = best;
                        wy = max(yb - S, 0);
                        wy1 = min(yb + S + 1, q.beh);
                        wx0 = max(xb - S, 0);
                        wx1 = min(xb + S + 1, q.bew);
                        wx = wx0;
                    } else if (q.do_rs) {
                        ph = RANDOM;
                    }
                }
            } else if (ph == WINDOW) {
                if (wy >= wy1) { ph = DONE; continue; }
                const int e = pt_xy(wx, wy);
                if (e != own && (!q.allowed || __ldg(q.allowed + (size_t) wy * q.bew + wx) == q.allowed_index)) c = e;
                if (++wx >= wx1) { wx = wx0; wy++; }
            } else {
                ph = DONE;
                c = random_neighbour(q, pass, p, pt_x(best), pt_y(best));
            }
        }
        return c;
    }
};

/* Steps 1-3 for every patch ("choose"): the chosen match and its exact distance.  Each lane walks
   its own patch's candidates in the reference's order -- table entries, k-coherence neighbours,
   spatial or random search -- and the warp scores one candidate per lane at a time, so lanes may be
   at different steps of the walk.  The LEARNED instantiation replaces, for patches whose proposal
   confidence reaches the threshold, the table candidate by the network's proposals (best first)
   and, unless configured otherwise, skips k-coherence for them.
   LEAN: the table step only (no further tables, k-coherence, spatial or random search), one
   candidate per patch, without the registers of the walk. */
template<int TP, bool LEARNED, bool LEAN>
__device__ __forceinline__ void
choose_tile(const QPlan &c_q, float *at, const float *__restrict__ a, const int *cur_pos,
            const float *cur_d, const int *tcand, const int2 *__restrict__ kcoh, int do_table,
            int *ch_pos, float *ch_d, int *kc_done, int use_done, unsigned long long *counters, const LearnedArgs &la,
            int x0, int y0, int y1) {
    const unsigned FULL = 0xffffffffu;
    AQuery aq;
    int x, y;
    tile_lane<TP, false>(c_q, at, x0, y0, x, y, aq);
    const bool live = x < c_q.ew && y < y1;
    const int p = live ? y * c_q.ew + x : 0;
    unsigned ne = 0, rows = 0, n_conf = 0, n_prop = 0;
    /* no state arrays: the initial field, x = b's ew + 1 and DIST_INFINITY (patchtable.h:3538-3547) */
    const int pos = cur_pos ? cur_pos[p] : pt_xy(c_q.bew + 1, 0);
    const float dstore = cur_d ? cur_d[p] : (float) PT_DIST_INF;
    auto entry = [&](int v) { return table_entry(c_q, v); };
    stage_a<TP>(at, a, c_q.aw, c_q.ah, x0, y0);
    if constexpr (LEAN) {
        int cand = -1;
        if (live && do_table) {
            cand = entry(tcand[p]);
            if (cand == pos) cand = -1;
        }
        stage_wait();
        __syncthreads();
        const float dbest = (float) ((double) dstore * c_q.prop_scale);
        const float d = dist32<TP, false, false>(aq, c_q, cand, cand >= 0, dbest, rows);
        const bool take = cand >= 0 && d < dbest;
        if (live) { ch_pos[p] = take ? cand : pos; ch_d[p] = take ? d : dstore; }
        count_work(counters, cand >= 0, rows);
        return;
    }
    bool confident = false;
    unsigned keep = 0;                    /* the network's proposals still to score, repeats dropped */
    if (LEARNED && live) {
        confident = la.conf[p] >= la.threshold;
        if (confident && do_table && la.cand) {
            const int4 *cp = reinterpret_cast<const int4 *>(la.cand + (size_t) p * PT_PROP_TOPK);
            const int4 c0 = cp[0], c1 = cp[1];
            const int raw[PT_PROP_TOPK] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
            int cand[PT_PROP_TOPK];
#pragma unroll
            for (int j = 0; j < PT_PROP_TOPK; j++) {
                cand[j] = raw[j] >= 0 ? entry(raw[j]) : -1;
                bool dup = cand[j] < 0 || cand[j] == pos;
#pragma unroll
                for (int t = 0; t < j; t++) dup |= ((keep >> t) & 1) && cand[t] == cand[j];
                if (!dup) keep |= 1u << j;
            }
            n_prop = __popc(keep);
            n_conf = 1;
        }
    }
    const bool table = do_table && !(LEARNED && confident && la.cand);
    const bool kc_here = !LEARNED || !confident || la.kcoh_confident;
    Walk<true> w;
    w.start(c_q, live, pos, dstore);
    for (bool staged = false;;) {
        int cand = -1;
        if (LEARNED && keep) {
            const int j = __ffs(keep) - 1;
            keep &= keep - 1;
            cand = entry(la.cand[(size_t) p * PT_PROP_TOPK + j]);
        }
        if (cand < 0) cand = w.next(c_q, kcoh, kc_done, use_done, c_q.do_kcoh, c_q.pass, kc_here, p, table, tcand);
        if (!staged) {
            /* later passes find nothing new for most patches: a tile without a candidate ends here */
            stage_wait();
            if (!__syncthreads_or(cand >= 0)) break;
            staged = true;
        }
        if (!__any_sync(FULL, cand >= 0)) break;
        const float d = dist32<TP, false, true, CHOOSE_D>(aq, c_q, cand, cand >= 0, w.dbest, rows);
        if (cand >= 0) {
            ne++;
            w.offer(cand, d);
        }
    }
    if (live) { ch_pos[p] = w.best; ch_d[p] = w.dch; }
    count_work(counters, ne, rows);
    if (LEARNED && la.counters) {
        unsigned c = __reduce_add_sync(FULL, n_conf), n = __reduce_add_sync(FULL, n_prop);
        if ((threadIdx.x & 31) == 0) { atomicAdd(la.counters, (unsigned long long) c); atomicAdd(la.counters + 1, (unsigned long long) n); }
    }
}

template<int TP, bool LEARNED, bool LEAN = false>
__global__ void __launch_bounds__(TP, min_ctas(LEAN ? CHOOSE_LEAN_LANES : CHOOSE_LANES, TP))
k_choose_tile(const QPlan c_q, const float *__restrict__ a, const int *cur_pos,
              const float *cur_d, const int *tcand, const int2 *__restrict__ kcoh, int do_table,
              int *ch_pos, float *ch_d, int *kc_done, int use_done, unsigned long long *counters, const LearnedArgs la) {
    extern __shared__ float at[];
    pdl_trigger();
    pdl_wait();
    choose_tile<TP, LEARNED, LEAN>(c_q, at, a, cur_pos, cur_d, tcand, kcoh, do_table, ch_pos, ch_d, kc_done, use_done,
                                   counters, la, blockIdx.x * tile_w(TP), blockIdx.y * tile_h(TP) + c_q.row0,
                                   c_q.row0 + c_q.rows);
}

/* Step 4 as a pull: the best of the stored match and every neighbour's chosen offset applied to
   this patch.  The patch's own choice comes first; the distinct neighbour candidates follow in
   increasing order of the distance their neighbour achieved with them (the likeliest good ones
   first, so the running best -- the early-exit bound -- tightens soonest).
   Neighbours sit `step` patches apart; passes with decreasing steps (jump flooding) carry an
   offset across a region in a logarithmic number of passes, where the reference's sequential
   sweep carries it along a whole row in one sweep. */
/* ONE: a single neighbour candidate per patch (pull_max 1).  The candidate is the one the
   general path would sort first -- among distinct candidates keyed by their first occurrence, the
   smallest key, the earliest on ties -- found in one streaming pass, and it is scored alone. */
/* NX: also the next pass's choose (c_q.nx) where asked for; without it the general pull's registers
   are its own (-speed 1 at 540 x 960: 1.675 ms, 1.714 with the code in the kernel but unused). */
template<int TP, int R, bool DESC, bool ONE, bool NX, int D = 1, int WPT = 1>
__device__ __forceinline__ void
pull_tile(const QPlan &c_q, float *at, const float *__restrict__ a, const int *cur_pos,
          const float *cur_d, const int *ch_pos, const float *ch_d, int *nxt_pos,
          float *nxt_d, unsigned long long *counters, int x0, int y0, int y1) {
    const unsigned FULL = 0xffffffffu;
    if constexpr (!DESC) stage_a<TP, TP * WPT>(at, a, c_q.aw, c_q.ah, x0, y0);
    AQuery aq;
    int x, y;
    tile_lane<TP, DESC, WPT>(c_q, at, x0, y0, x, y, aq);
    const bool live = x < c_q.ew && y < y1;
    const int p = live ? y * c_q.ew + x : 0;
    /* the match found: the next pass's state, or the float64 NNF of the final field (k_output fused) */
    auto finish = [&](int pos, float d) {
        if (c_q.ann) {
            double *o = c_q.ann + 3 * (size_t) p;
            o[0] = pt_x(pos);
            o[1] = pt_y(pos);
            o[2] = d;
        } else {
            nxt_pos[p] = pos;
            nxt_d[p] = d;
        }
    };
    auto staged = [&]() {
        if constexpr (!DESC) {
            stage_wait();
            __syncthreads();
        }
    };
    if constexpr (DESC) pt_desc_load(c_q.adesc + (size_t) p * c_q.ds4, 4 * c_q.ds4, aq.v);
    unsigned ne = 0, rows = 0;
    int bpos = cur_pos ? cur_pos[p] : pt_xy(c_q.bew + 1, 0);      /* null: the initial field */
    float bd = cur_d ? cur_d[p] : (float) PT_DIST_INF;
    {
        const int cp = ch_pos[p];
        const float cd = ch_d[p];
        if (pt_x(cp) < c_q.bew && pt_y(cp) < c_q.beh && cp != bpos && cd < bd) { bd = cd; bpos = cp; }
    }
    constexpr int MAXC = (2 * R + 1) * (2 * R + 1) - 1;
    const int S = c_q.step;
    int nc = 0;
    /* calls fn(candidate, the neighbour's own distance) for every neighbour's offset inside b */
    auto neighbours = [&](auto &&fn) {
#pragma unroll
        for (int dy = -R; dy <= R; dy++) {
#pragma unroll
            for (int dx = -R; dx <= R; dx++) {
                if (dx == 0 && dy == 0) continue;
                const int ny = y + S * dy, nx = x + S * dx;
                if (!live || ny < 0 || ny >= c_q.eh || nx < 0 || nx >= c_q.ew) continue;
                const int n = ny * c_q.ew + nx;
                const int cp = ch_pos[n];
                const int xs = pt_x(cp) - S * dx, ys = pt_y(cp) - S * dy;
                if (xs < 0 || ys < 0 || xs >= c_q.bew || ys >= c_q.beh) continue;
                if (c_q.allowed && __ldg(c_q.allowed + (size_t) ys * c_q.bew + xs) != c_q.allowed_index) continue;
                fn(pt_xy(xs, ys), ch_d + n);
            }
        }
    };
    if constexpr (ONE) {
        /* the distinct candidates seen so far, newest first (fixed register slots) */
        int seen[MAXC];
#pragma unroll
        for (int t = 0; t < MAXC; t++) seen[t] = -1;
        int best = -1;
        float bestk = finf();
        neighbours([&](int c, const float *kp) {
            bool dup = c == bpos;
#pragma unroll
            for (int t = 0; t < MAXC; t++) dup |= seen[t] == c;
            if (dup) return;
#pragma unroll
            for (int t = MAXC - 1; t > 0; t--) seen[t] = seen[t - 1];
            seen[0] = c;
            const float k = *kp;
            if (k < bestk) { bestk = k; best = c; }   /* the general sort's insertion rule */
        });
        staged();
        const float d = dist32<TP, DESC, true, D>(aq, c_q, best, best >= 0, bd, rows);
        if (best >= 0) {
            ne = 1;
            if (d < bd) { bd = d; bpos = best; }
        }
    } else {
        /* distinct neighbour candidates sorted by the neighbour's own distance (ties keep the
           neighbour order), kept in registers: every slot index is known at compile time.  A neighbour
           whose distance is +inf or NaN (the seed of a field may be) has no place in the order: the
           insertion leaves its offset out and it is not counted, or the walk would score the empty
           slots at the list's end. */
        int cand[MAXC];
        float key[MAXC];
#pragma unroll
        for (int t = 0; t < MAXC; t++) { cand[t] = -1; key[t] = finf(); }
        neighbours([&](int c, const float *kp) {
            bool dup = c == bpos;
#pragma unroll
            for (int t = 0; t < MAXC; t++) dup |= cand[t] == c;
            if (dup) return;
            float k = *kp;
            const bool finite = k < finf();
#pragma unroll
            for (int t = 0; t < MAXC; t++) {
                if (k < key[t]) {
                    const float tk = key[t]; key[t] = k; k = tk;
                    const int tc = cand[t]; cand[t] = c; c = tc;
                }
            }
            nc += finite;
        });
        if (nc > c_q.pull_max) nc = c_q.pull_max;   /* the best-first prefix of the list */
        ne = nc;
        staged();
        if constexpr (DESC) {
            float d[MAXC];                          /* every candidate's loads in flight at once */
#pragma unroll
            for (int t = 0; t < MAXC; t++) d[t] = dist32<TP, DESC, false>(aq, c_q, cand[t], t < nc, bd, rows);
#pragma unroll
            for (int t = 0; t < MAXC; t++)
                if (t < nc && d[t] < bd) { bd = d[t]; bpos = cand[t]; }
        } else {
            auto shift = [&]() {
#pragma unroll
                for (int t = 0; t + 1 < MAXC; t++) cand[t] = cand[t + 1];
            };
            /* with WPT warps on the tile, warp v scores candidates v, v + WPT, ... of the list */
            const int v = WPT > 1 ? threadIdx.x >> 5 : 0;
            int from = -1;
            for (int t = 0; t < v; t++) shift();
            for (int t0 = v; __any_sync(FULL, t0 < nc); t0 += WPT) {
                const int c = cand[0];
                const float d = dist32<TP, DESC, true, D>(aq, c_q, c, t0 < nc, bd, rows);
                if (t0 < nc && d < bd) { bd = d; bpos = c; from = t0; }
#pragma unroll
                for (int t = 0; t < WPT; t++) shift();
            }
            if constexpr (WPT > 1) {
                /* the smallest distance, the earliest in the list on ties: what one warp going through
                   the whole list keeps */
                __shared__ float s_d[WPT][32];
                __shared__ int s_pos[WPT][32], s_from[WPT][32];
                const int lane = threadIdx.x & 31;
                s_d[v][lane] = bd;
                s_pos[v][lane] = bpos;
                s_from[v][lane] = from;
                __syncthreads();
                if (v > 0) { count_work(counters, 0, rows); return; }
#pragma unroll
                for (int u = 1; u < WPT; u++) {
                    const int f = s_from[u][lane];
                    const float d = s_d[u][lane];
                    if (f >= 0 && (d < bd || (d == bd && from >= 0 && f < from))) { bd = d; bpos = s_pos[u][lane]; from = f; }
                }
            }
            if (live) finish(bpos, bd);
            count_work(counters, ne, rows);
            if constexpr (!NX) return;
            if (!c_q.nx.ch_pos) return;
            /* The next pass's choose for the match just found: its k-coherence neighbours and searches
               (the table step belongs to the first pass).  A choose launch of its own reads the state
               again and stages the tile for few candidates (0.02 per patch after the first pass of the
               default schedule): 48 x 64 92 us with, 80 without them, 355 x 611 472 and 444, 540 x 960
               959 and 918.  Walking on inside the loop above, lane by lane, keeps both candidate
               lists' state in registers and spills: 1080p 4.3 ms instead of 3.5. */
            Walk<false> w;
            w.start(c_q, live, bpos, bd);
            for (;;) {
                const int c = w.next(c_q, c_q.nx.kcoh, c_q.nx.kc_done, c_q.nx.use_done, c_q.nx.do_kcoh, c_q.nx.pass, true, p);
                if (!__any_sync(FULL, c >= 0)) break;
                const float d = dist32<TP, DESC, true, D>(aq, c_q, c, c >= 0, w.dbest, rows);
                if (c >= 0) w.offer(c, d);
            }
            if (live) { c_q.nx.ch_pos[p] = w.best; c_q.nx.ch_d[p] = w.dch; }
            return;
        }
    }
    if (live) finish(bpos, bd);
    count_work(counters, ne, rows);
}

template<int TP, int R, bool DESC, bool ONE = false, bool NX = false, int D = 1, int WPT = 1>
__global__ void __launch_bounds__(TP * WPT, min_ctas(WPT > 1 ? 2 * TP * WPT : ONE ? PULL_ONE_LANES : PULL_LANES, TP * WPT))
k_pull_tile(const QPlan c_q, const float *__restrict__ a, const int *cur_pos,
            const float *cur_d, const int *ch_pos, const float *ch_d,
            int *nxt_pos, float *nxt_d, unsigned long long *counters) {
    extern __shared__ float at[];
    if constexpr (DESC || ONE || WPT > 1) {      /* the others are launched in order */
        pdl_trigger();
        pdl_wait();
    }
    pull_tile<TP, R, DESC, ONE, NX, D, WPT>(c_q, at, a, cur_pos, cur_d, ch_pos, ch_d, nxt_pos, nxt_d, counters,
                                blockIdx.x * cta_w(TP, DESC), blockIdx.y * cta_h(TP, DESC) + c_q.row0, c_q.row0 + c_q.rows);
}

/* ---- launchers ---- */

/* The specialised variants apply: the choose of a pass with only the table step, the pull of a
   schedule with one neighbour candidate (image mode; descriptor mode keeps the general kernels). */
inline bool lean_choose(const QPlan &q) {
    return pt_lean_kernels() && !q.adesc && !q.do_kcoh && q.ntc == 0 && q.spatial == 0 &&
           !q.do_rs;
}
/* (a pull that does the next pass's choose is a general one) */
inline bool one_pull(const QPlan &q) { return pt_lean_kernels() && !q.adesc && q.pull_max == 1; }

/* Whether a launch may start while the kernel before it in the stream ends: descriptor mode always
   (540 x 960 208 -> 194 us), one candidate per patch up to 24 tiles per SM (48 x 64 27.7 -> 22.6 us, 180 x
   260 29.8 -> 26.7, 290 x 440 43.0 -> 41.5, 355 x 611 59.0 and 59.1), candidate lists up to 4 (48 x 64 79.9
   -> 73.9, 100 x 150 89.7 -> 83.7, 140 x 200 143 and 149, 228 x 350 200 and 256: the early CTAs leave the
   SMs unevenly loaded). */
inline bool early(const QuerySetup &s, const QPlan &q, bool single) {
    if (!s.pdl) return false;
    if (q.adesc) return true;
    const long long tiles = (long long) ((q.ew + WTW - 1) / WTW) * ((q.rows + WTH - 1) / WTH);
    return tiles <= (long long) (single ? 24 : SPLIT_TILES) * sm_count();
}

/* A launch that may start early or not (the kernel waits for the one before it by itself). */
template<class... KA, class... A>
inline cudaError_t launch(bool pdl, void (*kernel)(KA...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, KA(args)...);
}

inline dim3 tile_grid(const QPlan &q, int tp) {
    const int w = cta_w(tp, q.adesc != nullptr), h = cta_h(tp, q.adesc != nullptr);
    return dim3((q.ew + w - 1) / w, (q.rows + h - 1) / h);
}

inline pt_status make_qplan(const QuerySetup &s, QPlan &q) {
    memset(&q, 0, sizeof(q));
    q.aw = s.aw; q.ah = s.ah; q.ew = s.aw - 7; q.eh = s.ah - 7;
    q.bw = s.bw; q.bh = s.bh; q.bew = s.bw - 7; q.beh = s.bh - 7;
    q.prop_scale = s.prop_scale;
    q.triangle = s.triangle_factor;
    q.kc = s.kcoherence;
    q.kc_try = (s.kc_try > 0 && s.kc_try < s.kcoherence) ? s.kc_try : s.kcoherence;
    q.ks = s.kcoherence_step;
    q.radius = s.radius;
    q.do_kcoh = s.kcoherence > 0;
    q.step = s.step < 1 ? 1 : s.step;
    q.pull_max = s.pull_max > 0 ? s.pull_max : 1 << 30;
    q.tile = s.tile > 0 ? s.tile : TILE_DEFAULT;
    q.auto_tile = s.tile <= 0;
    q.row0 = s.rows > 0 ? s.row0 : 0;
    q.rows = s.rows > 0 ? s.rows : q.eh;
    if (s.rows > 0 && (q.row0 < 0 || q.row0 + q.rows > q.eh))
        return pt_fail(PT_BAD_ARG, "query rows [%d, %d) outside 0..%d", q.row0, q.row0 + q.rows, q.eh);
    if (q.tile != 32 && q.tile != 64 && q.tile != 128 && q.tile != 256)
        return pt_fail(PT_BAD_ARG, "gpu_tile %d: query patches per CTA must be 32, 64, 128 or 256", s.tile);
    q.brow = s.brow;
    q.nline = pt_row_lines(s.bw);
    q.allowed = s.allowed;
    q.allowed_index = s.allowed_index;
    q.adesc = reinterpret_cast<const float4 *>(s.adesc);
    q.bdesc = reinterpret_cast<const float4 *>(s.bdesc);
    q.ds4 = s.ds / 4;
    q.nd = s.nd;
    q.tcand_more = s.ntcand_more > 0 ? s.tcand_more : nullptr;
    q.ntc = q.tcand_more ? s.ntcand_more : 0;
    q.spatial = s.spatial > 0 ? s.spatial : 0;
    q.do_rs = s.do_rs;
    q.pass = s.pass;
    q.ann = s.ann;
    q.nx.kcoh = s.nx_kcoh;
    q.nx.kc_done = s.nx_kc_done;
    q.nx.use_done = s.nx_use_done;
    q.nx.do_kcoh = s.nx_do_kcoh;
    q.nx.pass = s.nx_pass;
    q.nx.ch_pos = s.nx_ch_pos;
    q.nx.ch_d = s.nx_ch_d;
    if (q.adesc) {
        if (!q.bdesc || (s.ds != 8 && s.ds != 16) || q.nd < 3 || q.nd > s.ds)
            return pt_fail(PT_BAD_ARG, "descriptor query: store of %d floats for %d dimensions", s.ds, q.nd);
    } else if (!q.brow) {
        return pt_fail(PT_BAD_ARG, "query without the row store of the table image");
    }
    if (q.radius > 2) return pt_fail(PT_UNSUPPORTED, "propagation radius %d > 2 on the GPU path", q.radius);
    return PT_OK;
}

/* The choose and the pull of a single image in CTAs of TP patches. */
template<int TP>
inline pt_status choose_width(const QuerySetup &s, const QPlan &q, const float *a, const int *cur_pos, const float *cur_d,
                              const int *tcand, const int2 *kcoh, int do_table, int *ch_pos, float *ch_d, int *kc_done,
                              int use_done, unsigned long long *evals, cudaStream_t st) {
    LearnedArgs none;
    memset(&none, 0, sizeof(none));
    const dim3 grid = tile_grid(q, TP);
    const bool lean = lean_choose(q);
    if (lean)
        PT_CUDA(launch(early(s, q, lean), (k_choose_tile<TP, false, true>), grid, TP, atile_bytes(TP), st, q, a, cur_pos,
                       cur_d, tcand, kcoh, do_table, ch_pos, ch_d, kc_done, use_done, evals, none));
    else
        PT_CUDA(launch(early(s, q, lean), (k_choose_tile<TP, false>), grid, TP, atile_bytes(TP), st, q, a, cur_pos, cur_d,
                       tcand, kcoh, do_table, ch_pos, ch_d, kc_done, use_done, evals, none));
    PT_LAUNCHED();
    return PT_OK;
}

template<int TP, int R>
inline pt_status pull_width(const QuerySetup &s, const QPlan &q, const float *a, const int *cur_pos, const float *cur_d,
                            const int *ch_pos, const float *ch_d, int *nxt_pos, float *nxt_d, unsigned long long *evals,
                            cudaStream_t st) {
    const dim3 grid = tile_grid(q, TP);
    if (q.nx.ch_pos)
        PT_CUDA(launch(false, (k_pull_tile<TP, R, false, false, true>), grid, TP, atile_bytes(TP), st, q, a, cur_pos, cur_d,
                       ch_pos, ch_d, nxt_pos, nxt_d, evals));
    else if (one_pull(q))
        PT_CUDA(launch(early(s, q, true), (k_pull_tile<TP, R, false, true>), grid, TP, atile_bytes(TP), st, q, a, cur_pos,
                       cur_d, ch_pos, ch_d, nxt_pos, nxt_d, evals));
    else
        PT_CUDA(launch(false, (k_pull_tile<TP, R, false>), grid, TP, atile_bytes(TP), st, q, a, cur_pos, cur_d, ch_pos, ch_d,
                       nxt_pos, nxt_d, evals));
    PT_LAUNCHED();
    return PT_OK;
}

}  // namespace

/* The choose and the pull of a CTA width that was asked for, and of descriptor mode. */
pt_status pt_choose_tiles(const QuerySetup &s, const float *a, const int *cur_pos, const float *cur_d, const int *tcand,
                          const int2 *kcoh, int do_table, int *ch_pos, float *ch_d, int *kc_done, int use_done,
                          unsigned long long *evals, cudaStream_t st);
pt_status pt_pull_tiles(const QuerySetup &s, const float *a, const int *cur_pos, const float *cur_d, const int *ch_pos,
                        const float *ch_d, int *nxt_pos, float *nxt_d, unsigned long long *evals, cudaStream_t st);
pt_status pt_choose_desc(const QuerySetup &s, const int *cur_pos, const float *cur_d, const int *tcand, const int2 *kcoh,
                         int do_table, int *ch_pos, float *ch_d, int *kc_done, int use_done, unsigned long long *evals,
                         cudaStream_t st);
pt_status pt_pull_desc(const QuerySetup &s, const float *a, const int *cur_pos, const float *cur_d, const int *ch_pos,
                       const float *ch_d, int *nxt_pos, float *nxt_d, unsigned long long *evals, cudaStream_t st);
