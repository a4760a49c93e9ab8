/* Descriptor mode: the choose and the pull over caller-supplied descriptor images. */
#include "k_query.cuh"

namespace {

/* ---- descriptor mode: each lane works on its patch alone (a candidate is one or two sectors of the
   descriptor store, nothing to share), rows of TILE_DESC patches per CTA ---- */

/* A patch's search state: its descriptor, the best match so far, the distance to beat and the
   choice's distance. */
struct DescLane {
    float4 av[4];
    int best;
    float dbest, dch;
    unsigned ne;

    __device__ __forceinline__ void start(const QPlan &q, int pos, float dstore) {
        best = pos;
        dch = dstore;
        dbest = (float) ((double) dstore * q.prop_scale);
        ne = 0;
    }
    __device__ __forceinline__ float dist(const QPlan &q, int c) const {
        return pt_desc_dist(av, q.bdesc + ((size_t) pt_y(c) * q.bew + pt_x(c)) * q.ds4, q.nd);
    }
    __device__ __forceinline__ bool offer(int c, float d) {
        ne++;
        if (!(d < dbest)) return false;
        dbest = dch = d;
        best = c;
        return true;
    }
    __device__ __forceinline__ bool inside(const QPlan &q) const { return pt_x(best) < q.bew && pt_y(best) < q.beh; }

    /* The choose after its table step: k-coherence neighbours, two at a time so that the walk waits for
       memory once per pair, then spatial or random search. */
    __device__ __forceinline__ void walk(const QPlan &q, const int2 *__restrict__ kcoh, int *kc_done, int use_done,
                                         int do_kcoh, int pass, int p) {
        const int src = best;
        bool accepted = false, repeat = false;
        if (do_kcoh) {
            repeat = use_done && kc_done[p] == src;
            if (!repeat && inside(q)) {
                const int ks = q.ks, xb = pt_x(best), yb = pt_y(best);
                const int2 *kp = kcoh + ((size_t) (yb / ks) * q.bew + (xb / ks)) * q.kc;
                const int kdx = ks > 1 ? xb % ks : 0, kdy = ks > 1 ? yb % ks : 0;
                auto near = [&](const int2 &e) { return (double) __int_as_float(e.y) < q.triangle * (double) dbest; };
                auto place = [&](const int2 &e) { return pt_xy(min(pt_x(e.x) + kdx, q.bew - 1), min(pt_y(e.x) + kdy, q.beh - 1)); };
                for (int k = 0; k < q.kc_try; k += 2) {
                    const int2 e0 = kp[k], e1 = k + 1 < q.kc_try ? kp[k + 1] : e0;
                    if (!near(e0)) break;
                    const int c0 = place(e0), c1 = place(e1);
                    const bool two = k + 1 < q.kc_try && near(e1);
                    const float d0 = dist(q, c0), d1 = two ? dist(q, c1) : 0.f;
                    accepted |= offer(c0, d0);
                    if (!two || !near(e1)) break;
                    accepted |= offer(c1, d1);
                }
            }
            kc_done[p] = (repeat || !accepted) ? src : -1;
        }
        if (!inside(q)) return;
        if (q.spatial > 0) {
            const int S = q.spatial, xb = pt_x(best), yb = pt_y(best);
            for (int ys = max(yb - S, 0); ys < min(yb + S + 1, q.beh); ys++)
                for (int xs = max(xb - S, 0); xs < min(xb + S + 1, q.bew); xs++) {
                    if (xs == xb && ys == yb) continue;
                    if (q.allowed && __ldg(q.allowed + (size_t) ys * q.bew + xs) != q.allowed_index) continue;
                    offer(pt_xy(xs, ys), dist(q, pt_xy(xs, ys)));
                }
        } else if (q.do_rs) {
            const int c = random_neighbour(q, pass, p, pt_x(best), pt_y(best));
            if (c >= 0) offer(c, dist(q, c));
        }
    }
};

/* The choose in descriptor mode.  (The lockstep walk of choose_tile measured 0.129 against 0.124 ms
   here: 540 x 960, 8 channels, the four chooses of the default schedule.) */
__global__ void __launch_bounds__(TILE_DESC, 10 * 64 / TILE_DESC)
k_choose_desc(const QPlan q, const int *cur_pos, const float *cur_d,
              const int *tcand, const int2 *__restrict__ kcoh, int do_table, int *ch_pos, float *ch_d,
              int *kc_done, int use_done, unsigned long long *counters) {
    pdl_trigger();
    pdl_wait();
    const int x = blockIdx.x * TILE_DESC + threadIdx.x, y = blockIdx.y + q.row0;
    DescLane l;
    l.ne = 0;
    if (x < q.ew) {
        const int p = y * q.ew + x;
        pt_desc_load(q.adesc + (size_t) p * q.ds4, 4 * q.ds4, l.av);
        l.start(q, cur_pos ? cur_pos[p] : pt_xy(q.bew + 1, 0), cur_d ? cur_d[p] : (float) PT_DIST_INF);
        if (do_table) {
            int prev = 0;
            for (int k = 0; k <= q.ntc; k++) {
                const int v = k == 0 ? tcand[p] : q.tcand_more[(size_t) (k - 1) * q.ew * q.eh + p];
                const int c = table_entry(q, v);
                if (c >= 0 && c != l.best && (k == 0 || v != prev)) l.offer(c, l.dist(q, c));
                prev = v;
            }
        }
        l.walk(q, kcoh, kc_done, use_done, q.do_kcoh, q.pass, p);
        ch_pos[p] = l.best;
        ch_d[p] = l.dch;
    }
    count_work(counters, l.ne, l.ne);
}

/* The pull in descriptor mode with every neighbour's candidate scored, and the next pass's choose.
   Distances are always complete, so the list need not be sorted: the smallest distance wins, and on
   ties the candidate whose neighbour achieved less with it, the order in which the sorted walk
   (pull_tile) meets them.  Only candidates equal in both (flat regions) are put through that walk's
   insertion, whose order of equal keys depends on what came between.  Loads of eight candidates are
   in flight together.  540 x 960, 8 channels, the default schedule with the chooses that follow: 249 us
   with a sorted list and chooses of their own, 203 so. */
template<int R>
__global__ void __launch_bounds__(TILE_DESC)
k_pull_desc(const QPlan q, const int *cur_pos, const float *cur_d,
            const int *ch_pos, const float *ch_d, int *nxt_pos, float *nxt_d,
            unsigned long long *counters) {
    constexpr int W = 2 * R + 1, MAXC = W * W - 1, G = 8;
    pdl_trigger();
    pdl_wait();
    const int x = blockIdx.x * TILE_DESC + threadIdx.x, y = blockIdx.y + q.row0;
    const bool live = x < q.ew;
    unsigned ne = 0;
    DescLane l;
    l.ne = 0;
    if (live) {
        const int p = y * q.ew + x;
        pt_desc_load(q.adesc + (size_t) p * q.ds4, 4 * q.ds4, l.av);
        int bpos = cur_pos ? cur_pos[p] : pt_xy(q.bew + 1, 0);
        float bd = cur_d ? cur_d[p] : (float) PT_DIST_INF;
        {
            const int cp = ch_pos[p];
            const float cd = ch_d[p];
            if (pt_x(cp) < q.bew && pt_y(cp) < q.beh && cp != bpos && cd < bd) { bd = cd; bpos = cp; }
        }
        const int own = bpos;
        int cand[MAXC];                   /* neighbour i's candidate, -1: none, or an earlier one's */
        float key[MAXC];
#pragma unroll
        for (int i = 0; i < MAXC; i++) {
            const int o = i < MAXC / 2 ? i : i + 1, dy = o / W - R, dx = o % W - R;
            const int ny = y + q.step * dy, nx = x + q.step * dx;
            cand[i] = -1;
            key[i] = 0.f;
            if (ny < 0 || ny >= q.eh || nx < 0 || nx >= q.ew) continue;
            const int n = ny * q.ew + nx;
            const int cp = ch_pos[n];
            key[i] = ch_d[n];
            const int xs = pt_x(cp) - q.step * dx, ys = pt_y(cp) - q.step * dy;
            if (xs < 0 || ys < 0 || xs >= q.bew || ys >= q.beh) continue;
            if (q.allowed && __ldg(q.allowed + (size_t) ys * q.bew + xs) != q.allowed_index) continue;
            const int c = pt_xy(xs, ys);
            bool dup = c == own || !(key[i] < finf());      /* as the sorted list: finite keys only */
#pragma unroll
            for (int t = 0; t < i; t++) dup |= cand[t] == c;
            if (!dup) cand[i] = c;
        }
        bool from = false, tie = false;   /* bpos is a neighbour's candidate, with key kb; another equals it */
        float kb = 0.f;
#pragma unroll
        for (int i0 = 0; i0 < MAXC; i0 += G) {
            float d[G];
#pragma unroll
            for (int i = 0; i < G; i++) d[i] = cand[i0 + i] >= 0 ? l.dist(q, cand[i0 + i]) : 0.f;
#pragma unroll
            for (int i = 0; i < G; i++) {
                if (cand[i0 + i] < 0) continue;
                ne++;
                if (d[i] < bd || (d[i] == bd && from && key[i0 + i] < kb)) {
                    bd = d[i];
                    bpos = cand[i0 + i];
                    kb = key[i0 + i];
                    from = true;
                    tie = false;
                } else if (d[i] == bd && from && key[i0 + i] == kb) {
                    tie = true;
                }
            }
        }
        if (tie) {
            int sc[MAXC];
            float sk[MAXC];
#pragma unroll
            for (int t = 0; t < MAXC; t++) { sc[t] = -1; sk[t] = finf(); }
#pragma unroll
            for (int i = 0; i < MAXC; i++) {
                if (cand[i] < 0) continue;
                int c = cand[i];
                float k = key[i];
#pragma unroll
                for (int t = 0; t < MAXC; t++) {
                    if (k < sk[t]) {
                        const float tk = sk[t]; sk[t] = k; k = tk;
                        const int tc = sc[t]; sc[t] = c; c = tc;
                    }
                }
            }
            bool found = false;
#pragma unroll
            for (int t = 0; t < MAXC; t++)
                if (!found && sc[t] >= 0 && l.dist(q, sc[t]) == bd) { bpos = sc[t]; found = true; }
        }
        if (q.ann) {
            double *o = q.ann + 3 * (size_t) p;
            o[0] = pt_x(bpos);
            o[1] = pt_y(bpos);
            o[2] = bd;
        } else {
            nxt_pos[p] = bpos;
            nxt_d[p] = bd;
        }
        if (q.nx.ch_pos) {
            l.start(q, bpos, bd);
            l.walk(q, q.nx.kcoh, q.nx.kc_done, q.nx.use_done, q.nx.do_kcoh, q.nx.pass, p);
            q.nx.ch_pos[p] = l.best;
            q.nx.ch_d[p] = l.dch;
        }
    }
    count_work(counters, ne, ne);
}

}  // namespace

pt_status pt_choose_desc(const QuerySetup &s, const int *cur_pos, const float *cur_d, const int *tcand, const int2 *kcoh,
                         int do_table, int *ch_pos, float *ch_d, int *kc_done, int use_done, unsigned long long *evals,
                         cudaStream_t st) {
    QPlan q;
    PT_TRY(make_qplan(s, q));
    constexpr int T = TILE_DESC;
    const dim3 grid = tile_grid(q, T);
    PT_CUDA(launch(early(s, q, false), k_choose_desc, grid, T, 0, st, q, cur_pos, cur_d, tcand, kcoh, do_table,
                   ch_pos, ch_d, kc_done, use_done, evals));
    PT_LAUNCHED();
    return PT_OK;
}

pt_status pt_pull_desc(const QuerySetup &s, const float *a, const int *cur_pos, const float *cur_d, const int *ch_pos,
                       const float *ch_d, int *nxt_pos, float *nxt_d, unsigned long long *evals, cudaStream_t st) {
    QPlan q;
    PT_TRY(make_qplan(s, q));
    const bool r1 = q.radius <= 1;
    constexpr int T = TILE_DESC;
    const dim3 grid = tile_grid(q, T);
    if (q.pull_max >= 24) {              /* every neighbour's candidate */
        if (r1) PT_CUDA(launch(early(s, q, false), k_pull_desc<1>, grid, T, 0, st, q, cur_pos, cur_d, ch_pos, ch_d,
                               nxt_pos, nxt_d, evals));
        else PT_CUDA(launch(early(s, q, false), k_pull_desc<2>, grid, T, 0, st, q, cur_pos, cur_d, ch_pos, ch_d,
                            nxt_pos, nxt_d, evals));
    }
    else if (r1) PT_CUDA(launch(early(s, q, false), (k_pull_tile<T, 1, true>), grid, T, 0, st, q, a, cur_pos, cur_d,
                        ch_pos, ch_d, nxt_pos, nxt_d, evals));
    else PT_CUDA(launch(early(s, q, false), (k_pull_tile<T, 2, true>), grid, T, 0, st, q, a, cur_pos, cur_d,
                        ch_pos, ch_d, nxt_pos, nxt_d, evals));
    PT_LAUNCHED();
    return PT_OK;
}
