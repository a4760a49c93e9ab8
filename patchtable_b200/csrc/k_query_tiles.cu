/* The choose and the pull of a single image in CTAs of 32, 64 or 256 patches (gpu_tile), and the choose
   with the learned network's proposals. */
#include "k_query.cuh"

pt_status pt_choose_tiles(const QuerySetup &s, const float *a, const int *cur_pos, const float *cur_d, const int *tcand,
                          const int2 *kcoh, int do_table, int *ch_pos, float *ch_d, int *kc_done, int use_done,
                          unsigned long long *evals, cudaStream_t st) {
    QPlan q;
    PT_TRY(make_qplan(s, q));
#define PT_CHOOSE_T(T) return choose_width<T>(s, q, a, cur_pos, cur_d, tcand, kcoh, do_table, ch_pos, ch_d, kc_done, use_done, \
                                              evals, st)
    switch (q.tile) {
        case 32: PT_CHOOSE_T(32);
        case 64: PT_CHOOSE_T(64);
        default: PT_CHOOSE_T(256);
    }
#undef PT_CHOOSE_T
}

pt_status pt_pull_tiles(const QuerySetup &s, const float *a, const int *cur_pos, const float *cur_d, const int *ch_pos,
                        const float *ch_d, int *nxt_pos, float *nxt_d, unsigned long long *evals, cudaStream_t st) {
    QPlan q;
    PT_TRY(make_qplan(s, q));
#define PT_PULL_T(T) return q.radius <= 1 \
        ? pull_width<T, 1>(s, q, a, cur_pos, cur_d, ch_pos, ch_d, nxt_pos, nxt_d, evals, st) \
        : pull_width<T, 2>(s, q, a, cur_pos, cur_d, ch_pos, ch_d, nxt_pos, nxt_d, evals, st)
    switch (q.tile) {
        case 32: PT_PULL_T(32);
        case 64: PT_PULL_T(64);
        default: PT_PULL_T(256);
    }
#undef PT_PULL_T
}

pt_status pt_launch_choose_learned(const QuerySetup &s, const float *a, const int *cur_pos,
                                   const float *cur_d, const int *tcand, const int2 *kcoh, int do_table, int *ch_pos,
                                   float *ch_d, int *kc_done, int use_done, const int *lcand, const float *lconf,
                                   float threshold, int kcoh_confident, unsigned long long *evals,
                                   unsigned long long *lcounters, cudaStream_t st) {
    QPlan q;
    PT_TRY(make_qplan(s, q));
    if (!lconf) return pt_fail(PT_BAD_ARG, "learned choose without confidences");
    if (q.adesc) return pt_fail(PT_UNSUPPORTED, "learned proposals in descriptor mode");
    LearnedArgs la;
    la.cand = lcand;
    la.conf = lconf;
    la.threshold = threshold;
    la.kcoh_confident = kcoh_confident;
    la.counters = lcounters;
#define PT_CHOOSE_L(T) { const dim3 grid = tile_grid(q, T); \
        k_choose_tile<T, true><<<grid, T, atile_bytes(T), st>>>(q, a, cur_pos, cur_d, tcand, kcoh, \
                                                                                   do_table, ch_pos, ch_d, kc_done, use_done, \
                                                                                   evals, la); }
    switch (q.tile) {
        case 32: PT_CHOOSE_L(32) break;
        case 64: PT_CHOOSE_L(64) break;
        case 128: PT_CHOOSE_L(128) break;
        default: PT_CHOOSE_L(256) break;
    }
#undef PT_CHOOSE_L
    PT_LAUNCHED();
    return PT_OK;
}
