/* Query kernels of single images at the default CTA width, the initial and the final fields, and the row
   store of the table image. */
#include <algorithm>

#include "k_query.cuh"

namespace {

/* The row store of a table image: for every image row and every even pixel 2c, the 32 floats
   (10 pixels and 2 floats of the next) from that pixel on, as one 128-byte line with the floats of
   equal index mod 4 together: float i of the run is at 8 * (i & 3) + i / 4.  A patch row at column
   x starts at float 3 * (x & 1) of line x / 2, so its float e = j + 4 n of SSE lane j lies in the
   8-float group (i0 & 3) at i0 / 4 + n with i0 = 3 * (x & 1) + j: one 32-byte load per lane, the
   four lanes of a quad reading one whole line, and one select per float.  64 bytes per pixel (the
   two RGBA copies that single-lane gathers needed took 32).  A line per third pixel takes 43 bytes
   but two selects per float: 1080p query at one pass 0.500 against 0.462 ms, default schedule 4.40
   against 4.02; a line per pixel (128 bytes, no select) gains 2 % more. */
__global__ void k_row_store(const float4 *__restrict__ b, int bw, int bh, int nline, float *out) {
    const long long t = blockIdx.x * (long long) NT + threadIdx.x;
    if (t >= (long long) bh * nline * 32) return;
    const long long line = t >> 5;
    const int y = (int) (line / nline), c = (int) (line - (long long) y * nline);
    const int g = (int) (t & 31) >> 3, m = (int) t & 7, i = 4 * m + g;
    const int x = 2 * c + i / 3, ch = i % 3;
    float v = 0.f;
    if (x < bw) {
        const float4 px = __ldg(b + (size_t) y * bw + x);
        v = ch == 0 ? px.x : ch == 1 ? px.y : px.z;
    }
    out[t] = v;
}

/* Initial field from the previous frame's NNF (patchtable.h:3548-3585): its matches (clamped to
   the table image when sanitize is set) with either their distance recomputed and scaled by
   scale_sv[p] (when given) or temporal_scale, or the previous distance times temporal_scale.
   orig[p] keeps what the end of the lookup restores for a patch that kept this match and this
   distance (patchtable.h:4178-4193): the scaled distance divided by temporal_scale. */
template<bool DESC>
__global__ void __launch_bounds__(TILE_DEFAULT)
k_init_temporal(const QPlan q, const double *__restrict__ prev, const float *__restrict__ scale_sv, int recalc,
                int sanitize, double temporal_scale, const float *__restrict__ a, int *cur_pos, float *cur_d, double *orig,
                int *bad) {
    constexpr int TP = TILE_DEFAULT;
    __shared__ float at[atile_bytes(TP) / sizeof(float)];
    const int x0 = blockIdx.x * cta_w(TP, DESC), y0 = blockIdx.y * cta_h(TP, DESC);
    if constexpr (!DESC) {
        if (recalc) {
            stage_a<TP>(at, a, q.aw, q.ah, x0, y0);
            stage_wait();
            __syncthreads();
        }
    }
    AQuery aq;
    int x, y;
    tile_lane<TP, DESC>(q, at, x0, y0, x, y, aq);
    const bool live = x < q.ew && y < q.eh;
    const int p = live ? y * q.ew + x : 0;
    int xs = 0, ys = 0;
    if (live) {
        xs = (int) prev[3 * (size_t) p];
        ys = (int) prev[3 * (size_t) p + 1];
        if (xs < 0 || ys < 0 || xs >= q.bew || ys >= q.beh) {
            if (!sanitize) atomicExch(bad, 1);
            xs = min(max(xs, 0), q.bew - 1);
            ys = min(max(ys, 0), q.beh - 1);
        }
    }
    double scaled = 0.0;
    if (recalc) {
        if constexpr (DESC) pt_desc_load(q.adesc + (size_t) p * q.ds4, 4 * q.ds4, aq.v);
        unsigned rows = 0;
        const float dcur = dist32<TP, DESC, false>(aq, q, pt_xy(xs, ys), live, finf(), rows);
        if (live) scaled = (double) dcur * (scale_sv ? (double) scale_sv[p] : temporal_scale);
    } else if (live) {
        scaled = prev[3 * (size_t) p + 2] * temporal_scale;
    }
    if (!live) return;
    cur_pos[p] = pt_xy(xs, ys);
    cur_d[p] = (float) scaled;
    orig[p] = scaled / temporal_scale;
}

/* init_random (patchtable.h:3522-3537): a random match per patch with its distance; the match
   comes from a hash of the patch index instead of two rand() calls. */
template<bool DESC>
__global__ void __launch_bounds__(TILE_DEFAULT)
k_init_random(const QPlan q, const float *__restrict__ a, int *cur_pos, float *cur_d) {
    constexpr int TP = TILE_DEFAULT;
    __shared__ float at[atile_bytes(TP) / sizeof(float)];
    const int x0 = blockIdx.x * cta_w(TP, DESC), y0 = blockIdx.y * cta_h(TP, DESC);
    if constexpr (!DESC) {
        stage_a<TP>(at, a, q.aw, q.ah, x0, y0);
        stage_wait();
        __syncthreads();
    }
    AQuery aq;
    int x, y;
    tile_lane<TP, DESC>(q, at, x0, y0, x, y, aq);
    const bool live = x < q.ew && y < q.eh;
    const int p = live ? y * q.ew + x : 0;
    unsigned hsh = mix32((unsigned) p * 0x9e3779b1u + 0x85ebca6bu);
    const int xs = (int) (hsh % (unsigned) q.bew);
    hsh = mix32(hsh ^ 0x27d4eb2fu);
    const int ys = (int) (hsh % (unsigned) q.beh);
    if constexpr (DESC) pt_desc_load(q.adesc + (size_t) p * q.ds4, 4 * q.ds4, aq.v);
    unsigned rows = 0;
    const float d = dist32<TP, DESC, false>(aq, q, pt_xy(xs, ys), live, finf(), rows);
    if (!live) return;
    cur_pos[p] = pt_xy(xs, ys);
    cur_d[p] = d;
}

/* The float64 NNF; a patch whose match and distance are still the initial temporal ones gets the
   unscaled distance back (patchtable.h:4178-4193). */
__global__ void k_output_temporal(int n, const int *__restrict__ pos, const float *__restrict__ d,
                                  const int *__restrict__ pos0, const float *__restrict__ d0,
                                  const double *__restrict__ orig, double *ann) {
    const int p = blockIdx.x * NT + threadIdx.x;
    if (p >= n) return;
    const int v = pos[p];
    ann[3 * (size_t) p + 0] = pt_x(v);
    ann[3 * (size_t) p + 1] = pt_y(v);
    ann[3 * (size_t) p + 2] = (v == pos0[p] && d[p] == d0[p]) ? orig[p] : (double) d[p];
}

__global__ void k_init(int n, int pos, float d, int *cur_pos, float *cur_d) {
    int p = blockIdx.x * NT + threadIdx.x;
    if (p < n) { cur_pos[p] = pos; cur_d[p] = d; }
}

/* The packed form of a float64 NNF whose distances are float values (every lookup but the
   temporal one): position x | y << 16 and the float distance, both exact. */
__global__ void k_pack_nnf(long long n, const double *__restrict__ ann, int *pos, float *d) {
    const long long p = blockIdx.x * (long long) NT + threadIdx.x;
    if (p >= n) return;
    pos[p] = pt_xy((int) ann[3 * p], (int) ann[3 * p + 1]);
    d[p] = (float) ann[3 * p + 2];
}

__global__ void k_output(int n, const int *__restrict__ pos, const float *__restrict__ d, double *ann) {
    int p = blockIdx.x * NT + threadIdx.x;
    if (p >= n) return;
    int v = pos[p];
    ann[3 * (size_t) p + 0] = pt_x(v);
    ann[3 * (size_t) p + 1] = pt_y(v);
    ann[3 * (size_t) p + 2] = d[p];
}

}  // namespace

static std::atomic<int> g_lean_kernels{1};

bool pt_lean_kernels() { return g_lean_kernels.load(std::memory_order_relaxed); }

/* Schedules whose later chooses have much to do (a spatial search) or whose pulls have (24 neighbours)
   gain from the launches saved only while the image is small: -speed 1, in us, 355 x 611 829 apart and
   797 together, 540 x 960 1,675 and 1,705; -speed 6 653 and 649, 1,491 and 1,505. */
bool pt_pull_chooses(const QuerySetup &s, long long patches) {
    if (s.adesc) return s.pull_max <= 0 || s.pull_max >= 24;
    if (pt_lean_kernels() && s.pull_max == 1) return false;
    return (s.spatial <= 0 && s.radius <= 1) || patches <= 64ll * 32 * sm_count();
}

extern "C" int pt_set_lean_kernels(int on) { return g_lean_kernels.exchange(on ? 1 : 0); }

int pt_row_lines(int bw) { return (bw - 7 + 1) / 2; }       /* lines of patch columns 0 .. bw - 8 */

size_t pt_row_store_floats(int bw, int bh) { return (size_t) pt_row_lines(bw) * bh * 32; }

void pt_row_image(const float *row, int bw, float *rgb) {
    const int last = pt_row_lines(bw) - 1;
    for (int x = 0; x < bw; x++) {
        const int line = std::min(x / 2, last);
        for (int ch = 0; ch < 3; ch++) {
            const int i = 3 * (x - 2 * line) + ch;
            rgb[3 * x + ch] = row[32 * (size_t) line + 8 * (i & 3) + i / 4];
        }
    }
}

pt_status pt_launch_row_store(const float4 *b, int bw, int bh, float *out, cudaStream_t st) {
    const long long n = (long long) pt_row_store_floats(bw, bh);
    k_row_store<<<(unsigned) ((n + NT - 1) / NT), NT, 0, st>>>(b, bw, bh, pt_row_lines(bw), out);
    PT_LAUNCHED();
    return PT_OK;
}

pt_status pt_launch_init(int n, int pos, float d, int *cur_pos, float *cur_d, cudaStream_t st) {
    k_init<<<(n + NT - 1) / NT, NT, 0, st>>>(n, pos, d, cur_pos, cur_d);
    PT_LAUNCHED();
    return PT_OK;
}

pt_status pt_launch_choose(const QuerySetup &s, int n, const float *a, const int *cur_pos, const float *cur_d,
                           const int *tcand, const int2 *kcoh, int do_table, int *ch_pos,
                           float *ch_d, int *kc_done, int use_done, unsigned long long *evals, cudaStream_t st) {
    QPlan q;
    PT_TRY(make_qplan(s, q));
    (void) n;
    if (q.adesc)
        return pt_choose_desc(s, cur_pos, cur_d, tcand, kcoh, do_table, ch_pos, ch_d, kc_done, use_done, evals, st);
    if (q.tile != TILE_DEFAULT)
        return pt_choose_tiles(s, a, cur_pos, cur_d, tcand, kcoh, do_table, ch_pos, ch_d, kc_done, use_done, evals, st);
    return choose_width<TILE_DEFAULT>(s, q, a, cur_pos, cur_d, tcand, kcoh, do_table, ch_pos, ch_d, kc_done, use_done, evals,
                                      st);
}

pt_status pt_launch_pull(const QuerySetup &s, int n, const float *a, const int *cur_pos, const float *cur_d,
                         const int *ch_pos, const float *ch_d, int *nxt_pos, float *nxt_d,
                         unsigned long long *evals, cudaStream_t st) {
    QPlan q;
    PT_TRY(make_qplan(s, q));
    (void) n;
    const bool r1 = q.radius <= 1;
    if (q.adesc) return pt_pull_desc(s, a, cur_pos, cur_d, ch_pos, ch_d, nxt_pos, nxt_d, evals, st);
    const bool one = one_pull(q) && !q.nx.ch_pos;
    /* Small images leave most of the chip idle and wait for one warp's rounds of candidates: four
       warps share a tile's list.  The four pulls of the default schedule, in us: 48 x 64 98 -> 58,
       100 x 150 (2.8 tiles per SM) 119 -> 66, 140 x 200 (5.4) 124 -> 107, 180 x 260 (9.2) 137 -> 159. */
    const dim3 tiles = tile_grid(q, 32);
    if (q.auto_tile && !one && (long long) tiles.x * tiles.y <= (long long) SPLIT_TILES * sm_count()) {
        constexpr int T = 32;
        if (r1)
            PT_CUDA(launch(early(s, q, one), (k_pull_tile<T, 1, false, false, true, SPLIT_D, SPLIT_W>), tiles, T * SPLIT_W,
                           atile_bytes(T), st, q, a, cur_pos, cur_d, ch_pos, ch_d, nxt_pos, nxt_d, evals));
        else
            PT_CUDA(launch(early(s, q, one), (k_pull_tile<T, 2, false, false, true, SPLIT_D, SPLIT_W>), tiles, T * SPLIT_W,
                           atile_bytes(T), st, q, a, cur_pos, cur_d, ch_pos, ch_d, nxt_pos, nxt_d, evals));
        PT_LAUNCHED();
        return PT_OK;
    }
    if (q.tile != TILE_DEFAULT) return pt_pull_tiles(s, a, cur_pos, cur_d, ch_pos, ch_d, nxt_pos, nxt_d, evals, st);
    return r1 ? pull_width<TILE_DEFAULT, 1>(s, q, a, cur_pos, cur_d, ch_pos, ch_d, nxt_pos, nxt_d, evals, st)
              : pull_width<TILE_DEFAULT, 2>(s, q, a, cur_pos, cur_d, ch_pos, ch_d, nxt_pos, nxt_d, evals, st);
}

pt_status pt_launch_pack_nnf(long long n, const double *ann, int *pos, float *d, cudaStream_t st) {
    if (n <= 0) return PT_OK;
    k_pack_nnf<<<(unsigned) ((n + NT - 1) / NT), NT, 0, st>>>(n, ann, pos, d);
    PT_LAUNCHED();
    return PT_OK;
}

pt_status pt_launch_output(int n, const int *pos, const float *d, double *ann, cudaStream_t st) {
    k_output<<<(n + NT - 1) / NT, NT, 0, st>>>(n, pos, d, ann);
    PT_LAUNCHED();
    return PT_OK;
}

pt_status pt_launch_init_temporal(const QuerySetup &s, const double *prev, const float *scale_sv, int recalc, int sanitize,
                                  double temporal_scale, const float *a, int *cur_pos, float *cur_d,
                                  double *orig, int *bad, cudaStream_t st) {
    QPlan q;
    PT_TRY(make_qplan(s, q));
    const dim3 grid = tile_grid(q, TILE_DEFAULT);
    if (q.adesc)
        k_init_temporal<true><<<grid, TILE_DEFAULT, 0, st>>>(q, prev, scale_sv, recalc, sanitize, temporal_scale, a, cur_pos,
                                                             cur_d, orig, bad);
    else
        k_init_temporal<false><<<grid, TILE_DEFAULT, 0, st>>>(q, prev, scale_sv, recalc, sanitize, temporal_scale, a, cur_pos,
                                                              cur_d, orig, bad);
    PT_LAUNCHED();
    return PT_OK;
}

pt_status pt_launch_output_temporal(int n, const int *pos, const float *d, const int *pos0, const float *d0,
                                    const double *orig, double *ann, cudaStream_t st) {
    k_output_temporal<<<(n + NT - 1) / NT, NT, 0, st>>>(n, pos, d, pos0, d0, orig, ann);
    PT_LAUNCHED();
    return PT_OK;
}

pt_status pt_launch_init_random(const QuerySetup &s, const float *a, int *cur_pos, float *cur_d,
                                cudaStream_t st) {
    QPlan q;
    PT_TRY(make_qplan(s, q));
    const dim3 grid = tile_grid(q, TILE_DEFAULT);
    if (q.adesc) k_init_random<true><<<grid, TILE_DEFAULT, 0, st>>>(q, a, cur_pos, cur_d);
    else k_init_random<false><<<grid, TILE_DEFAULT, 0, st>>>(q, a, cur_pos, cur_d);
    PT_LAUNCHED();
    return PT_OK;
}
