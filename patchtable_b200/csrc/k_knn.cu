/* Exact k-nearest-neighbour search in descriptor space for the k-coherence step.

   Ranking (shared with the CPU oracle): squared L2 in float, dimensions summed in index order,
   each product and sum rounded (no fused operations); ties by the smaller point index.

   Structure: train points are sorted along a Hilbert curve through their quantised descriptors and cut into
   buckets of 32 consecutive points, with axis-aligned boxes over the buckets and over groups of 32
   boxes, level by level.  Queries are processed in the same order, 32 to a warp; the warp walks the
   boxes together (k_knn_mma) and screens a bucket's 32 x 32 pairs with tensor-core products whose
   rounding is bounded, so that only pairs which may enter a list are evaluated exactly.  A subtree,
   bucket or pair is dropped only when its lower bound exceeds the current k-th distance by more
   than the rounding could account for -- so the result equals an exhaustive search.  Lists longer
   than 64 walk a binary tree of the same buckets (k_knn_wide). */
#include <cuda_runtime.h>
#include <cub/cub.cuh>
#include <cuda_fp16.h>

#include "pt_internal.h"
#include "pt_kernels.h"

namespace {

constexpr int NT = 128;
constexpr int BUCKET = 32;

__global__ void k_range(const float *__restrict__ pts, int N, int nd, float *mn, float *mx) {
    __shared__ float smin[PT_DESC_MAX][NT], smax[PT_DESC_MAX][NT];
    float a[PT_DESC_MAX], b[PT_DESC_MAX];
    for (int d = 0; d < nd; d++) { a[d] = __int_as_float(0x7f800000); b[d] = -__int_as_float(0x7f800000); }
    for (int i = blockIdx.x * NT + threadIdx.x; i < N; i += gridDim.x * NT)
        for (int d = 0; d < nd; d++) { float v = pts[(size_t) i * nd + d]; a[d] = fminf(a[d], v); b[d] = fmaxf(b[d], v); }
    for (int d = 0; d < nd; d++) { smin[d][threadIdx.x] = a[d]; smax[d][threadIdx.x] = b[d]; }
    __syncthreads();
    if (threadIdx.x < nd) {
        int d = threadIdx.x;
        float u = smin[d][0], v = smax[d][0];
        for (int i = 1; i < NT; i++) { u = fminf(u, smin[d][i]); v = fmaxf(v, smax[d][i]); }
        mn[blockIdx.x * PT_DESC_MAX + d] = u;
        mx[blockIdx.x * PT_DESC_MAX + d] = v;
    }
}

struct Quant {
    int nd, bits;
    float mn[PT_DESC_MAX], scale[PT_DESC_MAX];
};

/* Position of a point on the Hilbert curve through the quantised cells (J. Skilling, "Programming the
   Hilbert curve", AIP Conf. Proc. 707, 2004): unlike a Morton code's, its runs never jump, so 32
   consecutive points lie together wherever the points are dense. */
__global__ void k_curve(const Quant qz, const float *__restrict__ pts, int N, unsigned long long *codes, int *idx) {
    int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= N) return;
    unsigned q[PT_DESC_MAX];
    const unsigned top = (1u << qz.bits) - 1;
#pragma unroll
    for (int d = 0; d < PT_DESC_MAX; d++) {
        q[d] = 0;
        if (d < qz.nd) {
            float t = (pts[(size_t) i * qz.nd + d] - qz.mn[d]) * qz.scale[d];
            t = fminf(fmaxf(t, 0.f), (float) top);
            q[d] = (unsigned) t;
        }
    }
    /* undo the curve's exchanges and inversions, level by level, then Gray-encode */
    for (unsigned Q = 1u << (qz.bits - 1); Q > 1; Q >>= 1) {
        const unsigned P = Q - 1;
#pragma unroll
        for (int d = 0; d < PT_DESC_MAX; d++) {
            if (d < qz.nd) {
                if (q[d] & Q) {
                    q[0] ^= P;
                } else {
                    const unsigned t = (q[0] ^ q[d]) & P;
                    q[0] ^= t;
                    q[d] ^= t;
                }
            }
        }
    }
    unsigned last = q[0];
#pragma unroll
    for (int d = 1; d < PT_DESC_MAX; d++)
        if (d < qz.nd) { q[d] ^= q[d - 1]; last = q[d]; }
    unsigned flip = 0;
    for (unsigned Q = 1u << (qz.bits - 1); Q > 1; Q >>= 1)
        if (last & Q) flip ^= Q - 1;
    unsigned long long c = 0;
    for (int b = qz.bits - 1; b >= 0; b--) {
#pragma unroll
        for (int d = 0; d < PT_DESC_MAX; d++)
            if (d < qz.nd) c = (c << 1) | (((q[d] ^ flip) >> b) & 1u);
    }
    codes[i] = c;
    idx[i] = i;
}

__global__ void k_reorder(const float *__restrict__ pts, int N, int nd, const int *__restrict__ perm, float *sp) {
    long long t = blockIdx.x * 256ll + threadIdx.x;
    if (t >= (long long) N * nd) return;
    int i = (int) (t / nd), d = (int) (t % nd);
    sp[t] = pts[(size_t) perm[i] * nd + d];
}

/* Leaf boxes (heap nodes L .. 2L-1); empty leaves get an inverted box. */
__global__ void k_leaf_box(const float *__restrict__ sp, int N, int nd, int L, float *lo, float *hi) {
    int j = blockIdx.x * 256 + threadIdx.x;
    if (j >= L) return;
    int node = L + j;
    for (int d = 0; d < nd; d++) {
        float a = __int_as_float(0x7f800000), b = -__int_as_float(0x7f800000);
        for (int i = j * BUCKET; i < min(N, (j + 1) * BUCKET); i++) { float v = sp[(size_t) i * nd + d]; a = fminf(a, v); b = fmaxf(b, v); }
        lo[(size_t) node * nd + d] = a;
        hi[(size_t) node * nd + d] = b;
    }
}

__global__ void k_inner_box(int first, int count, int nd, float *lo, float *hi) {
    int j = blockIdx.x * 256 + threadIdx.x;
    if (j >= count) return;
    int node = first + j;
    for (int d = 0; d < nd; d++) {
        lo[(size_t) node * nd + d] = fminf(lo[(size_t) (2 * node) * nd + d], lo[(size_t) (2 * node + 1) * nd + d]);
        hi[(size_t) node * nd + d] = fmaxf(hi[(size_t) (2 * node) * nd + d], hi[(size_t) (2 * node + 1) * nd + d]);
    }
}

/* Squared distance from q to a box, rounded down enough to be a lower bound of the squared distance. */
__device__ __forceinline__ float box_lb(const float (&q)[PT_DESC_MAX], const float *lo, const float *hi, int nd) {
    float s = 0.f;
#pragma unroll
    for (int d = 0; d < PT_DESC_MAX; d++) {          /* unrolled: q stays in registers */
        if (d < nd) {
            float e = fmaxf(fmaxf(lo[d] - q[d], q[d] - hi[d]), 0.f);
            s += e * e;
        }
    }
    return s * (1.0f - 1e-5f);
}

__device__ __forceinline__ bool before(float d, int i, float d2, int i2) { return d < d2 || (d == d2 && i < i2); }

constexpr int KNN_STACK = 64;
constexpr int PSTRIDE = PT_DESC_MAX + 1;            /* staged point stride (odd: no bank conflicts) */

/* ---- screened search ---- */

constexpr int KNN_NT = 64;                          /* threads per CTA of the screened search */
constexpr int KNN_SUB = 4;                          /* boxes around a warp's queries, 8 each */
constexpr int KNN_LEVELS = 4;                       /* box levels above the buckets: 32^5 points per top box */

/* Boxes of every level, dimension-major: lo of dimension d at box[l] + d * stride[l], hi nd rows
   further; level 0 = buckets.  Row strides are multiples of 32 and padded with inverted boxes.
   bucket: the buckets' boxes again, one row of dp lower and dp upper bounds each. */
struct KnnTree {
    const float *bucket;
    const float *box[KNN_LEVELS + 1];
    int count[KNN_LEVELS + 1], stride[KNN_LEVELS + 1];
};

/* Bucket boxes from the sorted points (padded rows of dp floats), level 0 of the tree. */
__global__ void k_bucket_box(const float *__restrict__ sp, int N, int nd, int dp, int n, int stride, float *box,
                             float *rows) {
    const int j = blockIdx.x * 256 + threadIdx.x;
    if (j >= stride) return;
    for (int d = 0; d < nd; d++) {
        float a = __int_as_float(0x7f800000), b = -__int_as_float(0x7f800000);
        if (j < n)
            for (int i = j * BUCKET; i < min(N, (j + 1) * BUCKET); i++) {
                const float v = sp[(size_t) i * dp + d];
                a = fminf(a, v);
                b = fmaxf(b, v);
            }
        box[(size_t) d * stride + j] = a;
        box[(size_t) (nd + d) * stride + j] = b;
        if (j < n) {
            rows[(size_t) j * 2 * dp + d] = a;
            rows[(size_t) j * 2 * dp + dp + d] = b;
        }
    }
    if (j < n)
        for (int d = nd; d < dp; d++) rows[(size_t) j * 2 * dp + d] = rows[(size_t) j * 2 * dp + dp + d] = 0.f;
}

/* Keys that put the warps whose queries lie farthest apart (the diagonals of their boxes) first,
   since those open the most buckets: a sort of 30 us with its keys for 64,000 warps. */
__global__ void k_warp_spread(const float *__restrict__ qdesc, const int *__restrict__ qorder, int Q, int nd,
                              unsigned long long *key, int *warp) {
    const int t = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31;
    if (t - lane >= Q) return;
    const int q = qorder[min(t, Q - 1)];
    float sum = 0.f;
    for (int d = 0; d < nd; d++) {
        float a = qdesc[(size_t) q * nd + d], b = a;
        for (int o = 16 / KNN_SUB; o; o >>= 1) {
            a = fminf(a, __shfl_xor_sync(0xffffffffu, a, o));
            b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
        }
        sum += (b - a) * (b - a);
    }
    for (int o = 16 / KNN_SUB * 2; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) {
        key[t >> 5] = 0xffffffffu - __float_as_uint(sum);
        warp[t >> 5] = t >> 5;
    }
}

/* Boxes of level l + 1 from groups of 32 boxes of level l: one warp per box. */
__global__ void k_group_box(const float *__restrict__ in, int nd, int sin, int n, int stride, float *box) {
    const int j = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (j >= stride) return;
    for (int d = 0; d < nd; d++) {
        float a = __int_as_float(0x7f800000), b = -__int_as_float(0x7f800000);
        if (j < n) {
            a = in[(size_t) d * sin + 32 * j + lane];
            b = in[(size_t) (nd + d) * sin + 32 * j + lane];
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            a = fminf(a, __shfl_xor_sync(0xffffffffu, a, o));
            b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
        }
        if (lane == 0) {
            box[(size_t) d * stride + j] = a;
            box[(size_t) (nd + d) * stride + j] = b;
        }
    }
}

/* Points in sorted order as rows of dp floats (8 or 16), zero-padded. */
__global__ void k_reorder_pad(const float *__restrict__ pts, int N, int nd, int dp, const int *__restrict__ perm, float *sp) {
    const long long t = blockIdx.x * 256ll + threadIdx.x;
    if (t >= (long long) N * dp) return;
    const int i = (int) (t / dp), d = (int) (t % dp);
    sp[t] = d < nd ? pts[(size_t) perm[i] * nd + d] : 0.f;
}

/* D += A * B, 16 x 8 x 8, half operands and float sums. */
__device__ __forceinline__ void mma_16x8x8(float (&d)[4], unsigned a0, unsigned a1, unsigned b) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(b));
}

__device__ __forceinline__ unsigned half_pair(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const unsigned *>(&h);
}

/* A float with the 11 leading significand bits kept: exact in half precision (down to 2^-24). */
__device__ __forceinline__ float cut11(float x) { return __uint_as_float(__float_as_uint(x) & 0xffffe000u); }

/* Sum over the four lanes of a quad. */
__device__ __forceinline__ float quad_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

/* State of one warp's search: 32 queries; lane l owns query l.  In the products query 4 g + i is row
   g + 8 i, so the rows a quad g of lanes holds results of belong to its own lanes' queries. */
template<int K, int KS>
struct KnnWarp {
    static constexpr int DP = KS == 1 ? 8 : 16;      /* floats per point row */
    const float *sp;
    const int *sidx;
    const KnnTree &tr;
    int N, nd;
    float scale;
    const float *gbox;                    /* shared: boxes of the warp's queries, KNN_SUB x (lo[d], hi[d]) */
    float qv[DP];                         /* the lane's query */
    unsigned long long key[K];            /* its list, ascending: distance bits << 32 | point index */
    float kd;                             /* K-th distance (+inf until full; -1: no query) */
    float kdmax[KNN_SUB];                 /* the largest kd of each of the warp's boxes */
    float qn, ext;                        /* |q'|^2 of the rounded query, |q'| bounded above */
    float T;                              /* the lane's screening threshold */
    float cen[KS][2];                     /* centre coordinates of the lane's two dimensions per step */
    unsigned afrag[KS][2][2];             /* queries, -2 q', 1, 1 as A operands of the two 16-row tiles */

    __device__ __forceinline__ void thresholds() {
        /* A point whose float distance does not exceed kd has, in scaled units, true distance at
           most r = sqrt(kd) * scale * (1 + 2^-16).  Its rounded coordinates and the query's are off by
           at most 2^-10 of their own size (plus 2^-25 each, below half's normal range), |p'| <= |q'| + r,
           and the split of |p'|^2, the products and the float sums are off by at most 2^-17 of the
           squares involved (plus 2^-24): the screened value then cannot exceed T. */
        const float r = sqrtf(kd) * scale * (1.f + 1.0f / 65536.f);
        const float m = r + 1.002f / 1024.f * (2.f * ext + r) + 1e-6f;
        const float w = ext + m;
        T = kd < 0.f ? -__int_as_float(0x7f800000)
                     : (scale > 0.f && kd < __int_as_float(0x7f800000)) ? m * m * 1.0001f + (w * w + ext * ext) * (1.f / 131072.f) + 2.5e-7f - qn
                                                                       : __int_as_float(0x7f800000);
    }

    /* kdmax from the lanes' kd (the ordering of non-negative floats' bits is theirs; -1 is below) */
    __device__ __forceinline__ void bounds() {
        int v = __float_as_int(kd);
#pragma unroll
        for (int o = 16 / KNN_SUB; o; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
#pragma unroll
        for (int i = 0; i < KNN_SUB; i++) kdmax[i] = __int_as_float(__shfl_sync(0xffffffffu, v, 32 / KNN_SUB * i));
    }

    __device__ __forceinline__ void bucket(int j) {
        const unsigned FULL = 0xffffffffu;
        const int lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
        /* a lane's own bound against the bucket's box, unless every query of the warp is far */
        {
            const float4 *b0 = reinterpret_cast<const float4 *>(tr.bucket + (size_t) j * 2 * DP);
            float s = 0.f;
#pragma unroll
            for (int u = 0; u < DP / 4; u++) {
                const float4 lo = __ldg(b0 + u), hi = __ldg(b0 + DP / 4 + u);
                const float l[4] = {lo.x, lo.y, lo.z, lo.w}, h[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    if (4 * u + e < nd) {
                        const float v = fmaxf(fmaxf(l[e] - qv[4 * u + e], qv[4 * u + e] - h[e]), 0.f);
                        s += v * v;
                    }
                }
            }
            if (!__any_sync(FULL, !(s * (1.0f - 1e-5f) > kd))) return;
        }
        const int base = j * BUCKET, cnt = min(BUCKET, N - base);
        float acc[2][4][4];
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int t = 0; t < 4; t++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[m][t][e] = 0.f;
#pragma unroll
        for (int t = 0; t < 4; t++) {
            float x[KS][2], n2 = 0.f;
            const float *row = sp + (size_t) (base + min(8 * t + g, cnt - 1)) * DP;
#pragma unroll
            for (int k = 0; k < KS; k++) {
                const int d = 8 * k + 2 * c;
                float2 v = make_float2(cen[k][0], cen[k][1]);
                if (d < DP) v = __ldg(reinterpret_cast<const float2 *>(row + d));
                x[k][0] = cut11((v.x - cen[k][0]) * scale);
                x[k][1] = cut11((v.y - cen[k][1]) * scale);
                n2 += x[k][0] * x[k][0] + x[k][1] * x[k][1];
            }
            n2 = quad_sum(n2);
            if (c == 3) {                 /* the last two slots: |p'|^2 as a half and its remainder */
                x[KS - 1][0] = cut11(n2);
                x[KS - 1][1] = n2 - cut11(n2);
            }
#pragma unroll
            for (int k = 0; k < KS; k++) {
                const unsigned b = half_pair(x[k][0], x[k][1]);
                mma_16x8x8(acc[0][t], afrag[k][0][0], afrag[k][0][1], b);
                mma_16x8x8(acc[1][t], afrag[k][1][0], afrag[k][1][1], b);
            }
        }
        /* row i of the lane's quad: acc[i / 2][t][2 (i % 2) + 0, 1], points 8 t + 2 c + 0, 1 */
        unsigned hit[4];
        bool any = false;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float Ti = __shfl_sync(FULL, T, (lane & ~3) | i);
            hit[i] = 0;
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const float u = acc[i >> 1][t][2 * (i & 1)], v = acc[i >> 1][t][2 * (i & 1) + 1];
                if (!(u > Ti)) hit[i] |= 1u << (8 * t);
                if (!(v > Ti)) hit[i] |= 2u << (8 * t);
            }
            any |= hit[i] != 0;
        }
        if (!__any_sync(FULL, any)) return;
        /* to the owners: lane i of the quad gathers row i's bits from its four lanes */
#pragma unroll
        for (int i = 0; i < 4; i++) hit[i] <<= 2 * c;
        const bool b0 = lane & 1, b1 = lane & 2;
        const unsigned u0 = (b0 ? hit[1] : hit[0]) | __shfl_xor_sync(FULL, b0 ? hit[0] : hit[1], 1);
        const unsigned u1 = (b0 ? hit[3] : hit[2]) | __shfl_xor_sync(FULL, b0 ? hit[2] : hit[3], 1);
        unsigned mine = (b1 ? u1 : u0) | __shfl_xor_sync(FULL, b1 ? u0 : u1, 2);
        if (cnt < BUCKET) mine &= (1u << cnt) - 1;
        bool changed = false;
        while (mine) {
            const int m = __ffs(mine) - 1;
            mine &= mine - 1;
            const float4 *row = reinterpret_cast<const float4 *>(sp + (size_t) (base + m) * DP);
            float dsum = 0.f;
#pragma unroll
            for (int u = 0; u < DP / 4; u++) {
                const float4 pv = __ldg(row + u);
                const float pc[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    if (4 * u + e < nd) {
                        const float df = __fsub_rn(qv[4 * u + e], pc[e]);
                        dsum = __fadd_rn(dsum, __fmul_rn(df, df));
                    }
                }
            }
            if (!(dsum <= kd)) continue;
            unsigned long long x = ((unsigned long long) __float_as_uint(dsum) << 32) | (unsigned) sidx[base + m];
            if (x >= key[K - 1]) continue;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const bool lt = x < key[k];
                const unsigned long long lo = lt ? x : key[k];
                x = lt ? key[k] : x;
                key[k] = lo;
            }
            kd = __uint_as_float((unsigned) (key[K - 1] >> 32));
            changed = true;
        }
        __syncwarp();
        if (__any_sync(FULL, changed)) {
            thresholds();
            bounds();
        }
    }

    /* The children of box j of level LEVEL, nearest to the warp's queries first. */
    template<int LEVEL>
    __device__ __forceinline__ void visit(int j) {
        const unsigned FULL = 0xffffffffu;
        const int lane = threadIdx.x & 31, st = tr.stride[LEVEL - 1];
        const float *b0 = tr.box[LEVEL - 1] + 32 * j + lane;
        float s[KNN_SUB];
#pragma unroll
        for (int i = 0; i < KNN_SUB; i++) s[i] = 0.f;
#pragma unroll
        for (int d = 0; d < DP; d++) {
            if (d < nd) {
                const float lo = b0[d * st], hi = b0[(nd + d) * st];
#pragma unroll
                for (int i = 0; i < KNN_SUB; i++) {
                    const float e = fmaxf(fmaxf(lo - gbox[(2 * i + 1) * DP + d], gbox[2 * i * DP + d] - hi), 0.f);
                    s[i] += e * e;
                }
            }
        }
        bool open = 32 * j + lane < tr.count[LEVEL - 1];
        for (;;) {
            float near = __int_as_float(0x7f800000);      /* nearest of the boxes that admit the child */
            bool in = false;
#pragma unroll
            for (int i = 0; i < KNN_SUB; i++)
                if (!(s[i] * (1.0f - 1e-5f) > kdmax[i])) { in = true; near = fminf(near, s[i]); }
            open = open && in;
            const unsigned m = __ballot_sync(FULL, open);
            if (!m) return;
            const unsigned best = __reduce_min_sync(FULL, open ? __float_as_uint(near) : 0xffffffffu);
            const int w = __ffs(__ballot_sync(FULL, open && __float_as_uint(near) == best)) - 1;
            if (w < 0) return;
            if (lane == w) open = false;
            if constexpr (LEVEL == 1) bucket(32 * j + w);
            else visit<LEVEL - 1>(32 * j + w);
        }
    }
};

/* The search, 32 queries of the curve to a warp.  Boxes are tested 32 at a time, a child per lane,
   against four boxes around eight of the warp's queries each (one box around all 32 opens ten
   times the buckets for the few warps whose queries are scattered, and those warps end last); an
   open bucket is tested by every lane against its own query, screened by the tensor cores, and its
   surviving pairs go to the lanes that own the queries, which keep their lists sorted in registers
   as 64-bit keys (distance bits, then index: the ranking).

   Bound: instruction issue, of which the list insertions take the largest part (214 per query); at
   1920x1080 (2.05 M queries, 12 neighbours, 6 dimensions) a warp opens 480 buckets, screens 247 and
   inserts from 95 of them.  24.1 ms, against 109 ms for the exact evaluation of every point of the
   1,500 buckets a binary tree's bounds left open.  The heaviest warps run for half of that time, so
   they start first (worder); started in the curve's order 27.7 ms (with two boxes 27.9, with eight
   30.5, with a Morton order and one box 53.8). */
template<int K, int KS>
__global__ void __launch_bounds__(KNN_NT)
k_knn_mma(const float *__restrict__ sp, const int *__restrict__ sidx, int N, int nd, const KnnTree tr, float scale,
          const float *__restrict__ qdesc, const int *__restrict__ qorder, const int *__restrict__ worder, int Q,
          int *out) {
    typedef KnnWarp<K, KS> W;
    constexpr int DP = W::DP;
    const unsigned FULL = 0xffffffffu;
    __shared__ float gbox_s[KNN_NT / 32][2 * KNN_SUB * DP];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int slot = blockIdx.x * (KNN_NT / 32) + wid;
    if (32ll * slot >= Q) return;
    const int t = worder[slot] * 32 + lane;
    const bool active = t < Q;
    const int q = qorder[active ? t : t - lane];
    W w{sp, sidx, tr, N, nd, scale, gbox_s[wid]};
    float mid[DP];
    float n2 = 0.f;
#pragma unroll
    for (int d = 0; d < DP; d++) {
        w.qv[d] = d < nd ? qdesc[(size_t) q * nd + d] : 0.f;
        float a = w.qv[d], b = w.qv[d];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            if (o == 32 / KNN_SUB && lane % o == 0) {
                gbox_s[wid][2 * (lane / o) * DP + d] = a;
                gbox_s[wid][(2 * (lane / o) + 1) * DP + d] = b;
            }
            a = fminf(a, __shfl_xor_sync(FULL, a, o));
            b = fmaxf(b, __shfl_xor_sync(FULL, b, o));
        }
        mid[d] = a + 0.5f * (b - a);
        const float x = cut11((w.qv[d] - mid[d]) * scale);
        n2 += x * x;
    }
    __syncwarp();
    w.qn = n2;
    w.ext = sqrtf(n2) * 1.002f + 1e-6f;
#pragma unroll
    for (int k = 0; k < K; k++) w.key[k] = (0x7f800000ull << 32) | 0x7fffffffu;
    w.kd = active ? __int_as_float(0x7f800000) : -1.f;
#pragma unroll
    for (int i = 0; i < KNN_SUB; i++) w.kdmax[i] = __int_as_float(0x7f800000);
    /* A operands: element (row, col) of tile m = query row's -2 q' (or 1 in the last two columns);
       the lane holds rows g and g + 8 of each tile, columns 2 c and 2 c + 1 of each step */
    const int g = lane >> 2, c = lane & 3;
#pragma unroll
    for (int k = 0; k < KS; k++) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
            float v = 0.f;
#pragma unroll
            for (int d = 8 * k; d < 8 * k + 8; d++)
                if (d < DP && d == 8 * k + 2 * c + e) v = mid[d];
            w.cen[k][e] = v;
        }
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                /* row g + 8 (2 m + h): query 4 g + 2 m + h */
                float x[2] = {0.f, 0.f};
#pragma unroll
                for (int d = 8 * k; d < 8 * k + 8; d++) {
                    if (d < DP) {
                        const float v = __shfl_sync(FULL, w.qv[d], 4 * g + 2 * m + h);
                        if (d == 8 * k + 2 * c) x[0] = -2.f * cut11((v - mid[d]) * scale);
                        if (d == 8 * k + 2 * c + 1) x[1] = -2.f * cut11((v - mid[d]) * scale);
                    }
                }
                if (k == KS - 1 && c == 3) x[0] = x[1] = 1.f;
                w.afrag[k][m][h] = half_pair(x[0], x[1]);
            }
    }
    w.thresholds();
    for (int j = 0; j < tr.count[KNN_LEVELS]; j++) w.template visit<KNN_LEVELS>(j);
    if (active)
        for (int k = 0; k < K; k++) {
            const int id = (int) (unsigned) w.key[k];
            out[(size_t) q * K + k] = id == 0x7fffffff ? -1 : id;
        }
}

/* The same search for K = 128 .. 1024 (sets that need that many neighbours: thin images, or
   narrow flat regions where the nearest descriptors all lie within kcoherence_min_dist).  The
   sorted list lives in global memory (wd: distances, out: indices, K per query); a leaf's
   admissible points are first sorted in a 32-entry buffer and then merged into the list from the
   back in one pass, keeping the K smallest.  Traversal, rounding and tie rule are those of
   k_knn_mma, so its first 64 entries equal that kernel's result. */
__global__ void __launch_bounds__(NT)
k_knn_wide(const float *__restrict__ sp, const int *__restrict__ sidx, int N, int nd, int L,
           const float *__restrict__ lo, const float *__restrict__ hi, const float *__restrict__ qdesc,
           const int *__restrict__ qorder, int Q, int K, float *wd, int *out) {
    __shared__ int stk_s[NT / 32][KNN_STACK];
    __shared__ float pts_s[NT / 32][BUCKET * PSTRIDE];
    __shared__ int pid_s[NT / 32][BUCKET];
    const unsigned FULL = 0xffffffffu;
    const float INF = __int_as_float(0x7f800000);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int t = blockIdx.x * NT + threadIdx.x;
    const bool active = t < Q;
    const int q = active ? qorder[t] : 0;
    float qv[PT_DESC_MAX];
#pragma unroll
    for (int d = 0; d < PT_DESC_MAX; d++) qv[d] = (active && d < nd) ? qdesc[(size_t) q * nd + d] : 0.f;
    float *ld = wd + (size_t) q * K;
    int *li = out + (size_t) q * K;
    if (active)
        for (int j = 0; j < K; j++) { ld[j] = INF; li[j] = 0x7fffffff; }
    float worst_d = INF;
    int worst_i = 0x7fffffff;
    int *stk = stk_s[wid];
    float *pts = pts_s[wid];
    int *pid = pid_s[wid];
    if (lane == 0) stk[0] = 1;
    __syncwarp();
    int top = 1;
    while (top > 0) {
        const int node = stk[--top];
        __syncwarp();
        const float lb = active ? box_lb(qv, lo + (size_t) node * nd, hi + (size_t) node * nd, nd) : 0.f;
        const bool want = active && !(lb > worst_d);
        if (!__any_sync(FULL, want)) continue;
        if (node >= L) {
            const int base = (node - L) * BUCKET;
            const int cnt = min(BUCKET, N - base);
            if (lane < cnt) {
                const float *src = sp + (size_t) (base + lane) * nd;
                for (int d = 0; d < nd; d++) pts[lane * PSTRIDE + d] = src[d];
                pid[lane] = sidx[base + lane];
            }
            __syncwarp();
            if (want) {
                float bd[BUCKET];
                int bi[BUCKET];
                int nb = 0;
                for (int m = 0; m < cnt; m++) {
                    const float *pv = pts + m * PSTRIDE;
                    float dsum = 0.f;
#pragma unroll
                    for (int d = 0; d < PT_DESC_MAX; d++) {
                        if (d < nd) {
                            const float e = __fsub_rn(qv[d], pv[d]);
                            dsum = __fadd_rn(dsum, __fmul_rn(e, e));
                        }
                    }
                    const int id = pid[m];
                    if (!before(dsum, id, worst_d, worst_i)) continue;
                    int s2 = nb++;
                    while (s2 > 0 && before(dsum, id, bd[s2 - 1], bi[s2 - 1])) { bd[s2] = bd[s2 - 1]; bi[s2] = bi[s2 - 1]; s2--; }
                    bd[s2] = dsum;
                    bi[s2] = id;
                }
                if (nb > 0) {
                    /* backward merge: the union's largest go to virtual slots K .. K+nb-1 and drop out */
                    int ia = K - 1, ib = nb - 1;
                    for (int p = K + nb - 1; ib >= 0; p--) {
                        if (ia < 0 || before(ld[ia], li[ia], bd[ib], bi[ib])) {
                            if (p < K) { ld[p] = bd[ib]; li[p] = bi[ib]; }
                            ib--;
                        } else {
                            if (p < K) { ld[p] = ld[ia]; li[p] = li[ia]; }
                            ia--;
                        }
                    }
                    worst_d = ld[K - 1];
                    worst_i = li[K - 1];
                }
            }
            __syncwarp();                        /* the next leaf restages the points */
            continue;
        }
        const int c0 = 2 * node, c1 = 2 * node + 1;
        float l0 = 0.f, l1 = 0.f;
        if (want) {
            l0 = box_lb(qv, lo + (size_t) c0 * nd, hi + (size_t) c0 * nd, nd);
            l1 = box_lb(qv, lo + (size_t) c1 * nd, hi + (size_t) c1 * nd, nd);
        }
        float s0 = l0, s1 = l1;
#pragma unroll
        for (int o = 16; o; o >>= 1) { s0 += __shfl_xor_sync(FULL, s0, o); s1 += __shfl_xor_sync(FULL, s1, o); }
        if (top + 2 > KNN_STACK) continue;        /* cannot happen: depth <= 31 */
        if (lane == 0) {
            if (s0 <= s1) { stk[top] = c1; stk[top + 1] = c0; }
            else { stk[top] = c0; stk[top + 1] = c1; }
        }
        __syncwarp();
        top += 2;
    }
    if (active)
        for (int j = 0; j < K; j++)
            if (li[j] == 0x7fffffff) li[j] = -1;
}

}  // namespace

/* Exact top-K (K in {12, 16, 24, 32, 48, 64}, or a power of two up to PT_KNN_WIDE_MAX) train
   indices of every query, ascending (dist, index). */
pt_status pt_launch_knn(const float *train, int N, int nd, const float *qdesc, int Q, int K, int *out, cudaStream_t st) {
    if (N < 1 || Q < 1) return PT_OK;
    if (nd < 1 || nd > PT_DESC_MAX) return pt_fail(PT_UNSUPPORTED, "knn: %d dims", nd);
    /* range of the train and query points */
    const int NB = 2 * 148;
    DevBuf<float> pmn(st), pmx(st);
    PT_CUDA(pmn.reserve(NB * PT_DESC_MAX));
    PT_CUDA(pmx.reserve(NB * PT_DESC_MAX));
    k_range<<<NB / 2, NT, 0, st>>>(train, N, nd, pmn.p, pmx.p);
    PT_LAUNCHED();
    k_range<<<NB / 2, NT, 0, st>>>(qdesc, Q, nd, pmn.p + NB / 2 * PT_DESC_MAX, pmx.p + NB / 2 * PT_DESC_MAX);
    PT_LAUNCHED();
    std::vector<float> a(NB * PT_DESC_MAX), b(NB * PT_DESC_MAX);
    PT_CUDA(cudaMemcpyAsync(a.data(), pmn.p, sizeof(float) * a.size(), cudaMemcpyDeviceToHost, st));
    PT_CUDA(cudaMemcpyAsync(b.data(), pmx.p, sizeof(float) * b.size(), cudaMemcpyDeviceToHost, st));
    PT_CUDA(cudaStreamSynchronize(st));
    Quant qz;
    memset(&qz, 0, sizeof(qz));
    qz.nd = nd;
    qz.bits = std::min(10, 63 / nd);
    /* One scale for every dimension (that of the widest range): the curve then splits the
       dimensions in proportion to their spread, so a bucket's box is about as wide in every
       dimension in distance units, which is what the Euclidean lower bounds prune with.  (The
       search is exact whatever the order; only its pruning depends on the boxes.) */
    float rmax = 0.f;
    for (int d = 0; d < nd; d++) {
        float mn = a[d], mx = b[d];
        for (int i = 1; i < NB; i++) { mn = std::min(mn, a[i * PT_DESC_MAX + d]); mx = std::max(mx, b[i * PT_DESC_MAX + d]); }
        qz.mn[d] = mn;
        rmax = std::max(rmax, mx - mn);
    }
    for (int d = 0; d < nd; d++) qz.scale[d] = rmax > 0.f ? (float) ((1u << qz.bits) - 1) / rmax : 0.f;
    /* sort train points and queries along the curve */
    DevBuf<unsigned long long> codes(st), codes2(st);
    DevBuf<int> idx(st), perm(st), qorder(st);
    DevBuf<float> sp(st);
    PT_CUDA(codes.reserve(std::max(N, Q)));
    PT_CUDA(codes2.reserve(std::max(N, Q)));
    PT_CUDA(idx.reserve(std::max(N, Q)));
    PT_CUDA(perm.reserve(N));
    PT_CUDA(qorder.reserve(Q));
    const bool wide = K > 64;
    const int dp = wide ? nd : nd <= 6 ? 8 : 16;         /* floats per sorted point row */
    PT_CUDA(sp.reserve((size_t) N * dp));
    size_t tb = 0;
    PT_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, codes.p, codes2.p, idx.p, perm.p, std::max(N, Q), 0, 64, st));
    DevBuf<unsigned char> tmp(st);
    PT_CUDA(tmp.reserve(tb));
    k_curve<<<(N + 255) / 256, 256, 0, st>>>(qz, train, N, codes.p, idx.p);
    PT_LAUNCHED();
    PT_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, codes.p, codes2.p, idx.p, perm.p, N, 0, 64, st));
    pt_count_launches(4);
    k_curve<<<(Q + 255) / 256, 256, 0, st>>>(qz, qdesc, Q, codes.p, idx.p);
    PT_LAUNCHED();
    PT_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, codes.p, codes2.p, idx.p, qorder.p, Q, 0, 64, st));
    pt_count_launches(4);
    const int nbk = (N + BUCKET - 1) / BUCKET;
    dim3 grid((Q + NT - 1) / NT);
    if (wide) {
        if (K > PT_KNN_WIDE_MAX || (K & (K - 1))) return pt_fail(PT_UNSUPPORTED, "knn K=%d", K);
        k_reorder<<<(unsigned) (((long long) N * nd + 255) / 256), 256, 0, st>>>(train, N, nd, perm.p, sp.p);
        PT_LAUNCHED();
        /* bucket boxes and the binary tree above them */
        int L = 1;
        while (L < nbk) L <<= 1;
        DevBuf<float> lo(st), hi(st);
        PT_CUDA(lo.reserve((size_t) 2 * L * nd));
        PT_CUDA(hi.reserve((size_t) 2 * L * nd));
        k_leaf_box<<<(L + 255) / 256, 256, 0, st>>>(sp.p, N, nd, L, lo.p, hi.p);
        PT_LAUNCHED();
        for (int first = L / 2; first >= 1; first /= 2) {
            k_inner_box<<<(first + 255) / 256, 256, 0, st>>>(first, first, nd, lo.p, hi.p);
            PT_LAUNCHED();
        }
        DevBuf<float> wd(st);
        PT_CUDA(wd.reserve((size_t) Q * K));
        k_knn_wide<<<grid, NT, 0, st>>>(sp.p, perm.p, N, nd, L, lo.p, hi.p, qdesc, qorder.p, Q, K, wd.p, out);
        PT_LAUNCHED();
        PT_CUDA(cudaStreamSynchronize(st));
        return PT_OK;
    }
    k_reorder_pad<<<(unsigned) (((long long) N * dp + 255) / 256), 256, 0, st>>>(train, N, nd, dp, perm.p, sp.p);
    PT_LAUNCHED();
    /* boxes, level by level (rows padded to whole groups of 32) */
    KnnTree tr;
    size_t off[KNN_LEVELS + 1], total = 0;
    for (int l = 0, n = nbk; l <= KNN_LEVELS; l++, n = (n + 31) / 32) {
        tr.count[l] = n;
        tr.stride[l] = (n + 31) / 32 * 32;
        off[l] = total;
        total += (size_t) 2 * nd * tr.stride[l];
    }
    DevBuf<float> boxes(st), rows(st);
    PT_CUDA(boxes.reserve(total));
    PT_CUDA(rows.reserve((size_t) nbk * 2 * dp));
    tr.bucket = rows.p;
    for (int l = 0; l <= KNN_LEVELS; l++) tr.box[l] = boxes.p + off[l];
    k_bucket_box<<<(tr.stride[0] + 255) / 256, 256, 0, st>>>(sp.p, N, nd, dp, tr.count[0], tr.stride[0], boxes.p,
                                                         rows.p);
    PT_LAUNCHED();
    for (int l = 1; l <= KNN_LEVELS; l++) {
        k_group_box<<<(tr.stride[l] * 32 + 255) / 256, 256, 0, st>>>(tr.box[l - 1], nd, tr.stride[l - 1], tr.count[l],
                                                                      tr.stride[l], boxes.p + off[l]);
        PT_LAUNCHED();
    }
    /* Coordinates are scaled so that a squared distance of the whole range stays a finite half.
       Without a scale (0: ranges whose squares leave float's range) every pair is evaluated exactly. */
    const float reach = sqrtf(60000.f / nd);
    const float scale = rmax > 1e-10f && rmax < 1e30f ? reach / rmax : 0.f;
    const int nw = (Q + 31) / 32;
    DevBuf<int> worder(st);
    PT_CUDA(worder.reserve(nw));
    k_warp_spread<<<(Q + 255) / 256, 256, 0, st>>>(qdesc, qorder.p, Q, nd, codes.p, idx.p);
    PT_LAUNCHED();
    PT_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, codes.p, codes2.p, idx.p, worder.p, nw, 0, 32, st));
    pt_count_launches(4);
    const dim3 mgrid((Q + KNN_NT - 1) / KNN_NT);
#define PT_KNN_K(KK) case KK: \
        if (nd <= 6) k_knn_mma<KK, 1><<<mgrid, KNN_NT, 0, st>>>(sp.p, perm.p, N, nd, tr, scale, qdesc, qorder.p, worder.p, Q, out); \
        else if (nd <= 14) k_knn_mma<KK, 2><<<mgrid, KNN_NT, 0, st>>>(sp.p, perm.p, N, nd, tr, scale, qdesc, qorder.p, worder.p, Q, out); \
        else k_knn_mma<KK, 3><<<mgrid, KNN_NT, 0, st>>>(sp.p, perm.p, N, nd, tr, scale, qdesc, qorder.p, worder.p, Q, out); \
        break;
    switch (K) {
        PT_KNN_K(12) PT_KNN_K(16) PT_KNN_K(24) PT_KNN_K(32) PT_KNN_K(48) PT_KNN_K(64)
        default: return pt_fail(PT_UNSUPPORTED, "knn K=%d", K);
    }
#undef PT_KNN_K
    PT_LAUNCHED();
    PT_CUDA(cudaStreamSynchronize(st));
    return PT_OK;
}
