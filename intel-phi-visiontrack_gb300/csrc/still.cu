/* still.cu -- one camera's still picture on the GPU: the running mean of the frames each 16 x 8 cell has held still,
 * gated by the camera's own per-cell vectors from that mean to the newest frame.
 *
 * Reference: still_vectors, still_decide, still_update and still_finish (src/kern/still.c:116-251), run in that order
 * once a frame (src/kern/still.h:11; src/host/m3_ref.c:272-277), the vectors skipped on the first frame.
 *
 * A frame is two launches on one stream, no host round trip:
 *   vectors   lk.cu's per-cell kernel: LK from the mean to the frame at every cell's centre, one level, a 15 x 15
 *             patch, 6 iterations, forward-backward 0.25 px (still.c:14-19), the cell's mean |frame - mean|, counted in a
 *             histogram in 1/16 grey (the caller's own cells, and the first frame's, are counted by still_hist_kernel);
 *   decide    a CTA 8 x 4 cells: the noise median from the histogram, the limits (every CTA for itself), the evidence of
 *             its cells and the ring around them, the 3 x 3 vote, the counts, weights and states, the mean under its cells
 *             (still_decide, still_update: still.c:143-246), and its share of the drift statistics; the last CTA (an atomic
 *             ticket) finishes those and the state. FP64, a small fraction of F32's rate on GB300, is left to the cells that F32
 *             cannot decide and to that one thread.
 *
 * Exactness against the reference's long double:
 *   - the histogram, the median, the noise and its limit, the votes, the counts and the mean are exact;
 *   - the weight 1/n rounds to the same F32 through long double, double or an IEEE F32 division for every n up to
 *     65,535, so an F32 division gives it;
 *   - "a good vector longer than max(12 sigma, motion_px)" is decided exactly as the x87 does it: u^2 + v^2 is formed
 *     as an exact double-double, rounded to a 64-bit significand, and compared exactly with (12 sigma)^2;
 *   - the usual noise, a running mean over frames, is kept in FP64 (the reference: long double); it only enters the
 *     comparison of the median with three times itself;
 *   - the drift sums are exact fixed-point integers (units of 2^-60), divided and rounded to F32 once.
 * The last two agree with the reference's F32 results except where a value lies within 2^-53 of an F32 rounding
 * boundary. */
#include <math.h>
#include <stdint.h>

#include <new>

#include "vtg_ctx.h"
#include "vtg_internal.cuh"

#define STILL_MAX_SIDE 4096 /* up to 256 x 512 cells */
#define STILL_HIST VTG_STILL_BINS
#define STILL_TX 8 /* cells a CTA of the decision */
#define STILL_TY 4

/* The decision's state across frames, its newest statistics and the launches' hand-offs, in device memory. */
struct StillScal {
    double noise_usual;
    vtg_still_motion motion;
    unsigned ticket;   /* CTAs done in the decision; 0 between frames, like the sums below */
    int tracked, moving, good;
    unsigned long long counts;
    unsigned long long sums[3][3]; /* the drift sums' 42-bit pieces (StillFix) added up */
    int hist[STILL_HIST];
};

/* a double-double: hi + lo, |lo| at most half an ulp of hi */
struct DD {
    double hi, lo;
};

struct vtg_still {
    vtg_ctx *ctx;
    cudaStream_t stream;
    char *mem;
    size_t bytes;
    vtg_still_config c;
    int cols, rows, n, pitch;
    float *mean;
    vtg_cell *cells;
    unsigned *count;
    StillScal *scal;
    unsigned long long frames;
};

struct StillPrm {
    int cols, rows, n, avg;
    float motion_px, motion_grey;
    unsigned long long frames; /* before this one */
};

/* ---- double-double helpers: -fmad=false keeps every a * b + c here two roundings unless fma is written ---- */

__device__ __forceinline__ double two_sum_err(double a, double b, double s)
{
    const double bb = s - a;
    return (a - (s - bb)) + (b - bb);
}

__device__ __forceinline__ DD dd_add(DD a, DD b)
{
    const double s = a.hi + b.hi;
    const double e = two_sum_err(a.hi, b.hi, s) + (a.lo + b.lo);
    const double hi = s + e;
    return DD{hi, e - (hi - s)};
}

__device__ __forceinline__ DD dd_of(double a) { return DD{a, 0.0}; }

/* a / n, n > 0: a quotient and one correction term */
__device__ __forceinline__ DD dd_div(DD a, double n)
{
    const double q1 = a.hi / n;
    const double r = fma(-q1, n, a.hi) + a.lo;
    const double q2 = r / n;
    const double hi = q1 + q2;
    return DD{hi, q2 - (hi - q1)};
}

__device__ __forceinline__ DD dd_sqr(DD a)
{
    const double p = a.hi * a.hi;
    const double e = fma(a.hi, a.hi, -p) + 2.0 * a.hi * a.lo;
    const double hi = p + e;
    return DD{hi, e - (hi - p)};
}

__device__ __forceinline__ DD dd_neg(DD a) { return DD{-a.hi, -a.lo}; }

/* Whether a good vector moved (still.c:178-182): u^2 + v^2, rounded to a 64-bit significand as the x87 rounds the
 * long double sum, greater than need = max((12 sigma)^2, px^2), which is exact (56 bits at most). Both sides are
 * canonical double-doubles (head = the double nearest the sum), so they compare as (head, tail) pairs. */
__device__ __noinline__ bool still_longer_exact(float u, float v, float sigma, float px)
{
    const double a = (double)u * (double)u, b = (double)v * (double)v; /* exact: 48-bit products */
    double s = a + b, t = two_sum_err(a, b, s);
    if (t != 0.0) {
        int e;
        const double m = frexp(s, &e); /* s = m 2^e, m in [0.5, 1): a 64-bit significand's unit is 2^(e - 64) */
        int k = 64 - e;
        if (m == 0.5 && t < 0.0)
            k++; /* just below a power of two: the binade below, half the unit */
        const double t64 = ldexp(rint(ldexp(t, k)), -k);
        const double s2 = s + t64;
        t = two_sum_err(s, t64, s2);
        s = s2;
    }
    const double sg = (double)sigma * 12.0; /* VEC_OVER_SIGMA, still.c:21; exact */
    double np = sg * sg, ne = fma(sg, sg, -np);
    const double p2 = (double)px * (double)px;
    if (p2 > np || (p2 == np && ne < 0.0)) {
        np = p2;
        ne = 0.0;
    }
    return s > np || (s == np && t > ne);
}

/* The same, by F32 where the two sides differ by more than F32's rounding of them (a few parts in 2^24; no square under- or
 * overflows there). */
__device__ __forceinline__ bool still_longer(float u, float v, float sigma, float px)
{
    const float s = __fmaf_rn(u, u, v * v), sg = sigma * 12.0f, need = fmaxf(sg * sg, px * px);
    if (s > 1e-30f && s < 1e30f && need > 1e-30f && need < 1e30f) {
        if (s > need * 1.000002f)
            return true;
        if (s < need * 0.999998f)
            return false;
    }
    return still_longer_exact(u, v, sigma, px);
}

/* The drift sums (su += u, sv += v, suu += u^2 + v^2, still.c:206-211) exactly: each F32 u, and its square (exact
 * in 48 bits), as an integer in units of 2^-60. A good vector lies on its plane (|u| < 2^13), so a square needs at
 * most 87 bits and 131,072 cells' sums fit 128; bits below 2^-60 (|u| < 2^-37, a square below 2^-60) are dropped. */
__device__ __forceinline__ __int128 fix60(float f)
{
    const unsigned b = __float_as_uint(f);
    const int ex = (int)((b >> 23) & 0xffu);
    if (ex == 0)
        return 0; /* zero, or below 2^-126 */
    const unsigned long long m = (b & 0x7fffffu) | 0x800000u;
    const int sh = min(ex - 90, 80); /* u = m 2^(ex - 150), in units of 2^-60: m 2^(ex - 90) */
    const __int128 v = sh >= 0 ? (__int128)m << sh : (__int128)(sh > -64 ? m >> -sh : 0ull);
    return (b >> 31) ? -v : v;
}

__device__ __forceinline__ __int128 fix60_sq(float f)
{
    const unsigned b = __float_as_uint(f);
    const int ex = (int)((b >> 23) & 0xffu);
    if (ex == 0)
        return 0;
    const unsigned long long m = (b & 0x7fffffu) | 0x800000u, m2 = m * m; /* 48 bits */
    const int sh = min(2 * ex - 240, 72);                                 /* u^2 = m2 2^(2 ex - 300) */
    return sh >= 0 ? (__int128)m2 << sh : (__int128)(sh > -64 ? m2 >> -sh : 0ull);
}

__device__ __forceinline__ __int128 warp_sum_i128(__int128 v)
{
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        const unsigned long long lo = __shfl_xor_sync(VTG_FULL, (unsigned long long)v, d);
        const long long hi = __shfl_xor_sync(VTG_FULL, (long long)(v >> 64), d);
        v += ((__int128)hi << 64) | (__int128)lo;
    }
    return v;
}

/* v x 2^-60 as a double-double: three 42-bit pieces of |v|, each exact in a double */
__device__ DD dd_of_fix60(__int128 v)
{
    const bool neg = v < 0;
    const unsigned __int128 a = neg ? (unsigned __int128)(-v) : (unsigned __int128)v;
    const unsigned long long k = (1ull << 42) - 1ull;
    const double c0 = (double)(unsigned long long)(a & k), c1 = (double)(unsigned long long)((a >> 42) & k);
    const double c2 = (double)(unsigned long long)(a >> 84);
    DD r = dd_add(dd_add(dd_of(c2 * 0x1p24), dd_of(c1 * 0x1p-18)), dd_of(c0 * 0x1p-60));
    return neg ? dd_neg(r) : r;
}

/* A CTA's 128-bit sum into the frame's: its 42-bit pieces, the top one signed, each added up by a 64-bit atomic (at most
 * 131,072 cells' worth: 17 bits more). */
__device__ __forceinline__ void still_add(unsigned long long *to, __int128 v)
{
    const unsigned long long k = (1ull << 42) - 1ull;
    if (v) {
        atomicAdd(to + 0, (unsigned long long)v & k);
        atomicAdd(to + 1, (unsigned long long)(v >> 42) & k);
        atomicAdd(to + 2, (unsigned long long)(long long)(v >> 84));
    }
}
__device__ __forceinline__ __int128 still_sum(unsigned long long *from)
{
    const __int128 v = (__int128)__ldcg(from) + ((__int128)__ldcg(from + 1) << 42) + ((__int128)(long long)__ldcg(from + 2) << 84);
    from[0] = from[1] = from[2] = 0ull; /* ready for the next frame */
    return v;
}

/* The cells' differences counted, where lk_still_kernel did not. */
__global__ void __launch_bounds__(256) still_hist_kernel(int n, const vtg_cell *cells, int *hist)
{
    __shared__ int s_hist[STILL_HIST];
    const int i = (int)(blockIdx.x * 256 + threadIdx.x);
    s_hist[threadIdx.x] = 0;
    __syncthreads();
    if (i < n)
        atomicAdd(&s_hist[vtg_still_bin(cells[i].diff)], 1);
    __syncthreads();
    if (s_hist[threadIdx.x])
        atomicAdd(hist + threadIdx.x, s_hist[threadIdx.x]);
}

/* The decision and the mean (above). wide: the frame's rows may be read 16 bytes at a time. */
__global__ void __launch_bounds__(256) still_decide_kernel(StillPrm q, vtg_cell *cells, unsigned *__restrict__ count,
                                                           StillScal *sc, float *__restrict__ mean, int mpitch,
                                                           const float *__restrict__ cur, int cpitch, int w, int h, bool wide)
{
    __shared__ float s_limit, s_noise; /* exact: 16ths of grey, three times as many, or the caller's F32 */
    __shared__ int s_all;
    __shared__ unsigned char s_raw[STILL_TY + 2][STILL_TX + 2];
    __shared__ float s_w[STILL_TY][STILL_TX];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tiles_x = (q.cols + STILL_TX - 1) / STILL_TX;
    const int c0 = (int)(blockIdx.x % tiles_x) * STILL_TX, r0 = (int)(blockIdx.x / tiles_x) * STILL_TY;
    vtg_grid_dependency_wait();
    /* the frame's and the mean's pixels on their way while the decision is made: four rows of four a thread */
    const int x = c0 * 16 + 4 * lane;
    const bool quad = wide && x + 4 <= w;
    float4 fv[4], mv[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int y = r0 * 8 + 8 * k + warp;
        if (quad && y < h) {
            fv[k] = __ldg(reinterpret_cast<const float4 *>(cur + (size_t)y * cpitch + x));
            mv[k] = *reinterpret_cast<const float4 *>(mean + (size_t)y * mpitch + x);
        }
    }
    if (warp == 0) {
        /* med = the first bin whose running count reaches n / 2, at most 255 (the reference's walk) */
        const int half = q.n / 2;
        int c[8], sum = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            c[j] = __ldcg(&sc->hist[8 * lane + j]);
            sum += c[j];
        }
        int inc = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(VTG_FULL, inc, d);
            inc += lane >= d ? v : 0;
        }
        int run = inc - sum, first = STILL_HIST - 1;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            run += c[j];
            if (run >= half && 8 * lane + j < first)
                first = 8 * lane + j;
        }
        first = __reduce_min_sync(VTG_FULL, first);
        if (lane == 0) {
            const float noise = (float)first * 0.0625f, three = noise * 3.0f, grey = q.motion_grey; /* DIFF_OVER_NOISE */
            const double usual3 = sc->noise_usual * 3.0;
            s_noise = noise;
            s_limit = three > grey ? three : grey;
            s_all = q.frames >= 2 && noise > grey && (double)noise > usual3; /* above the larger of the two */
        }
    }
    __syncthreads();
    /* each cell's own evidence, the ring around the CTA's cells too (outside the grid: none): a good vector that moved, a lost
     * patch (LK_RESIDUAL), or a difference past the limit */
    if (tid < (STILL_TY + 2) * (STILL_TX + 2)) {
        const int a = tid / (STILL_TX + 2), b = tid - a * (STILL_TX + 2), r = r0 - 1 + a, c = c0 - 1 + b;
        bool e = false;
        if (r >= 0 && r < q.rows && c >= 0 && c < q.cols) {
            const vtg_cell *p = cells + r * q.cols + c;
            /* another CTA may store this cell's state now: its low byte stays */
            const unsigned lk = __ldcg(&p->state) & 0xffu;
            const bool moved = lk == 0 && still_longer(__ldcg(&p->u), __ldcg(&p->v), __ldcg(&p->sigma), q.motion_px);
            e = moved || (lk & 4u) != 0 || __ldcg(&p->diff) > s_limit;
        }
        s_raw[a][b] = (unsigned char)e;
    }
    __syncthreads();
    /* a cell moves when two cells of its 3 x 3 have evidence (EVIDENCE_MIN) or everything moved: its mean restarts;
     * otherwise its count grows to avg */
    int tracked = 0, moving = 0, good = 0, counts = 0, ci = 0;
    if (warp == 0) {
        const int a = lane / STILL_TX, b = lane % STILL_TX, r = r0 + a, c = c0 + b;
        if (r < q.rows && c < q.cols) {
            ci = r * q.cols + c;
            int votes = 0;
#pragma unroll
            for (int k = 0; k < 9; k++)
                votes += s_raw[a + k / 3][b + k % 3];
            const bool any = votes >= 2 || s_all, own = s_raw[a + 1][b + 1] != 0;
            const unsigned grown = count[ci] + 1u, n = any ? 1u : grown < (unsigned)q.avg ? grown : (unsigned)q.avg;
            count[ci] = n;
            s_w[a][b] = __fdiv_rn(1.0f, (float)n);
            const unsigned lk = __ldcg(&cells[ci].state) & 0xffu;
            cells[ci].state = lk | (own ? 0x100u : 0u) | (any ? 0x200u : 0u) | (n << 16);
            tracked = lk == 0;
            moving = any;
            counts = (int)n;
            good = lk == 0 && !any;
        }
    }
    __syncthreads();
    /* the mean: f where the weight is 1, else m + weight (f - m) as one fused multiply-add */
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int y = r0 * 8 + 8 * k + warp;
        if (y >= h || x >= w)
            continue;
        const float wt = s_w[k][lane >> 2];
        float *m = mean + (size_t)y * mpitch + x;
        auto mix = [&](float f, float o) { return wt == 1.0f ? f : __fmaf_rn(f - o, wt, o); };
        if (quad) {
            *reinterpret_cast<float4 *>(m) = make_float4(mix(fv[k].x, mv[k].x), mix(fv[k].y, mv[k].y), mix(fv[k].z, mv[k].z),
                                                         mix(fv[k].w, mv[k].w));
        } else {
            const float *f = cur + (size_t)y * cpitch + x;
            for (int e = 0; e < 4 && x + e < w; e++)
                m[e] = mix(__ldg(f + e), m[e]);
        }
    }
    if (warp != 0)
        return;
    /* the CTA's share of the statistics */
    {
        __int128 su = 0, sv = 0, suu = 0;
        if (good) {
            const float u = __ldcg(&cells[ci].u), v = __ldcg(&cells[ci].v);
            su = fix60(u);
            sv = fix60(v);
            suu = fix60_sq(u) + fix60_sq(v);
        }
        tracked = __reduce_add_sync(VTG_FULL, tracked);
        moving = __reduce_add_sync(VTG_FULL, moving);
        good = __reduce_add_sync(VTG_FULL, good);
        counts = __reduce_add_sync(VTG_FULL, counts); /* 32 x 65,535 at most */
        su = warp_sum_i128(su);
        sv = warp_sum_i128(sv);
        suu = warp_sum_i128(suu);
        if (lane < 3)
            still_add(sc->sums[lane], lane == 0 ? su : lane == 1 ? sv : suu);
        if (lane == 0) {
            atomicAdd(&sc->tracked, tracked);
            atomicAdd(&sc->moving, moving);
            atomicAdd(&sc->good, good);
            atomicAdd(&sc->counts, (unsigned long long)counts);
        }
    }
    /* the last CTA: the frame's statistics and state. A CTA takes its ticket when its share is added and it has read the
     * state that this changes. */
    unsigned last = 0u;
    __threadfence();
    __syncwarp();
    if (lane == 0)
        last = atomicAdd(&sc->ticket, 1u) == gridDim.x - 1;
    if (!__shfl_sync(VTG_FULL, last, 0))
        return;
    __threadfence();
#pragma unroll
    for (int j = 0; j < 8; j++)
        sc->hist[8 * lane + j] = 0; /* ready for the next frame, like the sums and the ticket */
    /* lane k: the k-th sum's mean over the good cells */
    const int all_good = __ldcg(&sc->good);
    const DD mine = all_good > 0 && lane < 3 ? dd_div(dd_of_fix60(still_sum(sc->sums[lane])), (double)all_good) : DD{0.0, 0.0};
    if (all_good <= 0 && lane < 3)
        still_sum(sc->sums[lane]);
    const DD mv2{__shfl_sync(VTG_FULL, mine.hi, 1), __shfl_sync(VTG_FULL, mine.lo, 1)};
    const DD muu{__shfl_sync(VTG_FULL, mine.hi, 2), __shfl_sync(VTG_FULL, mine.lo, 2)};
    if (lane != 0)
        return;
    vtg_still_motion &m = sc->motion;
    m.cols = (uint32_t)q.cols;
    m.rows = (uint32_t)q.rows;
    m.tracked = (uint32_t)__ldcg(&sc->tracked);
    m.moving = (uint32_t)__ldcg(&sc->moving);
    m.count_mean = (float)((double)__ldcg(&sc->counts) / (double)q.n);
    m.drift_u = m.drift_v = m.drift_rms = 0.0f;
    if (all_good > 0) {
        const DD var = dd_add(dd_add(muu, dd_neg(dd_sqr(mine))), dd_neg(dd_sqr(mv2)));
        m.drift_u = (float)(mine.hi + mine.lo);
        m.drift_v = (float)(mv2.hi + mv2.lo);
        const double vv = var.hi + var.lo;
        m.drift_rms = vv > 0.0 ? (float)sqrt(vv) : 0.0f;
    }
    m.diff_median = s_noise;
    m.diff_limit = s_limit;
    m.frames = q.frames + 1;
    const double nu = sc->noise_usual, noise = (double)s_noise;
    if (!s_all && q.frames >= 1)
        sc->noise_usual = q.frames == 1 ? noise : nu + (noise - nu) / 32.0; /* NOISE_FRAMES */
    sc->tracked = sc->moving = sc->good = 0;
    sc->counts = 0ull;
    sc->ticket = 0u;
}

/* ---- the C ABI ---- */

#define CU(call)                                                                                                       \
    do {                                                                                                               \
        const cudaError_t e_ = (call);                                                                                 \
        if (e_ != cudaSuccess) {                                                                                       \
            vtg_set_cuda_error(e_);                                                                                    \
            return VTG_ECUDA;                                                                                          \
        }                                                                                                              \
    } while (0)

static size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

struct StillLayout {
    size_t mean, cells, count, scal, bytes;
};

static bool still_cfg_ok(const vtg_still_config *c)
{
    return c && c->w >= 32 && c->h >= 32 && c->w <= STILL_MAX_SIDE && c->h <= STILL_MAX_SIDE && c->avg >= 1 &&
           c->avg <= 65535 && c->motion_px >= 0.0f && c->motion_grey >= 0.0f;
}

static StillLayout still_layout(const vtg_still_config *c)
{
    const int cols = (c->w + 15) / 16, rows = (c->h + 7) / 8, n = cols * rows;
    StillLayout L;
    size_t b = 0;
    L.mean = b;
    b += up256(sizeof(float) * (size_t)vtg_pitch(c->w) * (size_t)c->h);
    L.cells = b;
    b += up256(sizeof(vtg_cell) * (size_t)n);
    L.count = b;
    b += up256(sizeof(unsigned) * (size_t)n);
    L.scal = b;
    b += up256(sizeof(StillScal));
    L.bytes = b;
    return L;
}

extern "C" size_t vtg_still_bytes(const struct vtg_still_config *c)
{
    return still_cfg_ok(c) ? still_layout(c).bytes : 0;
}

extern "C" int vtg_still_create(vtg_ctx *ctx, const struct vtg_still_config *c, vtg_still **out)
{
    if (!ctx || !out || !still_cfg_ok(c))
        return VTG_EINVAL;
    *out = nullptr;
    const StillLayout L = still_layout(c);
    const int charged = vtg_ctx_charge(ctx, L.bytes);
    if (charged != VTG_OK)
        return charged;
    vtg_still *s = new (std::nothrow) vtg_still;
    if (!s) {
        vtg_ctx_release(ctx, L.bytes);
        return VTG_ENOMEM;
    }
    s->ctx = ctx;
    s->bytes = L.bytes;
    s->c = *c;
    s->cols = (c->w + 15) / 16;
    s->rows = (c->h + 7) / 8;
    s->n = s->cols * s->rows;
    s->pitch = vtg_pitch(c->w);
    s->frames = 0;
    cudaError_t e = cudaSetDevice(vtg_ctx_device(ctx));
    if (e == cudaSuccess)
        e = cudaMalloc(&s->mem, L.bytes);
    if (e != cudaSuccess) {
        vtg_set_cuda_error(e);
        vtg_ctx_release(ctx, L.bytes);
        delete s;
        return VTG_ENOMEM;
    }
    e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
    /* every field starts at zero, as still_create leaves them (still.c:82-87): the mean, the cells, the counts */
    if (e == cudaSuccess)
        e = cudaMemsetAsync(s->mem, 0, L.bytes, s->stream);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s->stream);
    if (e != cudaSuccess) {
        vtg_set_cuda_error(e);
        if (s->stream)
            cudaStreamDestroy(s->stream);
        cudaFree(s->mem);
        vtg_ctx_release(ctx, L.bytes);
        delete s;
        return VTG_ECUDA;
    }
    s->mean = (float *)(s->mem + L.mean);
    s->cells = (vtg_cell *)(s->mem + L.cells);
    s->count = (unsigned *)(s->mem + L.count);
    s->scal = (StillScal *)(s->mem + L.scal);
    vtg_ctx_track(ctx, s->stream, true);
    *out = s;
    return VTG_OK;
}

extern "C" void vtg_still_destroy(vtg_still *s)
{
    if (!s)
        return;
    cudaSetDevice(vtg_ctx_device(s->ctx));
    cudaStreamSynchronize(s->stream);
    vtg_ctx_track(s->ctx, s->stream, false);
    cudaStreamDestroy(s->stream);
    cudaFree(s->mem);
    vtg_ctx_release(s->ctx, s->bytes);
    delete s;
}

extern "C" void *vtg_still_stream(const vtg_still *s) { return s ? (void *)s->stream : nullptr; }

extern "C" int vtg_still_frame(vtg_still *s, const float *cur, int pitch, const struct vtg_cell *cells_in, int where,
                               void *stream)
{
    if (!s || !cur || pitch < s->c.w || (cells_in && where != VTG_HOST && where != VTG_DEVICE))
        return VTG_EINVAL;
    const cudaStream_t st = stream ? (cudaStream_t)stream : s->stream;
    CU(cudaSetDevice(vtg_ctx_device(s->ctx)));
    const int w = s->c.w, h = s->c.h;
    const bool vectors = !cells_in && s->frames > 0;
    if (cells_in)
        CU(cudaMemcpyAsync(s->cells, cells_in, sizeof(vtg_cell) * (size_t)s->n,
                           where == VTG_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, st));
    if (vectors) {
        /* still_vectors (still.c:116-141): the mean to the frame, one level; PATCH, LK_ITER, LK_EPS, LK_MIN_EIG,
         * LK_MAX_RESIDUAL, FB_MAX (still.c:14-19) */
        LkPrm p;
        p.W = 15;
        p.H = 15;
        p.max_iter = 6;
        p.eps2 = 0.01f * 0.01f;
        p.min_eig = 0.1f;
        p.max_residual = 16.0f;
        p.fb_max2 = 0.25f * 0.25f;
        p.area = 225.0f;
        p.pitch = 0;
        CellGrid g;
        g.cell_w = 16;
        g.cell_h = 8;
        g.cols = s->cols;
        g.rows = s->rows;
        g.n = s->n;
        CU(vtg_launch_still_cells(DevLevel{s->mean, w, h, s->pitch}, DevLevel{cur, w, h, pitch}, p, g, s->cells, s->scal->hist, st));
    } else {
        still_hist_kernel<<<(s->n + 255) / 256, 256, 0, st>>>(s->n, s->cells, s->scal->hist);
        CU(cudaGetLastError());
    }
    StillPrm q;
    q.cols = s->cols;
    q.rows = s->rows;
    q.n = s->n;
    q.avg = s->c.avg;
    q.motion_px = s->c.motion_px;
    q.motion_grey = s->c.motion_grey;
    q.frames = s->frames;
    const bool wide = (((uintptr_t)cur | (sizeof(float) * (uintptr_t)pitch)) & 15) == 0;
    const int tiles = ((s->cols + STILL_TX - 1) / STILL_TX) * ((s->rows + STILL_TY - 1) / STILL_TY);
    CU(vtg_launch_k(still_decide_kernel, dim3(tiles), dim3(256), 0, st, true, q, s->cells, s->count, s->scal, s->mean, s->pitch, cur,
                    pitch, w, h, wide));
    CU(cudaGetLastError());
    s->frames++; /* still_finish (still.c:248-251) */
    return VTG_OK;
}

extern "C" int vtg_still_read(vtg_still *s, struct vtg_cell *cells, struct vtg_still_motion *motion, float *mean,
                              int mean_pitch, int where, void *stream)
{
    if (!s || (where != VTG_HOST && where != VTG_DEVICE) || (mean && mean_pitch < s->c.w))
        return VTG_EINVAL;
    const cudaStream_t st = stream ? (cudaStream_t)stream : s->stream;
    const cudaMemcpyKind k = where == VTG_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
    CU(cudaSetDevice(vtg_ctx_device(s->ctx)));
    if (cells)
        CU(cudaMemcpyAsync(cells, s->cells, sizeof(vtg_cell) * (size_t)s->n, k, st));
    if (motion)
        CU(cudaMemcpyAsync(motion, &s->scal->motion, sizeof(vtg_still_motion), k, st));
    if (mean)
        CU(cudaMemcpy2DAsync(mean, sizeof(float) * (size_t)mean_pitch, s->mean, sizeof(float) * (size_t)s->pitch,
                             sizeof(float) * (size_t)s->c.w, (size_t)s->c.h, k, st));
    if (where == VTG_HOST)
        CU(cudaStreamSynchronize(st));
    return VTG_OK;
}

extern "C" int vtg_still_mean(const vtg_still *s, const float **plane, int *pitch)
{
    if (!s || !plane || !pitch)
        return VTG_EINVAL;
    *plane = s->mean;
    *pitch = s->pitch;
    return VTG_OK;
}
