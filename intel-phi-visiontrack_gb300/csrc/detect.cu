/* detect.cu -- corners inside a rectangle of a Q6 plane: the Harris response over Sobel gradients on a 5 x 5 box of
 * the structure tensor, each 16 x 16 cell's strongest response, and the selection of the strongest corners at a
 * spacing.
 *
 * Reference: detect_begin, detect_tensor, detect_response, detect_cells and detect_finish (src/kern/detect.h:21-37,
 * src/kern/detect.c:28-258), run in that order by the tracker's seed_at (src/kern/track.c:988-992).
 *
 * The response is the reference's bit for bit: every step is an IEEE F32 operation in the reference's order (the
 * Sobel sums of whole numbers, a fused multiply-add, the 1/512 scale, three rounded products, the five rows added top
 * to bottom, the box as (v + (v_-1 + v_+1)) + (v_-2 + v_+2) with the columns outside the region's 16-column groups
 * reading 0, and det - 0.04 trace^2 as two fused multiply-subtracts). No sqrt or division, so no arithmetic differs.
 *
 * Pipeline, one stream, no host round trip, four launches, each after the first a programmatic dependent:
 *   det_response  a CTA a tile of 16 rows x 64 columns: the plane tile, the tensor, the row sums and the box in
 *                 shared memory; the response out, the four cells' strongest (floored at 0)
 *   det_count     the best cell; a CTA a row, a warp an eighth of it: the local maxima above max(quality x the strongest of their 3 x 3
 *                 cells, 2500), counted
 *   det_collect   a CTA a row: its first place in scan order from the rows' counts (tall regions: det_scan, a launch of
 *                 its own), then the candidates in scan order, the first 8,192 kept (DETECT_MAX_CANDIDATES), each
 *                 scored v / local + 0.001 v / best in FP64 and rounded to F32 (the reference's long double rounds to
 *                 the same F32 but where the sum lies within 2^-53 of a rounding boundary)
 *   det_select    one CTA: the greedy spacing over the candidates by (score descending, scan order), in blocks of the best
 *                 up to 256 left: a block's members by a histogram of their keys, its order by counting the lesser keys, its
 *                 conflicts as bit masks, settled 32 at a time by one warp with the in-order result, until max corners are
 *                 taken. The corners taken sit in a grid of linked lists (cells at least the spacing wide), so a candidate
 *                 looks at 3 x 3 grid cells only.
 * The threshold needs no long double: local x quality is an exact product of two F32s, so its F32 rounding is the
 * reference's (float)(rel) and max(fl(rel), 2500) equals its (float)(rel > 2500 ? rel : 2500). */
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <new>

#include "vtg_ctx.h"
#include "vtg_internal.cuh"

#define DET_MAX_CAND 8192   /* DETECT_MAX_CANDIDATES, src/kern/detect.h:12 */
#define DET_TX 64           /* a response tile: four cells wide ... */
#define DET_TY 16           /* ... and one cell row high */
#define DET_SELECT_THREADS 1024
#define DET_SEGS 8          /* a row's candidate columns in this many segments, a warp each */
#define DET_GRID_MAX 16384  /* the taken corners' grid: at most this many cells */
#define DET_BLOCK 256       /* candidates a block of the selection, at most */
#define DET_BINS 2048       /* of its histogram: two a thread */
#define DET_SCAN_ROWS 2048  /* regions of more rows scan the rows' counts in a launch of their own */
static_assert(DET_BINS == 2 * DET_SELECT_THREADS, "two bins a thread");

struct DetGeo {
    int x0, y0, x1, y1, ax, cols, rows, nv, cell_rows;
};

struct DetPrm {
    const float *p; /* the plane, w x h, rows pitch floats apart */
    int w, h, pitch;
    DetGeo g;
    float quality;
    int need; /* ceil(min_dist^2): the spacing test on whole-pixel places */
    int max;
    int gs, gw, gh; /* the grid of corners taken: cells gs pixels square (gs^2 >= need), gw x gh of them */
};

struct vtg_detector {
    vtg_ctx *ctx;
    cudaStream_t stream;
    char *mem;
    size_t bytes;
    int max_w, max_h, max_cols, max_cells;
    float *resp, *cell, *best;
    int *rowcount, *rowbase, *ncand; /* counts a segment; counts a row, or (tall regions) first places a segment */
    unsigned *keys;
    int2 *cxy;
    struct Host {
        int count;
        float xs[512], ys[512];
    } *host, *host_dev; /* pinned host memory that det_select writes: a host caller's corners need no copy */
};

/* ---- the response and the cells ---- */

__global__ void __launch_bounds__(256) det_response(DetPrm q, float *__restrict__ resp, float *__restrict__ cell,
                                                    float *__restrict__ best)
{
    __shared__ float s_p[DET_TY + 6][DET_TX + 6];   /* image rows y0 - 3 + r0 + i, columns ax + c0 - 3 + j */
    __shared__ float s_t[3][DET_TY + 4][DET_TX + 4]; /* tensor rows r0 + i, region columns c0 - 2 + j */
    __shared__ float s_v[3][DET_TY][DET_TX + 4];     /* the five-row sums */
    __shared__ float s_m[8][4];                      /* each warp's strongest in the tile's four cells */
    const DetGeo &g = q.g;
    const int tid = threadIdx.x;
    const int r0 = blockIdx.y * DET_TY, c0 = blockIdx.x * DET_TX;
    vtg_grid_launch_dependents();
    if (tid == 0 && blockIdx.x == 0 && blockIdx.y == 0)
        *best = 0.0f; /* det_count's maximum starts here */
    /* a whole number of cell rows leaves one more, empty, at the region's foot */
    if (g.rows % DET_TY == 0 && blockIdx.y == gridDim.y - 1 && tid < 4 && 4 * (int)blockIdx.x + tid < g.nv)
        cell[gridDim.y * g.nv + 4 * blockIdx.x + tid] = 0.0f;
    for (int i = tid; i < (DET_TY + 6) * (DET_TX + 6); i += blockDim.x) {
        const int a = i / (DET_TX + 6), b = i - a * (DET_TX + 6);
        const int y = min(max(g.y0 - 3 + r0 + a, 0), q.h - 1), x = min(max(g.ax + c0 - 3 + b, 0), q.w - 1);
        s_p[a][b] = __ldg(q.p + (size_t)y * q.pitch + x);
    }
    __syncthreads();
    /* the tensor at region row r0 + a (image row y0 - 2 + r0 + a: staged row a + 1) and region column c0 - 2 + b
     * (staged column b + 1); 0 outside the region's columns, as the box's zero vectors read */
    for (int i = tid; i < (DET_TY + 4) * (DET_TX + 4); i += blockDim.x) {
        const int a = i / (DET_TX + 4), b = i - a * (DET_TX + 4);
        const int c = c0 - 2 + b;
        float xx = 0.0f, xy = 0.0f, yy = 0.0f;
        if (c >= 0 && c < g.cols) {
            const float *U = &s_p[a][b], *M = &s_p[a + 1][b], *D = &s_p[a + 2][b];
            const float dxu = U[2] - U[0], dxm = M[2] - M[0], dxd = D[2] - D[0];
            const float gx = __fmaf_rn(dxm, 2.0f, dxu + dxd) * (1.0f / 512.0f);
            const float dyl = D[0] - U[0], dyc = D[1] - U[1], dyr = D[2] - U[2];
            const float gy = __fmaf_rn(dyc, 2.0f, dyl + dyr) * (1.0f / 512.0f);
            xx = gx * gx;
            xy = gx * gy;
            yy = gy * gy;
        }
        s_t[0][a][b] = xx;
        s_t[1][a][b] = xy;
        s_t[2][a][b] = yy;
    }
    __syncthreads();
    for (int i = tid; i < 3 * DET_TY * (DET_TX + 4); i += blockDim.x) {
        const int t = i / (DET_TY * (DET_TX + 4)), rem = i - t * DET_TY * (DET_TX + 4);
        const int a = rem / (DET_TX + 4), b = rem - a * (DET_TX + 4);
        s_v[t][a][b] = (((s_t[t][a][b] + s_t[t][a + 1][b]) + s_t[t][a + 2][b]) + s_t[t][a + 3][b]) + s_t[t][a + 4][b];
    }
    __syncthreads();
    /* four outputs a thread: row a = tid / 16, columns j .. j + 3, all in cell j / 16 */
    const int a = tid >> 4, j = 4 * (tid & 15);
    const int r = r0 + a;
    float m = 0.0f;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const int b = j + e + 2; /* s_v column of region column c0 + j + e */
        const float *A = &s_v[0][a][b], *B = &s_v[1][a][b], *C = &s_v[2][a][b];
        const float va = (A[0] + (A[-1] + A[1])) + (A[-2] + A[2]);
        const float vb = (B[0] + (B[-1] + B[1])) + (B[-2] + B[2]);
        const float vc = (C[0] + (C[-1] + C[1])) + (C[-2] + C[2]);
        const float tr = va + vc;
        const float v = __fmaf_rn(-0.04f, tr * tr, __fmaf_rn(-vb, vb, va * vc));
        const int c = c0 + j + e;
        if (r < g.rows && c < g.cols) {
            resp[(size_t)r * g.cols + c] = v;
            m = fmaxf(m, v);
        }
    }
    /* the lanes of a cell: 4 a half-warp row, the two rows of the warp */
    m = fmaxf(m, __shfl_xor_sync(VTG_FULL, m, 1));
    m = fmaxf(m, __shfl_xor_sync(VTG_FULL, m, 2));
    m = fmaxf(m, __shfl_xor_sync(VTG_FULL, m, 16));
    const int lane = tid & 31, warp = tid >> 5;
    if (lane < 16 && (lane & 3) == 0)
        s_m[warp][lane >> 2] = m;
    __syncthreads();
    if (tid < 4) {
        float c = 0.0f;
        for (int w = 0; w < 8; w++)
            c = fmaxf(c, s_m[w][tid]);
        const int k = 4 * blockIdx.x + tid;
        if (k < g.nv)
            cell[blockIdx.y * g.nv + k] = c;
    }
}

/* ---- the selection ---- */

/* The strongest response of the 3 x 3 cells around region row r, column c (detect_finish's neighbourhood). */
__device__ __forceinline__ float det_near(const DetGeo &g, const float *cell, int r, int c)
{
    const int cr = r >> 4, k = c >> 4;
    float m = 0.0f;
#pragma unroll
    for (int a = -1; a <= 1; a++)
#pragma unroll
        for (int b = -1; b <= 1; b++)
            if (cr + a >= 0 && cr + a < g.cell_rows && k + b >= 0 && k + b < g.nv)
                m = fmaxf(m, __ldca(cell + (cr + a) * g.nv + k + b));
    return m;
}

/* A corner candidate: inside the rectangle's lanes, above its threshold (at least 2500: tried first), and no smaller than
 * any of its 8 neighbours (those past the region's columns read 0). near: its neighbourhood's strongest, when it is one. */
__device__ __forceinline__ bool det_candidate(const DetPrm &q, const float *resp, const float *cell, int r, int c, float &near)
{
    const DetGeo &g = q.g;
    const float *me = resp + (size_t)r * g.cols + c;
    const float v = __ldca(me);
    if (!(2500.0f < v))
        return false;
    const float *up = me - g.cols, *dn = me + g.cols;
    const bool lo = c > 0, hi = c + 1 < g.cols;
    const float n[8] = {lo ? __ldca(up - 1) : 0.0f, __ldca(up), hi ? __ldca(up + 1) : 0.0f, lo ? __ldca(me - 1) : 0.0f,
                        hi ? __ldca(me + 1) : 0.0f, lo ? __ldca(dn - 1) : 0.0f, __ldca(dn), hi ? __ldca(dn + 1) : 0.0f};
    bool top = true;
#pragma unroll
    for (int k = 0; k < 8; k++)
        top = top && n[k] <= v;
    if (!top)
        return false;
    near = det_near(g, cell, r, c);
    return fmaxf(near * q.quality, 2500.0f) < v;
}

__device__ __forceinline__ void det_lanes(const DetGeo &g, int &lo, int &hi)
{
    lo = g.x0 - g.ax > 1 ? g.x0 - g.ax : 1;
    hi = g.x1 - g.ax < g.cols - 1 ? g.x1 - g.ax : g.cols - 1;
}

/* Segment s of a row's candidate columns [lo, hi): [a, b), consecutive segments in column order. */
__device__ __forceinline__ void det_segment(const DetGeo &g, int s, int &a, int &b)
{
    int lo, hi;
    det_lanes(g, lo, hi);
    const int len = hi > lo ? hi - lo : 0, per = (len + DET_SEGS - 1) / DET_SEGS;
    a = lo + s * per;
    b = min(a + per, lo + len);
}

/* A CTA a row; rowtotal (regions up to DET_SCAN_ROWS) gets the row's count, rowcount its segments'. The first row of each cell
 * row finds its best cell too: an integer atomicMax on the F32 bits orders them as the floats, all being >= 0. */
__global__ void __launch_bounds__(32 * DET_SEGS) det_count(DetPrm q, const float *resp, const float *cell, float *best,
                                                        int *rowcount, int *rowtotal)
{
    __shared__ int s_n[DET_SEGS];
    const int r = blockIdx.x, sg = threadIdx.x >> 5, lane = threadIdx.x & 31;
    vtg_grid_launch_dependents();
    vtg_grid_dependency_wait();
    if (r % 16 == 0 && sg == 0) {
        unsigned m = 0u;
        for (int k = lane; k < q.g.nv; k += 32)
            m = max(m, __float_as_uint(__ldca(cell + (r >> 4) * q.g.nv + k)));
        m = __reduce_max_sync(VTG_FULL, m);
        if (lane == 0 && m > 0u)
            atomicMax(reinterpret_cast<int *>(best), (int)m);
    }
    int cnt = 0;
    if (r >= 1 && r < q.g.rows - 1) {
        int a, b;
        float near;
        det_segment(q.g, sg, a, b);
        for (int c0 = a; c0 < b; c0 += 32) {
            const int c = c0 + lane;
            cnt += __popc(__ballot_sync(VTG_FULL, c < b && det_candidate(q, resp, cell, r, c, near)));
        }
    }
    if (lane == 0)
        rowcount[r * DET_SEGS + sg] = s_n[sg] = cnt;
    if (!rowtotal)
        return;
    __syncthreads();
    if (threadIdx.x == 0) {
        int n = 0;
        for (int k = 0; k < DET_SEGS; k++)
            n += s_n[k];
        rowtotal[r] = n;
    }
}

/* Tall regions: each segment's first place in scan order (an exclusive scan), and the candidates kept: at most 8,192. */
__global__ void __launch_bounds__(1024) det_scan(int rows, const int *rowcount, int *__restrict__ rowbase,
                                                 int *__restrict__ ncand)
{
    __shared__ int s[1024];
    const int tid = threadIdx.x, per = (rows + 1023) / 1024, a = tid * per, b = min(a + per, rows);
    vtg_grid_launch_dependents();
    vtg_grid_dependency_wait();
    int sum = 0;
    for (int r = a; r < b; r++)
        sum += __ldca(rowcount + r);
    s[tid] = sum;
    __syncthreads();
    for (int d = 1; d < 1024; d <<= 1) {
        const int v = tid >= d ? s[tid - d] : 0;
        __syncthreads();
        s[tid] += v;
        __syncthreads();
    }
    int run = s[tid] - sum;
    for (int r = a; r < b; r++) {
        rowbase[r] = run;
        run += __ldca(rowcount + r);
    }
    if (tid == 1023)
        *ncand = min(s[1023], DET_MAX_CAND);
}

/* v / local + 0.001 v / best in FP64, rounded to F32. GB300's FP64 rate is a small fraction of its F32 rate (8,192 scores
 * bound the kernel by it: 22 us over a 1080p frame), so the sum is formed in pairs of F32s first (each quotient and its
 * remainder's, 0.001 as two F32s: within 2^-44), which decides the rounding unless it lies within 2^-40 of halfway between two
 * F32s; only then, or where a value is out of the pairs' range, are the FP64 divisions made. */
__device__ __forceinline__ float det_score(float v, float local, float best)
{
    const float rl = __frcp_rn(local), rb = __frcp_rn(best);
    const float q = v * rl, q1 = __fmaf_rn(-q, local, v) * rl;
    const float C0 = 0.001f, C1 = (float)(0.001 - (double)0.001f);
    const float p = C0 * v, p1 = __fmaf_rn(C0, v, -p) + C1 * v;
    const float t = p * rb, t1 = (__fmaf_rn(-t, best, p) + p1) * rb;
    /* q + t (q is the larger: local <= best), then everything below it */
    const float s = q + t, e = (t - (s - q)) + (q1 + t1);
    const float hi = s + e, lo = e - (hi - s);
    /* how far hi + lo is from halfway to hi's neighbour on lo's side */
    const float step = fabsf(__int_as_float(__float_as_int(hi) + (lo < 0.0f ? -1 : 1)) - hi);
    if (v < 1e30f && best < 1e30f && fabsf(fabsf(lo) - 0.5f * step) > 1e-12f * hi)
        return hi;
    const double x = (double)v;
    return (float)(x / (double)local + 0.001 * x / (double)best);
}

/* A CTA a row: the candidates of its segments from their first places on. scanned: rowbase holds the segments' places
 * (det_scan); otherwise it holds the rows' counts, and the row's place is the sum of those before it (a regular load a
 * thread for every 256 rows; at 2,048 rows this costs less than the launch it saves), the last row's CTA then knowing the
 * number kept. */
__global__ void __launch_bounds__(32 * DET_SEGS) det_collect(DetPrm q, const float *resp, const float *cell, const float *best,
                                                          const int *rowcount, const int *rowbase, bool scanned,
                                                          unsigned *__restrict__ keys, int2 *__restrict__ cxy,
                                                          int *__restrict__ ncand)
{
    __shared__ int s_n[DET_SEGS];
    const int r = blockIdx.x, sg = threadIdx.x >> 5, lane = threadIdx.x & 31;
    vtg_grid_launch_dependents();
    vtg_grid_dependency_wait();
    int pos;
    if (scanned) {
        pos = __ldca(rowbase + r * DET_SEGS + sg);
    } else {
        int sum = 0;
        for (int k = threadIdx.x; k < r; k += 32 * DET_SEGS)
            sum += __ldca(rowbase + k);
        sum = __reduce_add_sync(VTG_FULL, sum);
        if (lane == 0)
            s_n[sg] = sum;
        __syncthreads();
        pos = 0;
#pragma unroll
        for (int k = 0; k < DET_SEGS; k++)
            pos += s_n[k];
        if (r == q.g.rows - 1 && threadIdx.x == 0)
            *ncand = min(pos + __ldca(rowbase + r), DET_MAX_CAND);
#pragma unroll
        for (int k = 0; k < DET_SEGS; k++)
            pos += k < sg ? __ldca(rowcount + r * DET_SEGS + k) : 0;
    }
    if (r < 1 || r >= q.g.rows - 1 || pos >= DET_MAX_CAND)
        return;
    const float bst = __ldca(best);
    int a, b;
    det_segment(q.g, sg, a, b);
    for (int c0 = a; c0 < b && pos < DET_MAX_CAND; c0 += 32) {
        const int c = c0 + lane;
        float near = 0.0f;
        const bool f = c < b && det_candidate(q, resp, cell, r, c, near);
        const unsigned m = __ballot_sync(VTG_FULL, f);
        const int p = pos + __popc(m & ((1u << lane) - 1u));
        if (f && p < DET_MAX_CAND) {
            const float score = det_score(__ldca(resp + (size_t)r * q.g.cols + c), near, bst);
            keys[p] = ~__float_as_uint(score); /* ascending: the best first; the place is the index */
            cxy[p] = make_int2(q.g.ax + c, q.g.y0 + r);
        }
        pos += __popc(m);
    }
}

/* Whether the corner at (x, y) keeps the spacing from every corner in the grid: the 3 x 3 grid cells around its own
 * (a cell's side is at least the spacing, so no corner farther out can be too close). The whole warp asks together, a lane
 * without a corner with far = false, and steps through the lists by votes, so that no lane can leave a list on its own. With
 * nested loops left by a return, compiled into det_select, a lane was measured to come back after the warp's next ballots and
 * barriers: det_select then counted a block twice and wrote past its arrays. */
__device__ __forceinline__ bool det_far(const DetPrm &q, const int *s_head, const int *s_next, const int *s_tx,
                                        const int *s_ty, int x, int y, bool far)
{
    const int gx = (x - q.g.ax) / q.gs, gy = (y - q.g.y0) / q.gs;
    int h[9];
#pragma unroll
    for (int j = 0; j < 9; j++) {
        const int a = gx + j % 3 - 1, b = gy + j / 3 - 1;
        h[j] = far && a >= 0 && a < q.gw && b >= 0 && b < q.gh ? s_head[b * q.gw + a] : -1;
    }
#pragma unroll
    for (int j = 0; j < 9; j++) {
        int t = far ? h[j] : -1;
        while (__any_sync(VTG_FULL, t >= 0)) {
            if (t >= 0) {
                const int dx = s_tx[t] - x, dy = s_ty[t] - y;
                far = dx * dx + dy * dy >= q.need;
                t = far ? s_next[t] : -1;
            }
            __syncwarp();
        }
    }
    return far;
}

struct DetSelectSmem {
    int head[DET_GRID_MAX]; /* the taken corners' grid: the newest of each cell */
    int tx[512], ty[512], next[512];
    int hist[DET_BINS];
    unsigned long long list[DET_SELECT_THREADS]; /* a block's members: key << 13 | place in scan order */
    unsigned long long order[DET_SELECT_THREADS];
    int2 xy[DET_BLOCK]; /* those of them that keep the spacing from every corner taken before it, in order */
    unsigned mask[DET_BLOCK / 32][DET_BLOCK]; /* [k][i]: which of candidates 32 k .. 32 k + 31 before i are too close to i */
    unsigned got[DET_BLOCK / 32];
    int wsum[32], cut, below, upto;
    unsigned lo, hi;
};

/* The greedy spacing. The reference sorts the candidates by (score descending, scan order) and takes each that keeps the
 * spacing from every corner taken; the result of walking them in blocks, in that order, is the same. A key is ~score bits << 13
 * | place in scan order: 45 bits, all different. Eight keys a thread stay in registers. A block is the keys below a limit,
 * found by a histogram over the range of those left (2,048 bins; a range whose first bin holds more than a block is zoomed
 * into, which ends as keys differ), so nothing is ordered that the walk never reaches; the histogram's prefix sums also place
 * the members, a bin's few among themselves by counting. Whatever of it is too close to a corner
 * taken before it is out at once, a thread a member; up to 256 may be left (a block with more is tried again with fewer
 * members; the share left sets the next block's size). Those are settled by conflict masks, 32 candidates at a time by one warp:
 * a candidate is taken once no earlier one in conflict with it is taken or open, out once
 * one is taken. 128 corners of a 384 x 307 box (2,673 candidates): 16 us, where four radix passes over the candidates and
 * blocks settled in passes took 32. Latency of one SM's barriers and shared memory bounds it. */
__global__ void __launch_bounds__(DET_SELECT_THREADS, 1) det_select(DetPrm q, const int *ncand, const float *best, const unsigned *keys,
                                                                 const int2 *cxy, float *__restrict__ xs,
                                                                 float *__restrict__ ys, int *__restrict__ count)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    DetSelectSmem &S = *reinterpret_cast<DetSelectSmem *>(s_raw);
    constexpr int KEYS = DET_MAX_CAND / DET_SELECT_THREADS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < q.gw * q.gh; i += DET_SELECT_THREADS)
        S.head[i] = -1;
    if (tid == 0) {
        S.lo = ~0u;
        S.hi = 0u;
    }
    vtg_grid_dependency_wait();
    const int n = __ldca(best) > 0.0f ? __ldca(ncand) : 0;
    unsigned key[KEYS], lo = ~0u, hi = 0u;
#pragma unroll
    for (int k = 0; k < KEYS; k++) {
        const int i = tid + k * DET_SELECT_THREADS;
        key[k] = i < n ? __ldca(keys + i) : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KEYS; k++)
        if (tid + k * DET_SELECT_THREADS < n) {
            lo = min(lo, key[k]);
            hi = max(hi, key[k]);
        }
    lo = __reduce_min_sync(VTG_FULL, lo);
    hi = __reduce_max_sync(VTG_FULL, hi);
    if (lane == 0) {
        atomicMin(&S.lo, lo);
        atomicMax(&S.hi, hi);
    }
    __syncthreads();
    auto whole = [&](int k) { return ((unsigned long long)key[k] << 13) | (unsigned)(tid + k * DET_SELECT_THREADS); };
    /* keys below `from` are done with; the last one */
    unsigned long long from = (unsigned long long)S.lo << 13;
    const unsigned long long last = ((unsigned long long)S.hi << 13) | 8191ull;
    int taken = 0, left = n;
    int size = min(DET_BLOCK, max(64, 2 * q.max)); /* members of the next block: the greedy rarely looks further */
    while (left > 0 && taken < q.max) {
        const int cap = size <= DET_BLOCK ? DET_BLOCK : DET_SELECT_THREADS, want = min(left, size);
        unsigned long long a = from, b = last, limit;
        int shift, members;
        for (;;) {
            shift = max(0, 64 - __clzll((long long)(b - a)) - 11);
            S.hist[2 * tid] = 0;
            S.hist[2 * tid + 1] = 0;
            __syncthreads();
#pragma unroll
            for (int k = 0; k < KEYS; k++)
                if (tid + k * DET_SELECT_THREADS < n && whole(k) >= a && whole(k) <= b)
                    atomicAdd(&S.hist[(int)((whole(k) - a) >> shift)], 1);
            __syncthreads();
            const int h0 = S.hist[2 * tid], h1 = S.hist[2 * tid + 1];
            int inc = h0 + h1;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int v = __shfl_up_sync(VTG_FULL, inc, d);
                inc += lane >= d ? v : 0;
            }
            if (lane == 31)
                S.wsum[warp] = inc;
            __syncthreads();
            const int w = S.wsum[lane];
            const int base = __reduce_add_sync(VTG_FULL, lane < warp ? w : 0);
            const int e1 = base + inc, e0 = e1 - h1, s0 = e0 - h0; /* up to and with the thread's bins; before them */
            /* the bin where the count reaches what is wanted: one thread has it (the range holds as many) */
            if (s0 < want && want <= e1) {
                const bool first = want <= e0;
                S.cut = 2 * tid + (first ? 0 : 1);
                S.below = first ? s0 : e0;
                S.upto = first ? e0 : e1;
            }
            __syncthreads();
            const int cut = S.cut, below = S.below, upto = S.upto;
            S.hist[2 * tid] = s0; /* where each bin's members go */
            S.hist[2 * tid + 1] = e0;
            __syncthreads();
            if (upto <= cap) {
                limit = a + ((unsigned long long)(cut + 1) << shift);
                members = upto;
                break;
            }
            if (below > 0) {
                limit = a + ((unsigned long long)cut << shift);
                members = below;
                break;
            }
            b = a + ((unsigned long long)(cut + 1) << shift) - 1ull;
            a += (unsigned long long)cut << shift;
        }
        /* the members (none lies before a) by their bins, then in order: bin k's end where the next one's began */
#pragma unroll
        for (int k = 0; k < KEYS; k++)
            if (tid + k * DET_SELECT_THREADS < n && whole(k) >= a && whole(k) < limit)
                S.list[atomicAdd(&S.hist[(int)((whole(k) - a) >> shift)], 1)] = whole(k);
        __syncthreads();
        if (tid < members) {
            const unsigned long long k = S.list[tid];
            const int bin = (int)((k - a) >> shift), end = S.hist[bin];
            int at = bin ? S.hist[bin - 1] : 0;
            for (int j = at, e = end; j < e; j++)
                at += S.list[j] < k;
            S.order[at] = k;
        }
        __syncthreads();
        /* of them, those clear of every corner taken */
        int2 me = make_int2(0, 0);
        if (tid < members)
            me = __ldca(cxy + (int)(S.order[tid] & 8191ull));
        const bool clear = det_far(q, S.head, S.next, S.tx, S.ty, me.x, me.y, tid < members);
        const unsigned bal = __ballot_sync(VTG_FULL, clear);
        if (lane == 0)
            S.wsum[warp] = __popc(bal);
        __syncthreads();
        const int wc = S.wsum[lane];
        const int M = __reduce_add_sync(VTG_FULL, wc), slot = __reduce_add_sync(VTG_FULL, lane < warp ? wc : 0) +
                                                              __popc(bal & ((1u << lane) - 1u));
        __syncthreads();
        if (M > DET_BLOCK) { /* only when size > DET_BLOCK */
            size = max(DET_BLOCK, size / 2);
            continue;
        }
        from = limit;
        left -= members;
        /* the next block: three quarters of a full one clear, by this one's share */
        size = min(DET_SELECT_THREADS, max(DET_BLOCK, DET_BLOCK * 3 / 4 * members / max(M, 1)));
        if (clear)
            S.xy[slot] = me;
        __syncthreads();
        /* the conflicts: thread (i, part) compares candidate i with 64 of those before it */
        {
            const int i = tid % DET_BLOCK, part = tid / DET_BLOCK;
            unsigned m0 = 0u, m1 = 0u;
            if (64 * part <= (i | 31) && 64 * part < M) { /* uniform in a warp */
                const int2 p = S.xy[min(i, M - 1)];
#pragma unroll 4
                for (int j = 0; j < 32; j++) {
                    const int2 u = S.xy[64 * part + j], v = S.xy[64 * part + 32 + j];
                    const int ux = u.x - p.x, uy = u.y - p.y, vx = v.x - p.x, vy = v.y - p.y;
                    m0 |= ux * ux + uy * uy < q.need ? 1u << j : 0u;
                    m1 |= vx * vx + vy * vy < q.need ? 1u << j : 0u;
                }
            }
            /* only those before i */
            auto before = [&](int k) { return k > (i >> 5) ? 0u : k < (i >> 5) ? ~0u : (1u << (i & 31)) - 1u; };
            S.mask[2 * part][i] = m0 & before(2 * part);
            S.mask[2 * part + 1][i] = m1 & before(2 * part + 1);
        }
        __syncthreads();
        if (warp == 0) {
            unsigned got = 0u; /* lane k: the taken ones of word k */
            for (int k = 0; 32 * k < M; k++) {
                const int i = 32 * k + lane;
                unsigned hit = 0u;
                for (int e = 0; e < k; e++)
                    hit |= S.mask[e][i] & __shfl_sync(VTG_FULL, got, e);
                const unsigned own = S.mask[k][i];
                unsigned open = __ballot_sync(VTG_FULL, i < M && !hit), yes = 0u;
                while (open) {
                    const bool here = (open >> lane) & 1u;
                    const bool now = here && !(own & (open | yes));
                    const bool out = here && (own & yes);
                    yes |= __ballot_sync(VTG_FULL, now);
                    open &= ~__ballot_sync(VTG_FULL, now || out);
                }
                got = lane == k ? yes : got;
            }
            if (lane < DET_BLOCK / 32)
                S.got[lane] = got;
        }
        __syncthreads();
        /* the taken ones in order, those past max dropped */
        int total = 0, rank = 0;
#pragma unroll
        for (int k = 0; k < DET_BLOCK / 32; k++) {
            const int c = __popc(S.got[k]);
            rank += k < (tid >> 5) ? c : 0;
            total += c;
        }
        if (tid < M) {
            rank += __popc(S.got[tid >> 5] & ((1u << lane) - 1u));
            if (((S.got[tid >> 5] >> lane) & 1u) && taken + rank < q.max) {
                const int t = taken + rank;
                const int2 c = S.xy[tid];
                S.tx[t] = c.x;
                S.ty[t] = c.y;
                xs[t] = (float)c.x;
                ys[t] = (float)c.y;
                S.next[t] = atomicExch(&S.head[((c.y - q.g.y0) / q.gs) * q.gw + (c.x - q.g.ax) / q.gs], t);
            }
        }
        taken = min(taken + total, q.max);
        __syncthreads();
    }
    if (tid == 0)
        *count = taken;
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

/* detect_begin's layout (src/kern/detect.c:28-66); false when nothing of the rectangle lies inside the margin. */
static bool det_geometry(int w, int h, float rx, float ry, float rw, float rh, int margin, DetGeo &g)
{
    /* a region past any plane (or not a number) holds nothing; so does a negative margin's outside */
    const float lim = 1.0e8f;
    if (margin < 0 || !(fabsf(rx) < lim && fabsf(ry) < lim && fabsf(rw) < lim && fabsf(rh) < lim))
        return false;
    int x0 = (int)rx, y0 = (int)ry, x1 = (int)(rx + rw), y1 = (int)(ry + rh);
    x0 = x0 < margin ? margin : x0;
    y0 = y0 < margin ? margin : y0;
    x1 = x1 > w - margin ? w - margin : x1;
    y1 = y1 > h - margin ? h - margin : y1;
    if (x1 <= x0 || y1 <= y0)
        return false;
    g.x0 = x0;
    g.y0 = y0;
    g.x1 = x1;
    g.y1 = y1;
    g.ax = x0 & ~15;
    g.cols = (x1 - g.ax + 15) & ~15;
    g.rows = y1 - y0;
    g.nv = g.cols / 16;
    g.cell_rows = g.rows / 16 + 1;
    return true;
}

static size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

struct DetLayout {
    size_t resp, cell, best, rowcount, rowbase, ncand, keys, cxy, bytes;
};

static DetLayout det_layout(int max_w, int max_h, int &max_cols, int &max_cells)
{
    max_cols = ((max_w + 15) & ~15) + 16;
    max_cells = (max_h / 16 + 1) * (max_cols / 16);
    DetLayout L;
    size_t b = 0;
    L.resp = b;
    b += up256(sizeof(float) * (size_t)max_cols * max_h);
    L.cell = b;
    b += up256(sizeof(float) * (size_t)max_cells);
    L.best = b;
    b += 256;
    L.rowcount = b;
    b += up256(sizeof(int) * (size_t)max_h * DET_SEGS);
    L.rowbase = b;
    b += up256(sizeof(int) * (size_t)max_h * DET_SEGS);
    L.ncand = b;
    b += 256;
    L.keys = b;
    b += up256(sizeof(unsigned) * DET_MAX_CAND);
    L.cxy = b;
    b += up256(sizeof(int2) * DET_MAX_CAND);
    L.bytes = b;
    return L;
}

extern "C" size_t vtg_detector_bytes(int max_w, int max_h)
{
    if (max_w < 1 || max_h < 1 || max_w > 16384 || max_h > 16384)
        return 0;
    int mc, mcl;
    return det_layout(max_w, max_h, mc, mcl).bytes;
}

extern "C" int vtg_detector_create(vtg_ctx *ctx, int max_w, int max_h, vtg_detector **out)
{
    if (!ctx || !out || max_w < 1 || max_h < 1 || max_w > 16384 || max_h > 16384)
        return VTG_EINVAL;
    *out = nullptr;
    int max_cols, max_cells;
    const DetLayout L = det_layout(max_w, max_h, max_cols, max_cells);
    const int charged = vtg_ctx_charge(ctx, L.bytes);
    if (charged != VTG_OK)
        return charged;
    vtg_detector *d = new (std::nothrow) vtg_detector;
    if (!d) {
        vtg_ctx_release(ctx, L.bytes);
        return VTG_ENOMEM;
    }
    d->ctx = ctx;
    d->bytes = L.bytes;
    d->max_w = max_w;
    d->max_h = max_h;
    d->max_cols = max_cols;
    d->max_cells = max_cells;
    cudaError_t e = cudaSetDevice(vtg_ctx_device(ctx));
    if (e == cudaSuccess)
        e = cudaMalloc(&d->mem, L.bytes);
    if (e != cudaSuccess) {
        vtg_set_cuda_error(e);
        vtg_ctx_release(ctx, L.bytes);
        delete d;
        return VTG_ENOMEM;
    }
    d->host = nullptr;
    e = cudaHostAlloc(&d->host, sizeof *d->host, cudaHostAllocMapped);
    if (e == cudaSuccess)
        e = cudaHostGetDevicePointer(&d->host_dev, d->host, 0);
    if (e == cudaSuccess)
        e = cudaStreamCreateWithFlags(&d->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        vtg_set_cuda_error(e);
        cudaFreeHost(d->host);
        cudaFree(d->mem);
        vtg_ctx_release(ctx, L.bytes);
        delete d;
        return VTG_ECUDA;
    }
    d->resp = (float *)(d->mem + L.resp);
    d->cell = (float *)(d->mem + L.cell);
    d->best = (float *)(d->mem + L.best);
    d->rowcount = (int *)(d->mem + L.rowcount);
    d->rowbase = (int *)(d->mem + L.rowbase);
    d->ncand = (int *)(d->mem + L.ncand);
    d->keys = (unsigned *)(d->mem + L.keys);
    d->cxy = (int2 *)(d->mem + L.cxy);
    vtg_ctx_track(ctx, d->stream, true);
    *out = d;
    return VTG_OK;
}

extern "C" void vtg_detector_destroy(vtg_detector *d)
{
    if (!d)
        return;
    cudaSetDevice(vtg_ctx_device(d->ctx));
    cudaStreamSynchronize(d->stream);
    vtg_ctx_track(d->ctx, d->stream, false);
    cudaStreamDestroy(d->stream);
    cudaFree(d->mem);
    cudaFreeHost(d->host);
    vtg_ctx_release(d->ctx, d->bytes);
    delete d;
}

extern "C" void *vtg_detector_stream(const vtg_detector *d) { return d ? (void *)d->stream : nullptr; }

extern "C" int vtg_detect(vtg_detector *d, const float *plane, int w, int h, int pitch, float rx, float ry, float rw,
                          float rh, int margin, int max, float min_dist, float quality, float *xs, float *ys, int *count,
                          int where, void *stream)
{
    if (!d || !plane || w < 1 || h < 1 || pitch < w || max < 0 || max > 512 || !(min_dist >= 0.0f) ||
        !(quality >= 0.0f) || (max > 0 && (!xs || !ys)) || !count || (where != VTG_HOST && where != VTG_DEVICE) ||
        !(rx == rx && ry == ry && rw == rw && rh == rh))
        return VTG_EINVAL;
    const cudaStream_t st = stream ? (cudaStream_t)stream : d->stream;
    CU(cudaSetDevice(vtg_ctx_device(d->ctx)));
    DetPrm q;
    q.p = plane;
    q.w = w;
    q.h = h;
    q.pitch = pitch;
    q.quality = quality;
    q.max = max;
    /* exact: a product of two F32s; past 2^30 no two places in a 16384 x 16384 region are that far apart */
    const double min2 = (double)min_dist * (double)min_dist;
    q.need = min2 < (double)(1 << 30) ? (int)ceil(min2) : 1 << 30;
    const bool any = det_geometry(w, h, rx, ry, rw, rh, margin, q.g);
    if (any && (q.g.rows > d->max_h || q.g.cols > d->max_cols || q.g.nv * q.g.cell_rows > d->max_cells))
        return VTG_EINVAL;
    if (any) {
        /* the smallest side whose square reaches need, grown until the region's grid fits DET_GRID_MAX cells */
        long long gs = (long long)sqrt((double)q.need);
        while (gs * gs < q.need)
            gs++;
        gs = gs < 1 ? 1 : gs;
        while (((q.g.cols + gs - 1) / gs) * ((q.g.rows + gs - 1) / gs) > DET_GRID_MAX)
            gs++;
        q.gs = (int)gs;
        q.gw = (int)((q.g.cols + gs - 1) / gs);
        q.gh = (int)((q.g.rows + gs - 1) / gs);
    }
    if (!any || max == 0) {
        if (where == VTG_HOST) {
            *count = 0;
            return VTG_OK;
        }
        CU(cudaMemsetAsync(count, 0, sizeof(int), st));
        return VTG_OK;
    }
    const DetGeo &g = q.g;
    float *oxs = where == VTG_DEVICE ? xs : d->host_dev->xs, *oys = where == VTG_DEVICE ? ys : d->host_dev->ys;
    int *ocount = where == VTG_DEVICE ? count : &d->host_dev->count;
    const bool scan = g.rows > DET_SCAN_ROWS;
    const dim3 rows(g.rows), threads(32 * DET_SEGS);
    const float *resp = d->resp, *cell = d->cell, *best = d->best;
    const int *rowcount = d->rowcount, *rowbase = d->rowbase;
    det_response<<<dim3((g.cols + DET_TX - 1) / DET_TX, (g.rows + DET_TY - 1) / DET_TY), 256, 0, st>>>(q, d->resp,
                                                                                                   d->cell, d->best);
    CU(vtg_launch_k(det_count, rows, threads, 0, st, true, q, resp, cell, d->best, d->rowcount,
                    scan ? (int *)nullptr : d->rowbase));
    if (scan)
        CU(vtg_launch_k(det_scan, dim3(1), dim3(1024), 0, st, true, g.rows * DET_SEGS, rowcount, d->rowbase, d->ncand));
    CU(vtg_launch_k(det_collect, rows, threads, 0, st, true, q, resp, cell, best, rowcount, rowbase, scan, d->keys, d->cxy,
                    d->ncand));
    const int smem = (int)sizeof(DetSelectSmem);
    CU(cudaFuncSetAttribute(det_select, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    CU(vtg_launch_k(det_select, dim3(1), dim3(DET_SELECT_THREADS), smem, st, true, q, (const int *)d->ncand, best,
                    (const unsigned *)d->keys, (const int2 *)d->cxy, oxs, oys, ocount));
    CU(cudaGetLastError());
    if (where == VTG_HOST) {
        CU(cudaStreamSynchronize(st));
        *count = d->host->count;
        memcpy(xs, d->host->xs, sizeof(float) * (size_t)*count);
        memcpy(ys, d->host->ys, sizeof(float) * (size_t)*count);
    }
    return VTG_OK;
}

/* The stages' planes, for checking: resp (rows x cols) and cells (cell_rows x nv) of the last vtg_detect, and its
 * layout (x0, y0, x1, y1, ax, cols, rows, nv, cell_rows). Waits for the detector's stream. */
extern "C" int vtg_detect_maps(vtg_detector *d, float rx, float ry, float rw, float rh, int w, int h, int margin,
                               int *geo, float *resp, float *cells)
{
    if (!d || !geo)
        return VTG_EINVAL;
    DetGeo g;
    if (!det_geometry(w, h, rx, ry, rw, rh, margin, g) || g.rows > d->max_h || g.cols > d->max_cols ||
        g.nv * g.cell_rows > d->max_cells)
        return VTG_EINVAL;
    const int v[9] = {g.x0, g.y0, g.x1, g.y1, g.ax, g.cols, g.rows, g.nv, g.cell_rows};
    for (int k = 0; k < 9; k++)
        geo[k] = v[k];
    CU(cudaSetDevice(vtg_ctx_device(d->ctx)));
    CU(cudaStreamSynchronize(d->stream));
    if (resp)
        CU(cudaMemcpy(resp, d->resp, sizeof(float) * (size_t)g.rows * g.cols, cudaMemcpyDeviceToHost));
    if (cells)
        CU(cudaMemcpy(cells, d->cell, sizeof(float) * (size_t)g.nv * g.cell_rows, cudaMemcpyDeviceToHost));
    return VTG_OK;
}
