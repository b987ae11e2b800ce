/* framegen.cu -- a generated frame between two real ones on the GPU: the motion field of FidelityFX Optical Flow as
 * the reference restates it (block SAD search, filter, upscale over a pyramid), the vectors at the middle instant, and
 * the blended frame.
 *
 * Reference: src/kern/framegen.c (fg_hist_section, fg_scene_verdict, fg_search, fg_filter, fg_upscale,
 * fg_mid_vectors, fg_blend) and img_q6_to_u8_vx (src/kern/img_vx.c:36-47), run in the order of tk_generate_make
 * (src/kern/track.c:847-888).
 *
 * Every plane holds whole-number Q6 values, so every SAD is an exact F32 sum in any order and the fields are the
 * reference's bit for bit. The blend keeps the reference's six fused multiply-adds in their order (its sums pass 2^24)
 * and rounds to the nearest, ties to even. The reference reads replicated padding; here a read is a clamped index,
 * except the search window's origin, which the reference clamps into its padding (that moves the offsets searched)
 * and which is clamped here the same way.
 *
 * One call, on one stream; each launch after the first a programmatic dependent of the one before:
 *   fg_reduce3_kernel     three levels of the field's pyramid of both frames at once: level 0 is the frames' half size
 *                         (once more for each further three levels); beside the second, the scene test: 64-bin
 *                         histograms of nine sections of both frames' level 1, the last CTA's verdict
 *   fg_search_kernel      once a level, coarsest first: a warp an 8 x 8 block. Its estimate from the coarser level (the
 *                         coarser fields' filter and the upscale, a few lanes' work each), then the 24 x 24 window in
 *                         shared memory, a lane 8 of the 256 offsets
 *   fg_mid_kernel         a warp a block: the finest field's filter, then the vectors at the middle instant
 *   fg_blend_kernel       a warp a 16 x 16 tile of the full-size frame: the frame (Q6) and its bytes */
#include <math.h>
#include <stdint.h>

#include <new>

#include "vtg_ctx.h"
#include "vtg_internal.cuh"

#define FG_LEVELS 7 /* FG_MAX_LEVELS, src/kern/framegen.h:20 */
#define FG_WARPS 4  /* blocks a CTA in the search and the middle vectors */

/* one level of the field: both frames' planes there and its three fields */
struct FgLevel {
    const float *a, *b; /* older, newer */
    int w, h, pitch, bw, bh;
    short2 *raw, *fil, *up;
};

struct vtg_framegen {
    vtg_ctx *ctx;
    cudaStream_t stream;
    char *mem;
    size_t bytes;
    int w, h, levels, out_pitch;
    FgLevel L[FG_LEVELS];
    float *pa[FG_LEVELS], *pb[FG_LEVELS];
    short2 *mid;
    unsigned *hist; /* 2 x 9 x 64 */
    int *scene;     /* [0] the verdict, [1] the hist kernel's ticket */
    float *out;
    unsigned char *pic;
};

/* Coherent loads: what a launch before this one wrote was not read-only while this one, its dependent, ran. */
__device__ __forceinline__ float fg_at(const float *p, int pitch, int w, int h, int x, int y)
{
    return __ldca(p + (size_t)min(max(y, 0), h - 1) * pitch + min(max(x, 0), w - 1));
}

__device__ __forceinline__ float fg_warp_sum(float v)
{
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1)
        v += __shfl_xor_sync(VTG_FULL, v, d);
    return v;
}

/* Three pyramid steps of both frames (img_reduce, src/kern/img_ref.c:98-114: the 5 x 5 binomial, (sum + 128) >> 8, clamped
 * borders) in one launch. A CTA owns a 64 x 32 block of the first level made and the 32 x 16 and 16 x 8 blocks under it. The
 * first level's vertical sums come straight from the source, a thread a column and eleven rows of them (25 loads in
 * flight), for the 73 x 41 values that the levels above need; the rest runs in shared memory. A level reads the one below at
 * the reference's clamped indices, which always fall inside the computed halo. At 1080p, both frames, levels 0 to 2: 14 us
 * where a launch a level took 12 + 6 + 4 (25 loads a value); issue at half, between barriers, bounds it. */
#define FR_X 64
#define FR_Y 32
#define FR_A_C 73 /* the first level computed: columns X0 - 6 .. X0 + 66, rows Y0 - 6 .. Y0 + 34 */
#define FR_A_R 41
#define FR_S_C (2 * FR_A_C + 3) /* its source columns, from 2 X0 - 14 */
#define FR_S_P 152              /* 16-byte rows, and the last pair's eight values */
#define FR_B_C 35
#define FR_B_R 19
#define FR_C_C 16
#define FR_C_R 8
#define FR_SEG 11 /* rows of vertical sums a thread: four segments */

struct FgReduce {
    const float *s[2];
    int sw, sh, sp[2];
    int n; /* levels to make, 1 to 3 */
    float *d[3][2];
    int w[3], h[3], p[3];
    int bx, by; /* blocks */
};

struct FgReduceSmem {
    __align__(16) int v[FR_A_R][FR_S_P]; /* the first level's vertical sums */
    int a[FR_A_R][FR_A_C + 1];
    int v2[FR_B_R][FR_A_C];
    int b[FR_B_R][FR_B_C];
    int v3[FR_C_R][FR_B_C];
};

__device__ __forceinline__ int fg_tap5(int a, int b, int c, int d, int e) { return a + e + 4 * (b + d) + 6 * c; }

/* EDGE: some index of the block's needs its clamp. */
template <bool EDGE>
__device__ __forceinline__ void fg_reduce_block(const FgReduce &q, int f, int X0, int Y0, FgReduceSmem &S)
{
    const int tid = threadIdx.x, nt = blockDim.x;
    const float *src = q.s[f];
    auto clamp = [](int v, int n) { return EDGE ? min(max(v, 0), n - 1) : v; };
    for (int i = tid; i < 4 * FR_S_C; i += nt) {
        const int g = i / FR_S_C, c = i - g * FR_S_C, r0 = g * FR_SEG;
        const float *col = src + clamp(2 * X0 - 14 + c, q.sw);
        int v[2 * FR_SEG + 3];
#pragma unroll
        for (int k = 0; k < 2 * FR_SEG + 3; k++)
            v[k] = (int)__ldca(col + (size_t)clamp(2 * (Y0 - 6 + r0) - 2 + k, q.sh) * q.sp[f]);
#pragma unroll
        for (int r = 0; r < FR_SEG; r++)
            if (r0 + r < FR_A_R)
                S.v[r0 + r][c] = fg_tap5(v[2 * r], v[2 * r + 1], v[2 * r + 2], v[2 * r + 3], v[2 * r + 4]);
    }
    __syncthreads();
    /* two columns a thread, from eight vertical sums (column 73, past the last, is computed and not used) */
    for (int i = tid; i < FR_A_R * ((FR_A_C + 1) / 2); i += nt) {
        const int y = i / ((FR_A_C + 1) / 2), x = 2 * (i - y * ((FR_A_C + 1) / 2));
        const int4 u = *reinterpret_cast<const int4 *>(&S.v[y][2 * x]), t = *reinterpret_cast<const int4 *>(&S.v[y][2 * x + 4]);
        const int o0 = (fg_tap5(u.x, u.y, u.z, u.w, t.x) + 128) >> 8, o1 = (fg_tap5(u.z, u.w, t.x, t.y, t.z) + 128) >> 8;
        S.a[y][x] = o0;
        S.a[y][x + 1] = o1;
        const int gy = Y0 - 6 + y, gx = X0 - 6 + x; /* x and the block's edges are even */
        if (y >= 6 && y < 6 + FR_Y && x >= 6 && x < 6 + FR_X && (!EDGE || (gy < q.h[0] && gx < q.w[0]))) {
            float *d = q.d[0][f] + (size_t)gy * q.p[0] + gx;
            if (!EDGE || gx + 1 < q.w[0])
                *reinterpret_cast<float2 *>(d) = make_float2((float)o0, (float)o1);
            else
                *d = (float)o0;
        }
    }
    if (q.n < 2)
        return;
    __syncthreads();
    for (int i = tid; i < FR_B_R * FR_A_C; i += nt) {
        const int y = i / FR_A_C, x = i - y * FR_A_C;
        int v[5];
#pragma unroll
        for (int t = 0; t < 5; t++)
            v[t] = S.a[clamp(2 * (Y0 / 2 - 2 + y) - 2 + t, q.h[0]) - (Y0 - 6)][x];
        S.v2[y][x] = fg_tap5(v[0], v[1], v[2], v[3], v[4]);
    }
    __syncthreads();
    for (int i = tid; i < FR_B_R * FR_B_C; i += nt) {
        const int y = i / FR_B_C, x = i - y * FR_B_C;
        int v[5];
#pragma unroll
        for (int t = 0; t < 5; t++)
            v[t] = S.v2[y][clamp(2 * (X0 / 2 - 2 + x) - 2 + t, q.w[0]) - (X0 - 6)];
        const int o = (fg_tap5(v[0], v[1], v[2], v[3], v[4]) + 128) >> 8;
        S.b[y][x] = o;
        const int gy = Y0 / 2 - 2 + y, gx = X0 / 2 - 2 + x;
        if (y >= 2 && y < 2 + FR_Y / 2 && x >= 2 && x < 2 + FR_X / 2 && (!EDGE || (gy < q.h[1] && gx < q.w[1])))
            q.d[1][f][(size_t)gy * q.p[1] + gx] = (float)o;
    }
    if (q.n < 3)
        return;
    __syncthreads();
    for (int i = tid; i < FR_C_R * FR_B_C; i += nt) {
        const int y = i / FR_B_C, x = i - y * FR_B_C;
        int v[5];
#pragma unroll
        for (int t = 0; t < 5; t++)
            v[t] = S.b[clamp(2 * (Y0 / 4 + y) - 2 + t, q.h[1]) - (Y0 / 2 - 2)][x];
        S.v3[y][x] = fg_tap5(v[0], v[1], v[2], v[3], v[4]);
    }
    __syncthreads();
    for (int i = tid; i < FR_C_R * FR_C_C; i += nt) {
        const int y = i / FR_C_C, x = i - y * FR_C_C;
        const int gy = Y0 / 4 + y, gx = X0 / 4 + x;
        if (EDGE && (gy >= q.h[2] || gx >= q.w[2]))
            continue;
        int v[5];
#pragma unroll
        for (int t = 0; t < 5; t++)
            v[t] = S.v3[y][clamp(2 * gx - 2 + t, q.w[1]) - (X0 / 2 - 2)];
        q.d[2][f][(size_t)gy * q.p[2] + gx] = (float)((fg_tap5(v[0], v[1], v[2], v[3], v[4]) + 128) >> 8);
    }
}

__device__ void fg_reduce_any(const FgReduce &q, int block, FgReduceSmem &S)
{
    const int f = block / (q.bx * q.by), at = block - f * q.bx * q.by;
    const int X0 = (at % q.bx) * FR_X, Y0 = (at / q.bx) * FR_Y;
    /* every source row and column that the block reads lies inside the source: rows 2 Y0 - 14 .. + 4 FR_SEG x 2 + 2 */
    if (X0 > 0 && Y0 > 0 && 2 * X0 - 14 + FR_S_C <= q.sw && 2 * Y0 - 14 + 8 * FR_SEG + 3 <= q.sh)
        fg_reduce_block<false>(q, f, X0, Y0, S);
    else
        fg_reduce_block<true>(q, f, X0, Y0, S);
}

/* fg_hist_section (framegen.c:85-101): part `part` of FG_HIST_SPLIT of the sampled rows of section s of frame f, counted
 * a warp and added into the global counts; the last CTA of the test compares the frames (fg_scene_verdict,
 * framegen.c:103-113: more than half the samples in other bins, i.e. sum |a - b| > sum b) and zeroes the counts for
 * the next call. */
#define FG_HIST_SPLIT 8
#define FG_HIST_CTAS (18 * FG_HIST_SPLIT)
struct FgHistSmem {
    unsigned h[8][64];
    unsigned long long sum[8][2];
    bool last;
};

__device__ void fg_hist_part(const FgLevel &lv, int k0, unsigned *__restrict__ hist, int *scene, FgHistSmem &S)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int s = k0 % 9, f = (k0 / 9) % 2, part = k0 / 18;
    for (int i = tid; i < 8 * 64; i += 256)
        S.h[i >> 6][i & 63] = 0u;
    __syncthreads();
    const float *p = f ? lv.b : lv.a;
    const int sx = s % 3, sy = s / 3;
    const int x0 = (lv.w * sx / 3) & ~15, x1 = (lv.w * (sx + 1) / 3) & ~15;
    const int y0 = lv.h * sy / 3, y1 = lv.h * (sy + 1) / 3;
    const int cols = x1 - x0, rows = (y1 - y0 + 1) / 2;
    for (int k = part * 256 + tid; k < cols * rows; k += FG_HIST_SPLIT * 256) {
        const int y = y0 + 2 * (k / cols), x = x0 + k % cols;
        atomicAdd(&S.h[warp][(int)(__ldca(p + (size_t)y * lv.pitch + x) * (1.0f / 256.0f)) & 63], 1u);
    }
    __syncthreads();
    if (tid < 64) {
        unsigned n = 0u;
#pragma unroll
        for (int w = 0; w < 8; w++)
            n += S.h[w][tid];
        if (n)
            atomicAdd(&hist[(f * 9 + s) * 64 + tid], n);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0)
        S.last = atomicAdd(&scene[1], 1) == FG_HIST_CTAS - 1;
    __syncthreads();
    if (!S.last)
        return;
    __threadfence();
    unsigned long long diff = 0, total = 0;
    for (int i = tid; i < 9 * 64; i += 256) {
        const unsigned a = __ldcg(&hist[i]), b = __ldcg(&hist[9 * 64 + i]);
        diff += a > b ? a - b : b - a;
        total += b;
        hist[i] = 0;
        hist[9 * 64 + i] = 0;
    }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        diff += __shfl_xor_sync(VTG_FULL, diff, d);
        total += __shfl_xor_sync(VTG_FULL, total, d);
    }
    if (lane == 0) {
        S.sum[warp][0] = diff;
        S.sum[warp][1] = total;
    }
    __syncthreads();
    if (tid == 0) {
        diff = total = 0;
        for (int w = 0; w < 8; w++) {
            diff += S.sum[w][0];
            total += S.sum[w][1];
        }
        scene[0] = total && diff > total;
        scene[1] = 0;
    }
}

/* The levels' CTAs first, then (hist) the scene test's on level 1, which an earlier launch made. */
__global__ void __launch_bounds__(256) fg_reduce3_kernel(FgReduce q, int reduces, FgLevel l1, unsigned *hist, int *scene)
{
    __shared__ union {
        FgReduceSmem r;
        FgHistSmem h;
    } S;
    vtg_grid_launch_dependents();
    vtg_grid_dependency_wait();
    if ((int)blockIdx.x < reduces)
        fg_reduce_any(q, blockIdx.x, S.r);
    else
        fg_hist_part(l1, (int)blockIdx.x - reduces, hist, scene, S.h);
}

/* fg_filter (framegen.c:218-247) of the block at (bx, by): of the 3 x 3 around it (clamped; candidate 3 column + row), the
 * vector with the least sum of squared differences from the nine; the first on a tie. A lane reads all nine, and again, by
 * its own index, those it sums for. */
struct FgNine {
    int v[9]; /* packed short2 */
};

__device__ __forceinline__ int fg_raw_at(const FgLevel &lv, int bx, int by, int a)
{
    const int xx = a / 3, yy = a - 3 * xx;
    return __ldca(reinterpret_cast<const int *>(lv.raw) + min(max(by + yy - 1, 0), lv.bh - 1) * lv.bw +
                  min(max(bx + xx - 1, 0), lv.bw - 1));
}
__device__ __forceinline__ FgNine fg_nine(const FgLevel &lv, int bx, int by)
{
    FgNine n;
    const int *raw = reinterpret_cast<const int *>(lv.raw);
    int row[3], col[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        row[k] = min(max(by + k - 1, 0), lv.bh - 1) * lv.bw;
        col[k] = min(max(bx + k - 1, 0), lv.bw - 1);
    }
#pragma unroll
    for (int a = 0; a < 9; a++)
        n.v[a] = __ldca(raw + row[a % 3] + col[a / 3]);
    return n;
}
__device__ __forceinline__ unsigned fg_apart(int a, int b)
{
    const int dx = (short)(a & 0xffff) - (short)(b & 0xffff), dy = (a >> 16) - (b >> 16);
    return (unsigned)(dx * dx + dy * dy);
}
__device__ __forceinline__ unsigned fg_sum_apart(const FgNine &n, int me)
{
    unsigned d = 0u;
#pragma unroll
    for (int b = 0; b < 9; b++)
        d += fg_apart(me, n.v[b]);
    return d;
}
/* the lesser of two (sum, candidate) with their vectors */
__device__ __forceinline__ void fg_lesser(unsigned &d, int &a, int &v, unsigned od, int oa, int ov)
{
    const bool o = od < d || (od == d && oa < a);
    d = o ? od : d;
    a = o ? oa : a;
    v = o ? ov : v;
}
/* Eight lanes a block, lane j candidate j. Candidate 8's sum is that of the eight lanes' distances from it. */
__device__ __forceinline__ int fg_filtered8(const FgLevel &lv, int bx, int by, int j)
{
    const FgNine n = fg_nine(lv, bx, by);
    int v = fg_raw_at(lv, bx, by, j), a = j;
    unsigned d = fg_sum_apart(n, v), d8 = fg_apart(v, n.v[8]);
#pragma unroll
    for (int k = 1; k < 8; k <<= 1) {
        d8 += __shfl_xor_sync(VTG_FULL, d8, k);
        fg_lesser(d, a, v, __shfl_xor_sync(VTG_FULL, d, k), __shfl_xor_sync(VTG_FULL, a, k), __shfl_xor_sync(VTG_FULL, v, k));
    }
    return d8 < d ? n.v[8] : v;
}
/* Three lanes a block (lanes 3 k, 3 k + 1, 3 k + 2), lane j candidates 3 j .. 3 j + 2; the first lane ends with the vector. */
__device__ __forceinline__ int fg_filtered3(const FgLevel &lv, int bx, int by, int j)
{
    const FgNine n = fg_nine(lv, bx, by);
    int v = fg_raw_at(lv, bx, by, 3 * j), a = 3 * j;
    unsigned d = fg_sum_apart(n, v);
#pragma unroll
    for (int k = 1; k < 3; k++) {
        const int u = fg_raw_at(lv, bx, by, 3 * j + k);
        fg_lesser(d, a, v, fg_sum_apart(n, u), 3 * j + k, u);
    }
    const int lane = threadIdx.x & 31;
    const unsigned d1 = __shfl_sync(VTG_FULL, d, lane + 1), d2 = __shfl_sync(VTG_FULL, d, lane + 2);
    const int a1 = __shfl_sync(VTG_FULL, a, lane + 1), a2 = __shfl_sync(VTG_FULL, a, lane + 2);
    const int v1 = __shfl_sync(VTG_FULL, v, lane + 1), v2 = __shfl_sync(VTG_FULL, v, lane + 2);
    fg_lesser(d, a, v, d1, a1, v1);
    fg_lesser(d, a, v, d2, a2, v2);
    return v;
}

/* fg_upscale (framegen.c:251-288) for block (gx, gy) of the level under `lv`, a warp: of the four nearest blocks' filtered
 * vectors, the one with the least SAD over the 4 x 4 of lv that the block covers (the first on a tie), doubled. Eight lanes
 * a candidate: its filter, then two pixels each. The block whose own coarse block is candidate 3 (both places even) stores
 * that filtered vector: every coarse block has one. */
__device__ __forceinline__ short2 fg_upscaled(const FgLevel &lv, int gx, int gy, int lane)
{
    const int n = lane >> 3;
    const int cx = gx / 2 + n % 2 - 1 + gx % 2, cy = gy / 2 + n / 2 - 1 + gy % 2;
    const int px = gx * 4 + (lane & 3), py = gy * 4 + ((lane >> 2) & 1);
    const float c0 = fg_at(lv.b, lv.pitch, lv.w, lv.h, px, py), c1 = fg_at(lv.b, lv.pitch, lv.w, lv.h, px, py + 2);
    const int f = fg_filtered8(lv, min(max(cx, 0), lv.bw - 1), min(max(cy, 0), lv.bh - 1), lane & 7);
    const short2 v = make_short2((short)(f & 0xffff), (short)(f >> 16));
    if (lane == 24 && !(gx & 1) && !(gy & 1))
        lv.fil[(gy / 2) * lv.bw + gx / 2] = v;
    float s = fabsf(c0 - fg_at(lv.a, lv.pitch, lv.w, lv.h, px + v.x, py + v.y)) +
              fabsf(c1 - fg_at(lv.a, lv.pitch, lv.w, lv.h, px + v.x, py + 2 + v.y));
#pragma unroll
    for (int d = 1; d < 8; d <<= 1)
        s += __shfl_xor_sync(VTG_FULL, s, d);
    int pick = n, at = f;
#pragma unroll
    for (int d = 8; d < 32; d <<= 1) {
        const float os = __shfl_xor_sync(VTG_FULL, s, d);
        const int op = __shfl_xor_sync(VTG_FULL, pick, d), oa = __shfl_xor_sync(VTG_FULL, at, d);
        const bool o = os < s || (os == s && op < pick);
        s = o ? os : s;
        pick = o ? op : pick;
        at = o ? oa : at;
    }
    return make_short2((short)(2 * (short)(at & 0xffff)), (short)(2 * (at >> 16)));
}

/* fg_search (framegen.c:117-214) at one level: a warp an 8 x 8 block, from the coarser level's estimate (lv.up; none at the
 * top). The 256 offsets x0 - px + dx, wy + dy - 8 (dx, dy < 16) cost |dx - 8| + |dy - 8| plus the block's SAD; the
 * first lowest in row order wins. On the finest level a block the estimate explains (SAD <= 8192) is not searched, and
 * no motion wins when its SAD is no more than the best cost. */
#define FG_BIAS 12582912.0f /* 1.5 x 2^23: whole numbers below 2^22 of either sign keep one exponent with it */
#define FG_INT 5 /* of a row's eight differences, those taken as integers */
__global__ void __launch_bounds__(32 * FG_WARPS) fg_search_kernel(FgLevel lv, FgLevel coarse, bool top, int level,
                                                                  const int *__restrict__ scene)
{
    /* rows of 28: a quarter warp's eight rows of 16 bytes fall in different banks */
    __shared__ __align__(16) float s_win[FG_WARPS][24][28];
    __shared__ __align__(16) float s_blk[FG_WARPS][8][8];
    vtg_grid_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = (int)blockIdx.x * FG_WARPS + warp;
    vtg_grid_dependency_wait();
    if (i >= lv.bw * lv.bh)
        return;
    const int gx = i % lv.bw, gy = i / lv.bw;
    if (__ldca(scene)) {
        if (lane == 0) {
            lv.raw[i] = make_short2(0, 0);
            if (!top) {
                lv.up[i] = make_short2(0, 0);
                if (!(gx & 1) && !(gy & 1))
                    coarse.fil[(gy / 2) * coarse.bw + gx / 2] = make_short2(0, 0);
            }
        }
        return;
    }
    const int px = gx * 8, py = gy * 8;
    short2 want = make_short2(0, 0);
    if (!top) {
        want = fg_upscaled(coarse, gx, gy, lane);
        if (lane == 0)
            lv.up[i] = want;
    }
    const int wx = want.x, wy = want.y;
    const int lanes = (lv.w + 15) & ~15;
    const int x0 = min(max(px + wx - 8, -32), lanes), y0 = py + wy - 8;
    {
        /* every load of the window (a lane a column) and of the block in flight before the first store */
        float wv[24], bv[2];
        const float *col = lv.a + min(max(x0 + min(lane, 23), 0), lv.w - 1);
#pragma unroll
        for (int r = 0; r < 24; r++)
            wv[r] = __ldca(col + (size_t)(min(max(y0 + r, 0), lv.h - 1) * lv.pitch));
#pragma unroll
        for (int j = 0; j < 2; j++)
            bv[j] = fg_at(lv.b, lv.pitch, lv.w, lv.h, px + (lane & 7), py + (lane >> 3) + 4 * j);
        if (lane < 24)
#pragma unroll
            for (int r = 0; r < 24; r++)
                s_win[warp][r][lane] = wv[r] + FG_BIAS;
#pragma unroll
        for (int j = 0; j < 2; j++)
            s_blk[warp][(lane >> 3) + 4 * j][lane & 7] = bv[j] + FG_BIAS;
    }
    __syncwarp();
    if (level == 0) {
        /* the estimate's place is the window's centre: (x0 + 8, y0 + 8) */
        float s = 0.0f;
        for (int k = lane; k < 64; k += 32)
            s += fabsf(s_blk[warp][k >> 3][k & 7] - s_win[warp][8 + (k >> 3)][8 + (k & 7)]);
        s = fg_warp_sum(s);
        if (s <= 8192.0f) { /* FG_ENOUGH */
            if (lane == 0)
                lv.raw[i] = make_short2((short)(x0 - px + 8), (short)wy);
            return;
        }
    }
    /* The staged values carry FG_BIAS, so their bits as integers differ by the values' difference: five of a row's eight
     * absolute differences take one integer instruction each (sum of absolute differences, on the ALU pipe), three take two
     * F32 ones (on the FMA pipe), which keeps both pipes and the issue busy. A generated 1080p frame with 0, 3, 4, 5, 6, 8 of
     * them as integers: 46.0, 43.5, 42.5, 42.2, 42.5, 43.5 us. */
    const int dy = lane & 15, dx0 = (lane >> 4) * 8;
    float c[8];
    unsigned ci[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        c[k] = 0.0f;
        ci[k] = (unsigned)(abs(dx0 + k - 8) + abs(dy - 8)); /* FG_TIE_UNIT */
    }
#pragma unroll
    for (int r = 0; r < 8; r++) {
        float wv[16], bv[8];
#pragma unroll
        for (int k = 0; k < 4; k++)
            *reinterpret_cast<float4 *>(&wv[4 * k]) = *reinterpret_cast<const float4 *>(&s_win[warp][dy + r][dx0 + 4 * k]);
#pragma unroll
        for (int k = 0; k < 2; k++)
            *reinterpret_cast<float4 *>(&bv[4 * k]) = *reinterpret_cast<const float4 *>(&s_blk[warp][r][4 * k]);
#pragma unroll
        for (int k = 0; k < 8; k++)
#pragma unroll
            for (int n = 0; n < 8; n++)
                if (n < FG_INT)
                    ci[k] = __usad(__float_as_uint(wv[k + n]), __float_as_uint(bv[n]), ci[k]);
                else
                    c[k] += fabsf(wv[k + n] - bv[n]);
    }
#pragma unroll
    for (int k = 0; k < 8; k++)
        c[k] += (float)ci[k];
    float best = c[0];
    int bi = dy * 16 + dx0;
#pragma unroll
    for (int k = 1; k < 8; k++)
        if (c[k] < best) {
            best = c[k];
            bi = dy * 16 + dx0 + k;
        }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        const float ob = __shfl_xor_sync(VTG_FULL, best, d);
        const int oi = __shfl_xor_sync(VTG_FULL, bi, d);
        if (ob < best || (ob == best && oi < bi)) {
            best = ob;
            bi = oi;
        }
    }
    int vx = x0 - px + (bi & 15), vy = wy + (bi >> 4) - 8;
    if (level == 0) {
        float s = 0.0f;
        for (int k = lane; k < 64; k += 32)
            s += fabsf(s_blk[warp][k >> 3][k & 7] -
                       (fg_at(lv.a, lv.pitch, lv.w, lv.h, px + (k & 7), py + (k >> 3)) + FG_BIAS));
        s = fg_warp_sum(s);
        if (s <= best)
            vx = vy = 0;
    }
    if (lane == 0)
        lv.raw[i] = make_short2((short)vx, (short)vy);
}

/* fg_mid_vectors (framegen.c:292-328) on the finest level: no motion first, favoured by one grey level over the block
 * (FG_MID_FAVOUR_ZERO), then each vector of the 3 x 3 (row by row) that agrees better when each frame moves half way.
 * A warp a block, a lane two of its pixels. The 3 x 3's filtered vectors first, three lanes each. */
__global__ void __launch_bounds__(32 * FG_WARPS) fg_mid_kernel(FgLevel lv, short2 *__restrict__ mid)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = (int)blockIdx.x * FG_WARPS + warp;
    vtg_grid_launch_dependents();
    vtg_grid_dependency_wait();
    if (i >= lv.bw * lv.bh)
        return;
    const int bx = i % lv.bw, by = i / lv.bw, px = bx * 8, py = by * 8;
    const int nb = min(lane / 3, 8); /* the 3 x 3's block of this lane, row by row */
    const int fv = fg_filtered3(lv, min(max(bx + nb % 3 - 1, 0), lv.bw - 1), min(max(by + nb / 3 - 1, 0), lv.bh - 1), lane % 3);
    if (lane == 12)
        lv.fil[i] = make_short2((short)(fv & 0xffff), (short)(fv >> 16));
    auto sad = [&](int vx, int vy) {
        const int ax = vx >> 1, ay = vy >> 1, qx = vx - ax, qy = vy - ay;
        float s = 0.0f;
        for (int k = lane; k < 64; k += 32) {
            const int r = k >> 3, c = k & 7;
            s += fabsf(fg_at(lv.a, lv.pitch, lv.w, lv.h, px + c + ax, py + r + ay) -
                       fg_at(lv.b, lv.pitch, lv.w, lv.h, px + c - qx, py + r - qy));
        }
        return fg_warp_sum(s);
    };
    float best = sad(0, 0) - 64.0f;
    int vx = 0, vy = 0;
    for (int k = 0; k < 9; k++) {
        const int q = __shfl_sync(VTG_FULL, fv, 3 * k), qx = (short)(q & 0xffff), qy = q >> 16;
        if ((qx == vx && qy == vy) || (qx == 0 && qy == 0))
            continue;
        const float s = sad(qx, qy);
        if (s < best) {
            best = s;
            vx = qx;
            vy = qy;
        }
    }
    if (lane == 0)
        mid[i] = make_short2((short)vx, (short)vy);
}

/* fg_blend (framegen.c:332-357) and img_q6_to_u8_vx: a warp a 16 x 16 tile, a lane eight of its pixels (a column's every
 * second row), so that a lane has many loads in flight. */
#define FG_BLEND_WARPS 8
__global__ void __launch_bounds__(32 * FG_BLEND_WARPS) fg_blend_kernel(const float *__restrict__ a0, int pa,
                                                                       const float *__restrict__ b0, int pb, int w, int h,
                                                                       const short2 *mid, int bw, int bh,
                                                                       float *__restrict__ out, int po,
                                                                       unsigned char *__restrict__ pic)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tx = (int)blockIdx.x * FG_BLEND_WARPS + warp, ty = blockIdx.y;
    vtg_grid_dependency_wait();
    if (16 * tx >= w)
        return;
    /* lane k < 9: the 3 x 3's vector k, row by row; the others the first one again */
    const int nk = lane < 9 ? lane : 0;
    const int near = __ldca(reinterpret_cast<const int *>(mid) + min(max(ty + nk / 3 - 1, 0), bh - 1) * bw +
                            min(max(tx + nk % 3 - 1, 0), bw - 1));
    const int first = __shfl_sync(VTG_FULL, near, 0);
    const bool same = __all_sync(VTG_FULL, near == first);
    const int k = lane & 15, x = tx * 16 + k;
    auto store = [&](int y, float v) {
        out[(size_t)y * po + x] = v;
        if (pic) {
            const float q = rintf(v * (1.0f / 64.0f));
            pic[(size_t)y * w + x] = q <= 0.0f ? 0 : q >= 255.0f ? 255 : (unsigned char)q;
        }
    };
    auto at = [&](const float *p, int pitch, int xx, int yy) {
        return __ldg(p + (size_t)min(max(yy, 0), h - 1) * pitch + min(max(xx, 0), w - 1));
    };
    if (same) {
        const int vx = (short)(first & 0xffff), vy = first >> 16;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int y = ty * 16 + 2 * j + (lane >> 4);
            v[j] = rintf((at(a0, pa, x + vx, y + vy) + at(b0, pb, x - vx, y - vy)) * 0.5f);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int y = ty * 16 + 2 * j + (lane >> 4);
            if (x < w && y < h)
                store(y, v[j]);
        }
        return;
    }
    /* in 32nds: across, the left, own and right blocks; down, the own row and the one above or below */
    const float wl = k < 8 ? (float)(15 - 2 * k) : 0.0f, wr = k < 8 ? 0.0f : (float)(2 * k - 15);
    const float ws = k < 8 ? (float)(17 + 2 * k) : (float)(47 - 2 * k);
    const float wh[3] = {wl, ws, wr};
    /* a tile whose every read lies inside the frame takes them without clamps: six places of each frame, a column's rows
     * two rows apart */
    const int reach_x = (int)__reduce_max_sync(VTG_FULL, (unsigned)abs((int)(short)(near & 0xffff)));
    const int reach_y = (int)__reduce_max_sync(VTG_FULL, (unsigned)abs(near >> 16));
    const bool inside = tx * 16 >= reach_x && tx * 16 + 16 + reach_x <= w && ty * 16 >= reach_y && ty * 16 + 16 + reach_y <= h;
#pragma unroll
    for (int half = 0; half < 2; half++) { /* the tile's upper rows blend with the row of blocks above, the lower below */
        int q[2][3];
#pragma unroll
        for (int b = 0; b < 3; b++) {
            q[0][b] = __shfl_sync(VTG_FULL, near, 3 + b);
            q[1][b] = __shfl_sync(VTG_FULL, near, 6 * half + b);
        }
        const int s0 = 8 * half + (lane >> 4), y0 = ty * 16 + s0;
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) {
                const int ex = (short)(q[a][b] & 0xffff), ey = q[a][b] >> 16;
                float sum[4];
                if (inside) {
                    const float *fa = a0 + (ptrdiff_t)(y0 + ey) * pa + (x + ex), *fb = b0 + (ptrdiff_t)(y0 - ey) * pb + (x - ex);
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        sum[j] = __ldg(fa + 2 * j * pa) + __ldg(fb + 2 * j * pb);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        sum[j] = at(a0, pa, x + ex, y0 + 2 * j + ey) + at(b0, pb, x - ex, y0 + 2 * j - ey);
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int s = s0 + 2 * j, wo = s < 8 ? 15 - 2 * s : 2 * s - 15;
                    acc[j] = __fmaf_rn(sum[j], wh[b] * (float)(a == 0 ? 32 - wo : wo), acc[j]);
                }
            }
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (x < w && y0 + 2 * j < h)
                store(y0 + 2 * j, rintf(acc[j] * (1.0f / 2048.0f)));
    }
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

static bool fg_size_ok(int w, int h) { return w >= 64 && h >= 64 && w <= 8192 && h <= 8192; }

/* The field's levels (src/kern/track.c:547-556): the frames' half size, then halves, while both sides are >= 16. */
static int fg_shapes(int w, int h, int lw[FG_LEVELS], int lh[FG_LEVELS])
{
    int n = 0, x = (w + 1) / 2, y = (h + 1) / 2;
    while (n < FG_LEVELS && x >= 16 && y >= 16) {
        lw[n] = x;
        lh[n] = y;
        n++;
        x = (x + 1) / 2;
        y = (y + 1) / 2;
    }
    return n;
}

static size_t fg_layout(int w, int h, size_t off_plane_a[FG_LEVELS], size_t off_plane_b[FG_LEVELS],
                        size_t off_f[FG_LEVELS][3], size_t *off_mid, size_t *off_hist, size_t *off_scene,
                        size_t *off_out, size_t *off_pic)
{
    int lw[FG_LEVELS], lh[FG_LEVELS];
    const int n = fg_shapes(w, h, lw, lh);
    size_t b = 0;
    for (int L = 0; L < n; L++) {
        const size_t plane = up256(sizeof(float) * (size_t)vtg_pitch(lw[L]) * (size_t)lh[L]);
        const size_t field = up256(sizeof(short2) * (size_t)((lw[L] + 7) / 8) * (size_t)((lh[L] + 7) / 8));
        off_plane_a[L] = b;
        b += plane;
        off_plane_b[L] = b;
        b += plane;
        for (int k = 0; k < 3; k++) {
            off_f[L][k] = b;
            b += field;
        }
    }
    *off_mid = b;
    b += up256(sizeof(short2) * (size_t)((lw[0] + 7) / 8) * (size_t)((lh[0] + 7) / 8));
    *off_hist = b;
    b += up256(sizeof(unsigned) * 2 * 9 * 64);
    *off_scene = b;
    b += 256;
    *off_out = b;
    b += up256(sizeof(float) * (size_t)vtg_pitch(w) * (size_t)h);
    *off_pic = b;
    b += up256((size_t)w * (size_t)h);
    return b;
}

extern "C" size_t vtg_framegen_bytes(int w, int h)
{
    if (!fg_size_ok(w, h))
        return 0;
    size_t a[FG_LEVELS], b[FG_LEVELS], f[FG_LEVELS][3], m, hi, s, o, p;
    return fg_layout(w, h, a, b, f, &m, &hi, &s, &o, &p);
}

extern "C" int vtg_framegen_create(vtg_ctx *ctx, int w, int h, vtg_framegen **out)
{
    if (!ctx || !out || !fg_size_ok(w, h))
        return VTG_EINVAL;
    *out = nullptr;
    size_t oa[FG_LEVELS], ob[FG_LEVELS], of[FG_LEVELS][3], om, oh, os, oo, op;
    const size_t bytes = fg_layout(w, h, oa, ob, of, &om, &oh, &os, &oo, &op);
    const int charged = vtg_ctx_charge(ctx, bytes);
    if (charged != VTG_OK)
        return charged;
    vtg_framegen *g = new (std::nothrow) vtg_framegen;
    if (!g) {
        vtg_ctx_release(ctx, bytes);
        return VTG_ENOMEM;
    }
    g->ctx = ctx;
    g->bytes = bytes;
    g->w = w;
    g->h = h;
    g->out_pitch = vtg_pitch(w);
    int lw[FG_LEVELS], lh[FG_LEVELS];
    g->levels = fg_shapes(w, h, lw, lh);
    g->stream = nullptr;
    cudaError_t e = cudaSetDevice(vtg_ctx_device(ctx));
    if (e == cudaSuccess)
        e = cudaMalloc(&g->mem, bytes);
    if (e != cudaSuccess) {
        vtg_set_cuda_error(e);
        vtg_ctx_release(ctx, bytes);
        delete g;
        return VTG_ENOMEM;
    }
    e = cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(g->mem, 0, bytes, g->stream);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(g->stream);
    if (e != cudaSuccess) {
        vtg_set_cuda_error(e);
        if (g->stream)
            cudaStreamDestroy(g->stream);
        cudaFree(g->mem);
        vtg_ctx_release(ctx, bytes);
        delete g;
        return VTG_ECUDA;
    }
    for (int L = 0; L < g->levels; L++) {
        FgLevel &v = g->L[L];
        g->pa[L] = (float *)(g->mem + oa[L]);
        g->pb[L] = (float *)(g->mem + ob[L]);
        v.a = g->pa[L];
        v.b = g->pb[L];
        v.w = lw[L];
        v.h = lh[L];
        v.pitch = vtg_pitch(lw[L]);
        v.bw = (lw[L] + 7) / 8;
        v.bh = (lh[L] + 7) / 8;
        v.raw = (short2 *)(g->mem + of[L][0]);
        v.fil = (short2 *)(g->mem + of[L][1]);
        v.up = (short2 *)(g->mem + of[L][2]);
    }
    g->mid = (short2 *)(g->mem + om);
    g->hist = (unsigned *)(g->mem + oh);
    g->scene = (int *)(g->mem + os);
    g->out = (float *)(g->mem + oo);
    g->pic = (unsigned char *)(g->mem + op);
    vtg_ctx_track(ctx, g->stream, true);
    *out = g;
    return VTG_OK;
}

extern "C" void vtg_framegen_destroy(vtg_framegen *g)
{
    if (!g)
        return;
    cudaSetDevice(vtg_ctx_device(g->ctx));
    cudaStreamSynchronize(g->stream);
    vtg_ctx_track(g->ctx, g->stream, false);
    cudaStreamDestroy(g->stream);
    cudaFree(g->mem);
    vtg_ctx_release(g->ctx, g->bytes);
    delete g;
}

extern "C" void *vtg_framegen_stream(const vtg_framegen *g) { return g ? (void *)g->stream : nullptr; }

extern "C" int vtg_framegen_levels(const vtg_framegen *g) { return g ? g->levels : 0; }

extern "C" int vtg_framegen_run(vtg_framegen *g, const float *older, int older_pitch, const float *newer,
                                int newer_pitch, float *out, int out_pitch, uint8_t *pic, int where, void *stream)
{
    if (!g || !older || !newer || older_pitch < g->w || newer_pitch < g->w || (out && out_pitch < g->w) ||
        (pic && where != VTG_HOST && where != VTG_DEVICE))
        return VTG_EINVAL;
    const cudaStream_t st = stream ? (cudaStream_t)stream : g->stream;
    CU(cudaSetDevice(vtg_ctx_device(g->ctx)));
    /* the field's pyramid: level 0 from the frames, each next from the last, three levels a launch; the scene test with the
     * launch after level 1's */
    FgReduce q = {};
    q.s[0] = older;
    q.s[1] = newer;
    q.sw = g->w;
    q.sh = g->h;
    q.sp[0] = older_pitch;
    q.sp[1] = newer_pitch;
    bool hist = false;
    for (int L = 0; L < g->levels || !hist; L += 3) {
        q.n = min(3, g->levels - L);
        int reduces = 0;
        if (q.n > 0) {
            for (int k = 0; k < q.n; k++) {
                q.d[k][0] = g->pa[L + k];
                q.d[k][1] = g->pb[L + k];
                q.w[k] = g->L[L + k].w;
                q.h[k] = g->L[L + k].h;
                q.p[k] = g->L[L + k].pitch;
            }
            q.bx = (q.w[0] + FR_X - 1) / FR_X;
            q.by = (q.h[0] + FR_Y - 1) / FR_Y;
            reduces = 2 * q.bx * q.by;
        }
        const bool test = L > 0 && !hist;
        CU(vtg_launch_k(fg_reduce3_kernel, dim3(reduces + (test ? FG_HIST_CTAS : 0)), dim3(256), 0, st, L > 0, q, reduces, g->L[1],
                        g->hist, g->scene));
        hist = hist || test;
        if (q.n == 3) {
            q.s[0] = g->pa[L + 2];
            q.s[1] = g->pb[L + 2];
            q.sw = q.w[2];
            q.sh = q.h[2];
            q.sp[0] = q.sp[1] = q.p[2];
        }
    }
    for (int L = g->levels - 1; L >= 0; L--) {
        const FgLevel &v = g->L[L];
        const bool top = L == g->levels - 1;
        CU(vtg_launch_k(fg_search_kernel, dim3((v.bw * v.bh + FG_WARPS - 1) / FG_WARPS), dim3(32 * FG_WARPS), 0, st, true, v,
                        g->L[top ? L : L + 1], top, L, (const int *)g->scene));
    }
    const FgLevel &z = g->L[0];
    CU(vtg_launch_k(fg_mid_kernel, dim3((z.bw * z.bh + FG_WARPS - 1) / FG_WARPS), dim3(32 * FG_WARPS), 0, st, true, z, g->mid));
    float *dst = out ? out : g->out;
    const int dp = out ? out_pitch : g->out_pitch;
    unsigned char *pd = pic ? (where == VTG_DEVICE ? (unsigned char *)pic : g->pic) : nullptr;
    CU(vtg_launch_k(fg_blend_kernel, dim3((g->w + 16 * FG_BLEND_WARPS - 1) / (16 * FG_BLEND_WARPS), (g->h + 15) / 16),
                    dim3(32 * FG_BLEND_WARPS), 0, st, true, older, older_pitch, newer, newer_pitch, g->w, g->h,
                    (const short2 *)g->mid, z.bw, z.bh, dst, dp, pd));
    CU(cudaGetLastError());
    if (pic && where == VTG_HOST) {
        CU(cudaMemcpyAsync(pic, g->pic, (size_t)g->w * (size_t)g->h, cudaMemcpyDeviceToHost, st));
        CU(cudaStreamSynchronize(st));
    }
    return VTG_OK;
}

extern "C" int vtg_framegen_fields(vtg_framegen *g, int level, struct vtg_fg_vec *raw, struct vtg_fg_vec *fil,
                                   struct vtg_fg_vec *up, struct vtg_fg_vec *mid, int *scene, int where, void *stream)
{
    if (!g || level < 0 || level >= g->levels || (where != VTG_HOST && where != VTG_DEVICE))
        return VTG_EINVAL;
    const cudaStream_t st = stream ? (cudaStream_t)stream : g->stream;
    const cudaMemcpyKind k = where == VTG_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
    CU(cudaSetDevice(vtg_ctx_device(g->ctx)));
    const FgLevel &v = g->L[level];
    const size_t n = sizeof(short2) * (size_t)v.bw * (size_t)v.bh;
    if (raw)
        CU(cudaMemcpyAsync(raw, v.raw, n, k, st));
    if (fil)
        CU(cudaMemcpyAsync(fil, v.fil, n, k, st));
    if (up)
        CU(cudaMemcpyAsync(up, v.up, n, k, st));
    if (mid)
        CU(cudaMemcpyAsync(mid, g->mid, sizeof(short2) * (size_t)g->L[0].bw * (size_t)g->L[0].bh, k, st));
    if (scene)
        CU(cudaMemcpyAsync(scene, g->scene, sizeof(int), k, st));
    if (where == VTG_HOST)
        CU(cudaStreamSynchronize(st));
    return VTG_OK;
}

extern "C" int vtg_framegen_frame(const vtg_framegen *g, const float **plane, int *pitch)
{
    if (!g || !plane || !pitch)
        return VTG_EINVAL;
    *plane = g->out;
    *pitch = g->out_pitch;
    return VTG_OK;
}
