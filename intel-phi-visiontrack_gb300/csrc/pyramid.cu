/* pyramid.cu -- the Gaussian pyramid of an 8-bit frame, bit-exact to the reference's Q6 planes.
 *
 * Reference: tk_build (src/kern/track.c:584-629) runs img_u8_to_q6 (src/kern/img_ref.c:32-40, img_vx.c:24-34) and
 * img_pad_rows / img_pad_tb (img_ref.c:9-30) for level 0, then img_reduce (img_ref.c:98-114, img_vx.c:129-162) per
 * level: the 5 x 5 binomial (1 4 6 4 1)^2 at every second pixel of every second row, rounded as (sum + 128) >> 8,
 * reading a replicated border. Every value is a whole number below 2^24, so the reference's F32 sums are exact; here
 * they are int32 sums, the border is a clamped index, and the results are the same bits.
 *
 * Levels 0 to 3 in one launch (pyr_fused_kernel, pyr_fused_batch_kernel; pyr_input_kernel where tk_build's input steps make
 * level 0): a CTA reads its block's bytes once and reduces level by level in shared memory, halos included (below). Levels
 * from 4 on take one launch per level (pyr_reduce_kernel, pyr_batch_kernel): a CTA of 256 threads makes a 64 x 16 tile of
 * its output level from a 136 x 36 source tile staged in shared memory, the vertical pass over the staged rows, the
 * horizontal pass over the vertical sums, as the reference's vert5 / shift8 do. */
#include <math.h>
#include <stddef.h>

#include "vtg_internal.cuh"
#include "x87.cuh"

#define RT_X 64 /* output tile */
#define RT_Y 16
#define RS_Y (2 * RT_Y + 4) /* source rows of a tile: two each side */
/* Staged columns: a tile's source columns are 2 ox - 2 .. 2 ox + 129; staging starts 16-byte aligned before them, at 2 ox - 4
 * (136 values). Column k of the vertical sums is source column 2 ox - 4 + k. */
#define SF_X 136
#define SF_P 140 /* row pitch of staged values and of the vertical sums: 16-byte aligned rows */

/* A whole number 0 <= v < 2^23 as a float without a conversion instruction: the bits of 2^23 + v, less 2^23. */
__device__ __forceinline__ float small_int_to_float(int v)
{
    return __int_as_float(0x4B000000 | v) - 8388608.0f;
}

/* Byte e of w times 64 (a Q6 value) as a float: the byte placed in the mantissa of 2^23 by one byte permute, then
 * (2^23 + b) x 64 - 2^29 = 64 b in one fused multiply-add, exact (2^29 + 64 b is a multiple of 64 below 2^30). */
__device__ __forceinline__ float q6_of(uint32_t w, int e)
{
    return __fmaf_rn(__int_as_float((int)__byte_perm(w, 0x4Bu, 0x4550u + (unsigned)e)), 64.0f, -536870912.0f);
}

/* One 64 x 16 tile of the output level at (ox, oy) from level L - 1 (F32 Q6, whole numbers), (h + 128) >> 8. The source's base and
 * pitch are 16-byte aligned. Staging reads whole 16-byte chunks inside the row and clamps the chunks that reach past an edge
 * element by element, so every read is inside the plane and the border is the reference's replicated edge. */
__device__ __forceinline__ void reduce_tile(const float *src, int sw, int sh, int spitch, float *__restrict__ dst, int dw, int dh,
                                            int dpitch, int ox, int oy, float (*s_f)[SF_P], float (*s_v)[SF_P])
{
    const int tid = threadIdx.x;
    const int sy0 = 2 * oy - 2, gx0 = 2 * ox - 4;
    /* coherent loads: the level below may have been written while this launch, its dependent, had begun */
    for (int i = tid; i < RS_Y * (SF_X / 4); i += blockDim.x) {
        const int r = i / (SF_X / 4), k = i - r * (SF_X / 4);
        const int gy = min(max(sy0 + r, 0), sh - 1), gx = gx0 + 4 * k;
        const float *row = src + (size_t)gy * spitch;
        float4 v;
        if (gx >= 0 && gx + 4 <= sw)
            v = __ldca(reinterpret_cast<const float4 *>(row + gx));
        else
            v = make_float4(__ldca(row + min(max(gx, 0), sw - 1)), __ldca(row + min(max(gx + 1, 0), sw - 1)),
                            __ldca(row + min(max(gx + 2, 0), sw - 1)), __ldca(row + min(max(gx + 3, 0), sw - 1)));
        *reinterpret_cast<float4 *>(&s_f[r][4 * k]) = v;
    }
    __syncthreads();
    for (int i = tid; i < RT_Y * (SF_X / 4); i += blockDim.x) {
        const int r = i / (SF_X / 4), g = i - r * (SF_X / 4);
        /* F32 as the reference sums: whole numbers below 2^24, so every sum is exact */
        float4 t[5];
#pragma unroll
        for (int q = 0; q < 5; q++)
            t[q] = *reinterpret_cast<const float4 *>(&s_f[2 * r + q][4 * g]);
        float4 o;
        o.x = t[0].x + t[4].x + 4.0f * (t[1].x + t[3].x) + 6.0f * t[2].x;
        o.y = t[0].y + t[4].y + 4.0f * (t[1].y + t[3].y) + 6.0f * t[2].y;
        o.z = t[0].z + t[4].z + 4.0f * (t[1].z + t[3].z) + 6.0f * t[2].z;
        o.w = t[0].w + t[4].w + 4.0f * (t[1].w + t[3].w) + 6.0f * t[2].w;
        *reinterpret_cast<float4 *>(&s_v[r][4 * g]) = o;
    }
    __syncthreads();
    /* horizontal: output x takes vertical sums 2 x + 2 .. 2 x + 6; four outputs a thread (sums 8 g .. 8 g + 15) */
    for (int i = tid; i < RT_Y * (RT_X / 4); i += blockDim.x) {
        const int r = i / (RT_X / 4), g = i - r * (RT_X / 4);
        const int gy = oy + r, gx = ox + 4 * g;
        if (gy >= dh || gx >= dw)
            continue;
        float f[16];
#pragma unroll
        for (int q = 0; q < 4; q++)
            *reinterpret_cast<float4 *>(&f[4 * q]) = *reinterpret_cast<const float4 *>(&s_v[r][8 * g + 4 * q]);
        float o[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int c = 2 * e + 4;
            const float h = f[c - 2] + f[c + 2] + 4.0f * (f[c - 1] + f[c + 1]) + 6.0f * f[c];
            o[e] = floorf((h + 128.0f) * (1.0f / 256.0f)); /* (h + 128) >> 8, exact */
        }
        float *d = dst + (size_t)gy * dpitch + gx;
        if (gx + 4 <= dw) {
            *reinterpret_cast<float4 *>(d) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
            for (int e = 0; e < 4 && gx + e < dw; e++)
                d[e] = o[e];
        }
    }
}

struct ReduceSmem {
    __align__(16) float f[RS_Y][SF_P], v[RT_Y][SF_P];
};

__global__ void __launch_bounds__(256) pyr_reduce_kernel(const float *src, int sw, int sh, int spitch, float *__restrict__ dst,
                                                         int dw, int dh, int dpitch)
{
    __shared__ ReduceSmem S;
    vtg_grid_dependency_wait(); /* the level below, when launched as a dependent of its launch */
    reduce_tile(src, sw, sh, spitch, dst, dw, dh, dpitch, blockIdx.x * RT_X, blockIdx.y * RT_Y, S.f, S.v);
}

/* Many frames at once: the launch's tiles are every job's tiles of this level, back to back; a block finds its job by
 * binary search over the tile offsets. */
__global__ void __launch_bounds__(256) pyr_batch_kernel(const PyrJob *__restrict__ jobs, const int *__restrict__ start,
                                                        int njobs, int level, int *__restrict__ reset)
{
    __shared__ ReduceSmem S;
    vtg_grid_dependency_wait(); /* the level below, when launched as a dependent of its launch */
    if (reset && blockIdx.x == 0 && threadIdx.x == 0)
        *reset = 0;
    const int b = blockIdx.x;
    int lo = 0, hi = njobs; /* start[lo] <= b < start[hi] */
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(start + mid) <= b)
            lo = mid;
        else
            hi = mid;
    }
    const PyrJob &j = jobs[lo];
    const int t = b - __ldg(start + lo);
    const int dw = j.lw[level], dh = j.lh[level];
    const int tiles_x = (dw + RT_X - 1) / RT_X;
    reduce_tile(j.lv[level - 1], j.lw[level - 1], j.lh[level - 1], j.pitch[level - 1], j.lv[level], dw, dh, j.pitch[level],
                (t % tiles_x) * RT_X, (t / tiles_x) * RT_Y, S.f, S.v);
}

/* ---- levels 0 to 3 from the bytes in one launch ----
 *
 * A CTA owns a 128 x 64 block of level 0 and the blocks of levels 1, 2 and 3 under it (64 x 32, 32 x 16, 16 x 8). It
 * stages the bytes the block's level 3 depends on (rows Y0 - 14 .. Y0 + 70, columns X0 - 16 .. X0 + 143, each clamped
 * into the frame: the reference's replicated border), writes level 0 from them, and reduces in shared memory: level 1
 * over 73 x 41 values (the block and the halo level 2 needs), level 2 over 35 x 19, level 3 over its 16 x 8. A level's
 * reduce reads the level below at the reference's clamped indices, which always fall inside the computed halo, so the
 * values outside a level's plane that the halo holds are never read. Every sum is an exact integer: (sum of the bytes'
 * taps + 2) >> 2 for level 1 ((64 h + 128) >> 8 of the Q6 values), (h + 128) >> 8 above. Level 1 is then never read
 * back from memory, and three launches become one. */
#define FP_X 128 /* a CTA's level-0 block */
#define FP_Y 64
#define FB_R 85  /* staged byte rows: Y0 - 14 .. Y0 + 70 */
#define FB_C 160 /* staged byte columns: X0 - 16 .. X0 + 143 (16-byte chunks) */
#define F1_R 41  /* level 1 computed: rows Y0 / 2 - 6 .. Y0 / 2 + 34 */
#define F1_C 73  /*                   columns X0 / 2 - 6 .. X0 / 2 + 66 */
#define F1_P 76
#define F2_R 19  /* level 2: rows Y0 / 4 - 2 .. Y0 / 4 + 16 */
#define F2_C 35  /*          columns X0 / 4 - 2 .. X0 / 4 + 32 */
#define F2_P 36
#define F3_R 8   /* level 3: the block, rows Y0 / 8 .. + 7 */
#define F3_C 16  /*          columns X0 / 8 .. + 15 */

struct FusedUpper {
    __align__(16) uint16_t l1[F1_R][F1_P]; /* level 1 (at most 16320) */
    __align__(16) int v2[F2_R][F1_P];      /* level 2's vertical sums of level 1 */
    __align__(16) uint16_t l2[F2_R][F2_P]; /* level 2 */
    __align__(16) int v3[F3_R][F2_P];      /* level 3's vertical sums of level 2 */
};

struct FusedSmem {
    __align__(16) uint8_t b[FB_R][FB_C];   /* the bytes */
    __align__(16) uint16_t v1[F1_R][FB_C]; /* level 1's vertical sums of the bytes (at most 16 x 255) */
    FusedUpper u;
};

/* One frame of a fused launch: the bytes (rows `stride` apart), and levels 0 .. min(levels, 4) - 1. */
struct FusedFrame {
    const uint8_t *src;
    int stride, w, h, levels;
    float *lv[4];
    int pitch[4];
};

__device__ __forceinline__ int tap5(int a, int b, int c, int d, int e) { return a + e + 4 * (b + d) + 6 * c; }

/* A block is interior when every byte it stages lies inside the frame. Then no index of any level needs a clamp, and
 * every write of its blocks lies inside their planes. */
__device__ __forceinline__ bool fused_interior(const FusedFrame &f, int X0, int Y0)
{
    return X0 >= 16 && X0 + 144 <= f.w && Y0 >= 14 && Y0 + 71 <= f.h;
}

/* Levels 1 to 3 of a block from level 1 in S.l1. */
template <bool EDGE>
__device__ __forceinline__ void fused_upper(const FusedFrame &f, int X0, int Y0, FusedUpper &S)
{
    const int tid = threadIdx.x, nt = blockDim.x;
    const int w1 = (f.w + 1) / 2, h1 = (f.h + 1) / 2, w2 = (w1 + 1) / 2, h2 = (h1 + 1) / 2, w3 = (w2 + 1) / 2,
              h3 = (h2 + 1) / 2;
    /* level 1's block (local rows and columns 6 ..), four columns a thread */
    const int o1x = X0 / 2 - 6, o1y = Y0 / 2 - 6; /* level 1's local origin */
    for (int i = tid; i < (FP_Y / 2) * (FP_X / 8); i += nt) {
        const int r = i / (FP_X / 8), c = 4 * (i - r * (FP_X / 8));
        const int gy = Y0 / 2 + r, gx = X0 / 2 + c;
        if (EDGE && (gy >= h1 || gx >= w1))
            continue;
        const uint32_t a = *reinterpret_cast<const uint32_t *>(&S.l1[r + 6][c + 6]);
        const uint32_t b = *reinterpret_cast<const uint32_t *>(&S.l1[r + 6][c + 8]);
        const float4 o = make_float4(small_int_to_float((int)(a & 0xFFFFu)), small_int_to_float((int)(a >> 16)),
                                     small_int_to_float((int)(b & 0xFFFFu)), small_int_to_float((int)(b >> 16)));
        float *d = f.lv[1] + (size_t)gy * f.pitch[1] + gx;
        if (!EDGE || gx + 4 <= w1) {
            *reinterpret_cast<float4 *>(d) = o;
        } else {
            d[0] = o.x;
            if (gx + 1 < w1)
                d[1] = o.y;
            if (gx + 2 < w1)
                d[2] = o.z;
        }
    }
    if (f.levels < 3)
        return;
    /* level 2's vertical sums over level 1's (clamped) rows */
    const int o2x = X0 / 4 - 2, o2y = Y0 / 4 - 2; /* level 2's local origin */
    if constexpr (!EDGE) { /* a thread two columns of a run of rows, two new ones an output */
        constexpr int PAIRS = (F1_C + 1) / 2, RUN = 4;
        const int run = tid / PAIRS, x = 2 * (tid - run * PAIRS), y0 = run * RUN;
        int a[5], b[5];
        auto take = [&](int slot, int r) {
            const uint32_t q = *reinterpret_cast<const uint32_t *>(&S.l1[r][x]);
            a[slot] = (int)(q & 0xffffu);
            b[slot] = (int)(q >> 16);
        };
        if (y0 < F2_R) {
#pragma unroll
            for (int t = 0; t < 3; t++)
                take(t, 2 * y0 + t);
#pragma unroll
            for (int k = 0; k < RUN; k++) {
                if (y0 + k >= F2_R)
                    break;
                const int c0 = 2 * k % 5, c1 = (2 * k + 1) % 5, c2 = (2 * k + 2) % 5, c3 = (2 * k + 3) % 5, c4 = (2 * k + 4) % 5;
                take(c3, 2 * (y0 + k) + 3);
                take(c4, 2 * (y0 + k) + 4);
                *reinterpret_cast<int2 *>(&S.v2[y0 + k][x]) =
                    make_int2(tap5(a[c0], a[c1], a[c2], a[c3], a[c4]), tap5(b[c0], b[c1], b[c2], b[c3], b[c4]));
            }
        }
    }
    for (int i = tid; EDGE && i < F2_R * F1_C; i += nt) {
        const int y = i / F1_C, x = i - y * F1_C;
        int a[5];
#pragma unroll
        for (int t = 0; t < 5; t++)
            a[t] = S.l1[min(max(2 * (o2y + y) - 2 + t, 0), h1 - 1) - o1y][x];
        S.v2[y][x] = tap5(a[0], a[1], a[2], a[3], a[4]);
    }
    __syncthreads();
    for (int i = tid; i < F2_R * F2_C; i += nt) {
        const int y = i / F2_C, x = i - y * F2_C;
        int a[5];
#pragma unroll
        for (int t = 0; t < 5; t++)
            a[t] = S.v2[y][EDGE ? min(max(2 * (o2x + x) - 2 + t, 0), w1 - 1) - o1x : 2 * x + t];
        S.l2[y][x] = (uint16_t)((tap5(a[0], a[1], a[2], a[3], a[4]) + 128) >> 8);
    }
    __syncthreads();
    for (int i = tid; i < (FP_Y / 4) * (FP_X / 4); i += nt) {
        const int r = i / (FP_X / 4), c = i - r * (FP_X / 4);
        const int gy = Y0 / 4 + r, gx = X0 / 4 + c;
        if (!EDGE || (gy < h2 && gx < w2))
            f.lv[2][(size_t)gy * f.pitch[2] + gx] = small_int_to_float(S.l2[r + 2][c + 2]);
    }
    if (f.levels < 4)
        return;
    for (int i = tid; i < F3_R * F2_C; i += nt) {
        const int y = i / F2_C, x = i - y * F2_C;
        int a[5];
#pragma unroll
        for (int t = 0; t < 5; t++)
            a[t] = S.l2[EDGE ? min(max(2 * (Y0 / 8 + y) - 2 + t, 0), h2 - 1) - o2y : 2 * y + t][x];
        S.v3[y][x] = tap5(a[0], a[1], a[2], a[3], a[4]);
    }
    __syncthreads();
    for (int i = tid; i < F3_R * F3_C; i += nt) {
        const int y = i / F3_C, x = i - y * F3_C;
        const int gy = Y0 / 8 + y, gx = X0 / 8 + x;
        if (EDGE && (gy >= h3 || gx >= w3))
            continue;
        int a[5];
#pragma unroll
        for (int t = 0; t < 5; t++)
            a[t] = S.v3[y][EDGE ? min(max(2 * gx - 2 + t, 0), w2 - 1) - o2x : 2 * x + t];
        f.lv[3][(size_t)gy * f.pitch[3] + gx] = small_int_to_float((tap5(a[0], a[1], a[2], a[3], a[4]) + 128) >> 8);
    }
}

/* Sixteen bytes at any alignment as four words: from five aligned words, shifted. They read up to three bytes before and after,
 * so the caller keeps p three bytes clear of its row's ends. */
__device__ __forceinline__ void load16(const uint8_t *p, uint32_t (&q)[4])
{
    const uint32_t *a = reinterpret_cast<const uint32_t *>((uintptr_t)p & ~(uintptr_t)3);
    const int sh = 8 * (int)((uintptr_t)p & 3);
    uint32_t w[5];
#pragma unroll
    for (int k = 0; k < 4; k++)
        w[k] = __ldg(a + k);
    w[4] = sh ? __ldg(a + 4) : 0u;
#pragma unroll
    for (int k = 0; k < 4; k++)
        q[k] = __funnelshift_r(w[k], w[k + 1], sh);
}

template <bool EDGE>
__device__ void fused_block(const FusedFrame &f, int X0, int Y0, FusedSmem &S)
{
    const int tid = threadIdx.x, nt = blockDim.x;
    const int w = f.w, h = f.h;
    const bool vec = (((uintptr_t)f.src | (uintptr_t)f.stride) & 15) == 0;
    /* the bytes: staged row r is frame row Y0 - 14 + r, staged column c frame column X0 - 16 + c, both clamped */
    for (int i = tid; i < FB_R * (FB_C / 16); i += nt) {
        const int r = i / (FB_C / 16), k = i - r * (FB_C / 16);
        const int gy = EDGE ? min(max(Y0 - 14 + r, 0), h - 1) : Y0 - 14 + r, gx = X0 - 16 + 16 * k;
        const uint8_t *row = f.src + (size_t)gy * f.stride;
        uint4 v;
        if (vec && (!EDGE || (gx >= 0 && gx + 16 <= w))) {
            v = __ldg(reinterpret_cast<const uint4 *>(row + gx));
        } else if (gx >= 3 && gx + 19 <= w) {
            uint32_t q[4];
            load16(row + gx, q);
            v = make_uint4(q[0], q[1], q[2], q[3]);
        } else {
            uint32_t q[4];
#pragma unroll
            for (int a = 0; a < 4; a++) {
                uint32_t x = 0;
#pragma unroll
                for (int e = 0; e < 4; e++)
                    x |= (uint32_t)__ldg(row + min(max(gx + 4 * a + e, 0), w - 1)) << (8 * e);
                q[a] = x;
            }
            v = make_uint4(q[0], q[1], q[2], q[3]);
        }
        *reinterpret_cast<uint4 *>(&S.b[r][16 * k]) = v;
    }
    __syncthreads();
    /* level 0: the block's rows (staged 14 ..) and columns (staged 16 ..), four a thread */
    for (int i = tid; i < FP_Y * (FP_X / 4); i += nt) {
        const int r = i / (FP_X / 4), g = i - r * (FP_X / 4);
        const int gy = Y0 + r, gx = X0 + 4 * g;
        if (EDGE && (gy >= h || gx >= w))
            continue;
        const uint32_t q = *reinterpret_cast<const uint32_t *>(&S.b[r + 14][16 + 4 * g]);
        const float4 o = make_float4(q6_of(q, 0), q6_of(q, 1), q6_of(q, 2), q6_of(q, 3));
        float *d = f.lv[0] + (size_t)gy * f.pitch[0] + gx;
        if (!EDGE || gx + 4 <= w) {
            *reinterpret_cast<float4 *>(d) = o;
        } else {
            d[0] = o.x;
            if (gx + 1 < w)
                d[1] = o.y;
            if (gx + 2 < w)
                d[2] = o.z;
        }
    }
    if (f.levels < 2)
        return;
    /* level 1's vertical sums: local row y (frame row of level 1 Y0 / 2 - 6 + y) takes staged rows 2 y .. 2 y + 4;
     * four columns a thread, even and odd bytes in the 16-bit halves of two words (no half carries: at most 4080). A thread
     * runs down its rows with the last five in registers: read again for each output, a 3840 x 2160 frame took 13.0 us, and
     * now 12.0 (three streams; level 2's sums the same way); 3001 x 2000, whose rows are unaligned, 14.6 and 11.7 */
    constexpr int GROUPS = FB_C / 4, RUNS = 256 / GROUPS, RUN = (F1_R + RUNS - 1) / RUNS;
    const int g4 = tid % GROUPS, y0 = tid / GROUPS * RUN;
    if (tid < RUNS * GROUPS) { /* a thread a run of rows, two new ones an output */
        uint32_t e[5], o[5];
        auto take = [&](int slot, int r) {
            const uint32_t q = *reinterpret_cast<const uint32_t *>(&S.b[r][4 * g4]);
            e[slot] = q & 0x00FF00FFu;
            o[slot] = (q >> 8) & 0x00FF00FFu;
        };
#pragma unroll
        for (int t = 0; t < 3; t++)
            take(t, 2 * y0 + t);
#pragma unroll
        for (int k = 0; k < RUN; k++) {
            if (y0 + k >= F1_R)
                break;
            const int c0 = 2 * k % 5, c1 = (2 * k + 1) % 5, c2 = (2 * k + 2) % 5, c3 = (2 * k + 3) % 5, c4 = (2 * k + 4) % 5;
            take(c3, 2 * (y0 + k) + 3);
            take(c4, 2 * (y0 + k) + 4);
            const uint32_t E = e[c0] + e[c4] + 4u * (e[c1] + e[c3]) + 6u * e[c2];
            const uint32_t O = o[c0] + o[c4] + 4u * (o[c1] + o[c3]) + 6u * o[c2];
            *reinterpret_cast<uint2 *>(&S.v1[y0 + k][4 * g4]) = make_uint2((E & 0xFFFFu) | (O << 16), (E >> 16) | (O & 0xFFFF0000u));
        }
    }
    __syncthreads();
    /* level 1: local column x (frame column X0 / 2 - 6 + x) centres on staged column 2 x + 4. Two columns a thread in
     * the halves of one word: with w_k = v1 columns 2 x + 2 + 2 k and 2 x + 3 + 2 k, column x takes (w_0 lo, w_0 hi,
     * w_1 lo, w_1 hi, w_2 lo) and column x + 1 the same one word on. A sum is at most 16 x 4080 = 65280 a half, and
     * (h + 2) >> 2 at most 16320, so the mask drops exactly what the high half shifts into the low one. */
    for (int i = tid; i < F1_R * ((F1_C + 1) / 2); i += nt) {
        const int y = i / ((F1_C + 1) / 2), x = 2 * (i - y * ((F1_C + 1) / 2));
        const uint32_t *v = reinterpret_cast<const uint32_t *>(&S.v1[y][2 * x + 2]);
        const uint32_t w0 = v[0], w1 = v[1], w2 = v[2], w3 = v[3];
        const uint32_t L0 = __byte_perm(w0, w1, 0x5410), H0 = __byte_perm(w0, w1, 0x7632);
        const uint32_t L1 = __byte_perm(w1, w2, 0x5410), H1 = __byte_perm(w1, w2, 0x7632);
        const uint32_t L2 = __byte_perm(w2, w3, 0x5410);
        const uint32_t hs = L0 + L2 + 4u * (H0 + H1) + 6u * L1;
        *reinterpret_cast<uint32_t *>(&S.u.l1[y][x]) = ((hs + 0x00020002u) >> 2) & 0x3FFF3FFFu;
    }
    __syncthreads();
    fused_upper<EDGE>(f, X0, Y0, S.u);
}

__device__ __forceinline__ void fused_any(const FusedFrame &f, int bx, int by, FusedSmem &S)
{
    const int X0 = bx * FP_X, Y0 = by * FP_Y;
    if (fused_interior(f, X0, Y0))
        fused_block<false>(f, X0, Y0, S);
    else
        fused_block<true>(f, X0, Y0, S);
}

__global__ void __launch_bounds__(256) pyr_fused_kernel(FusedFrame f)
{
    __shared__ FusedSmem S;
    fused_any(f, blockIdx.x, blockIdx.y, S);
}

/* Many frames: the launch's blocks are every job's blocks back to back; a CTA finds its job by binary search. */
__global__ void __launch_bounds__(256) pyr_fused_batch_kernel(const PyrJob *__restrict__ jobs, const int *__restrict__ start,
                                                              int njobs, int *__restrict__ reset)
{
    __shared__ FusedSmem S;
    if (reset && blockIdx.x == 0 && threadIdx.x == 0)
        *reset = 0;
    const int b = blockIdx.x;
    int lo = 0, hi = njobs; /* start[lo] <= b < start[hi] */
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(start + mid) <= b)
            lo = mid;
        else
            hi = mid;
    }
    const PyrJob &j = jobs[lo];
    if (j.opts) /* vtg_launch_build_input made these levels */
        return;
    FusedFrame f;
    f.src = j.src;
    f.stride = j.stride;
    f.w = j.w;
    f.h = j.h;
    f.levels = j.levels;
#pragma unroll
    for (int L = 0; L < 4; L++) {
        f.lv[L] = L < j.levels ? j.lv[L] : nullptr;
        f.pitch[L] = L < j.levels ? j.pitch[L] : 0;
    }
    const int t = b - __ldg(start + lo), bcols = (j.w + FP_X - 1) / FP_X;
    fused_any(f, t % bcols, t / bcols, S);
}

int vtg_pyr_fused_tiles(int w, int h) { return ((w + FP_X - 1) / FP_X) * ((h + FP_Y - 1) / FP_Y); }

/* ---- tk_build's optional input steps (src/kern/track.c:600-622) ----
 *
 * CONTRAST: the min and max of the frame (img_minmax_ref, img_ref.c:57-71), the gain 16320 / (max - min) and the offset
 * -min x gain in x87 extended precision (track.c:603-614), each rounded to F32, then per pixel
 * clamp(rint(Q6 x gain + offset), 0, 16320) (img_norm, img_ref.c:42-55). PRE_GAUSS: the 5 x 5 binomial of that with
 * (h + 128) >> 8 (img_gauss5, img_ref.c:83-96). The result is level 0. The stretch runs on the bytes through a table:
 * a frame has 256 byte values, each mapped once per CTA. */

/* tk_build's gain and offset (track.c:606-614) for Q6 minimum lo and maximum hi: gain = 16320 / (hi - lo) or 1, offset
 * = -lo x gain, both formed in extended precision and rounded to F32. */
__host__ __device__ static inline void contrast_gain(int lo, int hi, float *go)
{
    if (hi > lo) {
        const X87 g = x87_div(16320u, (uint32_t)(hi - lo));
        go[0] = x87_to_f32(g);
        go[1] = -x87_to_f32(x87_mul(g, (uint32_t)lo));
    } else {
        go[0] = 1.0f;
        go[1] = -(float)lo;
    }
}

extern "C" int vtg_contrast_gain(int lo, int hi, float *gain_offset)
{
    if (!gain_offset || lo < 0 || hi < lo || hi >= (1 << 24))
        return VTG_EINVAL;
    contrast_gain(lo, hi, gain_offset);
    return VTG_OK;
}

/* The minimum and maximum over a CTA of per-thread values (min in the low byte of the result, max in the next). */
__device__ __forceinline__ uint32_t block_minmax(uint32_t mn, uint32_t mx, uint32_t *s_w)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    mn = __reduce_min_sync(VTG_FULL, mn);
    mx = __reduce_max_sync(VTG_FULL, mx);
    if (lane == 0)
        s_w[warp] = mn | (mx << 8);
    __syncthreads();
    if (warp == 0) {
        const uint32_t v = lane < (int)(blockDim.x >> 5) ? s_w[lane] : 255u;
        mn = __reduce_min_sync(VTG_FULL, v & 255u);
        mx = __reduce_max_sync(VTG_FULL, (v >> 8) & 255u);
        if (lane == 0)
            s_w[32] = mn | (mx << 8);
    }
    __syncthreads();
    const uint32_t r = s_w[32];
    __syncthreads();
    return r;
}

/* The frame's byte min and max (x 64 = img_minmax of its Q6 plane): CTA b scans rows b, b + grid, ... four bytes at a
 * time (16 with an aligned frame) and writes its partial to mm[b]; the last CTA to finish (a ticket in
 * mm[VTG_MM_BLOCKS]) combines the partials, writes gain and offset to mm[VTG_MM_BLOCKS + 1 ..] and resets the ticket. */
__global__ void __launch_bounds__(256) pyr_minmax_kernel(const uint8_t *__restrict__ src, int w, int h, int stride,
                                                         uint32_t *__restrict__ mm)
{
    __shared__ uint32_t s_w[33];
    __shared__ bool s_last;
    uint32_t mn4 = 0xffffffffu, mx4 = 0u;
    const bool vec = (((uintptr_t)src | (uintptr_t)stride) & 15) == 0;
    for (int y = blockIdx.x; y < h; y += gridDim.x) {
        const uint8_t *row = src + (size_t)y * stride;
        for (int x = 16 * (int)threadIdx.x; x < w; x += 16 * (int)blockDim.x) {
            uint32_t v[4];
            if (vec && x + 16 <= w) {
                const uint4 q = __ldg(reinterpret_cast<const uint4 *>(row + x));
                v[0] = q.x;
                v[1] = q.y;
                v[2] = q.z;
                v[3] = q.w;
            } else if (x >= 3 && x + 19 <= w) {
                load16(row + x, v);
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    uint32_t word = 0;
#pragma unroll
                    for (int e = 0; e < 4; e++) /* past the row's end: its last byte again, which changes nothing */
                        word |= (uint32_t)__ldg(row + min(x + 4 * k + e, w - 1)) << (8 * e);
                    v[k] = word;
                }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                mn4 = __vminu4(mn4, v[k]);
                mx4 = __vmaxu4(mx4, v[k]);
            }
        }
    }
    uint32_t mn = min(min(mn4 & 255u, (mn4 >> 8) & 255u), min((mn4 >> 16) & 255u, mn4 >> 24));
    uint32_t mx = max(max(mx4 & 255u, (mx4 >> 8) & 255u), max((mx4 >> 16) & 255u, mx4 >> 24));
    const uint32_t part = block_minmax(mn, mx, s_w);
    if (threadIdx.x == 0) {
        mm[blockIdx.x] = part;
        __threadfence();
        s_last = atomicAdd(&mm[VTG_MM_BLOCKS], 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last)
        return;
    __threadfence();
    mn = 255u;
    mx = 0u;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
        const uint32_t p = __ldcg(&mm[i]);
        mn = min(mn, p & 255u);
        mx = max(mx, (p >> 8) & 255u);
    }
    const uint32_t all = block_minmax(mn, mx, s_w);
    if (threadIdx.x == 0) {
        float go[2];
        contrast_gain(64 * (int)(all & 255u), 64 * (int)((all >> 8) & 255u), go);
        reinterpret_cast<float *>(mm)[VTG_MM_BLOCKS + 1] = go[0];
        reinterpret_cast<float *>(mm)[VTG_MM_BLOCKS + 2] = go[1];
        mm[VTG_MM_BLOCKS] = 0u; /* the next frame's ticket; this kernel's CTAs have all taken theirs */
    }
}

/* Levels 0 to 3 under the input steps in one launch, blocks as above. The bytes (rows Y0 - 16 .. Y0 + 72, columns X0 - 16 ..
 * X0 + 143, clamped into the frame) are staged through the stretch's table (or x 64) as whole numbers; GAUSS then makes level 0
 * over the block and the halo that level 1 needs (rows Y0 - 14 .. Y0 + 70, columns X0 - 14 .. X0 + 134) by the binomial's two
 * passes, else the staged values are level 0. Past the frame's edge the levels read the clamped index, never the halo's own
 * value there. A value's bit 15 keeps the table's -0, which a level-0 store without GAUSS must (the sums mask it).
 * The vertical passes run down a column with the last five rows in
 * registers: a shared load and a tap sum an output, where each output read its five rows. Bound by its phases' issue: two CTAs an
 * SM. A 1281 x 719 frame with both steps (and the launch for the gain), three streams: 15.4 us as five launches, 9.8 as two, 9.3
 * with unaligned bytes by shifted words, 8.5 with the running columns. (Started early, under the minimum and maximum's launch, it
 * fetches its bytes sooner, but a frame alone took 22 us, not 16, at 640 x 480: not done.) */
#define PI_R 89
#define PI_C 160
#define P0_R 85 /* level 0 as level 1 reads it */
#define P0_C 149
#define P0_P 152
#define PI_T 512

struct InputSmem {
    uint32_t lut[256]; /* a byte's value; bit 15: it is -0 */
    union {
        __align__(16) uint16_t n[PI_R][PI_C]; /* the mapped bytes */
        FusedUpper u;                         /* once they are not needed */
    };
    union {
        __align__(16) int v0[P0_R][P0_P + 4]; /* GAUSS: vertical sums, columns X0 - 16 .. X0 + 139 */
        int v1[F1_R][P0_P];     /* level 1's vertical sums, columns X0 - 14 .. */
    };
    __align__(16) uint16_t l0[P0_R][P0_P]; /* GAUSS: level 0 (must stay last) */
};

#define PI_CHUNKS ((PI_R * (PI_C / 16) + PI_T - 1) / PI_T) /* 16-byte chunks of the staged bytes a thread takes */

template <bool EDGE>
__device__ __forceinline__ void input_fetch(const FusedFrame &f, int X0, int Y0, uint32_t (&q)[PI_CHUNKS][4])
{
    const int w = f.w, h = f.h;
    const bool vec = (((uintptr_t)f.src | (uintptr_t)f.stride) & 15) == 0;
#pragma unroll
    for (int j = 0; j < PI_CHUNKS; j++) {
        const int i = (int)threadIdx.x + j * PI_T;
        if (i >= PI_R * (PI_C / 16))
            break;
        const int r = i / (PI_C / 16), k = i - r * (PI_C / 16);
        const int gy = EDGE ? min(max(Y0 - 16 + r, 0), h - 1) : Y0 - 16 + r, gx = X0 - 16 + 16 * k;
        const uint8_t *row = f.src + (size_t)gy * f.stride;
        if (vec && (!EDGE || (gx >= 0 && gx + 16 <= w))) {
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(row + gx));
            q[j][0] = v.x;
            q[j][1] = v.y;
            q[j][2] = v.z;
            q[j][3] = v.w;
        } else if (gx >= 3 && gx + 19 <= w) {
            load16(row + gx, q[j]);
        } else {
#pragma unroll
            for (int a = 0; a < 4; a++) {
                q[j][a] = 0u;
#pragma unroll
                for (int e = 0; e < 4; e++)
                    q[j][a] |= (uint32_t)__ldg(row + (EDGE ? min(max(gx + 4 * a + e, 0), w - 1) : gx + 4 * a + e)) << (8 * e);
            }
        }
    }
}

template <bool GAUSS, bool EDGE>
__device__ __forceinline__ void input_block(const FusedFrame &f, int X0, int Y0, const uint32_t (&q)[PI_CHUNKS][4], InputSmem &S)
{
    const int tid = threadIdx.x, w = f.w, h = f.h;
#pragma unroll
    for (int j = 0; j < PI_CHUNKS; j++) {
        const int i = tid + j * PI_T;
        if (i >= PI_R * (PI_C / 16))
            break;
        const int r = i / (PI_C / 16), k = i - r * (PI_C / 16);
        uint32_t o[8];
#pragma unroll
        for (int a = 0; a < 8; a++) {
            const uint32_t two = q[j][a >> 1] >> (16 * (a & 1));
            o[a] = S.lut[two & 255u] | S.lut[(two >> 8) & 255u] << 16;
        }
        *reinterpret_cast<uint4 *>(&S.n[r][16 * k]) = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4 *>(&S.n[r][16 * k + 8]) = make_uint4(o[4], o[5], o[6], o[7]);
    }
    __syncthreads();
    /* two columns of a row of level 0's staged values, low and high half */
    auto l0_pair = [&](int r, int c) {
        return GAUSS ? *reinterpret_cast<const uint32_t *>(&S.l0[r][c]) :
                       *reinterpret_cast<const uint32_t *>(&S.n[r + 2][c + 2]) & 0x7fff7fffu;
    };
    if (GAUSS) {
        /* a thread two columns of a run of rows, the last five rows' values in registers */
        constexpr int PAIRS = (P0_P + 4) / 2, RUN = (P0_R + PI_T / PAIRS - 1) / (PI_T / PAIRS);
        const int run = tid / PAIRS, c = 2 * (tid - run * PAIRS), r0 = run * RUN;
        if (run < PI_T / PAIRS) {
            int a[5], b[5];
#pragma unroll
            for (int k = -4; k < RUN; k++) {
                if (r0 + k >= P0_R)
                    break;
                const uint32_t q = *reinterpret_cast<const uint32_t *>(&S.n[r0 + k + 4][c]);
                a[(k + 5) % 5] = (int)(q & 0x7fffu);
                b[(k + 5) % 5] = (int)((q >> 16) & 0x7fffu);
                if (k >= 0) /* rows r .. r + 4 sit from (k + 1) % 5 on */
                    *reinterpret_cast<int2 *>(&S.v0[r0 + k][c]) =
                        make_int2(tap5(a[(k + 1) % 5], a[(k + 2) % 5], a[(k + 3) % 5], a[(k + 4) % 5], a[k % 5]),
                                  tap5(b[(k + 1) % 5], b[(k + 2) % 5], b[(k + 3) % 5], b[(k + 4) % 5], b[k % 5]));
            }
        }
        __syncthreads();
        /* level 0's column c (frame column X0 - 14 + c) centres on vertical sum c + 2 */
        for (int i = tid; i < P0_R * P0_P / 4; i += PI_T) {
            const int r = i / (P0_P / 4), c = 4 * (i - r * (P0_P / 4));
            const int4 u = *reinterpret_cast<const int4 *>(&S.v0[r][c]), v = *reinterpret_cast<const int4 *>(&S.v0[r][c + 4]);
            const int o0 = (tap5(u.x, u.y, u.z, u.w, v.x) + 128) >> 8, o1 = (tap5(u.y, u.z, u.w, v.x, v.y) + 128) >> 8,
                      o2 = (tap5(u.z, u.w, v.x, v.y, v.z) + 128) >> 8, o3 = (tap5(u.w, v.x, v.y, v.z, v.w) + 128) >> 8;
            *reinterpret_cast<uint2 *>(&S.l0[r][c]) = make_uint2((uint32_t)o0 | (uint32_t)o1 << 16, (uint32_t)o2 | (uint32_t)o3 << 16);
        }
        __syncthreads();
    }
    /* level 0's block: its local rows and columns 14 .., two columns a thread */
    for (int i = tid; i < FP_Y * (FP_X / 2); i += PI_T) {
        const int r = i / (FP_X / 2), c = 2 * (i - r * (FP_X / 2));
        const int gy = Y0 + r, gx = X0 + c;
        if (EDGE && (gy >= h || gx >= w))
            continue;
        const uint32_t q = GAUSS ? *reinterpret_cast<const uint32_t *>(&S.l0[r + 14][c + 14])
                                 : *reinterpret_cast<const uint32_t *>(&S.n[r + 16][c + 16]);
        auto value = [](uint32_t u) { return __int_as_float(__float_as_int(small_int_to_float((int)(u & 0x7fffu))) | (int)((u >> 15 & 1u) << 31)); };
        float *d = f.lv[0] + (size_t)gy * f.pitch[0] + gx;
        if (!EDGE || gx + 2 <= w)
            *reinterpret_cast<float2 *>(d) = make_float2(value(q & 0xffffu), value(q >> 16));
        else
            *d = value(q & 0xffffu);
    }
    if (f.levels < 2)
        return;
    /* level 1: its local origin is X0 / 2 - 6, Y0 / 2 - 6, level 0's X0 - 14, Y0 - 14 */
    /* (v1 takes v0's place: nothing of v0 is read after the barrier above) */
    if constexpr (!EDGE) { /* runs of rows again: two new ones an output */
        constexpr int PAIRS = P0_P / 2, RUN = (F1_R + PI_T / PAIRS - 1) / (PI_T / PAIRS);
        const int run = tid / PAIRS, c = 2 * (tid - run * PAIRS), y0 = run * RUN;
        if (run < PI_T / PAIRS) {
            int a[5], b[5];
            auto take = [&](int slot, int r) {
                const uint32_t q = l0_pair(r, c);
                a[slot] = (int)(q & 0xffffu);
                b[slot] = (int)(q >> 16);
            };
#pragma unroll
            for (int t = 0; t < 3; t++)
                take(t, 2 * y0 + t);
#pragma unroll
            for (int k = 0; k < RUN; k++) {
                if (y0 + k >= F1_R)
                    break;
                take((2 * k + 3) % 5, 2 * (y0 + k) + 3);
                take((2 * k + 4) % 5, 2 * (y0 + k) + 4);
                *reinterpret_cast<int2 *>(&S.v1[y0 + k][c]) =
                    make_int2(tap5(a[2 * k % 5], a[(2 * k + 1) % 5], a[(2 * k + 2) % 5], a[(2 * k + 3) % 5], a[(2 * k + 4) % 5]),
                              tap5(b[2 * k % 5], b[(2 * k + 1) % 5], b[(2 * k + 2) % 5], b[(2 * k + 3) % 5], b[(2 * k + 4) % 5]));
            }
        }
    }
    for (int i = tid; EDGE && i < F1_R * (P0_P / 2); i += PI_T) {
        const int y = i / (P0_P / 2), c = 2 * (i - y * (P0_P / 2));
        int a[5], b[5];
#pragma unroll
        for (int t = 0; t < 5; t++) {
            const int r = EDGE ? min(max(2 * (Y0 / 2 - 6 + y) - 2 + t, 0), h - 1) - (Y0 - 14) : 2 * y + t;
            const uint32_t q = l0_pair(EDGE ? min(max(r, 0), P0_R - 1) : r, c);
            a[t] = (int)(q & 0xffffu);
            b[t] = (int)(q >> 16);
        }
        *reinterpret_cast<int2 *>(&S.v1[y][c]) = make_int2(tap5(a[0], a[1], a[2], a[3], a[4]), tap5(b[0], b[1], b[2], b[3], b[4]));
    }
    __syncthreads();
    for (int i = tid; i < F1_R * F1_C; i += PI_T) {
        const int y = i / F1_C, x = i - y * F1_C;
        int a[5];
#pragma unroll
        for (int t = 0; t < 5; t++) {
            const int c = EDGE ? min(max(2 * (X0 / 2 - 6 + x) - 2 + t, 0), w - 1) - (X0 - 14) : 2 * x + t;
            a[t] = S.v1[y][EDGE ? min(max(c, 0), P0_C - 1) : c];
        }
        S.u.l1[y][x] = (uint16_t)((tap5(a[0], a[1], a[2], a[3], a[4]) + 128) >> 8);
    }
    __syncthreads();
    fused_upper<EDGE>(f, X0, Y0, S.u);
}

template <bool GAUSS>
__global__ void __launch_bounds__(PI_T) pyr_input_kernel(FusedFrame f, bool contrast, const uint32_t *mm)
{
    extern __shared__ __align__(16) unsigned char s_input[];
    InputSmem &S = *reinterpret_cast<InputSmem *>(s_input);
    const int tid = threadIdx.x, X0 = blockIdx.x * FP_X, Y0 = blockIdx.y * FP_Y;
    const bool inside = X0 >= 16 && X0 + 144 <= f.w && Y0 >= 16 && Y0 + 73 <= f.h;
    /* the bytes, which were there before the minimum and maximum's launch (an ordinary one) */
    uint32_t q[PI_CHUNKS][4];
    if (inside)
        input_fetch<false>(f, X0, Y0, q);
    else
        input_fetch<true>(f, X0, Y0, q);
    vtg_grid_dependency_wait(); /* the gain and offset, when launched as that launch's dependent */
    if (tid < 256) {
        float v = (float)(64 * tid);
        if (contrast) {
            const float g = __ldcg(reinterpret_cast<const float *>(mm) + VTG_MM_BLOCKS + 1);
            const float o = __ldcg(reinterpret_cast<const float *>(mm) + VTG_MM_BLOCKS + 2);
            /* the reference's x87 form rounds Q6 x gain + offset to F32 from an exact extended sum (the product has 38
             * bits, the sum's lowest bit is at least 2^-23 and its size below 2^23); one fused multiply-add rounds the
             * same exact value once */
            v = rintf(__fmaf_rn(v, g, o));
            /* the reference's select, which keeps the -0 that rint gives a small negative value (the level's bits) */
            v = v < 0.0f ? 0.0f : v > 16320.0f ? 16320.0f : v;
        }
        S.lut[tid] = (uint32_t)fabsf(v) | (__float_as_uint(v) >> 31 << 15);
    }
    __syncthreads();
    if (inside)
        input_block<GAUSS, false>(f, X0, Y0, q, S);
    else
        input_block<GAUSS, true>(f, X0, Y0, q, S);
}

static FusedFrame fused_frame(const uint8_t *frame, int stride, int w, int h, float *const *levels, const int *pitches, int nlevels)
{
    FusedFrame f;
    f.src = frame;
    f.stride = stride;
    f.w = w;
    f.h = h;
    f.levels = nlevels;
    for (int L = 0; L < 4; L++) {
        f.lv[L] = L < nlevels ? levels[L] : nullptr;
        f.pitch[L] = L < nlevels ? pitches[L] : 0;
    }
    return f;
}

cudaError_t vtg_launch_build_input(const uint8_t *frame, int stride, int w, int h, int opts, uint32_t *mm, float *const *levels,
                                   const int *pitches, int nlevels, cudaStream_t s)
{
    const bool contrast = (opts & VTG_BUILD_CONTRAST) != 0, gauss = (opts & VTG_BUILD_PRE_GAUSS) != 0;
    if (contrast)
        pyr_minmax_kernel<<<min(h, VTG_MM_BLOCKS), 256, 0, s>>>(frame, w, h, stride, mm);
    const dim3 grid((w + FP_X - 1) / FP_X, (h + FP_Y - 1) / FP_Y);
    auto kernel = gauss ? pyr_input_kernel<true> : pyr_input_kernel<false>;
    const size_t smem = gauss ? sizeof(InputSmem) : offsetof(InputSmem, v1) + sizeof(InputSmem::v1);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
        e = vtg_launch_k(kernel, grid, dim3(PI_T), smem, s, contrast, fused_frame(frame, stride, w, h, levels, pitches, nlevels),
                         contrast, (const uint32_t *)mm);
    return e;
}

/* Levels 4 on, a launch each, as dependents of the one before. */
static cudaError_t launch_upper_levels(int w, int h, float *const *levels, const int *pitches, int nlevels, cudaStream_t s)
{
    int sw = w, sh = h;
    for (int L = 1; L < nlevels; L++) {
        const int dw = (sw + 1) / 2, dh = (sh + 1) / 2;
        if (L >= 4) {
            const cudaError_t e = vtg_launch_k(pyr_reduce_kernel, dim3((dw + RT_X - 1) / RT_X, (dh + RT_Y - 1) / RT_Y), dim3(256), 0, s,
                                               true, (const float *)levels[L - 1], sw, sh, pitches[L - 1], levels[L], dw, dh,
                                               pitches[L]);
            if (e != cudaSuccess)
                return e;
        }
        sw = dw;
        sh = dh;
    }
    return cudaGetLastError();
}

cudaError_t vtg_launch_pyramid_opts(const uint8_t *frame, int stride, int w, int h, float *const *levels,
                                    const int *pitches, int nlevels, int opts, uint32_t *mm, cudaStream_t s)
{
    if (!(opts & (VTG_BUILD_CONTRAST | VTG_BUILD_PRE_GAUSS)))
        return vtg_launch_pyramid(frame, stride, w, h, levels, pitches, nlevels, s);
    const cudaError_t e = vtg_launch_build_input(frame, stride, w, h, opts, mm, levels, pitches, nlevels, s);
    return e != cudaSuccess ? e : launch_upper_levels(w, h, levels, pitches, nlevels, s);
}

int vtg_pyr_tiles(int w, int h, int level)
{
    /* tiles of the launch that makes `level` (4 and up) of a w x h frame */
    int sw = w, sh = h;
    for (int L = 1; L < level; L++) {
        sw = (sw + 1) / 2;
        sh = (sh + 1) / 2;
    }
    const int dw = (sw + 1) / 2, dh = (sh + 1) / 2;
    return ((dw + RT_X - 1) / RT_X) * ((dh + RT_Y - 1) / RT_Y);
}

cudaError_t vtg_launch_pyramid_batch(const PyrJob *jobs, const int *starts, const int *tiles_total, int njobs,
                                     int max_levels, cudaStream_t s, int *reset, bool pdl)
{
    int last = 3; /* the last level launched */
    for (int L = 4; L < max_levels; L++)
        if (tiles_total[L - 1] > 0)
            last = L;
    /* levels 0 .. 3 of every job in one launch (row VTG_MAX_LEVELS - 1 of the tables), then levels 4 .. */
    cudaError_t e = vtg_launch_k(pyr_fused_batch_kernel, tiles_total[VTG_MAX_LEVELS - 1], 256, 0, s, false, jobs,
                                 (const int *)(starts + (size_t)(VTG_MAX_LEVELS - 1) * (njobs + 1)), njobs,
                                 last < 4 ? reset : (int *)nullptr);
    for (int L = 4; L < max_levels && e == cudaSuccess; L++)
        if (tiles_total[L - 1] > 0)
            e = vtg_launch_k(pyr_batch_kernel, tiles_total[L - 1], 256, 0, s, pdl, jobs, (const int *)(starts + (size_t)(L - 1) * (njobs + 1)),
                             njobs, L, L == last ? reset : (int *)nullptr);
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t vtg_launch_pyramid(const uint8_t *frame, int stride, int w, int h, float *const *levels, const int *pitches,
                               int nlevels, cudaStream_t s)
{
    /* Levels 0 .. 3 from the bytes in one launch, then one launch per further level. */
    pyr_fused_kernel<<<dim3((w + FP_X - 1) / FP_X, (h + FP_Y - 1) / FP_Y), 256, 0, s>>>(
        fused_frame(frame, stride, w, h, levels, pitches, nlevels));
    return launch_upper_levels(w, h, levels, pitches, nlevels, s);
}
