/* ncc_tc.cu -- the correlation map on the 5th-generation tensor cores: tcgen05.mma (kind::f16, BF16 or FP16 products,
 * F32 accumulation in tensor memory), operands brought into shared memory by asynchronous bulk copies and read through
 * matrix descriptors, the accumulator read back with tcgen05.ld, scored with exact int64 window sums and reduced to the
 * per-cell map in the epilogue.
 *
 * The correlation as a GEMM. A CTA owns a tile of corners: 1024 consecutive x (X0 + 8 m + s, m < 128, s < 8) by Q
 * consecutive y (Y0 + q, q < Q; Q = 16, or 8 for templates wider than 120). Then
 *     st(X0 + 8 m + s, Y0 + q) = sum over image rows r, columns c of  A_r[m][c] * B_r[(q, s)][c]
 * with A_r[m][c] = J[r][X0 + 8 m + c] and B_r[(q, s)][c] = t[r - Y0 - q][c - s] (zero outside the template): D =
 * sum_r A_r B_r^T with M = 128, N = 8 Q, and K = the tile's Q + T_h - 1 image rows times K_row = T_w + 8 rounded up
 * to 16.
 *   A needs no im2col. Consecutive rows of A_r start 8 elements (16 bytes) apart in the image row, so a K-major,
 *   no-swizzle descriptor with 16-byte core-matrix rows, a 16-byte leading (K) offset and a 128-byte stride (M) offset
 *   reads A_r straight from the row: address(m, k) = row + 2 (8 m + k). The picture is converted to 16 bits once per
 *   search (ncc_prep), shifted so that every tile's row segment starts on a 16-byte boundary.
 *   B_r depends only on r - Y0: the band (Q + T_h - 1 blocks of 8 Q x K_row) is built once per template in the canonical
 *   core-matrix layout.
 * Pipeline: three threads drive it. Six shared-memory stages (five when the CTA makes its factors too), each an image-row segment and a band
 * block, arrive by cp.async.bulk on a "full" mbarrier (expected bytes). A producer thread (warp 0) fills a stage again as soon as the
 * MMAs of its last use commit to its "empty" mbarrier. Two issuer threads (warps 1 and 2) take alternate stages, each
 * into its own accumulator: issuing a stage's MMAs takes a lone thread longer than the tensor core takes to run them,
 * so one issuer would leave it idle. Every wait is bounded by the global timer; past it the kernel records an error
 * word.
 * Factors: each corner's 1 / sqrt(norm var) from exact integer window sums, by ncc_prep or, where the tensor core is busy for
 * longer than that takes, by twelve more warps of the map's CTAs while it multiplies (tc_fused).
 * Epilogue: four warps cover the accumulator's 128 lanes, one row (8 x-corners by Q y-corners) a thread; with more warps
 * each of a lane quarter's reads its share of the row's columns. A thread sums the issuers' accumulators for its
 * row. Per corner: st = acc - J(x, y) sum t' (the reference's st is relative to the corner's first pixel), times the
 * corner's factor (0 for a near-blank window: the exact integer rule), the best
 * per 16 x 16 cell by value then scan order, merged across tiles by a 64-bit atomicMax on (ordered score, inverted scan
 * index). */
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "vtg_ncc.cuh"

#define TC_M 128
#define TC_QMAX 16 /* y-corners of a tile, at most */
#define TC_XS (8 * TC_M) /* x-corners of a tile */
#ifndef TC_ISSUERS
#define TC_ISSUERS 2 /* MMA-issuing threads, each with its own accumulator, taking every TC_ISSUERS-th stage */
#endif
#define TC_WAIT_NS 2000000000ull /* a wait gives up after 2 s of the global timer */
#define TC_MAX_KROW 144          /* T_w <= 128 */

static inline int tc_krow(int tw) { return ((tw + 8 + 15) / 16) * 16; }

/* y-corners of a tile (N = 8 Q). An MMA reads its A (4 KB) and B (16 N bytes) from shared memory at 128 bytes a cycle
 * and multiplies for N / 2 cycles, so below N = 128 the shared-memory reads bound it. Q = 16 while six stages of it fit
 * the shared memory (K_row <= 128), else 8. The band's zero rows (Q - 1 of every Q + th - 1 image rows) cost less than
 * the reads they save. */
#ifndef TC_Q_BIG
#define TC_Q_BIG 16
#endif
static inline int tc_q(int tw, int th)
{
    (void)th;
    return TC_Q_BIG == 16 && tc_krow(tw) > 128 ? 8 : TC_Q_BIG;
}

/* the band at its largest tile height: enough for either */
size_t vtg_ncc_band_bytes(int tw, int th) { return (size_t)(TC_QMAX + th - 1) * 8 * TC_QMAX * tc_krow(tw) * sizeof(uint16_t); }

/* The 16-bit picture: rows up to h + TC_QMAX + T_h (zeros past the picture), TC_XS-aligned tiles plus the last K row. */
static inline int conv_pitch(int w) { return ((w + TC_XS - 1) / TC_XS) * TC_XS + TC_MAX_KROW; }

size_t vtg_ncc_conv_elems(int max_w, int max_h, int max_th) { return (size_t)conv_pitch(max_w) * (size_t)(max_h + TC_QMAX + max_th); }

/* The corners' factors: rows of whole tiles (TC_XS corners), so a tile's factor loads stay inside its row. */
size_t vtg_ncc_fac_elems(int max_w, int max_h) { return (size_t)((max_w + TC_XS - 1) / TC_XS) * TC_XS * (size_t)max_h; }

/* ---- the band ---- */

__device__ __forceinline__ uint16_t to16(float v, int kind)
{
    return kind == VTG_NCC_BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
}

__device__ __forceinline__ float from16(uint16_t v, int kind)
{
    return kind == VTG_NCC_BF16 ? __bfloat162float(__ushort_as_bfloat16(v)) : __half2float(__ushort_as_half(v));
}

/* Band block k (image row Y0 + k of a tile), element (n = 8 q + s, c) at core matrix (c / 8, n / 8), row n % 8, column
 * c % 8: core matrices of 8 x 8 elements (128 bytes), K-chunks of 8 columns N / 8 matrices apart. */
__global__ void ncc_band_kernel(const float *__restrict__ app, int tw, int th, int kind, int krow, int rows, int nq,
                                uint16_t *__restrict__ band)
{
    const int N = 8 * nq;
    const size_t per = (size_t)N * krow;
    const size_t total = per * rows;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(idx / per);
        const int rem = (int)(idx - (size_t)k * per);
        const int n = rem / krow, c = rem - n * krow;
        const int q = n >> 3, s = n & 7;
        const int i = k - q, j = c - s;
        const float v = (i >= 0 && i < th && j >= 0 && j < tw) ? app[i * tw + j] : 0.0f;
        const size_t off = (size_t)k * per + ((size_t)(c >> 3) * (N / 8) + (n >> 3)) * 64 + (n & 7) * 8 + (c & 7);
        band[off] = to16(v, kind);
    }
}

/* What the band's rounding keeps and loses of the template, in double: h the 16-bit value, d = t - h (exact: a 16-bit
 * and an F32 value's difference). */
__global__ void ncc_band_sum(const float *__restrict__ app, int count, int kind, NccBandStats *__restrict__ out)
{
    __shared__ double s[4][256];
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
        const float t = app[i];
        const double h = (double)from16(to16(t, kind), kind), d = (double)t - h;
        a[0] += h;
        a[1] += d;
        a[2] += d * d;
        a[3] += (double)t * (double)t;
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
        s[k][threadIdx.x] = a[k];
    __syncthreads();
    for (int h = 128; h >= 1; h >>= 1) {
        if (threadIdx.x < h)
#pragma unroll
            for (int k = 0; k < 4; k++)
                s[k][threadIdx.x] += s[k][threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        *out = NccBandStats{(float)s[0][0], (float)s[1][0], (float)s[2][0], (float)s[3][0]};
}

cudaError_t vtg_launch_ncc_band(const float *app, int tw, int th, int kind, uint16_t *band, NccBandStats *stats,
                                cudaStream_t st)
{
    const int q = tc_q(tw, th), krow = tc_krow(tw), rows = q + th - 1;
    const size_t total = (size_t)8 * q * krow * rows;
    const int blocks = (int)((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
    ncc_band_kernel<<<blocks, 256, 0, st>>>(app, tw, th, kind, krow, rows, q, band);
    ncc_band_sum<<<1, 256, 0, st>>>(app, tw * th, kind, stats);
    return cudaGetLastError();
}

/* How far a corner's FP16 tensor-core score may lie from its F32 score (ncc_map_f32q's chains), on a byte picture. With v =
 * sum (J - mean)^2 over the window, a score is a sum over sqrt(norm v); f is the window's first pixel, sigma = sqrt(v / n),
 * d = t - h the template's FP16 rounding. By Cauchy-Schwarz, for any constant c,
 *     sum |t (J - c)| <= |t| sqrt(v + n (mean - c)^2) <= |t| sqrt(v) (1 + |mean - c| / sigma),
 * so errors relative to such a sum become, in the score, that many units of |t| / sqrt(norm) times the bracket:
 *   - the rounding: sum d (J - f) = sum (d - mean d)(J - mean) + sum d (mean - f), at most |d - mean d| / sqrt(norm) and
 *     |sum d| / sqrt(n norm) |mean - f| / sigma;
 *   - the tensor core's accumulation of t (J - 128) (the picture is converted less 128): each MMA of 16 products taken as
 *     rounded to 2^-21 of the sum of magnitudes, over the steps of one issuer. No public document states an MMA's rounding, so
 *     this part is an assumption, measured: with templates that FP16 holds exactly, where nothing but the accumulation and the
 *     chains is left, no corner was further off than 0.047 of the bound (128 x 128, random bytes; 0.039 at 64 x 64 over black and
 *     white noise), over scenes, noise, ramps, stripes, edges, dark, dim and bright pictures at 64 x 64 to 128 x 128 and 32 x 128;
 *     with the rounding's part, which is proven, no corner further than 0.53, of 10.9 million;
 *   - the F32 chains of t (J - f): n / 2 additions each, rounded to 2^-24;
 *   - the scores' own last operations: a few units in the last place of 1.
 * flt_a = -1 where FP16 does not hold the template (d infinite, or more than a hundredth of t). */
void vtg_ncc_filter_bound(NccPrm &p, const NccBandStats &b)
{
    const double n = p.n, sd = fabs((double)b.sum_d), norm = (double)p.norm;
    const double steps = ((p.th + TC_QMAX) / TC_ISSUERS + 2) * (double)(tc_krow(p.tw) / 16) + 16.0;
    const double spread = (double)b.sum_dd * 1.001 - sd * sd * 0.999 / n;
    const double t = sqrt((double)b.sum_tt / norm); /* 1 for a caller's true norm */
    const double core = t * steps * 0x1p-21, chain = t * (n * 0.5 + 16.0) * 0x1p-24;
    const double a = sqrt((spread <= 0.0 ? 0.0 : spread) / norm) + core + chain + 4e-6; /* NaN stays: a value past FP16's */
    const bool good = norm > 0.0 && a <= 0.01; /* false for NaN */
    p.flt_a = good ? (float)(a * 1.02) : -1.0f;
    p.flt_m = good ? (float)(core * 1.02) : 0.0f;
    p.flt_f = good ? (float)((chain + sd / sqrt(n * norm)) * 1.02) : 0.0f;
}

/* ---- per-search preparation ---- */

/* A word's four bytes less `centre`, as 16-bit values in two words. */
template <int KIND>
__device__ __forceinline__ uint2 conv4(uint32_t w, float centre)
{
    if (KIND == VTG_NCC_FP16) { /* 0x6400 | b is 1024 + b */
        const __half2 off = __float2half2_rn(1024.0f + centre);
        const uint32_t a = __byte_perm(w, 0x64646464u, 0x4140u), b = __byte_perm(w, 0x64646464u, 0x4342u);
        const __half2 x = __hsub2(*reinterpret_cast<const __half2 *>(&a), off), y = __hsub2(*reinterpret_cast<const __half2 *>(&b), off);
        return make_uint2(*reinterpret_cast<const uint32_t *>(&x), *reinterpret_cast<const uint32_t *>(&y));
    }
    /* bytes are BF16 values: the upper half of the F32, from 2^23 + b */
    const float off = 8388608.0f + centre;
    uint32_t f[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
        f[k] = __float_as_uint(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + k)) - off);
    return make_uint2(__byte_perm(f[0], f[1], 0x7632u), __byte_perm(f[2], f[3], 0x7632u));
}

/* conv[r][i] = 16-bit J[r][x0 + i] - centre (minus the centre past the picture), for rows 0 .. rows - 1 and columns 0 .. cpitch - 1:
 * the CTA (bx, by) of 256 threads converts row by, eight elements a thread and one 16-byte store (cpitch is a multiple of 8
 * and rows start 16-byte aligned: 2 cpitch = 2048 tiles_x + 288 bytes). Inside the row the bytes come as three aligned words,
 * shifted: the first starts up to three bytes before, the third ends up to twelve after. */
template <int KIND>
__device__ __forceinline__ void conv_cta(const uint8_t *__restrict__ plane, int pitch, int w, int h, int x0, int rows,
                                         int cpitch, float centre, uint16_t *__restrict__ conv, int bx, int by)
{
    const int r = by, i0 = 8 * (bx * 256 + (int)threadIdx.x);
    if (r >= rows || i0 >= cpitch)
        return;
    uint32_t v[2] = {0u, 0u};
    const int x = x0 + i0;
    const uint8_t *src = plane + (size_t)r * pitch + x;
    const bool whole = r < h && x >= 3 && x + 12 <= w;
    if (whole) {
        const uint32_t *q = reinterpret_cast<const uint32_t *>((uintptr_t)src & ~(uintptr_t)3);
        const int sh = 8 * (int)((uintptr_t)src & 3);
        const uint32_t q0 = __ldg(q), q1 = __ldg(q + 1), q2 = __ldg(q + 2);
        v[0] = __funnelshift_r(q0, q1, sh);
        v[1] = __funnelshift_r(q1, q2, sh);
    } else if (r < h) {
#pragma unroll
        for (int e = 0; e < 8; e++)
            if (x + e < w)
                v[e >> 2] |= (uint32_t)__ldg(src + e) << (8 * (e & 3));
    }
    const uint2 a = conv4<KIND>(v[0], centre), b = conv4<KIND>(v[1], centre);
    *reinterpret_cast<uint4 *>(conv + (size_t)r * cpitch + i0) = make_uint4(a.x, a.y, b.x, b.y);
}

/* fac[(y - y0) fpitch + (x - x0)] = 1 / sqrt(norm var) from the corner's exact window sums; 0 for a near-blank window
 * (n var <= n norm / 16) or norm <= 0 -- the reference's rule (src/kern/track.c:203-205) on exact integers.
 * The sums come straight from the bytes, nx x ny corners (nx + T_w - 1 <= NT, ny <= TY) by NT threads, tid their number: a CTA of
 * the preparation, or the warps of a map's CTA that do not drive its tensor core (tc_fused).
 *   - a thread a column, down its column: running sums over the template's T_h rows for the corner rows, into shared memory;
 *   - a thread NT / 16 columns of a row: its prefix sums, the row's 16 threads' totals scanned by shuffles;
 *   - a corner's window sums are then P(x + T_w) - P(x), four consecutive corners a thread by 16-byte reads.
 * Bytes keep every window sum in 32 bits (sum J^2 <= 255^2 x 128^2 < 2^31). A row's prefix of J^2 may pass 2^32, so
 * the prefixes are unsigned and wrap: their differences are still exact. n var is formed in 64 bits. The preparation's CTAs are
 * bound by issue and by their loads' latency: 16 us over a 1080p frame at 64 x 64; a shuffle scan of every row by every warp,
 * and a corner a thread, took 13M instructions where this takes 8M, and 23 us. */
#define BOX_NT 256 /* threads of a preparation's CTA */
/* corners of such a CTA across: the most, a multiple of 32, whose columns (+ T_w - 1) fit its threads */
static inline int bp_tx(int tw) { return ((BOX_NT + 1 - tw) / 32) * 32; }

template <int NT>
struct BoxSmem {
    __align__(16) unsigned p[2][TC_QMAX][NT + 4]; /* P[r][c]: columns 0 .. c - 1 of row r; of J and of J^2 */
};

/* a barrier of the NT threads (the CTA's own is 0) */
template <int NT>
__device__ __forceinline__ void box_sync()
{
    asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
}

template <int NT, int TY, bool TOL>
__device__ void box_sums(const uint8_t *__restrict__ plane, int pitch, const NccPrm &p, int fpitch, float *__restrict__ fac,
                                         uint16_t *__restrict__ tol, int tx0, int ty0, int nx, int ny, int tid, BoxSmem<NT> &S)
{
    constexpr int SEG = NT / 16;
    const int ncol = nx + p.tw - 1;
    {
        /* column tid's sums (0 past the tile's columns); every load of the sliding part in flight, before the first window's
         * rows are added */
        const bool in = tid < ncol;
        const uint8_t *col = plane + (size_t)(p.y0 + ty0) * pitch + (p.x0 + tx0 + min(tid, ncol - 1));
        unsigned leave[TY], enter[TY];
#pragma unroll
        for (int r = 1; r < TY; r++) {
            const int k = min(r, ny - 1) - (ny > 1 ? 1 : 0);
            leave[r] = __ldg(col + (size_t)k * pitch);
            enter[r] = __ldg(col + (size_t)(k + p.th) * pitch);
        }
        unsigned sa = 0, sb = 0;
#pragma unroll 16
        for (int i = 0; i < p.th; i++) {
            const unsigned v = __ldg(col + (size_t)i * pitch);
            sa += v;
            sb += v * v;
        }
        S.p[0][0][tid] = in ? sa : 0u;
        S.p[1][0][tid] = in ? sb : 0u;
#pragma unroll
        for (int r = 1; r < TY; r++) {
            sa += enter[r] - leave[r];
            sb += enter[r] * enter[r] - leave[r] * leave[r];
            S.p[0][r][tid] = in ? sa : 0u;
            S.p[1][r][tid] = in ? sb : 0u;
        }
    }
    box_sync<NT>();
    /* row tid / 16, columns SEG (tid % 16) ..: read, scanned, and written one place on (a row lies in one half of a warp) */
    const int row = tid >> 4, seg = tid & 15;
    if (row < TY) {
#pragma unroll
        for (int t = 0; t < 2; t++) {
            unsigned v[SEG];
            uint4 *const at = reinterpret_cast<uint4 *>(&S.p[t][row][SEG * seg]);
#pragma unroll
            for (int k = 0; k < SEG / 4; k++)
                *reinterpret_cast<uint4 *>(&v[4 * k]) = at[k];
#pragma unroll
            for (int k = 1; k < SEG; k++)
                v[k] += v[k - 1];
            unsigned before = v[SEG - 1];
#pragma unroll
            for (int d = 1; d < 16; d <<= 1) {
                const unsigned u = __shfl_up_sync(VTG_FULL, before, d, 16);
                before += seg >= d ? u : 0u;
            }
            before -= v[SEG - 1];
            __syncwarp();
            /* P[SEG seg] = before, P[SEG seg + 1 ..] = before + v[0] ..: the SEG places from there on, and NT */
#pragma unroll
            for (int k = 0; k < SEG / 4; k++)
                at[k] = make_uint4(k ? before + v[4 * k - 1] : before, before + v[4 * k], before + v[4 * k + 1], before + v[4 * k + 2]);
            if (seg == 15)
                S.p[t][row][NT] = before + v[SEG - 1];
        }
    }
    box_sync<NT>();
    /* four corners a thread of a row (tw is a multiple of 8: both ends 16-byte aligned); fac's rows hold whole tiles, so a
     * group's store stays inside, past the window's last corner too */
    const int groups = (nx + 3) / 4;
    for (int i = tid; i < ny * groups; i += NT) {
        const int r = i / groups, x = 4 * (i - r * groups);
        const uint4 l1 = *reinterpret_cast<const uint4 *>(&S.p[0][r][x]), h1 = *reinterpret_cast<const uint4 *>(&S.p[0][r][x + p.tw]);
        const uint4 l2 = *reinterpret_cast<const uint4 *>(&S.p[1][r][x]), h2 = *reinterpret_cast<const uint4 *>(&S.p[1][r][x + p.tw]);
        const unsigned w1[4] = {h1.x - l1.x, h1.y - l1.y, h1.z - l1.z, h1.w - l1.w};
        const unsigned w2[4] = {h2.x - l2.x, h2.y - l2.y, h2.z - l2.z, h2.w - l2.w};
        float f[4];
        uint32_t e[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const long long nvar = (long long)p.n * (long long)w2[k] - (long long)w1[k] * (long long)w1[k];
            /* 1 / sqrt(norm var) = sqrt(n / norm) / sqrt(n var) */
            const float rs = rsqrtf((float)nvar);
            f[k] = (nvar <= p.nthr || p.norm <= 0.0f) ? 0.0f : p.rnorm * rs;
            if constexpr (TOL) { /* |mean - c| / sigma = |sum J - n c| / sqrt(n var); rounded up */
                const int j = x + k < nx ? __ldg(plane + (size_t)(p.y0 + ty0 + r) * pitch + (p.x0 + tx0 + x + k)) : 0;
                const float zm = fabsf((float)((int)w1[k] - 128 * p.n)) * rs, zf = fabsf((float)((int)w1[k] - j * p.n)) * rs;
                e[k] = __half_as_ushort(__float2half_ru(p.flt_a + p.flt_m * zm + p.flt_f * zf));
            }
        }
        const size_t at = (size_t)(ty0 + r) * fpitch + tx0 + x;
        *reinterpret_cast<float4 *>(fac + at) = make_float4(f[0], f[1], f[2], f[3]);
        if constexpr (TOL)
            *reinterpret_cast<uint2 *>(tol + at) = make_uint2(e[0] | e[1] << 16, e[2] | e[3] << 16);
    }
}

/* The map's preparation in one launch of 256-thread CTAs: the picture converted, and the cells' words that the map merges into
 * and the status word zeroed. BOX: the first nbox sum the windows (the longer work, so they start first), where the map's CTAs do not. */
template <int KIND, bool FILTER, bool BOX>
__global__ void __launch_bounds__(BOX_NT) ncc_prep(const uint8_t *__restrict__ plane, int pitch, NccPrm p, int fw, int fpitch,
                                                int btx, int bgx, int nbox, float *__restrict__ fac,
                                                uint16_t *__restrict__ tol, int rows, int cpitch, int cgx, uint16_t *__restrict__ conv,
                                                unsigned long long *__restrict__ cellw, int cells, unsigned *__restrict__ ncand,
                                                int *__restrict__ err)
{
    vtg_grid_launch_dependents(); /* the map may start its setup as this launch's last CTAs run */
    const int b = (int)blockIdx.x;
    if constexpr (BOX) {
        __shared__ BoxSmem<BOX_NT> S;
        if (b < nbox) {
            const int x = b % bgx * btx, y = b / bgx * TC_QMAX;
            box_sums<BOX_NT, TC_QMAX, FILTER>(plane, pitch, p, fpitch, fac, tol, x, y, min(btx, fw - x),
                                              min(TC_QMAX, p.y1 - p.y0 + 1 - y), (int)threadIdx.x, S);
            return;
        }
    }
    const int k = b - nbox, g = k * 256 + (int)threadIdx.x;
    if (g < cells)
        cellw[g] = 0ull;
    if (g == 0)
        *err = 0; /* the map's, for this search */
    if (FILTER && g == 0)
        *ncand = 0u;
    conv_cta<KIND>(plane, pitch, p.w, p.h, p.x0, rows, cpitch, FILTER ? 128.0f : 0.0f, conv, k % cgx, k / cgx);
}

/* ---- PTX helpers ---- */

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

/* A tcgen05 shared-memory matrix descriptor, no swizzle: start, leading (K) and stride (M/N) byte offsets, all in
 * 16-byte units, and the fixed version bits 46-48 = 0b001. */
__device__ __forceinline__ uint64_t mdesc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}

__device__ __forceinline__ uint64_t globaltimer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

/* Bounded wait on an mbarrier phase: true when the phase with this parity completed, false after TC_WAIT_NS. */
__device__ __forceinline__ bool mbar_wait(uint32_t a, uint32_t parity)
{
    const uint64_t t0 = globaltimer();
    for (;;) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(a), "r"(parity), "r"(100000u)
                     : "memory");
        if (done)
            return true;
        if (globaltimer() - t0 > TC_WAIT_NS)
            return false;
    }
}

/* Arms a stage's full barrier for `bytes` and brings its two operands in by bulk copy. */
__device__ __forceinline__ void tc_fill(uint32_t mbar, uint32_t dst_a, const void *src_a, uint32_t bytes_a, uint32_t dst_b,
                                        const void *src_b, uint32_t bytes_b)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes_a + bytes_b) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_a),
                 "l"(src_a), "r"(bytes_a), "r"(mbar)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_b),
                 "l"(src_b), "r"(bytes_b), "r"(mbar)
                 : "memory");
}

__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(
                     tmem_d),
                 "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
                 : "memory");
}

__device__ __forceinline__ void tc_commit(uint32_t mbar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

/* 16 consecutive accumulator columns of the thread's row (lane = row within the warp's 32), not yet waited for */
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
                 "%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}

/* ---- the map ---- */

/* Tensor-memory columns a CTA allocates: the issuers' accumulators (8 Q columns each), rounded up to a power of two
 * of at least 32 as tcgen05.alloc requires. */
__host__ __device__ constexpr uint32_t tc_cols(int q)
{
    return 8u * q * TC_ISSUERS <= 32u ? 32u : 8u * q * TC_ISSUERS <= 64u ? 64u : 8u * q * TC_ISSUERS <= 128u ? 128u
           : 8u * q * TC_ISSUERS <= 256u ? 256u : 512u;
}
static_assert(8 * TC_QMAX * TC_ISSUERS <= 512, "the accumulators fit the tensor memory");
static_assert(TC_ISSUERS >= 1 && TC_ISSUERS <= 3, "issuers are warps 1 .. 3 of the CTA's four");

/* A CTA of the map. Four warps cover the accumulator's 128 lanes. Not FUSED: at Q = 16 eight warps, two to a lane quarter, each
 * reading half the columns. FUSED: sixteen, four to a quarter; while the tensor core multiplies, warps 4 to 15 make the tile's
 * factors (box_sums), 256 corners a round, with a stage fewer to leave them the shared memory. shares: warps to a quarter;
 * chunks: 16-column blocks a thread reads. */
#define TC_BOX_WARP 4
#define TC_BOX_X 256
template <int Q, bool FUSED> struct TcShape {
    static constexpr int threads = FUSED ? 512 : Q == 16 ? 256 : 128;
    static constexpr int shares = threads / 128;
    static constexpr int chunks = Q / 2 / shares;
    static constexpr int stages = FUSED ? 5 : 6;
    static constexpr int boxes = threads - 32 * TC_BOX_WARP; /* FUSED: the threads that make factors */
};

struct TcSmem {
    uint32_t a_bytes, b_bytes, stage_bytes, total;
};

static TcSmem tc_smem(int krow, int q, bool fused)
{
    TcSmem s;
    s.a_bytes = (uint32_t)(((TC_XS + krow) * 2 + 127) & ~127);
    s.b_bytes = (uint32_t)(8 * q * krow * 2);
    s.stage_bytes = s.a_bytes + s.b_bytes;
    /* + mbarriers and the tensor-memory address */
    s.total = (fused ? TcShape<16, true>::stages : TcShape<16, false>::stages) * s.stage_bytes + 256;
    if (fused)
        s.total += (uint32_t)sizeof(BoxSmem<TcShape<16, true>::boxes>);
    return s;
}

/* The checked build's failure: while on, the map's first CTA ends as if one of its waits had given up (all have ended by then).
 * Returns 1 there, 0 in the production build, which has no such word. */
#ifdef VTG_CHECKED
__device__ int g_vtg_give_up;
#endif
extern "C" int vtg_check_give_up(int on)
{
#ifdef VTG_CHECKED
    return cudaMemcpyToSymbol(g_vtg_give_up, &on, sizeof on) == cudaSuccess ? 1 : VTG_ECUDA;
#else
    (void)on;
    return 0;
#endif
}

/* FILTER: the F32 map's first half. Instead of a cell's best, the corners whose score may be it in F32 arithmetic go to
 * cand: a corner's F32 score lies within its tol of its score here (vtg_ncc_filter_bound), so only corners with score + tol
 * >= max over the cell's corners here of (score - tol) can be the cell's best or tie with it. (Of a cell over two tiles, Q
 * = 8, each tile's part is taken by itself, which can only keep more.) On the blurred-noise frames 1.0 to 1.3 corners a cell
 * are left of 256, at 64 x 64 (29 us for this map, where the F32 map took 728). A near-blank window scores exactly 0 either way: the
 * earliest of them goes straight to the cell's word. */
template <int KIND, int Q, bool FILTER, bool FUSED>
__global__ void __launch_bounds__(TcShape<Q, FUSED>::threads, 1) ncc_map_tc(NccPrm p, const uint8_t *__restrict__ plane, int pitch,
                                                     const uint16_t *__restrict__ band, int krow, int tiles_x,
                                                     uint32_t a_bytes, uint32_t stage_bytes,
                                                     const uint16_t *__restrict__ conv, int cpitch,
                                                     float *fac, int fpitch,
                                                     unsigned long long *__restrict__ cellw, int *__restrict__ err,
                                                     uint16_t *tol, unsigned *__restrict__ cand, unsigned *__restrict__ ncand)
{
    using Shape = TcShape<Q, FUSED>;
    constexpr int TC_STAGES = Shape::stages;
    extern __shared__ __align__(1024) uint8_t smem[];
    if (!FILTER)
        vtg_grid_launch_dependents(); /* the top-8 pass may take the SMs this launch leaves free and wait there */
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tx = blockIdx.x % tiles_x, ty = blockIdx.x / tiles_x;
    const int Y0 = p.y0 + ty * Q;
    const int nk = Q + p.th - 1;
    const int kchunks = krow / 16;
    uint8_t *ctl = smem + TC_STAGES * stage_bytes;
    const uint32_t full0 = smem_u32(ctl), empty0 = full0 + 8 * TC_STAGES;
    uint32_t *tmem_slot = (uint32_t *)(ctl + 16 * TC_STAGES);
    /* [0]: stages filled; [1 + i]: 1 + the last stage issuer i committed (0: none) */
    int *issued = (int *)(ctl + 16 * TC_STAGES + 8);
    const uint32_t a_copy = (uint32_t)((TC_XS + krow) * 2), b_copy = (uint32_t)((8 * Q) * krow * 2);

    if (tid == 0) {
        for (int s = 0; s < TC_STAGES; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(tc_cols(Q))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const int fh = p.y1 - p.y0 + 1;
    if constexpr (FUSED) {
        if (warp >= TC_BOX_WARP) {
            /* The tile's factors. They need not wait for the preparation: the picture was there before that started (an ordinary
             * launch), and whatever read the last search's factors was done. */
            const int nx = min(TC_XS, p.x1 - p.x0 + 1 - tx * TC_XS);
            BoxSmem<Shape::boxes> &S = *reinterpret_cast<BoxSmem<Shape::boxes> *>(ctl + 256);
            for (int x = 0; x < nx; x += TC_BOX_X) {
                if (x)
                    box_sync<Shape::boxes>(); /* the last round's sums are read */
                box_sums<Shape::boxes, Q, FILTER>(plane, pitch, p, fpitch, fac, tol, tx * TC_XS + x, ty * Q, min(TC_BOX_X, nx - x),
                                                  min(Q, fh - ty * Q), tid - 32 * TC_BOX_WARP, S);
            }
        }
    }
    /* Launched as a programmatic dependent of the preparation, the CTA got here (barriers, tensor memory) while that
     * drained; everything below reads what it wrote (the 16-bit rows, the factors, the cells' reset), with ordinary
     * coherent loads: that data was not read-only while this kernel ran. */
    vtg_grid_dependency_wait();

    /* The epilogue's inputs: before the MMAs start, so that they arrive while those run, or FUSED after them. Thread
     * (quad, lane) owns accumulator row m = 32 quad + lane, corners X0 + 8 m + s, and of its y-corners its share's 2 chunks.
     * A y-corner's eight picture values (the converted row holds the bytes exactly) and eight factors are one 16-byte and two
     * 16-byte loads. */
    constexpr int CH = Shape::chunks;
    const int m = (warp & 3) * 32 + lane, c0 = (warp >> 2) * CH;
    const int xr = tx * TC_XS + 8 * m; /* x - x0 of the thread's first corner */
    uint4 jr[2 * CH];
    float4 fr[4 * CH];
    uint4 er[FILTER ? 2 * CH : 1];
    auto inputs = [&]() {
#pragma unroll
        for (int i = 0; i < 2 * CH; i++) {
            const int yr = ty * Q + 2 * c0 + i;
            if (yr < fh) {
                const float4 *f = reinterpret_cast<const float4 *>(fac + (size_t)yr * fpitch + xr);
                jr[i] = __ldca(reinterpret_cast<const uint4 *>(conv + (size_t)(p.y0 + yr) * cpitch + xr));
                fr[2 * i] = f[0];
                fr[2 * i + 1] = f[1];
                if constexpr (FILTER)
                    er[i] = *reinterpret_cast<const uint4 *>(tol + (size_t)yr * fpitch + xr);
            } else {
                if constexpr (FILTER)
                    er[i] = make_uint4(0u, 0u, 0u, 0u);
                jr[i] = make_uint4(0u, 0u, 0u, 0u);
                fr[2 * i] = fr[2 * i + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        }
    };
    if constexpr (!FUSED)
        inputs();

    const int fmt = KIND == VTG_NCC_BF16 ? 1 : 0;
    const uint32_t idesc = (1u << 4) | ((uint32_t)fmt << 7) | ((uint32_t)fmt << 10) | ((uint32_t)((8 * Q) >> 3) << 17) |
                           ((uint32_t)(TC_M >> 4) << 24);
    int good = 1;
    /* conv row r holds picture row r from column p.x0 on: this tile's segment starts at column tx * TC_XS */
    const uint16_t *arow = conv + (size_t)Y0 * cpitch + (size_t)tx * TC_XS;
    if (warp == 0 && lane == 0) {
        /* the producer: stage k % TC_STAGES is filled with image row Y0 + k and band block k once the MMAs of its
         * previous use have completed (the commit to its empty barrier) */
        int k = 0;
        for (; k < nk; k++) {
            const int s = k % TC_STAGES;
            if (k >= TC_STAGES && !mbar_wait(empty0 + 8 * s, (uint32_t)((k / TC_STAGES - 1) & 1))) {
                good = 0;
                break;
            }
            uint8_t *sa = smem + s * stage_bytes;
            tc_fill(full0 + 8 * s, smem_u32(sa), arow + (size_t)k * cpitch, a_copy, smem_u32(sa + a_bytes),
                    band + (size_t)k * (8 * Q) * krow, b_copy);
        }
        issued[0] = k;
    } else if (warp >= 1 && warp <= TC_ISSUERS && lane == 0) {
        /* the MMA issuers: issuer i takes stages i, i + TC_ISSUERS, ... into its own accumulator (8 Q columns at
         * 8 Q i), each stage's MMAs as soon as its copies have landed; a commit frees the stage for the producer. A
         * lone thread spends most of a stage issuing its MMAs, so several threads shorten the tile's chain. */
        const int ia = warp - 1;
        const uint32_t acc = tmem + (uint32_t)(8 * Q * ia);
        int last = -1;
        for (int k = ia; k < nk; k += TC_ISSUERS) {
            const int s = k % TC_STAGES;
            if (!mbar_wait(full0 + 8 * s, (uint32_t)((k / TC_STAGES) & 1))) {
                good = 0;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            /* K chunk kc starts 32 bytes further into the row and 2 Q core matrices further into the band block: the
             * descriptors' start fields (16-byte units, no carry below 256 KB) step by 2 and by 16 Q */
            const uint32_t a0 = smem_u32(smem + s * stage_bytes), b0 = a0 + a_bytes;
            const uint64_t ad = mdesc(a0, 16, 128), bd = mdesc(b0, Q * 128, 128);
            for (int kc = 0; kc < kchunks; kc++)
                tc_mma(acc, ad + 2u * kc, bd + (uint64_t)(16 * Q) * kc, idesc, (k != ia || kc != 0) ? 1u : 0u);
            tc_commit(empty0 + 8 * s);
            last = k;
        }
        issued[1 + ia] = last + 1;
        /* an issuer's last commit covers every MMA it issued */
        if (good && last >= 0)
            good = mbar_wait(empty0 + 8 * (last % TC_STAGES), (uint32_t)((last / TC_STAGES) & 1)) ? 1 : 0;
    }
#ifdef VTG_CHECKED
    if (g_vtg_give_up && blockIdx.x == 0)
        good = 0;
#endif
    const int ok_all = __syncthreads_and(good);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!ok_all) {
        /* A wait gave up. Before the CTA frees its tensor memory and exits, what it started must be done: the MMAs of
         * every committed stage (the last commit tracks them all) and the bulk copies of every stage filled but not
         * consumed (each completes its full barrier's phase), else they would still write into tensor and shared
         * memory that the next CTA on this SM may own. These waits are bounded too; past them the engines themselves
         * have stopped and the context cannot be saved from here. */
        if (tid == 0) {
            atomicExch(err, 1);
            const int kp = issued[0];
            for (int i = 0; i < TC_ISSUERS; i++) {
                const int lk = issued[1 + i] - 1;
                if (lk >= 0)
                    mbar_wait(empty0 + 8 * (lk % TC_STAGES), (uint32_t)((lk / TC_STAGES) & 1));
            }
            /* a stage not committed by its issuer was not refilled: its barrier is still in that stage's phase */
            for (int k = 0; k < kp; k++)
                if (k >= issued[1 + k % TC_ISSUERS])
                    mbar_wait(full0 + 8 * (k % TC_STAGES), (uint32_t)((k / TC_STAGES) & 1));
        }
    } else {
        if constexpr (FUSED)
            inputs();
        /* epilogue. The step is a power of two dividing the cell, and X0 - x0 is a multiple of 16, so the corner (x, y)
         * is on the step grid when (8 m + s) and y - y0 are multiples of it. */
        const int sh = __ffs(p.step) - 1;
        const int per = NCC_CELL >> sh;
        const int ly0 = (ty % (NCC_CELL / Q)) * Q; /* this tile's first row inside its cell row */
        uint32_t xmask = 0;
#pragma unroll
        for (int s = 0; s < 8; s++)
            if (xr + s <= p.x1 - p.x0 && ((8 * m + s) & (p.step - 1)) == 0)
                xmask |= 1u << s;
        /* f(its number, q, s, score, factor, bound) over the thread's corners on the step grid */
        auto tol_of = [&](int i, int s) {
            if constexpr (FILTER) {
                const uint32_t ew[4] = {er[i].x, er[i].y, er[i].z, er[i].w};
                return __half2float(__ushort_as_half((uint16_t)(ew[s >> 1] >> (16 * (s & 1)))));
            } else {
                return 0.0f;
            }
        };
        auto corners = [&](auto f) {
#pragma unroll
            for (int cc = 0; cc < CH; cc++) {
                const int c = c0 + cc;
                /* columns 16 c .. 16 c + 15 (y-corners 2 c, 2 c + 1) of every issuer's accumulator, summed in issuer
                 * order */
                float v[16];
                {
                    const uint32_t row = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(16 * c);
                    uint32_t r[TC_ISSUERS][16];
#pragma unroll
                    for (int i = 0; i < TC_ISSUERS; i++)
                        tc_ld16(row + (uint32_t)(8 * Q * i), r[i]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int e = 0; e < 16; e++) {
                        v[e] = __uint_as_float(r[0][e]);
#pragma unroll
                        for (int i = 1; i < TC_ISSUERS; i++)
                            if (i < nk) /* an issuer with no stage left its accumulator unwritten */
                                v[e] += __uint_as_float(r[i][e]);
                    }
                }
#pragma unroll
                for (int qq = 0; qq < 2; qq++) {
                    const int q = 2 * c + qq, yr = ty * Q + q;
                    if (yr >= fh || (yr & (p.step - 1)))
                        continue;
                    const int i = 2 * cc + qq;
                    const uint32_t jw[4] = {jr[i].x, jr[i].y, jr[i].z, jr[i].w};
                    const float fq[8] = {fr[2 * i].x, fr[2 * i].y, fr[2 * i].z, fr[2 * i].w,
                                         fr[2 * i + 1].x, fr[2 * i + 1].y, fr[2 * i + 1].z, fr[2 * i + 1].w};
#pragma unroll
                    for (int s = 0; s < 8; s++) {
                        if (!((xmask >> s) & 1u))
                            continue;
                        const float j0 = from16((uint16_t)(jw[s >> 1] >> (16 * (s & 1))), KIND);
                        /* a near-blank window's factor is 0: + 0 makes its score +0 whatever the sign of the sum, the
                         * reference's 0 (a -0 would order below the other cells' +0 in the top-8 keys) */
                        f(8 * (2 * cc + qq) + s, q, s, (v[8 * qq + s] - j0 * p.sum_t) * fq[s] + 0.0f, fq[s], tol_of(i, s));
                    }
                }
            }
        };
        auto key_of = [&](int q, int s) { return ((ly0 + q) >> sh) * per + ((8 * (m & 1) + s) >> sh); };
        const int ccol = tx * (TC_XS / NCC_CELL) + (m >> 1), crow = (Y0 - p.y0) / NCC_CELL;
        const bool mine = ccol < p.ccols && crow < p.crows;
        if constexpr (FILTER) {
            float lb = -2.0f;
            int zkey = 1 << 30;
            corners([&](int, int q, int s, float score, float fac, float e) {
                if (fac > 0.0f) {
                    lb = fmaxf(lb, score - e);
                } else {
                    lb = fmaxf(lb, 0.0f);
                    zkey = min(zkey, key_of(q, s));
                }
            });
            lb = fmaxf(lb, __shfl_xor_sync(VTG_FULL, lb, 1));
            zkey = min(zkey, __shfl_xor_sync(VTG_FULL, zkey, 1));
            if constexpr (Shape::shares > 1) { /* the tile's other rows: the other shares' */
                __shared__ float s_lb[Shape::shares][128];
                s_lb[warp >> 2][m] = lb;
                __syncthreads();
#pragma unroll
                for (int k = 0; k < Shape::shares; k++)
                    lb = fmaxf(lb, s_lb[k][m]);
            }
            if ((m & 1) == 0 && mine && zkey < (1 << 30))
                atomicMax(cellw + (size_t)crow * p.ccols + ccol, ncc_cell_word(0.0f, zkey));
            unsigned long long keep = 0ull;
            corners([&](int k, int, int, float score, float fac, float e) {
                if (fac > 0.0f && score + e >= lb)
                    keep |= 1ull << k;
            });
            /* the warp's corners take a run of the list */
            const int cnt = __popcll(keep);
            int inc = cnt;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int u = __shfl_up_sync(VTG_FULL, inc, d);
                inc += lane >= d ? u : 0;
            }
            unsigned at = 0u;
            if (lane == 31 && inc > 0)
                at = atomicAdd(ncand, (unsigned)inc);
            at = __shfl_sync(VTG_FULL, at, 31) + (unsigned)(inc - cnt);
            while (keep) {
                const int k = __ffsll((long long)keep) - 1;
                keep &= keep - 1ull;
                cand[at++] = ((unsigned)(ty * Q + 2 * c0 + (k >> 3)) << 16) | (unsigned)(xr + (k & 7));
            }
        } else {
            float best = -2.0f;
            int bkey = 1 << 30;
            corners([&](int, int q, int s, float score, float, float) {
                const int key = key_of(q, s);
                if (score > best || (score == best && key < bkey)) {
                    best = score;
                    bkey = key;
                }
            });
            const float ob = __shfl_xor_sync(VTG_FULL, best, 1);
            const int okey = __shfl_xor_sync(VTG_FULL, bkey, 1);
            if (ob > best || (ob == best && okey < bkey)) {
                best = ob;
                bkey = okey;
            }
            if ((m & 1) == 0 && mine && bkey < (1 << 30))
                atomicMax(cellw + (size_t)crow * p.ccols + ccol, ncc_cell_word(best, bkey));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tc_cols(Q)) : "memory");
    }
}

/* A search's tiles and scratch sizes on the tensor-core map. */
struct TcGrid {
    int krow, q, fw, fh, tiles_x, tiles_y, cpitch, fpitch, rows;
};

static TcGrid tc_grid(const NccPrm &p)
{
    TcGrid g;
    g.krow = tc_krow(p.tw);
    g.q = tc_q(p.tw, p.th);
    g.fw = p.x1 - p.x0 + 1;
    g.fh = p.y1 - p.y0 + 1;
    g.tiles_x = (g.fw + TC_XS - 1) / TC_XS;
    g.tiles_y = (g.fh + g.q - 1) / g.q;
    g.cpitch = g.tiles_x * TC_XS + TC_MAX_KROW;
    g.fpitch = g.tiles_x * TC_XS;          /* every tile's 1,024 corners inside a factor row */
    g.rows = p.y0 + g.tiles_y * g.q + p.th; /* every row a tile's band reads */
    return g;
}

static bool tc_fits(const NccPrm &p, const NccScratch &s, const TcGrid &g)
{
    return s.band && s.conv && s.fac && s.cellw && p.tw <= 128 && (size_t)g.cpitch * g.rows <= s.conv_elems &&
           (size_t)g.fpitch * g.fh <= s.fac_elems && !(p.step & (p.step - 1)) && NCC_CELL % p.step == 0 &&
           /* the converting CTAs zero the cells' words */
           (long long)((g.cpitch / 8 + 255) / 256) * g.rows * 256 >= (long long)p.ccols * p.crows;
}

bool vtg_ncc_filters(const NccPrm &p, const NccScratch &s)
{
    if (!s.cand || !s.tol || !(p.flt_a >= 0.0f) || (p.step != 1 && p.step != 2) || p.w < 64)
        return false;
    const TcGrid g = tc_grid(p);
    /* The filter costs a preparation over the plane and two more launches; the map it replaces is one launch whose CTAs take
     * their whole template's products in one chain. Measured (whole searches, filter against map, us): 64 x 64 over 201 x
     * 201 corners 64 / 67, over a 1080p frame 80 / 748; 48 x 48 over 201 x 201 corners (9e7 products) 56 / 48, over 401 x 301
     * (2.8e8) 57 / 61; 32 x 21 over a 640 x 480 frame (1.9e8) 45 / 44, over 960 x 540 (3.2e8) 48 / 64; 16 x 16 over 960 x 540
     * (1.3e8) 47 / 43. So it takes every template from 4,096 pixels on, and smaller ones from 2e8 products. A plane under about 250
     * wide and much taller than its template keeps the map: a row of bounds is whole tiles, 1,024 corners, and their room is the
     * second integral image's, four bounds a pixel. */
    const double products = (double)g.fw * g.fh * p.n / (p.step * p.step);
    return (p.n >= 4096 || products >= 2.0e8) && tc_fits(p, s, g) && (size_t)g.fw * g.fh <= s.cand_elems &&
           (size_t)g.fpitch * g.fh <= s.tol_elems;
}

/* Whether the map's own CTAs make their tiles' factors, under the MMAs. They do when the tensor core is busy for longer than that
 * takes (cycles: an MMA of 8 Q columns takes 4 Q; a round of 256 corners measured some 4,000 and 90 a template row, its loads'
 * latency), or when the preparation would be long by itself: tall templates over most SMs' tiles. Otherwise the preparation,
 * whose CTAs fill the chip, is the shorter way. Whole searches, us, factors by the preparation / by the map: 96 x 96 over a 1080p
 * frame 90 / 82, 64 x 64 62.6 / 58.9, 128 x 128 130 / 118, 64 x 64 over 3840 x 2160 153 / 143, over 201 x 201 corners 49.7 /
 * 47.9; but over 960 x 540 53.5 / 57.7 (30 tiles of four rounds), 32 x 32 over 1080p 52.2 / 53.1, 32 x 21 over 3840 x 2160
 * 111 / 125. */
static bool tc_fused(const NccPrm &p, const TcGrid &g)
{
    const int rounds = ((g.fw < TC_XS ? g.fw : TC_XS) + TC_BOX_X - 1) / TC_BOX_X;
    const int mma = (g.q + p.th - 1) * (g.krow / 16) * 4 * g.q, box = rounds * (4000 + 90 * p.th);
    return mma >= box || (p.th >= 64 && p.tw >= 64 && g.tiles_x * g.tiles_y >= 100);
}

/* The preparation and the map. The map (and the passes after it) start as programmatic dependents, their launch and
 * setup overlapping the kernel before, except when events around the map time it alone. */
template <int KIND, bool FILTER, bool FUSED>
static cudaError_t tc_launch_as(const uint8_t *plane, int pitch, const NccPrm &p, const NccScratch &s, const TcGrid &g,
                                cudaStream_t st)
{
    const TcSmem sm = tc_smem(g.krow, g.q, FUSED);
    const int cells = p.ccols * p.crows;
    const int btx = bp_tx(p.tw), bgx = (g.fw + btx - 1) / btx, nbox = FUSED ? 0 : bgx * ((g.fh + TC_QMAX - 1) / TC_QMAX);
    const int cgx = (g.cpitch / 8 + 255) / 256, nconv = cgx * g.rows;
    ncc_prep<KIND, FILTER, !FUSED><<<nbox + nconv, BOX_NT, 0, st>>>(plane, pitch, p, g.fw, g.fpitch, btx, bgx, nbox, s.fac, s.tol,
                                                                    g.rows, g.cpitch, cgx, s.conv, s.cellw, cells, s.ncand, s.err);
    const bool pdl = !s.map_ev0;
    auto run = [&](auto kernel, int threads) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm.total);
        if (e == cudaSuccess && s.map_ev0)
            e = cudaEventRecord(s.map_ev0, st);
        if (e != cudaSuccess)
            return e;
        return vtg_launch_k(kernel, dim3(g.tiles_x * g.tiles_y), dim3(threads), sm.total, st, pdl, p, plane, pitch,
                            (const uint16_t *)s.band, g.krow, g.tiles_x, sm.a_bytes, sm.stage_bytes, (const uint16_t *)s.conv,
                            g.cpitch, s.fac, g.fpitch, s.cellw, s.err, s.tol, s.cand, s.ncand);
    };
    return g.q == 8 ? run(ncc_map_tc<KIND, 8, FILTER, FUSED>, TcShape<8, FUSED>::threads)
                    : run(ncc_map_tc<KIND, 16, FILTER, FUSED>, TcShape<16, FUSED>::threads);
}

template <int KIND, bool FILTER>
static cudaError_t tc_launch(const uint8_t *plane, int pitch, const NccPrm &p, const NccScratch &s, const TcGrid &g,
                             cudaStream_t st)
{
    return tc_fused(p, g) ? tc_launch_as<KIND, FILTER, true>(plane, pitch, p, s, g, st)
                          : tc_launch_as<KIND, FILTER, false>(plane, pitch, p, s, g, st);
}

cudaError_t vtg_launch_ncc_filter(const uint8_t *plane, int pitch, const NccPrm &p, const NccScratch &s, cudaStream_t st)
{
    return tc_launch<VTG_NCC_FP16, true>(plane, pitch, p, s, tc_grid(p), st);
}

cudaError_t vtg_launch_ncc_map_tc(const void *plane, int pitch, int elem_bytes, const NccPrm &p, const NccScratch &s,
                                  int kind, cudaStream_t st)
{
    const TcGrid g = tc_grid(p);
    if (elem_bytes != 1 || (kind != VTG_NCC_BF16 && kind != VTG_NCC_FP16) || !tc_fits(p, s, g))
        return cudaErrorInvalidValue;
    cudaError_t e = kind == VTG_NCC_BF16 ? tc_launch<VTG_NCC_BF16, false>((const uint8_t *)plane, pitch, p, s, g, st)
                                         : tc_launch<VTG_NCC_FP16, false>((const uint8_t *)plane, pitch, p, s, g, st);
    if (e == cudaSuccess && s.map_ev1)
        e = cudaEventRecord(s.map_ev1, st);
    if (e != cudaSuccess)
        return e;
    /* the cells from their words, and their best eight */
    return vtg_launch_ncc_top(p, s, true, st, !s.map_ev0);
}
