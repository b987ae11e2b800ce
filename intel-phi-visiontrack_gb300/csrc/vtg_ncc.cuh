/* vtg_ncc.cuh -- what the appearance search's kernels share (ncc.cu, ncc_tc.cu) and the C ABI (api_ncc.cu). */
#ifndef VTG_NCC_CUH
#define VTG_NCC_CUH

#include <math.h>

#include "vtg_internal.cuh"

#define NCC_CELL 16 /* SEARCH_CELL, src/kern/track.c:61: corners to a cell of the map */
#define NCC_TOP 8   /* SEARCH_TOP, src/kern/track.c:62: cells looked at again in half pixels */
#define NCC_HALF_MAX (NCC_TOP * 65 * 65) /* half-pixel scores of the candidates at the largest step (16), with
                                          * the ring around each window */

/* One search: the plane, the template and the clamped window of corners. */
struct NccPrm {
    int w, h;        /* the plane */
    int tw, th, n;   /* template, n = tw th */
    float norm;      /* sum of the template's squares */
    float sum_t;     /* sum of the template as the tensor-core map multiplies it (its rounded values) */
    int x0, x1, y0, y1, step;
    int ccols, crows; /* the map's cells */
    /* the near-blank rule on exact integers: n var <= nthr, 16 n var <= nthr16 (half pixels) */
    long long nthr, nthr16;
    float rnorm; /* sqrt(n / norm): the tensor-core map's factor is rnorm / sqrt(n var) */
    /* the F32 map by filter: how far a corner's FP16 tensor-core score may lie from its F32 score, flt_a + flt_m |its
     * window's mean - 128| / sigma + flt_f |mean - first pixel| / sigma (vtg_ncc_filter_bound); flt_a < 0: no bound */
    float flt_a, flt_m, flt_f;
};

/* What the 16-bit band loses of the template, summed in double (ncc_band_sum): h the rounded value, d = t - h. */
struct NccBandStats {
    float sum_h, sum_d, sum_dd, sum_tt; /* sum h, sum d, sum d^2, sum t^2 */
};

/* nthr = floor(n norm / 16) and nthr16 = floor(n norm): n norm is exact in double (n <= 2^14, norm an F32), so an
 * integer n var compares with them exactly as with n norm / 16 itself, and no kernel needs FP64 for the rule. */
static inline void ncc_thresholds(NccPrm &p)
{
    const double nn = (double)p.n * (double)p.norm;
    p.nthr = (long long)floor(nn * 0.0625);
    p.nthr16 = (long long)floor(nn);
    p.rnorm = p.norm > 0.0f ? (float)sqrt((double)p.n / (double)p.norm) : 0.0f;
}

/* Scratch of a search context, in device memory. */
struct NccScratch {
    long long *S1, *S2; /* integral images of J and J^2, (h + 1) rows of tp */
    int tp;
    float *map_v;
    int *map_x, *map_y;
    int *top, *ntop;
    float *half;          /* the candidates' half-pixel scores: NCC_TOP x (2 around + 3)^2, around <= 2 x 16 - 1 */
    const uint16_t *band; /* the template band for the tensor-core map (ncc_tc.cu), NULL if unset */
    int *err;             /* device status word of the tensor-core map: nonzero when a bounded wait gave up; each search resets it */
    /* the tensor-core map's own scratch: the 16-bit picture (shifted so a tile's row starts 16-byte aligned), each
     * corner's normalisation factor, and one 64-bit (score, corner) word per cell */
    uint16_t *conv;
    size_t conv_elems;
    float *fac;
    size_t fac_elems;
    unsigned long long *cellw;
    /* the top-8 pass's per-CTA lists (NCC_TOP keys a CTA, ncc_top_ctas(cells) CTAs) and two arrival counters, one for
     * it and one for the half-pixel pass: zero between searches, each reset by the CTA that arrives last */
    unsigned long long *topblk;
    int topblk_lists; /* lists topblk holds */
    unsigned *arrive;
    /* the F32 map by filter: the corners to score exactly ((y - y0) << 16 | (x - x0)), in the integral images' place
     * (that map uses none), room for every corner of the plane; and how many they are */
    unsigned *cand, *ncand;
    size_t cand_elems;
    uint16_t *tol; /* that map's bound a corner (FP16, rounded up), rows as fac's; beside the list */
    size_t tol_elems;
    /* vtg_search_profile: events recorded just before and just after the map kernel (NULL: none) */
    cudaEvent_t map_ev0, map_ev1;
};

/* The top-8 pass: NCC_TOPB_THREADS threads a CTA, NCC_TOPB_PER cells a thread; it needs ncc_top_ctas(cells) lists. */
#define NCC_TOPB_THREADS 256
#define NCC_TOPB_PER 4
static inline int ncc_top_ctas(int cells) { return (cells + NCC_TOPB_THREADS * NCC_TOPB_PER - 1) / (NCC_TOPB_THREADS * NCC_TOPB_PER); }

/* A cell's candidate as one orderable word: higher score first, then the earlier corner in scan order. 0: none. */
__device__ __forceinline__ unsigned long long ncc_cell_word(float v, int key)
{
    unsigned u = __float_as_uint(v);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ((unsigned long long)u << 32) | (unsigned long long)(0xFFFFFFFFu - (unsigned)key);
}

__device__ __forceinline__ float ncc_word_score(unsigned long long w)
{
    const unsigned u = (unsigned)(w >> 32);
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

/* A cell of the tensor-core map from its 64-bit word (ordered score, inverted scan index): value and corner, or -2 and
 * the cell's origin where no corner was scored (the F32 map's convention). */
__device__ __forceinline__ void ncc_cell_decode(const NccPrm &p, int cell, unsigned long long w, float &v, int &x, int &y)
{
    const int cx0 = p.x0 + (cell % p.ccols) * NCC_CELL, cy0 = p.y0 + (cell / p.ccols) * NCC_CELL;
    const int per = NCC_CELL / p.step;
    if (w == 0ull) {
        v = -2.0f;
        x = cx0;
        y = cy0;
        return;
    }
    const int key = (int)(0xFFFFFFFFu - (unsigned)(w & 0xFFFFFFFFull));
    v = ncc_word_score(w);
    x = cx0 + (key % per) * p.step;
    y = cy0 + (key / per) * p.step;
}

/* ---- the eight best cells: keys, a warp's best ---- */

/* A cell's key: its value in ascending float order as unsigned, then the inverted cell index (the earlier cell first
 * among equal values); 0 for no value (-2). */
__device__ __forceinline__ unsigned long long top_key(float v, int i)
{
    if (!(v > -2.0f))
        return 0ull;
    unsigned u = __float_as_uint(v);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u); /* ascending float order as unsigned */
    return ((unsigned long long)u << 32) | (unsigned long long)(0xFFFFFFFFu - (unsigned)i);
}

/* The NCC_TOP largest of a warp's keys, N a lane, best first: lane k (and k + 8, ..) ends with the k-th, 0 where there are fewer.
 * Each turn takes the largest by two 32-bit maxima over the warp and strikes it from its lane: about 60 cycles a turn, where
 * merging sorted lists by shuffles took six times that. Keys are distinct (the cell index is in their low bits). */
template <int N>
__device__ __forceinline__ unsigned long long top_of_warp(unsigned long long (&t)[N])
{
    unsigned long long mine = 0ull;
#pragma unroll
    for (int k = 0; k < NCC_TOP; k++) {
        unsigned long long m = t[0];
#pragma unroll
        for (int j = 1; j < N; j++)
            m = t[j] > m ? t[j] : m;
        const unsigned hi = __reduce_max_sync(VTG_FULL, (unsigned)(m >> 32));
        const unsigned lo = __reduce_max_sync(VTG_FULL, (unsigned)(m >> 32) == hi ? (unsigned)m : 0u);
        const unsigned long long best = ((unsigned long long)hi << 32) | lo;
        if (((threadIdx.x & 31) % NCC_TOP) == k)
            mine = best;
#pragma unroll
        for (int j = 0; j < N; j++)
            t[j] = t[j] == best ? 0ull : t[j];
    }
    return mine;
}

/* The last CTA of a top-8 pass, its warp 0: the best eight of the n CTAs' lists in blk (read through L2) into top /
 * ntop, and the arrival counter back to zero. */
__device__ __forceinline__ void ncc_top_final(const unsigned long long *blk, int n, unsigned *arrive, int *top, int *ntop)
{
    const int lane = threadIdx.x & 31;
    unsigned long long t[5] = {0ull, 0ull, 0ull, 0ull, 0ull}; /* [0]: the best so far, on lanes 0 .. 7 */
    for (int b = 0; b < n * NCC_TOP; b += 4 * 32) {
#pragma unroll
        for (int k = 0; k < 4; k++)
            t[1 + k] = b + 32 * k + lane < n * NCC_TOP ? __ldcg(blk + b + 32 * k + lane) : 0ull;
        const unsigned long long best = top_of_warp(t);
        t[0] = lane < NCC_TOP ? best : 0ull;
    }
    const unsigned found = __ballot_sync(VTG_FULL, lane < NCC_TOP && t[0] != 0ull);
    if (lane < NCC_TOP && t[0] != 0ull)
        top[lane] = (int)(0xFFFFFFFFu - (unsigned)(t[0] & 0xFFFFFFFFull));
    if (lane == 0) {
        *ntop = __popc(found);
        *arrive = 0u;
    }
}

/* Elements of the tensor-core map's scratch for planes up to max_w x max_h and templates up to max_tw x max_th. */
size_t vtg_ncc_conv_elems(int max_w, int max_h, int max_th);
size_t vtg_ncc_fac_elems(int max_w, int max_h);

/* The top-8 pass on its own launch: over map_v, or (words) over the tensor-core map's cell words, which it decodes;
 * with pdl as a programmatic dependent of the kernel before it. */
cudaError_t vtg_launch_ncc_top(const NccPrm &p, const NccScratch &s, bool words, cudaStream_t st, bool pdl);
cudaError_t vtg_launch_ncc(const void *plane, int pitch, int plane_type, const float *app, const NccPrm &p,
                           const NccScratch &s, int map_kind, vtg_found *out, cudaStream_t st);
cudaError_t vtg_launch_ncc_corners(const void *plane, int pitch, int plane_type, const float *app, const NccPrm &p,
                                   int count, const int *xs, const int *ys, float *out, cudaStream_t st);
/* The tensor-core map (ncc_tc.cu): the same map_v / map_x / map_y as ncc_map_f32, products in BF16 or FP16. */
cudaError_t vtg_launch_ncc_map_tc(const void *plane, int pitch, int elem_bytes, const NccPrm &p, const NccScratch &s,
                                  int kind, cudaStream_t st);
/* The F32 map by filter (U8 planes), first half: the FP16 tensor-core map, which leaves in s.cand the corners whose F32
 * score may be their cell's best and in s.cellw the near-blank corners' zeros. */
cudaError_t vtg_launch_ncc_filter(const uint8_t *plane, int pitch, const NccPrm &p, const NccScratch &s, cudaStream_t st);
/* Whether that map takes a search of these sizes: its scratch is there and large enough, the bound holds and the
 * search is large enough to gain by it. */
bool vtg_ncc_filters(const NccPrm &p, const NccScratch &s);
/* The bound's parts from the FP16 band's statistics; flt_a = -1 where it would let too many corners through. */
void vtg_ncc_filter_bound(NccPrm &p, const NccBandStats &b);
/* Builds the template band for the tensor-core map from a zero-mean template. */
cudaError_t vtg_launch_ncc_band(const float *app, int tw, int th, int kind, uint16_t *band, NccBandStats *stats,
                                cudaStream_t st);
size_t vtg_ncc_band_bytes(int tw, int th);

#endif
