/* vtg_search_create on a fake of the CUDA runtime in which the call named by argv[1] fails: whatever was made before must be given
 * back. Linked with the library's api_ncc.o; prints the status and what is left (allocations, pinned blocks, streams, charge). */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <cuda_runtime.h>

#include "vtg.h"

struct NccPrm;
struct NccScratch;
struct NccBandStats;

static const char *g_fail;
static int g_mem, g_pinned, g_streams;
static long g_charge;

static cudaError_t step(const char *name, cudaError_t bad = cudaErrorUnknown) { return g_fail && !strcmp(name, g_fail) ? bad : cudaSuccess; }

extern "C" {
cudaError_t cudaSetDevice(int) { return step("cudaSetDevice"); }
cudaError_t cudaMalloc(void **p, size_t)
{
    const cudaError_t e = step("cudaMalloc", cudaErrorMemoryAllocation);
    if (e == cudaSuccess) {
        *p = malloc(16);
        g_mem++;
    }
    return e;
}
cudaError_t cudaFree(void *p)
{
    g_mem -= p != nullptr;
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    const cudaError_t e = step("cudaHostAlloc", cudaErrorMemoryAllocation);
    if (e == cudaSuccess) {
        *p = malloc(n);
        g_pinned++;
    }
    return e;
}
cudaError_t cudaFreeHost(void *p)
{
    g_pinned -= p != nullptr;
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned)
{
    *d = h;
    return step("cudaHostGetDevicePointer");
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    const cudaError_t e = step("cudaStreamCreateWithFlags");
    if (e == cudaSuccess) {
        *s = (cudaStream_t)0x10;
        g_streams++;
    }
    return e;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { g_streams--; return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return step("cudaMemsetAsync"); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return step("cudaStreamSynchronize"); }
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMallocAsync(void **, size_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaFreeAsync(void *, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *) { return cudaErrorUnknown; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *, cudaEvent_t, cudaEvent_t) { return cudaErrorUnknown; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaErrorUnknown; }
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
}

int vtg_ctx_charge(vtg_ctx *, size_t n) { g_charge += (long)n; return VTG_OK; }
void vtg_ctx_release(vtg_ctx *, size_t n) { g_charge -= (long)n; }
int vtg_ctx_device(const vtg_ctx *) { return 0; }
void vtg_ctx_track(vtg_ctx *, cudaStream_t, bool) {}
void vtg_set_cuda_error(cudaError_t) {}
size_t vtg_ncc_fac_elems(int, int) { return 16; }
size_t vtg_ncc_band_bytes(int, int) { return 16; }
size_t vtg_ncc_conv_elems(int, int, int) { return 16; }
void vtg_ncc_filter_bound(NccPrm &, const NccBandStats &) {}
cudaError_t vtg_launch_ncc(const void *, int, int, const float *, const NccPrm &, const NccScratch &, int, vtg_found *, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t vtg_launch_ncc_band(const float *, int, int, int, unsigned short *, NccBandStats *, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t vtg_launch_ncc_corners(const void *, int, int, const float *, const NccPrm &, int, const int *, const int *, float *, cudaStream_t) { return cudaErrorUnknown; }

int main(int argc, char **argv)
{
    g_fail = argc > 1 ? argv[1] : nullptr;
    vtg_search *s = nullptr;
    const int rc = vtg_search_create((vtg_ctx *)0x20, 640, 480, 64, 64, &s);
    if (rc == VTG_OK) {
        g_fail = nullptr;
        vtg_search_destroy(s);
    }
    printf("%d %d %d %d %ld\n", rc, g_mem, g_pinned, g_streams, g_charge);
    return 0;
}
