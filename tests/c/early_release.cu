/* A caller's kernel that lets the stream's next kernel start before it has written what that one reads: out = src (n floats), some
 * time after griddepcontrol.launch_dependents. The wait before it is bounded by the clock. */
#include <cuda_runtime.h>

__global__ void early_release_kernel(float *out, const float *src, int n, long long cycles)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long start = clock64();
    while (clock64() - start < cycles)
        ;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = src[i];
}

extern "C" int early_release(float *out, const float *src, int n, long long cycles, void *stream)
{
    early_release_kernel<<<64, 256, 0, (cudaStream_t)stream>>>(out, src, n, cycles);
    return (int)cudaGetLastError();
}
