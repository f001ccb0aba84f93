// A block that waits for bytes which nothing copies: every thread gives up within
// seconds, sets the flag and returns, and the context is usable after it.  (The
// waits are those of the FP64 and FP32 steps.)
#include <cstdio>

#include "../../tmixer_b200/csrc/tmx_run.cuh"

__global__ void k_wait(int* error, int* returned)
{
    __shared__ unsigned long long full;
    const unsigned bar = tmx::smem_addr(&full);
    if (threadIdx.x == 0) {
        tmx::mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tmx::mbar_expect(bar, 16);
    }
    __syncthreads();
    if (!tmx::mbar_wait(bar, 0)) tmx::mbar_give_up(error, bar);
    atomicAdd(returned, 1);
}

int main()
{
    int* error;  // mapped host memory, as a handle's
    int *returned, n = 0;
    if (cudaHostAlloc((void**)&error, sizeof(int), cudaHostAllocMapped) != cudaSuccess) return 2;
    if (cudaMalloc((void**)&returned, sizeof(int)) != cudaSuccess) return 2;
    *error = 0;
    cudaMemset(returned, 0, sizeof(int));
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    cudaEventRecord(a);
    k_wait<<<1, 128>>>(error, returned);
    cudaEventRecord(b);
    const cudaError_t e = cudaDeviceSynchronize();
    float ms = 0;
    cudaEventElapsedTime(&ms, a, b);
    const cudaError_t m = cudaMemcpy(&n, returned, sizeof(int), cudaMemcpyDeviceToHost);
    std::printf("%s, %s, flag %d, %d threads back after %.0f ms\n", cudaGetErrorString(e), cudaGetErrorString(m), *error, n,
                ms);
    return e == cudaSuccess && m == cudaSuccess && *error == 1 && n == 128 && ms < 15000 ? 0 : 1;
}
