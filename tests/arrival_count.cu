// Rounds of n arrivals at one count of last_arrival, as the CTAs of the block-mean kernels make them, far past
// 2^32 in all, then one more round one arrival after the other: which[i] = 1 where the i-th was told it is the last.
#include "mdp_internal.cuh"

__global__ void arrive(uint32_t *count, uint32_t n, long long rounds, unsigned long long *lasts) {
    const long long    total = rounds * n, step = (long long) gridDim.x * blockDim.x;
    unsigned long long mine = 0;
    for (long long i = (long long) blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) mine += last_arrival(count, n);
    if (mine) atomicAdd(lasts, mine);
}
__global__ void one_round(uint32_t *count, uint32_t n, int *which) {
    for (uint32_t i = 0; i < n; i++) which[i] = last_arrival(count, n);
}

extern "C" int arrival_count(uint32_t n, long long rounds, unsigned long long *h_lasts, int *h_which) {
    uint32_t           *count = nullptr;
    unsigned long long *lasts = nullptr;
    int                *which = nullptr;
    cudaError_t         e = cudaMalloc(&count, 4);
    if (e == cudaSuccess) e = cudaMalloc(&lasts, 8);
    if (e == cudaSuccess) e = cudaMalloc(&which, 4 * n);
    if (e == cudaSuccess) e = cudaMemset(count, 0, 4);
    if (e == cudaSuccess) e = cudaMemset(lasts, 0, 8);
    if (e == cudaSuccess) {
        arrive<<<148, 256>>>(count, n, rounds, lasts);
        one_round<<<1, 1>>>(count, n, which);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(h_lasts, lasts, 8, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(h_which, which, 4 * n, cudaMemcpyDeviceToHost);
    cudaFree(count);
    cudaFree(lasts);
    cudaFree(which);
    return (int) e;
}
