// The quotient of the routing's softmax (route_token.cuh) against CUDA's division: how many of n pairs 2^-100 <= a <= 1, 1 <= b < 2^20 differ.
#include <cuda_runtime.h>

#include "../tqllm_b200/csrc/route_token.cuh"

__global__ void quotients_k(const float * a, const float * b, int n, int * differ) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && b2::quotient(a[i], b[i], 1.f / b[i]) != a[i] / b[i]) atomicAdd(differ, 1);
}
extern "C" __attribute__((visibility("default"))) int count_different(const void * a, const void * b, int n, void * differ, void * stream) {
    quotients_k<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const float *>(a), static_cast<const float *>(b), n, static_cast<int *>(differ));
    return int(cudaGetLastError());
}
