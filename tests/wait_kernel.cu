// One warp that tries a barrier nobody arrives at: how long a bounded wait of the grouped GEMM (tc_ptx.cuh) lasts.
#include <cuda_runtime.h>

#include "../tqllm_b200/csrc/tc_ptx.cuh"

__global__ void wait_k(int tries, unsigned long long * out) {
    __shared__ unsigned long long bar;
    const uint32_t at = b2::tc::saddr(&bar);
    if (threadIdx.x == 0) { b2::tc::bar_init(at, 1); b2::tc::bar_init_fence(); }
    __syncthreads();
    unsigned long long t0, t1;
    int passed = 0;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0)::"memory");
    for (int i = 0; i < tries; ++i) passed += b2::tc::bar_try(at, 0);
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1)::"memory");
    if (threadIdx.x == 0) { out[0] = t1 - t0; out[1] = passed; }
}
// out: two values on the device: nanoseconds of `tries` tries, how many of them succeeded
extern "C" __attribute__((visibility("default"))) int run_wait(int tries, void * out, void * stream) {
    wait_k<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(tries, static_cast<unsigned long long *>(out));
    return int(cudaGetLastError());
}
extern "C" __attribute__((visibility("default"))) unsigned wait_limit() { return b2::tc::WAIT_LIMIT; }
