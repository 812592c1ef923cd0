// smem_harness.cu - test harness: a launch whose kernel's limit of dynamic shared memory (allow_dynamic_smem,
// lsm_kernels.h) was asked for twice, by itself and then by another launch. Built by tests/test_gpu_threads.py;
// test infrastructure only.
#include <cuda_runtime.h>
#include <stddef.h>

#include "../../finoptions-engine_b200/csrc/lsm_kernels.h"

namespace {

__global__ void smem_kernel(int* out) {
    __shared__ int fixed[32];
    extern __shared__ int dynamic[];
    fixed[threadIdx.x] = int(threadIdx.x);
    if (threadIdx.x == 0) dynamic[0] = 1;
    __syncthreads();
    if (threadIdx.x == 0) *out = fixed[31] + dynamic[0];
}

}  // namespace

extern "C" int smem_allow(size_t bytes) {
    return int(fo::allow_dynamic_smem(reinterpret_cast<const void*>(smem_kernel), bytes));
}

// 0, or the CUDA error. `taken` is at least one int.
extern "C" int smem_check(size_t allowed, size_t other, size_t taken) {
    int* out = nullptr;
    cudaError_t e = cudaMalloc(&out, sizeof(int));
    if (e == cudaSuccess) e = cudaError_t(smem_allow(allowed));
    if (e == cudaSuccess) e = cudaError_t(smem_allow(other));
    if (e == cudaSuccess) {
        smem_kernel<<<1, 32, taken>>>(out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    cudaFree(out);
    return int(e);
}
