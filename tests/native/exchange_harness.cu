// exchange_harness.cu - test harness: the waits of the backward kernel on one CTA - the exchange of a grid's
// sums (lsm_exchange.cuh) with the other CTAs' lines laid out beforehand, some of them never, and the wait
// for a bulk copy (lsm_bulk_copy.cuh) that nothing completes. Built by tests/test_gpu_exchange.py; test
// infrastructure only.
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../finoptions-engine_b200/csrc/lsm_bulk_copy.cuh"
#include "../../finoptions-engine_b200/csrc/lsm_exchange.cuh"
#include "../../finoptions-engine_b200/csrc/lsm_kernels.h"

namespace {

constexpr int kWarps = 16;

struct Outcome {
    fo::dd total[fo::kExchangeSlots];
    int failed, warps_left;
    unsigned long long elapsed_ns;
};

// CTA `block` of `blocks` at exchange `seq`, whose own sums are red[warp][slot].
__global__ void __launch_bounds__(kWarps * 32) exchange_kernel(const double* red, double2* partials, int block, int blocks,
                                                               unsigned seq, fo::DeviceStatus* status,
                                                               unsigned long long limit_ns, Outcome* out) {
    __shared__ fo::ExchangeSmem<kWarps> sm;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) sm.failed = 0;
    if (threadIdx.x < kWarps * fo::kExchangeSlots)
        sm.red[threadIdx.x / fo::kExchangeSlots][threadIdx.x % fo::kExchangeSlots] = red[threadIdx.x];
    __syncthreads();
    const unsigned long long start = fo::global_timer_ns();
    if (warp < fo::kExchangeWarps) {
        const fo::dd total = fo::exchange_totals(sm, partials, block, blocks, seq, status, limit_ns);
        if (warp == 0 && lane < fo::kExchangeSlots) out->total[lane] = total;
    }
    __syncthreads();
    if (lane == 0) atomicAdd(&out->warps_left, 1);
    if (threadIdx.x != 0) return;
    out->failed = sm.failed;
    out->elapsed_ns = fo::global_timer_ns() - start;
}

// Waits for `bytes` to arrive: copied from `src`, or (copy 0) never.
__global__ void copy_kernel(const double* src, int words, int copy, fo::DeviceStatus* status, unsigned long long limit_ns,
                            Outcome* out) {
    __shared__ __align__(16) double buffer[256];
    __shared__ uint64_t bar;
    fo::mbarrier_init(&bar, 1);
    if (copy) fo::bulk_load(buffer, src, uint32_t(words * sizeof(double)), &bar);
    const unsigned long long start = fo::global_timer_ns();
    out->failed = fo::wait_bulk(&bar, 0, status, limit_ns) ? 0 : 1;
    out->elapsed_ns = fo::global_timer_ns() - start;
    out->warps_left = 1;
    double sum = 0.0;
    for (int i = 0; copy && i < words; ++i) sum += buffer[i];
    out->total[0] = fo::dd_make(sum);
}

}  // namespace

extern "C" int exchange_bytes() { return int(sizeof(Outcome)); }

// red: [16][8]. lines: exchange_words(blocks) words as the buffers stand when the CTA arrives, returned as it
// leaves them. Returns 0 or the CUDA error.
extern "C" int exchange_check(const double* red, double* lines, int block, int blocks, unsigned seq,
                              unsigned long long limit_ns, void* outcome, unsigned* timeout_flag) {
    const size_t words = size_t(fo::exchange_words(blocks));
    double* d_red = nullptr;
    double2* d_lines = nullptr;
    fo::DeviceStatus* st = nullptr;
    Outcome* out = nullptr;
    cudaError_t e = cudaMalloc(&d_red, sizeof(double) * kWarps * fo::kExchangeSlots);
    if (e == cudaSuccess) e = cudaMalloc(&d_lines, sizeof(double2) * words);
    if (e == cudaSuccess) e = cudaMalloc(&st, sizeof(*st));
    if (e == cudaSuccess) e = cudaMalloc(&out, sizeof(*out));
    if (e == cudaSuccess) e = cudaMemset(st, 0, sizeof(*st));
    if (e == cudaSuccess) e = cudaMemset(out, 0, sizeof(*out));
    if (e == cudaSuccess)
        e = cudaMemcpy(d_red, red, sizeof(double) * kWarps * fo::kExchangeSlots, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d_lines, lines, sizeof(double2) * words, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        exchange_kernel<<<1, kWarps * 32>>>(d_red, d_lines, block, blocks, seq, st, limit_ns, out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(outcome, out, sizeof(*out), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(lines, d_lines, sizeof(double2) * words, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess)
        e = cudaMemcpy(timeout_flag, reinterpret_cast<unsigned char*>(st) + offsetof(fo::DeviceStatus, barrier_timeout),
                       sizeof(unsigned), cudaMemcpyDeviceToHost);
    cudaFree(d_red);
    cudaFree(d_lines);
    cudaFree(st);
    cudaFree(out);
    return int(e);
}

// words: at most 256, even.
extern "C" int copy_check(const double* src, int words, int copy, unsigned long long limit_ns, void* outcome,
                          unsigned* timeout_flag) {
    double* d_src = nullptr;
    fo::DeviceStatus* st = nullptr;
    Outcome* out = nullptr;
    cudaError_t e = cudaMalloc(&d_src, sizeof(double) * 256);
    if (e == cudaSuccess) e = cudaMalloc(&st, sizeof(*st));
    if (e == cudaSuccess) e = cudaMalloc(&out, sizeof(*out));
    if (e == cudaSuccess) e = cudaMemset(st, 0, sizeof(*st));
    if (e == cudaSuccess) e = cudaMemset(out, 0, sizeof(*out));
    if (e == cudaSuccess) e = cudaMemcpy(d_src, src, sizeof(double) * words, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        copy_kernel<<<1, 1>>>(d_src, words, copy, st, limit_ns, out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(outcome, out, sizeof(*out), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess)
        e = cudaMemcpy(timeout_flag, reinterpret_cast<unsigned char*>(st) + offsetof(fo::DeviceStatus, barrier_timeout),
                       sizeof(unsigned), cudaMemcpyDeviceToHost);
    cudaFree(d_src);
    cudaFree(st);
    cudaFree(out);
    return int(e);
}
