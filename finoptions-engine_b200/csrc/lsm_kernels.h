// lsm_kernels.h - launch interface of the single-contract LSM kernels (host <-> device).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "lsm_device.cuh"

namespace fo {

constexpr int kBackwardThreads = 512;
constexpr int kEvalThreads = 256;
// The moments of every fitted row, and the backward pass's exchange buffer back at phase 0.
struct MomentArgs {
    DevicePlan plan;
    const double* slab;          // stored training rows [rows - first_stored_row, paths]
    double2* partials;           // [fitted rows][blocks][16] CTA totals (unused with one block a row)
    FitRecord* records;          // [rows]; `arrived` and `again` start at zero
    DeviceStatus* status;
    double2* exchange;           // BackwardArgs::partials
    int exchange_words;          // exchange_words(backward blocks)
    int relaunch;                // a second launch takes the rows again whose pivot was too far
};

struct BackwardArgs {
    DevicePlan plan;
    const double* slab;          // stored training rows [rows - first_stored_row, paths]
    double2* partials;           // [2][blocks][8] double-double CTA sums, by exchange parity and slot
    FitRecord* records;          // [rows]: moments_kernel's
    DeviceStatus* status;
    int ppt;                     // paths per thread
    double* values;              // NULL: values and spots on chip (shared memory); else [train paths]
                                 // values in HBM, spots read from the slab (populations beyond the
                                 // on-chip capacity)
};
constexpr int exchange_words(int blocks) { return 2 * 8 * blocks; }

struct EvalArgs {
    DevicePlan plan;
    PhiloxKeys keys;             // of plan.eval_seed
    const FitRecord* records;
    double2* partials;           // [blocks][2]
    unsigned* counts;            // [rows] stopping counts
    unsigned* itm_counts;        // [rows] active in-the-money paths at unsupported rows
    DeviceStatus* status;
    uint32_t* stops;             // optional [evaluation paths]: the row at which each path stopped
    double* result;              // price, second moment, standard deviation, standard error
};

// Pathwise adjoint Greeks of the fused evaluation (lsm_greeks.cu).
constexpr int kMaxGreekDividends = 8;
constexpr int kGreekSlots = 32;
enum GreekSlot : int {
    kGreekDelta = 0,     // sum of dP/dS0
    kGreekVega = 1,      // sum of dP/dsigma
    kGreekL0 = 2,        // sum of dP/dL_0 (drift of the first step)
    kGreekTerminal = 3,  // sum of dP/dL_N at expiry stops (discount + last drift)
    kGreekJump = 4,      // [kMaxGreekDividends]: sums of dP/dL at each cash-dividend node
    kGreekDividend = kGreekJump + kMaxGreekDividends,  // [kMaxGreekDividends]: sums of dP/dD_j
};

struct GreeksArgs {
    uint32_t dividends;                         // cash dividends of the schedule, in node order
    uint32_t div_node[kMaxGreekDividends];
    double div_amount[kMaxGreekDividends];
    double sigma;
    const double* sqrt_dt;                      // [intervals]
    const double* dt;                           // [intervals]
    double2* partials;                          // [blocks][kGreekSlots] double-double block sums
    double* sums;                               // [kGreekSlots]: their totals
};

// Launches a kernel that may start while the one ahead of it in the stream still runs (its sampler tables
// and its launch then take no time of their own: 4,096 paths of 12 dates, 78 -> 72 us for the kernels of a
// contract). The kernel calls await_prior_grid before it reads or writes global memory.
template <typename... P, typename... A>
cudaError_t launch_early(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, A... args) {
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, P(args)...);
}

// Lets a kernel take `bytes` of dynamic shared memory. The limit belongs to the kernel and not to a launch: set to
// what each launch needs, another thread's smaller one could lower it between this one's setting and its
// launch. So it is only ever raised, to all that a CTA has beside the kernel's static share. A kernel whose
// static share is at most `fixed` needs no leave for what fits 48 KB with it (a query takes half a microsecond).
inline cudaError_t allow_dynamic_smem(const void* kernel, size_t bytes, size_t fixed = 48 * 1024) {
    if (fixed + bytes <= 48 * 1024) return cudaSuccess;
    cudaFuncAttributes attr{};
    cudaError_t e = cudaFuncGetAttributes(&attr, kernel);
    if (e != cudaSuccess || size_t(attr.maxDynamicSharedSizeBytes) >= bytes) return e;
    int device = 0, most = 0;
    e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) return e;
    if (attr.sharedSizeBytes + bytes > size_t(most)) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                most - int(attr.sharedSizeBytes));
}

// Clears a plan's read-back region (a multiple of 16 bytes), its status words to "none" where they start so.
cudaError_t launch_reset(void* region, size_t bytes, DeviceStatus* status, int sms, cudaStream_t stream);
cudaError_t launch_normals(uint64_t seed, uint32_t domain, uint32_t path_start, uint64_t paths, uint32_t count,
                           double* out, unsigned long long* fail, cudaStream_t stream);
cudaError_t launch_simulate(const DevicePlan& plan, uint64_t paths, uint64_t seed, uint32_t domain, double* out,
                            uint32_t store_first_row, int reconstruct_escrowed, unsigned long long* fail,
                            int sms, cudaStream_t stream);
cudaError_t launch_replay(const DevicePlan& plan, uint64_t seed, uint32_t domain, uint32_t path, int want_row,
                          SimFailure* out, cudaStream_t stream);
// External normals ([intervals, paths], time-major): the first non-finite value's index, the
// simulation, and the replay of one failing path.
cudaError_t launch_first_nonfinite(const double* values, uint64_t n, unsigned long long* first, cudaStream_t stream);
cudaError_t launch_simulate_external(const DevicePlan& plan, uint64_t paths, const double* normals, double* out,
                                     unsigned long long* fail, cudaStream_t stream);
cudaError_t launch_replay_external(const DevicePlan& plan, uint64_t paths, const double* normals, uint64_t path,
                                   SimFailure* out, cudaStream_t stream);
// CTAs per row of the moments launch, at most what the workspace holds; what that many take.
int moment_blocks(uint64_t paths, uint32_t rows, int sms, size_t workspace_bytes);
size_t moment_workspace_bytes(uint32_t rows, int blocks);
cudaError_t launch_moments(const MomentArgs& args, int blocks, cudaStream_t stream);
int backward_max_blocks(int device);
int backward_max_ppt();
size_t backward_smem_bytes(int ppt);
cudaError_t launch_backward(const BackwardArgs& args, int blocks, int ppt, cudaStream_t stream);
cudaError_t launch_diagnose(const DevicePlan& plan, FitRecord* records, cudaStream_t stream);
size_t evaluate_smem_bytes(uint32_t rows);
cudaError_t launch_evaluate(const EvalArgs& args, int blocks, cudaStream_t stream);
size_t evaluate_greeks_smem_bytes(uint32_t rows);
cudaError_t launch_evaluate_greeks(const EvalArgs& args, const GreeksArgs& greeks, int blocks, cudaStream_t stream);

}  // namespace fo
