// lsm_kernels.cu - sm_100a kernels of the single-contract LSM path.
//
//   K1 simulate_kernel     Philox -> ZIGNOR -> GBM -> event phases, one thread per path; stores the
//                          observed rows time-major [rows, paths] with coalesced row stores
//                          (path/seeded.rs:399-474 fused with the transpose).
//   K2 the backward induction is in lsm_backward.cu.
//   K3 diagnose_kernel     rank / condition diagnostic per fitted row, off the critical path
//                          (regression.rs:540-577).
//   K4 evaluate_kernel     re-simulates the evaluation population and applies the fixed policy on
//                          the fly: no path storage (policy.rs:642-834).
//                          Its last CTA forms price and standard error (policy.rs:891-926).
//   replay_kernel          re-runs one failing path to recover the typed failure details.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "lsm_common.cuh"
#include "lsm_device.cuh"
#include "lsm_evaluate.cuh"
#include "lsm_kernels.h"

namespace fo {

constexpr int kSimulateThreads = 256;
constexpr int kSimulateCtasPerSm = 4;
constexpr int kReplayThreads = 32;

// ---------------------------------------------------------------------------------------------
// Normals export
// ---------------------------------------------------------------------------------------------

__global__ void __launch_bounds__(kSimulateThreads) normals_kernel(PhiloxKeys keys, uint32_t domain,
                                                                   uint32_t path_start, uint64_t paths,
                                                                   uint32_t count, double* out,
                                                                   unsigned long long* fail) {
    __shared__ NormalSmem<kSimulateThreads> normals;
    load_normal_tables(normals);
    for (uint64_t p = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; p < paths;
         p += uint64_t(gridDim.x) * blockDim.x) {
        NormalStream<kSimulateThreads> s;
        s.init(normals, domain, uint32_t(path_start + p));
        for (uint32_t k = 0; k < count; k += kChunkNormals) {
            double z[kChunkNormals];
            if (!s.next<kChunkNormals>(keys, k, count, z)) {
                atomicMin(fail, (unsigned long long)p);
                break;
            }
#pragma unroll
            for (uint32_t j = 0; j < kChunkNormals; ++j)
                if (k + j < count) out[p * count + k + j] = z[j];
        }
    }
}

// One kernel where two memsets were: each of them took the stream as long.
__global__ void __launch_bounds__(256) reset_kernel(uint4* region, size_t words, const void* status) {
    let_next_grid_start();
    const size_t none = (reinterpret_cast<uintptr_t>(status) - reinterpret_cast<uintptr_t>(region)) / sizeof(uint32_t);
    static_assert(kStatusNoneBytes % sizeof(uint32_t) == 0, "whole words start as none");
    const auto word = [&](size_t i) { return i - none < kStatusNoneBytes / sizeof(uint32_t) ? ~0u : 0u; };
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < words; i += size_t(gridDim.x) * blockDim.x)
        region[i] = make_uint4(word(4 * i), word(4 * i + 1), word(4 * i + 2), word(4 * i + 3));
}

// ---------------------------------------------------------------------------------------------
// K1: seeded simulation with time-major row stores.
// ---------------------------------------------------------------------------------------------

template <int C>
__global__ void __launch_bounds__(kSimulateThreads, kSimulateCtasPerSm) simulate_kernel(DevicePlan plan, uint64_t paths, PhiloxKeys keys,
                                                                    uint32_t domain, double* out,
                                                                    uint32_t store_first_row, int reconstruct_escrowed,
                                                                    unsigned long long* fail) {
    __shared__ NormalSmem<kSimulateThreads> normals;
    load_normal_tables(normals);
    await_prior_grid();
    for (uint64_t p = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; p < paths;
         p += uint64_t(gridDim.x) * blockDim.x) {
        auto store = [&](int row, double value) {
            if (uint32_t(row) < store_first_row) return;
            if (reconstruct_escrowed) {
                // Escrowed observations: origin -> S0; otherwise prepaid forward + prepaid cash.
                value = plan.row_node[row] == 0 ? plan.initial_spot : value + plan.escrow_cash[row];
            }
            out[uint64_t(row - store_first_row) * paths + p] = value;
        };
        const SimResult r = simulate_path<true, C>(plan, normals, keys, domain, uint32_t(p), store);
        if (r.code != 0) atomicMin(fail, (unsigned long long)p);
    }
}

// External normals: the lowest index of a non-finite value in the [intervals, paths] buffer.
__global__ void __launch_bounds__(256) first_nonfinite_kernel(const double* values, uint64_t n,
                                                              unsigned long long* first) {
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
        if (!fo_isfinite(values[i])) atomicMin(first, (unsigned long long)i);
}

// K1 driven by caller normals: one thread per path, time-major [rows, paths] stores.
__global__ void __launch_bounds__(256) simulate_external_kernel(DevicePlan plan, uint64_t paths, const double* normals,
                                                                double* out, unsigned long long* fail) {
    for (uint64_t p = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; p < paths;
         p += uint64_t(gridDim.x) * blockDim.x) {
        const SimResult r = simulate_path_external(plan, normals, paths, p,
                                                   [&](int row, double value) { out[uint64_t(row) * paths + p] = value; });
        if (r.code != 0) atomicMin(fail, (unsigned long long)p);
    }
}

__global__ void replay_external_kernel(DevicePlan plan, uint64_t paths, const double* normals, uint64_t path,
                                       SimFailure* out) {
    if (threadIdx.x != 0) return;
    const SimResult r = simulate_path_external(plan, normals, paths, path, [](int, double) {});
    out->code = r.code;
    out->interval = r.interval;
    out->spot = r.spot;
    out->normal = r.normal;
    out->observed = 0.0;
}

// Re-runs one path serially to recover the typed failure details and the state at `want_row`.
__global__ void replay_kernel(DevicePlan plan, uint64_t seed, uint32_t domain, uint32_t path, int want_row,
                              SimFailure* out) {
    __shared__ NormalSmem<kReplayThreads> normals;
    load_normal_tables(normals);
    if (threadIdx.x != 0) return;
    const PhiloxKeys keys = philox_keys(seed);
    double observed = 0.0;
    const SimResult r = simulate_path(plan, normals, keys, domain, path, [&](int row, double v) {
        if (row == want_row) observed = v;
    });
    out->code = r.code;
    out->interval = r.interval;
    out->spot = r.spot;
    out->normal = r.normal;
    out->observed = observed;
}

// ---------------------------------------------------------------------------------------------
// K3: diagnostics for regression rows.
// ---------------------------------------------------------------------------------------------

// One row a CTA, by one thread: rows of one warp would wait for each other's rotations and sweeps. Bound by
// its serial chain of divisions and square roots.
template <int D>
__global__ void __launch_bounds__(32) diagnose_kernel(DevicePlan plan, FitRecord* records) {
    const uint32_t row = blockIdx.x;
    FitRecord& rec = records[row];
    if (threadIdx.x != 0 || rec.kind != kRuleRegression) return;
    int rank = 0, aux = 0;
    double condition = 0.0;
    rec.diag_status =
        diagnose_design_d<D>(rec.model, plan.rank_tolerance, plan.condition_limit, &rank, &condition, &aux);
    rec.diag_rank = rank;
    rec.diag_condition = condition;
    rec.diag_aux = aux;
}

// ---------------------------------------------------------------------------------------------
// K4: fused re-simulation + fixed-policy evaluation.
// ---------------------------------------------------------------------------------------------

// Issue-bound like the simulation. At 52 weeks, 2^20 paths: 0.474 ms with a branch per observation and the
// stop's bookkeeping inside it, the steps in a loop of their own; 0.456 with the steps of a chunk unrolled;
// 0.435 with a row decided by signs and the bookkeeping after the path (4,096 paths: 53 -> 46 us). At three
// CTAs per SM, without spills, 0.438, and 262,144 paths take 146 us against 131.
template <int D, int C>
__global__ void __launch_bounds__(kEvalThreads, 4) evaluate_kernel(EvalArgs a) {
    extern __shared__ __align__(16) unsigned char eval_smem_raw[];
    const DevicePlan& plan = a.plan;
    const uint32_t rows = plan.rows;
    __shared__ NormalSmem<kEvalThreads> normals;
    __shared__ double red[32 * 2];
    EvalRow* rules = reinterpret_cast<EvalRow*>(eval_smem_raw);      // [rows]
    unsigned* counts = reinterpret_cast<unsigned*>(rules + rows);    // [rows]
    unsigned* itm_counts = counts + rows;                            // [rows]
    const double K = plan.strike;
    load_normal_tables(normals);
    await_prior_grid();
    for (uint32_t r = threadIdx.x; r < rows; r += blockDim.x) {
        rules[r] = make_eval_row(plan, a.records, r);
        counts[r] = 0;
        itm_counts[r] = 0;
    }
    __syncthreads();
    const uint64_t P = plan.eval_paths;
    const uint32_t last = rows - 1;
    const uint64_t tie = plan.tie_rule == 0 ? 0u : 1u;
    double sum = 0.0, sumsq = 0.0;
    for (uint64_t p = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; p < P; p += uint64_t(gridDim.x) * blockDim.x) {
        // The payoff is -1 until the policy stops the path: its sign says that it still runs.
        double payoff = -1.0;
        uint32_t stop_row = 0;
        const auto stop = [&](double paid, int row) {
            payoff = paid;
            stop_row = uint32_t(row);
        };
        auto observe = [&](int row, double spot) {
            const EvalRow& er = rules[row];
            const double below = K - spot;
            if (uint32_t(row) == last) {
                if (__double2hiint(payoff) < 0) stop((below < 0.0 ? -below : 0.0) * er.discount, row);
                return;
            }
            if (er.rule.general == 0 && within_rule(spot)) {
                // By the signs of K - spot, of the continuation less the excess (less one in the last bit where a
                // tie exercises: the difference is zero, and then positive, only at a tie) and of the payoff.
                const double kept = rule_continuation<D>(er.rule, -below) + below;
                const int keeps = int((double_to_bits(kept) - tie) >> 32);
                if ((__double2hiint(below) & keeps & __double2hiint(payoff)) < 0) stop(-below * er.discount, row);
            } else if (__double2hiint(payoff) < 0 && below < 0.0 &&
                       decide_row<D>(plan, a.records, a.status, er.rule, uint32_t(row), p, spot, -below, itm_counts)) {
                stop(fo_fabs(-below * er.discount), row);
            }
        };
        const SimResult r = simulate_path<true, C>(plan, normals, a.keys, plan.eval_domain, uint32_t(p), observe);
        if (r.code != 0) atomicMin(&a.status->eval_sim_fail, (unsigned long long)p);
        if (__double2hiint(payoff) < 0) {
            payoff = 0.0;  // the simulation failed before the path stopped
        } else {
            atomicAdd(&counts[stop_row], 1u);
            if (a.stops) a.stops[p] = stop_row;
            if (!fo_isfinite(payoff)) {
                if (stop_row == last) atomicMin(&a.status->eval_terminal_fail, (unsigned long long)p);
                else atomicMin(&a.status->eval_fail, ((unsigned long long)stop_row << 33) | (p << 1) | 1ull);
            }
        }
        sum += payoff;
        sumsq += payoff * payoff;
    }
    double acc[2] = {sum, sumsq};
    cta_reduce_to<2>(acc, red, a.partials + size_t(blockIdx.x) * 2);
    for (uint32_t r = threadIdx.x; r < rows; r += blockDim.x) {
        if (counts[r]) atomicAdd(&a.counts[r], counts[r]);
        if (itm_counts[r]) atomicAdd(&a.itm_counts[r], itm_counts[r]);
    }
    if (last_cta(a.status)) finalize_price(a.partials, int(gridDim.x), P, a.result);
}

// ---------------------------------------------------------------------------------------------
// Host-callable launchers
// ---------------------------------------------------------------------------------------------

cudaError_t launch_normals(uint64_t seed, uint32_t domain, uint32_t path_start, uint64_t paths, uint32_t count,
                           double* out, unsigned long long* fail, cudaStream_t stream) {
    const int threads = kSimulateThreads;
    const uint64_t blocks = (paths + threads - 1) / threads;
    normals_kernel<<<unsigned(blocks < 65535 * 16 ? blocks : 65535 * 16), threads, 0, stream>>>(
        philox_keys(seed), domain, path_start, paths, count, out, fail);
    return cudaGetLastError();
}

cudaError_t launch_reset(void* region, size_t bytes, DeviceStatus* status, int sms, cudaStream_t stream) {
    const size_t words = bytes / sizeof(uint4);
    const size_t blocks = std::min<size_t>((words + 255) / 256, size_t(sms));
    reset_kernel<<<unsigned(blocks), 256, 0, stream>>>(static_cast<uint4*>(region), words, status);
    return cudaGetLastError();
}

cudaError_t launch_simulate(const DevicePlan& plan, uint64_t paths, uint64_t seed, uint32_t domain, double* out,
                            uint32_t store_first_row, int reconstruct_escrowed, unsigned long long* fail,
                            int sms, cudaStream_t stream) {
    const int threads = kSimulateThreads;
    uint64_t blocks = (paths + threads - 1) / threads;
    // A CTA fills 15 KB of sampler tables first, about the work of eight steps: short paths share a CTA's
    // tables among several blocks of paths, down to one wave of CTAs.
    const uint64_t share = std::max<uint64_t>(1, 32 / std::max<uint32_t>(plan.intervals, 1));
    const uint64_t wave = uint64_t(kSimulateCtasPerSm) * uint64_t(sms);
    if (blocks > wave) blocks = std::max<uint64_t>(wave, (blocks + share - 1) / share);
    if (blocks > (1u << 20)) blocks = 1u << 20;
    const auto kernel = plan.intervals <= 2 ? simulate_kernel<2> : simulate_kernel<kChunkNormals>;
    return launch_early(kernel, dim3(unsigned(blocks)), threads, 0, stream, plan, paths, philox_keys(seed), domain, out,
                        store_first_row, reconstruct_escrowed, fail);
}

cudaError_t launch_first_nonfinite(const double* values, uint64_t n, unsigned long long* first, cudaStream_t stream) {
    const uint64_t blocks = std::min<uint64_t>((n + 255) / 256, 148u * 16u);
    first_nonfinite_kernel<<<unsigned(std::max<uint64_t>(blocks, 1)), 256, 0, stream>>>(values, n, first);
    return cudaGetLastError();
}

cudaError_t launch_simulate_external(const DevicePlan& plan, uint64_t paths, const double* normals, double* out,
                                     unsigned long long* fail, cudaStream_t stream) {
    uint64_t blocks = (paths + 255) / 256;
    if (blocks > (1u << 20)) blocks = 1u << 20;
    simulate_external_kernel<<<unsigned(blocks), 256, 0, stream>>>(plan, paths, normals, out, fail);
    return cudaGetLastError();
}

cudaError_t launch_replay_external(const DevicePlan& plan, uint64_t paths, const double* normals, uint64_t path,
                                   SimFailure* out, cudaStream_t stream) {
    replay_external_kernel<<<1, 32, 0, stream>>>(plan, paths, normals, path, out);
    return cudaGetLastError();
}

cudaError_t launch_replay(const DevicePlan& plan, uint64_t seed, uint32_t domain, uint32_t path, int want_row,
                          SimFailure* out, cudaStream_t stream) {
    replay_kernel<<<1, kReplayThreads, 0, stream>>>(plan, seed, domain, path, want_row, out);
    return cudaGetLastError();
}

cudaError_t launch_diagnose(const DevicePlan& plan, FitRecord* records, cudaStream_t stream) {
    if (plan.rows <= 1) return cudaSuccess;
    const unsigned rows = plan.rows - 1;
    switch (plan.degree) {  // validated to 0..4 on the host
        case 0: diagnose_kernel<0><<<rows, 32, 0, stream>>>(plan, records); break;
        case 1: diagnose_kernel<1><<<rows, 32, 0, stream>>>(plan, records); break;
        case 2: diagnose_kernel<2><<<rows, 32, 0, stream>>>(plan, records); break;
        case 3: diagnose_kernel<3><<<rows, 32, 0, stream>>>(plan, records); break;
        default: diagnose_kernel<4><<<rows, 32, 0, stream>>>(plan, records); break;
    }
    return cudaGetLastError();
}

size_t evaluate_smem_bytes(uint32_t rows) {
    return sizeof(EvalRow) * rows + sizeof(unsigned) * 2 * rows;
}

template <int D>
static cudaError_t launch_evaluate_d(const EvalArgs& args, int blocks, size_t smem, cudaStream_t stream) {
    const auto kernel = args.plan.intervals <= 2 ? evaluate_kernel<D, 2> : evaluate_kernel<D, kChunkNormals>;
    const cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem, sizeof(NormalSmem<kEvalThreads>) + 1024);
    if (e != cudaSuccess) return e;
    return launch_early(kernel, dim3(unsigned(blocks)), kEvalThreads, smem, stream, args);
}

cudaError_t launch_evaluate(const EvalArgs& args, int blocks, cudaStream_t stream) {
    const size_t smem = evaluate_smem_bytes(args.plan.rows);
    switch (args.plan.degree) {  // validated to 0..4 on the host
        case 0: return launch_evaluate_d<0>(args, blocks, smem, stream);
        case 1: return launch_evaluate_d<1>(args, blocks, smem, stream);
        case 2: return launch_evaluate_d<2>(args, blocks, smem, stream);
        case 3: return launch_evaluate_d<3>(args, blocks, smem, stream);
        default: return launch_evaluate_d<4>(args, blocks, smem, stream);
    }
}

}  // namespace fo
