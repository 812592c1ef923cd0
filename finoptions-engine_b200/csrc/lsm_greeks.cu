// lsm_greeks.cu - fused evaluation with pathwise adjoint Greeks for one contract (no reference
// counterpart: the reference obtains sensitivities by bump-and-reprice through price_lsm_call).
//
// The fitted exercise policy is held fixed. Each evaluation path is re-simulated exactly as in
// evaluate_kernel (same Philox stream, ZIGNOR normals and GBM / cash-dividend arithmetic), so the
// price partials are bitwise those of the plain evaluation. While simulating, the path keeps a
// few numbers per segment between cash-dividend nodes; when it stops (exercise or expiry) a short
// backward recurrence over those segments yields its contribution to delta, vega, the
// log-discount sensitivities and the cash-dividend sensitivities.
//
// With payoff P = (S_obs - K) exp(L_n) at the stopping node n and a = dP/dS the adjoint of the
// state, the GBM step S' = S exp(u_i), u_i = sigma sqrt(dt_i) Z_i + log_drift_i, is multiplicative,
// so w = a S is constant along a segment without cash dividends and
//   dP/du_i = w_segment(i),   dP/dsigma = sum_segments w_s sum_{i in s} (Z_i sqrt(dt_i) - sigma dt_i).
// Because log_drift_i = -(L_{i+1} - L_i) - (Q_{i+1} - Q_i) - sigma^2 dt_i / 2, the log-discount
// gradient is w at node 0, the jump of w at each cash-dividend node, and P - w_last at the
// stopping node (exactly -K exp(L_n) for an early exercise, which the host applies from the
// stopping counts). A cash jump S+ = h(S-) maps a+ to a- = a+ h'(S-) and contributes
// -a+ [S- > D] to dP/dD.
#include <cuda_runtime.h>
#include <stdint.h>

#include "lsm_adjoint.cuh"
#include "lsm_common.cuh"
#include "lsm_device.cuh"
#include "lsm_evaluate.cuh"
#include "lsm_kernels.h"

namespace fo {

template <int D, int C>  // D == plan.degree
__global__ void __launch_bounds__(kEvalThreads, 4) evaluate_greeks_kernel(EvalArgs a, GreeksArgs gk) {
    extern __shared__ __align__(16) unsigned char greeks_smem_raw[];
    __shared__ double gred[32 * kGreekSlots];
    __shared__ dd gtot[kGreekSlots];
    const DevicePlan& plan = a.plan;
    const uint32_t rows = plan.rows;
    __shared__ NormalSmem<kEvalThreads> normals;
    __shared__ double red[32 * 2];
    EvalRow* rules = reinterpret_cast<EvalRow*>(greeks_smem_raw);             // [rows]
    unsigned* counts = reinterpret_cast<unsigned*>(rules + rows);       // [rows]
    unsigned* itm_counts = counts + rows;                               // [rows]
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
    double sum = 0.0, sumsq = 0.0;
    GreekSums gs;
    gs.reset();
    for (uint64_t p = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; p < P; p += uint64_t(gridDim.x) * blockDim.x) {
        bool active = true;
        double payoff = 0.0, held = 0.0;  // the payoff and the state it was taken at
        uint32_t stop_row = 0;
        PathAdjoint adj;
        adj.reset();
        auto observe = [&](int row, double spot) {
            if (!active) return;
            const EvalRow& er = rules[row];
            if (uint32_t(row) == last) {
                const double d = spot - K;
                payoff = (d > 0.0 ? d : 0.0) * er.discount;
                if (!fo_isfinite(payoff)) atomicMin(&a.status->eval_terminal_fail, (unsigned long long)p);
                active = false;
                held = spot;
                stop_row = last;
                return;
            }
            const double excess = spot - K;
            if (!(excess > 0.0)) return;
            if (decide_row<D>(plan, a.records, a.status, er.rule, uint32_t(row), p, spot, excess, itm_counts)) {
                payoff = excess * er.discount;
                if (!fo_isfinite(payoff))
                    atomicMin(&a.status->eval_fail, ((unsigned long long)row << 33) | (p << 1) | 1ull);
                active = false;
                held = spot;
                stop_row = uint32_t(row);
            }
        };
        const auto step = [&](uint32_t i, const StepCoef&, double z, double g) {
            if (active) adj.step(g, z * gk.sqrt_dt[i] - gk.sigma * gk.dt[i]);
        };
        const auto cash = [&](uint32_t at, double before, double amount) {
            if (active) adj.cash(at, before, amount);
        };
        const SimResult r = simulate_path<false, C>(plan, normals, a.keys, plan.eval_domain, uint32_t(p), observe, step, cash);
        if (r.code != 0) atomicMin(&a.status->eval_sim_fail, (unsigned long long)p);
        // The backward recurrence after the path, where its sums are not live through the path's loop.
        if (!active) {
            atomicAdd(&counts[stop_row], 1u);
            adj.stop(gs, plan.row_node[stop_row], held, payoff, rules[stop_row].discount, stop_row == last,
                     plan.policy, 1.0);
        }
        sum += payoff;
        sumsq += payoff * payoff;
    }
    // Price partials exactly as evaluate_kernel forms them.
    double acc[2] = {sum, sumsq};
    cta_reduce_to<2>(acc, red, a.partials + size_t(blockIdx.x) * 2);
    for (uint32_t r = threadIdx.x; r < rows; r += blockDim.x) {
        if (counts[r]) atomicAdd(&a.counts[r], counts[r]);
        if (itm_counts[r]) atomicAdd(&a.itm_counts[r], itm_counts[r]);
    }
    double gacc[kGreekSlots];
    gs.to_slots(gacc);
    cta_reduce_dd<kGreekSlots>(gacc, gred, gtot);
    if (threadIdx.x < kGreekSlots)
        gk.partials[size_t(blockIdx.x) * kGreekSlots + threadIdx.x] = make_double2(gtot[threadIdx.x].hi, gtot[threadIdx.x].lo);
    if (!last_cta(a.status)) return;
    finalize_price(a.partials, int(gridDim.x), P, a.result);
    // Every slot's total over the blocks in a fixed order, a warp per slot.
    for (int slot = threadIdx.x >> 5; slot < kGreekSlots; slot += kEvalThreads / 32) {
        const dd total = sum_slot<kGreekSlots>(gk.partials, int(gridDim.x), slot);
        if ((threadIdx.x & 31) == 0) gk.sums[slot] = dd_round(total);
    }
}

size_t evaluate_greeks_smem_bytes(uint32_t rows) {
    return sizeof(EvalRow) * rows + sizeof(unsigned) * 2 * rows;
}

template <int D>
static cudaError_t launch_evaluate_greeks_d(const EvalArgs& args, const GreeksArgs& greeks, int blocks,
                                            cudaStream_t stream) {
    const size_t smem = evaluate_greeks_smem_bytes(args.plan.rows);
    const auto kernel =
        args.plan.intervals <= 2 ? evaluate_greeks_kernel<D, 2> : evaluate_greeks_kernel<D, kChunkNormals>;
    const cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    if (e != cudaSuccess) return e;
    return launch_early(kernel, dim3(unsigned(blocks)), kEvalThreads, smem, stream, args, greeks);
}

cudaError_t launch_evaluate_greeks(const EvalArgs& args, const GreeksArgs& greeks, int blocks, cudaStream_t stream) {
    switch (args.plan.degree) {  // validated to 0..4 on the host
        case 0: return launch_evaluate_greeks_d<0>(args, greeks, blocks, stream);
        case 1: return launch_evaluate_greeks_d<1>(args, greeks, blocks, stream);
        case 2: return launch_evaluate_greeks_d<2>(args, greeks, blocks, stream);
        case 3: return launch_evaluate_greeks_d<3>(args, greeks, blocks, stream);
        default: return launch_evaluate_greeks_d<4>(args, greeks, blocks, stream);
    }
}

}  // namespace fo
