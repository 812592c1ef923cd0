// lsm_persistent.cu - the launch interface of the batch kernels (lsm_persistent.cuh): the instance of a
// request's degree, and the summary kernel, which has none.
#include "lsm_persistent.cuh"

namespace fo {

// The phase executor's last kernel: every problem's summary, one warp per problem, once every
// evaluation partial is written (the evaluation kernel has finished).
__global__ void __launch_bounds__(kPersistentThreads) batch_summarize_kernel(BatchArgs a, BatchQueue, uint32_t, int) {
    const uint32_t warps = kPersistentThreads / 32;
    const uint32_t i = blockIdx.x * warps + (threadIdx.x >> 5);
    if (i < a.n_problems) summarize_problem(a, i, int(threadIdx.x & 31));
}

static cudaError_t prepare_phase(int phase, const BatchArgs& a, const BatchQueue& q, int strikes, uint32_t rule_rows,
                                 bool stage, int ctas_per_sm, PersistentLaunch* out) {
    *out = PersistentLaunch{};
    const bool greeks = a.greek_partials != nullptr;
    switch (a.degree) {  // validated to 0..4 on the host
        case 0: return prepare_batch_degree<0>(phase, greeks, strikes, q, rule_rows, stage, ctas_per_sm, out);
        case 1: return prepare_batch_degree<1>(phase, greeks, strikes, q, rule_rows, stage, ctas_per_sm, out);
        case 2: return prepare_batch_degree<2>(phase, greeks, strikes, q, rule_rows, stage, ctas_per_sm, out);
        case 3: return prepare_batch_degree<3>(phase, greeks, strikes, q, rule_rows, stage, ctas_per_sm, out);
        default: return prepare_batch_degree<4>(phase, greeks, strikes, q, rule_rows, stage, ctas_per_sm, out);
    }
}

cudaError_t prepare_batch_persistent(const BatchArgs& a, const BatchQueue& q, int strikes, uint32_t rule_rows,
                                     bool stage, int ctas_per_sm, PersistentLaunch* out) {
    return prepare_phase(kPhaseAll, a, q, strikes, rule_rows, stage, ctas_per_sm, out);
}

cudaError_t prepare_batch_phases(const BatchArgs& a, const BatchQueue (&q)[3], int strikes, uint32_t rule_rows,
                                 bool stage, PersistentLaunch (&out)[kBatchPhaseLaunches]) {
    cudaError_t e = prepare_phase(kPhaseSimulate, a, q[0], strikes, rule_rows, stage, 0, &out[0]);
    if (e == cudaSuccess) e = prepare_phase(kPhaseFit, a, q[1], strikes, rule_rows, stage, 0, &out[1]);
    if (e == cudaSuccess) e = prepare_phase(kPhaseEvaluate, a, q[2], strikes, rule_rows, stage, 0, &out[3]);
    const void* const diagnose[5] = {batch_diagnose_entry<0>(), batch_diagnose_entry<1>(), batch_diagnose_entry<2>(),
                                     batch_diagnose_entry<3>(), batch_diagnose_entry<4>()};
    out[2] = PersistentLaunch{diagnose[a.degree], 0, int(a.n_problems), kDiagnoseThreads};
    const uint32_t warps = kPersistentThreads / 32;
    out[4] = PersistentLaunch{reinterpret_cast<const void*>(batch_summarize_kernel), 0,
                              int((a.n_problems + warps - 1) / warps), kPersistentThreads};
    return e;
}

cudaError_t enqueue_batch_persistent(const PersistentLaunch& launch, const BatchArgs& a, const BatchQueue& q,
                                     uint32_t rule_rows, bool stage, cudaStream_t stream) {
    if (launch.grid <= 0) return cudaSuccess;
    BatchArgs args = a;
    BatchQueue queue = q;
    uint32_t rows = rule_rows;
    int stage_rules = stage ? 1 : 0;
    void* params[4] = {&args, &queue, &rows, &stage_rules};
    return cudaLaunchKernel(launch.kernel, dim3(unsigned(launch.grid)), dim3(unsigned(launch.threads)), params, launch.smem,
                            stream);
}

}  // namespace fo
