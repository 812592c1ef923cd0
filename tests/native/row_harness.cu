// row_harness.cu - test harness: a fitted row's coefficients and rule from its response sums as the backward
// kernel forms them (lsm_row_solve.cuh), beside the rule that the evaluation forms from the recorded
// coefficients. One warp per case. Built by tests/test_gpu_row_solve.py; test infrastructure only.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../finoptions-engine_b200/csrc/lsm_row_solve.cuh"

using namespace fo;

struct RowCase {
    double mean, scale, alpha[kMaxDegree], beta[kMaxDegree], norm[kMaxColumns], strike, response[kMaxColumns];
};
struct RowResult {
    ExerciseRule rule, recorded;
    double coef[kMaxColumns];
    int32_t kind, broken, bad_responses, pad;
};

template <int D>
__global__ void __launch_bounds__(32) row_kernel(const RowCase* cases, int n, RowResult* out) {
    __shared__ RowBasis basis;
    __shared__ RowSolution row;
    __shared__ FitRecord rec;
    const int i = int(blockIdx.x), lane = int(threadIdx.x);
    if (i >= n) return;
    const RowCase& c = cases[i];
    if (lane == 0) {
        rec = FitRecord{};
        rec.kind = kRuleRegression;
        rec.model.mean = c.mean;
        rec.model.scale = c.scale;
        rec.model.inv_scale = make_divisor(c.scale).inv;
        for (int j = 0; j < kMaxDegree; ++j) {
            rec.model.alpha[j] = c.alpha[j];
            rec.model.beta[j] = c.beta[j];
        }
        for (int j = 0; j < kMaxColumns; ++j) rec.model.norm[j] = c.norm[j];
    }
    __syncwarp();
    prepare_basis<D>(rec, c.strike, 1.0, &basis);
    __syncwarp();
    solve_row<D>(basis, lane < kMaxColumns ? c.response[lane] : 0.0, false, &row);
    __syncwarp();
    if (lane != 0) return;
    RowResult& r = out[i];
    r = RowResult{};
    r.rule = row.rule;
    r.kind = row.kind;
    r.broken = row.broken;
    r.bad_responses = row.bad_responses;
    for (int j = 0; j <= D; ++j) r.coef[j] = rec.model.coef[j] = row.coef[j];
    r.recorded = make_exercise_rule(rec.model, D, c.strike);
}

extern "C" int row_bytes(int which) { return which == 0 ? int(sizeof(RowCase)) : int(sizeof(RowResult)); }

// Solves n cases of one degree (host arrays); returns 0 or the CUDA error.
extern "C" int row_solve(const void* cases, int n, int degree, void* results) {
    RowCase* d_cases = nullptr;
    RowResult* d_out = nullptr;
    cudaError_t e = cudaMalloc(&d_cases, sizeof(RowCase) * size_t(n));
    if (e == cudaSuccess) e = cudaMalloc(&d_out, sizeof(RowResult) * size_t(n));
    if (e == cudaSuccess) e = cudaMemcpy(d_cases, cases, sizeof(RowCase) * size_t(n), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        switch (degree) {
            case 0: row_kernel<0><<<n, 32>>>(d_cases, n, d_out); break;
            case 1: row_kernel<1><<<n, 32>>>(d_cases, n, d_out); break;
            case 2: row_kernel<2><<<n, 32>>>(d_cases, n, d_out); break;
            case 3: row_kernel<3><<<n, 32>>>(d_cases, n, d_out); break;
            default: row_kernel<4><<<n, 32>>>(d_cases, n, d_out); break;
        }
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(results, d_out, sizeof(RowResult) * size_t(n), cudaMemcpyDeviceToHost);
    cudaFree(d_cases);
    cudaFree(d_out);
    return int(e);
}
