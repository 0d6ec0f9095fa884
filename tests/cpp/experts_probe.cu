// Ops::experts_grouped on tensors that a test provides (tests/test_experts_grouped_gpu.py).
#include <cuda_runtime.h>

#include <memory>
#include <string>
#include <vector>

#include "friday/capi.h"
#include "friday/ops.h"

using namespace friday;

static std::string g_error;

#define API extern "C" __attribute__((visibility("default")))

API const char* probe_error() { return g_error.c_str(); }

// counts: a number of choices per expert, or null; out in the residual's dtype, contiguous
API int probe_experts_grouped(const FridayTensor* h, const FridayTensor* ids, const FridayTensor* weights, const FridayTensor* w_gate_up,
                              const FridayTensor* w_down, const FridayTensor* residual, const int* counts, int experts, int top, int inner, int act,
                              float limit, float slope, FridayTensor* out, long long* launches) {
    try {
        Ops ops(0, nullptr);
        Arena arena(nullptr);
        ops.arena = &arena;
        Ops::Routing r;
        r.ids = *(const Tensor*)ids;
        r.weights = *(const Tensor*)weights;
        std::vector<int> known;
        if (counts) known.assign(counts, counts + experts);
        const Tensor result = ops.experts_grouped(*(const Tensor*)h, r, *(const Tensor*)w_gate_up, *(const Tensor*)w_down, *(const Tensor*)residual, top,
                                                  inner, act, limit, slope, counts ? &known : nullptr);
        *launches = ops.launches();
        cuda_check(cudaMemcpyAsync(out->data, result.data, result.bytes(), cudaMemcpyDeviceToDevice, ops.stream()), "cudaMemcpyAsync");
        cuda_check(cudaStreamSynchronize(ops.stream()), "cudaStreamSynchronize");
        ops.check_status();
        return 0;
    } catch (const std::exception& e) {
        g_error = e.what();
        return 1;
    }
}
