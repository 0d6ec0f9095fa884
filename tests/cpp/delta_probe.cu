// Ops::delta_step_ok for a step of one token per sequence (tests/test_delta_rule_gpu.py); nothing is launched.
#include <cuda_runtime.h>

#include "friday/ops.h"

using namespace friday;

extern "C" __attribute__((visibility("default"))) int probe_delta_step_ok(int heads, int qk_heads, int dk, int dv, int taps, int decode, int write) {
    Ops ops(0, nullptr);
    const int64_t channels = 2ll * qk_heads * dk + (int64_t)heads * dv;
    DeviceBuffer memory(4 * (size_t)((taps - 1) * channels + (int64_t)heads * dk * dv));
    Ops::DeltaSpec s;
    s.heads = heads;
    s.qk_heads = qk_heads;
    s.dk = dk;
    s.dv = dv;
    s.taps = taps;
    CacheView view;
    view.kind = CacheRequest::State;
    view.write = write != 0;
    view.state = Tensor::make(memory.get(), DType::F32, {1, (int64_t)(memory.bytes() / 4)});
    StepContext ctx;
    ctx.decode = decode != 0;
    ctx.n_seqs = 1;
    const Tensor rows = Tensor::make(memory.get(), DType::BF16, {1, channels}), raw = Tensor::make(memory.get(), DType::F32, {1, (int64_t)heads});
    return ops.delta_step_ok(rows, raw, rows, s, view, ctx) ? 1 : 0;
}
