// Ops::delta_scan of one prompt of zeros (tests/test_delta_rule_memory_gpu.py): what its arena holds afterwards, and the kernels it launched.
#include <cuda_runtime.h>

#include "friday/ops.h"

using namespace friday;

extern "C" __attribute__((visibility("default"))) int probe_delta_scan(int rows, int heads, int dv, long long* arena_bytes, long long* launches) {
    const int dk = 128, taps = 4;
    Ops ops(0, nullptr);
    Arena arena(nullptr);
    ops.arena = &arena;
    const int64_t channels = 2ll * dk + (int64_t)heads * dv, state = (taps - 1) * channels + (int64_t)heads * dk * dv;
    DeviceBuffer qkv(4 * (size_t)rows * channels, true), raw(4 * (size_t)rows * heads * dk, true), vec(4 * (size_t)heads * dk, true), mem(4 * (size_t)state, true);
    std::vector<int> geometry((size_t)rows + 3, 0);           // row_seq, then seq_start, seq_qlen, seq_slots
    geometry[(size_t)rows + 1] = rows;
    DeviceBuffer geo(4 * geometry.size());
    cuda_check(cudaMemcpy(geo.get(), geometry.data(), 4 * geometry.size(), cudaMemcpyHostToDevice), "cudaMemcpy");
    const int* g = geo.as<int>();
    Ops::DeltaSpec s;
    s.heads = heads;
    s.qk_heads = 1;
    s.dk = dk;
    s.dv = dv;
    s.taps = taps;
    s.per_channel = true;
    CacheView view;
    view.kind = CacheRequest::State;
    view.write = true;
    view.state = Tensor::make(mem.get(), DType::F32, {1, state});
    view.seq_slots = g + rows + 2;
    StepContext ctx;
    ctx.rows = rows;
    ctx.n_seqs = 1;
    ctx.max_q_len = rows;
    ctx.row_seq = g;
    ctx.seq_start = g + rows;
    ctx.seq_qlen = g + rows + 1;
    const long long before = ops.launches();
    ops.delta_scan(Tensor::make(qkv.get(), DType::F32, {rows, channels}), Tensor::make(raw.get(), DType::F32, {rows, (int64_t)heads * dk}),
                   Tensor::make(raw.get(), DType::F32, {rows, heads}), Tensor::make(vec.get(), DType::F32, {heads}),
                   Tensor::make(vec.get(), DType::F32, {(int64_t)heads * dk}), s, view, ctx);
    cuda_check(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
    *arena_bytes = (long long)arena.capacity();
    *launches = ops.launches() - before;
    return 0;
}
