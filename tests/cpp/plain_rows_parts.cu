// Parts of a user's own that read 32-bit rows where they lie (tests/test_plain_rows_gpu.py): in 32 bits the rows that a part is given, and the
// normed rows that a shipped part returns to it, are plain unless it says that it takes others.
//
//   feed_forward "toy_reads_rows"    residual + W h, from h.t
//   mixer "toy_wraps_attention"      the shipped attention, whose result's norm it makes anew from the rows that it got: they must be the same
// Architectures "ToyReadsForCausalLM" and "ToyWrapsForCausalLM": Qwen2's, with that part in every layer.
#include <cuda_runtime.h>

#include "friday/config.h"
#include "friday/ops.h"
#include "friday/parts.h"

using namespace friday;

namespace {

class ReadsRows : public FeedForward {
public:
    ReadsRows(const PartSpec&, const BuildEnv& e) : FeedForward(e) { declare("w.weight", {e.width, e.width}); }
    PartOut forward(Ops& ops, const Rows& h, const Tensor& residual, const StepContext&, Norm*) override {
        return PartOut(ops.linear(Rows(h.t), tensor("w.weight"), nullptr, &residual));
    }
};

class WrapsAttention : public Mixer {
public:
    WrapsAttention(const PartSpec& s, const BuildEnv& e) : Mixer(e) { inner_ = adopt("", build<Mixer>("mixer", s.part("inner"), e)); }
    CacheRequest cache_request() const override { return inner_->cache_request(); }
    PartOut forward(Ops& ops, const Rows& h, const Tensor& residual, const StepContext& ctx, const CacheView& view, Norm* then) override {
        PartOut out = inner_->forward(ops, h, residual, ctx, view, then);
        if (out.has_normed) out.normed = Rows(out.normed.t);
        return out;
    }

private:
    Mixer* inner_;
};

PartRegistrar t1("feed_forward", "toy_reads_rows", [](const PartSpec& s, const BuildEnv& e) -> Part* { return new ReadsRows(s, e); });
PartRegistrar t2("mixer", "toy_wraps_attention", [](const PartSpec& s, const BuildEnv& e) -> Part* { return new WrapsAttention(s, e); });

ModelSpec reads_spec(const Json& typed) {
    ModelSpec spec = qwen2_spec(typed);
    spec.architecture = "ToyReadsForCausalLM";
    for (PartSpec& layer : spec.layers) layer.parts["feed_forward"] = PartSpec("toy_reads_rows", Json::object(), "toy.");
    return spec;
}

ModelSpec wraps_spec(const Json& typed) {
    ModelSpec spec = qwen2_spec(typed);
    spec.architecture = "ToyWrapsForCausalLM";
    for (PartSpec& layer : spec.layers) {
        PartSpec inner = layer.parts["mixer"];
        PartSpec wrap("toy_wraps_attention", Json::object(), inner.prefix);
        inner.prefix = "";
        wrap.parts["inner"] = inner;
        layer.parts["mixer"] = wrap;
    }
    return spec;
}

struct RegisterToys {
    RegisterToys() {
        register_architecture({"ToyReadsForCausalLM", Qwen2Config::read, reads_spec});
        register_architecture({"ToyWrapsForCausalLM", Qwen2Config::read, wraps_spec});
    }
} register_toys;

}  // namespace
