"""What this library is timed on: generation through its public entry points (Engine, Engine.step, Engine.decoder).

A case is one model, one data type and one piece of a request's life:
  "decode"    one more token for every sequence of a batch that is being generated, from the captured step (the tokens
              are given, as a caller does that samples for itself), with its logits;
  "prompt"    new sequences are taken in by one call of the step function, which returns their last tokens' logits;
  "generate"  a whole batch from its prompts to its last token: slots, prompts, the decoder's steps, slots given back.
Models are the shapes that the benchmark and the tests of this repository use, with seeded random weights; a seed
gives other weights and other tokens.  exact() states the same models in 64-bit torch, without the library.
"""
import math
import random

import torch

from friday_inference_engine_b200 import Engine

# ---------------------------------------------------------------------------
# models
# ---------------------------------------------------------------------------
# Eight of the 7B shape's 28 layers, and its whole vocabulary.  The layers are alike, and random weights let bf16 rounding
# grow with the depth: at 28 layers two correct orders of summation differ by 0.026 to 0.037 of the logits' norm, which
# would tell nothing about a fault in one of them.
QWEN25_7B = {
    "architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "num_hidden_layers": 8, "hidden_size": 3584,
    "num_attention_heads": 28, "num_key_value_heads": 4, "head_dim": 128, "intermediate_size": 18944,
    "vocab_size": 152064, "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": False,
    "use_sliding_window": False, "max_position_embeddings": 32768, "torch_dtype": "bfloat16",
}
# Two layers of the 7B shape with a short vocabulary: what the 32-bit path is checked on at full layer sizes.
QWEN25_7B_LAYERS = dict(QWEN25_7B, num_hidden_layers=2, vocab_size=5000, max_position_embeddings=4096)
# The small model with a window on every layer that the 32-bit checks run from prompt to last token.
QWEN_SMALL = {
    "architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "num_hidden_layers": 3, "hidden_size": 96,
    "num_attention_heads": 3, "num_key_value_heads": 1, "head_dim": 32, "intermediate_size": 256, "vocab_size": 1000,
    "rope_theta": 1000000.0, "rms_norm_eps": 1e-5, "tie_word_embeddings": False, "use_sliding_window": True,
    "sliding_window": 24, "max_window_layers": 0, "max_position_embeddings": 256, "torch_dtype": "bfloat16",
}


def dapozen_config(width):
    """Seven layers, every third from the second on state space duality, the others attention within runs of 2,048
    positions; a gated feed-forward in the even layers, experts by token id in the odd ones."""
    heads, kv = width // 128, width // 512
    att = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "conv": 4, "scale": 128 ** -0.5,
           "rot": {"base": 10000.0, "dims": 64}, "mask": {"size": 2048}}
    ssd = {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 2, "norm_groups": 2, "conv": 4}
    dense = {"kind": "dense", "ff": 3 * width}
    moe = {"kind": "moe", "expert": {"ff": width, "limit": 7.0}, "router": {"experts": 8, "top": 2},
           "shared": {"ff": width, "limit": 7.0}}
    layers = [{"type": "mamba2" if i % 3 == 1 else "attention", "mixer": ssd if i % 3 == 1 else att,
               "mlp": dense if i % 2 == 0 else moe} for i in range(7)]
    return {"architecture": "Dapozen", "vocab": 32768, "width": width, "embedding": {"scale": 12.0},
            "norm": {"eps": 1e-6}, "layers": layers, "logit_softcap": 25.0}


def beletar_config(width):
    """Attention over a latent of 512, two delta-rule layers, one with a decay per key channel; a gated feed-forward
    everywhere; the last three layers run twice."""
    heads = width // 128
    latent = {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5,
              "rot": {"base": 10000.0, "dims": 64,
                      "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    delta = {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "conv": 4}
    kinds = [("latent_attention", latent), ("delta", delta), ("delta", delta),
             ("channel_delta", dict(delta, decay_rank=64, gate_rank=64))]
    layers = [{"type": kind, "mixer": mixer, "mlp": {"kind": "dense", "ff": 3 * width}} for kind, mixer in kinds]
    return {"architecture": "Beletar", "vocab": 32768, "width": width, "norm": {"eps": 1e-5},
            "embedding": {"scale": 1.0}, "layers": layers, "loop": {"start": 1, "stop": 4, "times": 2}}


def config_of(case):
    model = case["model"]
    if model == "dapozen":
        return dapozen_config(case["width"])
    if model == "beletar":
        return beletar_config(case["width"])
    return {"qwen7b": QWEN25_7B, "qwen7b_layers": QWEN25_7B_LAYERS, "qwen_small": QWEN_SMALL}[model]


def vocab_of(cfg):
    return cfg["vocab_size"] if "vocab_size" in cfg else cfg["vocab"]


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def qwen(what, batch, shortest, longest, new=0, model="qwen7b", dtype="bfloat16"):
    return {"model": model, "dtype": dtype, "what": what, "batch": batch, "shortest": shortest, "longest": longest,
            "new": new}


def hybrid(model, width, what, batch, shortest, longest, new=0):
    return dict(qwen(what, batch, shortest, longest, new, model), width=width)


def listed():
    return [
        # one user's chat: the latency of a token, bound by reading every weight once
        dict(qwen("decode", 1, 1024, 1024), name="qwen7b_decode_1"),
        # the benchmark's headline: a small batch in generation
        dict(qwen("decode", 8, 1024, 1024), name="qwen7b_decode_8"),
        # a busy server's batch
        dict(qwen("decode", 64, 1024, 1024), name="qwen7b_decode_64"),
        # long documents in generation: attention reads gigabytes of keys and values beside the weights
        dict(qwen("decode", 8, 8000, 8000), name="qwen7b_decode_8_long"),
        # a short question, no multiple of any tile: time to first token
        dict(qwen("prompt", 1, 100, 100), name="qwen7b_prompt_100"),
        # the benchmark's prompt
        dict(qwen("prompt", 1, 2048, 2048), name="qwen7b_prompt_2048"),
        # a batch of requests that start together with unequal lengths
        dict(qwen("prompt", 16, 64, 2048), name="qwen7b_prompts_16_unequal"),
        # the smallest model and the 32-bit path, where launches count: a replayed trace or a test's generation
        dict(qwen("generate", 4, 1, 64, 16, "qwen_small", "float32"), name="qwen_small_float32_generate"),
        # the 32-bit path at full layer sizes: checking a model's logits
        dict(qwen("prompt", 2, 33, 300, 0, "qwen7b_layers", "float32"), name="qwen7b_layers_float32_prompt"),
        # hybrid designs: a long prompt, and whole requests of a batch
        dict(hybrid("dapozen", 2048, "prompt", 1, 2048, 2048), name="dapozen_prompt_2048"),
        dict(hybrid("dapozen", 2048, "generate", 8, 64, 512, 16), name="dapozen_generate_8"),
        dict(hybrid("beletar", 2048, "generate", 8, 64, 512, 16), name="beletar_generate_8"),
    ]


def spread(rng, low, high):
    """A whole number of [low, high], even over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "float32", "dapozen", "beletar"])
    if kind == "decode":
        batch = spread(rng, 1, 64)
        longest = spread(rng, 65, min(8000, 65536 // batch))
        return qwen("decode", batch, max(64, longest // rng.randint(1, 3)), longest)
    if kind == "prompt":
        batch = spread(rng, 1, 16)
        longest = spread(rng, 65, min(2048, 18000 // batch))
        return qwen("prompt", batch, rng.randint(1, longest), longest)
    if kind == "float32":
        if rng.random() < 0.5:
            return qwen("generate", rng.randint(1, 8), 1, rng.randint(2, 128), rng.randint(1, 24), "qwen_small", "float32")
        return qwen("prompt", rng.randint(1, 4), 1, spread(rng, 16, 300), 0, "qwen7b_layers", "float32")
    width = rng.choice([1024, 2048])
    if rng.random() < 0.5:
        longest = spread(rng, 64, 2048)
        return hybrid(kind, width, "prompt", 1, longest, longest)
    return hybrid(kind, width, "generate", rng.randint(1, 8), rng.randint(1, 64), rng.randint(65, 512), rng.randint(2, 16))


def lengths_of(case):
    """The prompts' lengths: the longest and the shortest, the others between them, in no order."""
    n, low, high = case["batch"], case["shortest"], case["longest"]
    rng = random.Random(3 + 7 * n + 31 * low + 101 * high)
    lens = [high, low][:n] + [rng.randint(low, high) for _ in range(n - 2)]
    rng.shuffle(lens)
    return lens


WARM = 3            # steps that a decoder has done when a "decode" pass begins: it runs from its captured step by then
ROOM = 2048         # tokens that "decode" passes may add to a sequence


def sequences_of(case, seed):
    """Every sequence's tokens: its prompt and all that follow it in the first pass."""
    g = torch.Generator().manual_seed(1000003 * (seed + 1))
    more = WARM + 1 if case["what"] == "decode" else case["new"]
    vocab = vocab_of(config_of(case))
    return [torch.randint(0, vocab, (n + more,), generator=g).tolist() for n in lengths_of(case)]


def taken_in(eng, prompts, group=8):
    """Slots that hold the prompts."""
    slots = [eng.alloc_slot() for _ in prompts]
    for lo in range(0, len(prompts), group):
        part = slots[lo:lo + group]
        eng.step(part, prompts[lo:lo + group], [[]] * len(part))
    return slots


def prepare(case, seed):
    lens = lengths_of(case)
    longest = max(lens)
    room = ROOM if case["what"] == "decode" else case["new"] + 8
    pages = sum((n + room + 63) // 64 + 1 for n in lens)
    eng = Engine(config=config_of(case), seed=seed, dtype=case["dtype"], max_ctx=min(longest + room, 16384),
                 max_batch=case["batch"], max_tokens=64 * pages)
    seqs = sequences_of(case, seed)
    prompts = [s[:n] for s, n in zip(seqs, lens)]
    state = {"engine": eng, "what": case["what"], "prompts": prompts}
    if case["what"] == "decode":
        state["slots"] = taken_in(eng, prompts)
        state["decoder"] = eng.decoder(state["slots"], [s[n] for s, n in zip(seqs, lens)])
        for k in range(WARM):
            state["decoder"].step([s[n + k] for s, n in zip(seqs, lens)])
        state["tokens"] = [s[n + WARM] for s, n in zip(seqs, lens)]
    elif case["what"] == "generate":
        state["steps"] = [[s[n + k] for s, n in zip(seqs, lens)] for k in range(case["new"])]
    return state


def run(state):
    eng, what = state["engine"], state["what"]
    if what == "decode":
        state["decoder"].step(state["tokens"])
        return [state["decoder"].logits]
    prompts = state["prompts"]
    slots = [eng.alloc_slot() for _ in prompts]
    logits = eng.step(slots, prompts, [[len(p) - 1] for p in prompts])
    outputs = [logits]
    if what == "generate":
        decoder = eng.decoder(slots, state["steps"][0])
        for tokens in state["steps"]:
            decoder.step(tokens)
            outputs.append(decoder.logits)
        decoder.close()
    for slot in slots:
        eng.free_slot(slot)
    return outputs


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def seen_keys(first, last, window=None, run_size=None):
    """Sum over the positions first .. last - 1 of the keys that each one sees, itself included."""
    if run_size:
        return sum(p % run_size + 1 for p in range(first, last))
    if window:
        return sum(min(p + 1, window) for p in range(first, last))
    return (last * (last + 1) - first * (first + 1)) // 2


def model_work(cfg, dtype, spans, wanted):
    """(bytes, flops) of one call of the model: `spans` has each sequence's (first new position, end); `wanted` rows of
    logits.  Weights are read once, cached rows once, new rows and states written once."""
    size = 4 if dtype == "float32" else 2
    rows, batch = sum(e - f for f, e in spans), len(spans)
    width, vocab = cfg.get("hidden_size") or cfg["width"], vocab_of(cfg)
    weights = vocab * width
    move = 4 * wanted * vocab + size * rows * width
    flops = 2 * wanted * vocab * width
    if "hidden_size" in cfg:
        hd, inner = cfg["head_dim"], cfg["intermediate_size"]
        qd, kvd, n = cfg["num_attention_heads"] * hd, cfg["num_key_value_heads"] * hd, cfg["num_hidden_layers"]
        window = cfg["sliding_window"] if cfg["use_sliding_window"] else None
        matrices = (qd + 2 * kvd) * width + width * qd + 3 * inner * width
        weights += n * matrices
        flops += n * (2 * rows * matrices + 4 * qd * sum(seen_keys(f, e, window) for f, e in spans))
        move += n * 2 * kvd * size * sum(min(e, (window or e) + e - f) for f, e in spans)
        return weights * size + move, flops
    runs = run_order(cfg)
    counted = set()
    for i, _ in runs:
        m, mlp = cfg["layers"][i]["mixer"], cfg["layers"][i]["mlp"]
        heads, kind = m["heads"], cfg["layers"][i]["type"]
        if kind == "attention":
            d, dv, groups = m["dim"], m["vdim"], m["kv_heads"]
            mat = (heads * d + groups * (d + dv) + 2 * heads * dv) * width
            size_run = m["mask"]["size"]
            flops += 2 * heads * (d + dv) * sum(seen_keys(f, e, None, size_run) for f, e in spans)
            move += groups * (d + dv) * size * sum(min(e, (e - 1) % size_run + 1 + e - f) for f, e in spans)
            move += batch * 8 * (m["conv"] - 1) * (heads * d + groups * (d + dv))
        elif kind == "mamba2":
            inner, gn = heads * m["vdim"], m["groups"] * m["state"]
            mat = (2 * inner + 2 * gn + heads) * width + width * inner
            flops += 4 * rows * heads * m["state"] * m["vdim"]
            move += batch * 8 * (heads * m["state"] * m["vdim"] + (m["conv"] - 1) * (inner + 2 * gn))
        elif kind == "latent_attention":
            d, rd, dv, rank = m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            mat = (heads * (d + rd) + rank + rd + heads) * width + heads * (d + dv) * rank + width * heads * dv
            flops += 2 * heads * (d + rd + dv) * sum(seen_keys(f, e) for f, e in spans)
            move += (rank + rd) * size * sum(e for _, e in spans)
        else:
            groups, dk, dv = m["kv_heads"], m["dim"], m["vdim"]
            mat = (2 * groups * dk + heads * dv) * width + heads * width + width * heads * dv
            if kind == "channel_delta":
                mat += m["decay_rank"] * (width + heads * dk) + m["gate_rank"] * (width + heads * dv)
            else:
                mat += heads * width + heads * dv * width
            flops += 7 * rows * heads * dk * dv
            move += batch * 8 * (heads * dk * dv + (m["conv"] - 1) * (2 * groups * dk + heads * dv))
        used = 3 * mlp.get("ff", 0) * width
        read = used
        if mlp["kind"] == "moe":
            n, top, one = mlp["router"]["experts"], mlp["router"]["top"], 3 * mlp["expert"]["ff"] * width
            shared = 3 * mlp["shared"]["ff"] * width
            used, read = shared + top * one, shared + n * (1.0 - (1.0 - top / n) ** rows) * one
        flops += 2 * rows * (mat + used)
        if i not in counted:                 # a layer that runs twice need not be read twice by a large enough cache
            counted.add(i)
            weights += mat + read
    return weights * size + move, flops


def work(case):
    cfg, lens, dtype = config_of(case), lengths_of(case), case["dtype"]
    if case["what"] == "decode":
        total = [model_work(cfg, dtype, [(n + WARM, n + WARM + 1) for n in lens], len(lens))]
    else:
        total = [model_work(cfg, dtype, [(0, n) for n in lens], len(lens))]
        total += [model_work(cfg, dtype, [(n + k, n + k + 1) for n in lens], len(lens)) for k in range(case["new"])]
    return {"bytes": float(sum(b for b, _ in total)), "flops": float(sum(f for _, f in total))}


def tolerance(case):
    if case["dtype"] == "float32":
        # 3.5e-7 off the 64-bit values at the small model, 6.4e-6 where 18,944 terms are summed
        return {"rel": 2.5e-5, "max": 2.5e-4}
    if case["model"] == "qwen7b":
        # other splits of sums, other tiles and norms rounded by themselves: 0.011 to 0.019 from one another (largest 0.09)
        return {"rel": 0.03, "max": 0.35}
    # the same changes: 0.0063 (largest 0.03)
    return {"rel": 0.025, "max": 0.12}


# ---------------------------------------------------------------------------
# the models in 64 bits
# ---------------------------------------------------------------------------
MASK = 0xFFFFFFFF


def stream_key(seed, name):
    """The random weights' stream of a tensor: FNV-1a over the seed's bytes, a zero byte and the name, then a finalizer."""
    m = (1 << 64) - 1
    h = 1469598103934665603
    for b in int(seed).to_bytes(8, "little") + b"\0" + name.encode():
        h = ((h ^ b) * 1099511628211) & m
    h ^= h >> 30
    h = (h * 0xBF58476D1CE4E5B9) & m
    h ^= h >> 27
    h = (h * 0x94D049BB133111EB) & m
    return h ^ (h >> 31)


def philox(low, key):
    """The first two words of Philox-4x32-10 for counters (low, 0, 0, 0), `low` an int64 tensor below 2^32."""
    c0, c1, c2, c3 = low, torch.zeros_like(low), torch.zeros_like(low), torch.zeros_like(low)
    k0, k1 = key & MASK, key >> 32
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = ((p1 >> 32) & MASK) ^ c1 ^ k0, p1 & MASK, ((p0 >> 32) & MASK) ^ c3 ^ k1, p0 & MASK
        k0, k1 = (k0 + 0x9E3779B9) & MASK, (k1 + 0xBB67AE85) & MASK
    return c0, c1


class Weights:
    """The seeded tensors by name, made when they are asked for, in 64 bits (stored as bf16, as a checkpoint has them)."""

    def __init__(self, seed, prefix=""):
        self.seed, self.prefix = seed, prefix

    def sub(self, prefix):
        return Weights(self.seed, self.prefix + prefix)

    def __call__(self, name, *shape, mean=0.0):
        n = math.prod(shape)
        key = stream_key(self.seed, self.prefix + name)
        out = torch.empty((n + 1) // 2 * 2, dtype=torch.float64, device="cuda")
        step = 1 << 25
        for lo in range(0, (n + 1) // 2, step):
            pair = torch.arange(lo, min(lo + step, (n + 1) // 2), device="cuda")
            c0, c1 = philox(pair, key)
            r = torch.sqrt(-2.0 * torch.log(((c0 >> 8).double() + 0.5) / 16777216.0))
            a = (2.0 * math.pi) * ((c1 >> 8).double() / 16777216.0)
            z = torch.stack([r * torch.cos(a), r * torch.sin(a)], dim=1).reshape(-1).float()
            z = z * torch.tensor(0.02, dtype=torch.float32, device="cuda") + mean
            out[2 * lo:2 * lo + z.numel()] = z.bfloat16().double()
        return out[:n].reshape(shape)

    def ids(self, name, rows, cols, below):
        c0, _ = philox(torch.arange(rows, device="cuda"), stream_key(self.seed, self.prefix + name))
        return ((c0 >> 1)[:, None] + torch.arange(cols, device="cuda")) % below


def run_order(cfg):
    """(layer, whether the embedding is added before it) in the order in which the layers run."""
    n, loop = len(cfg["layers"]), cfg.get("loop")
    if not loop:
        return [(i, False) for i in range(n)]
    a, b = loop["start"], loop["stop"]
    span = [(i, t > 0 and i == a) for t in range(loop["times"]) for i in range(a, b)]
    return [(i, False) for i in range(a)] + span + [(i, False) for i in range(b, n)]


def unit_rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def layer_norm(x, w, b, eps):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w + b


def softmax_attention(q, k, v, scale, window=None, run_size=None, sink=None):
    """Causal attention of one sequence: q [T, heads, d], k [T, groups, d], v [T, groups, dv]; a query sees the last
    `window` keys, or those of its own run of positions; `sink` [heads] joins the denominator."""
    T, heads, _ = q.shape
    share = heads // k.shape[1]
    out = torch.empty(T, heads, v.shape[2], dtype=q.dtype, device=q.device)
    place = torch.arange(T, device=q.device)
    for lo in range(0, T, 1024):
        rows = place[lo:lo + 1024, None]
        hidden = place > rows
        if window:
            hidden |= place <= rows - window
        if run_size:
            hidden |= place < rows // run_size * run_size
        for g in range(k.shape[1]):
            s = torch.einsum("thd,kd->htk", q[lo:lo + 1024, g * share:(g + 1) * share], k[:, g]) * scale
            s = s.masked_fill(hidden, -math.inf)
            if sink is not None:
                extra = sink[g * share:(g + 1) * share, None, None].expand(-1, s.shape[1], 1)
                s = torch.cat([s, extra], dim=-1)
            p = torch.softmax(s, dim=-1)[..., :T]
            out[lo:lo + 1024, g * share:(g + 1) * share] = torch.einsum("htk,kd->thd", p, v[:, g])
    return out


def rotate_pairs(x, rot):
    """x [T, heads, d]: dimensions 2i and 2i + 1 among the first `dims` turn by position * frequency."""
    dims, base = rot["dims"], rot["base"]
    i = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
    f, mult = base ** (-2.0 * i / dims), 1.0
    if rot.get("scaling"):
        sc = rot["scaling"]

        def turn_dim(turns):
            return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        low, high = max(math.floor(turn_dim(sc["fast"])), 0), min(math.ceil(turn_dim(sc["slow"])), dims - 1)
        ramp = ((i - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
        f, mult = f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None, None] * f
    c, s = torch.cos(a) * mult, torch.sin(a) * mult
    out = x.clone()
    u, w = x[..., 0:dims:2], x[..., 1:dims:2]
    out[..., 0:dims:2], out[..., 1:dims:2] = u * c - w * s, w * c + u * s
    return out


def causal_conv(x, taps):
    """y_t = sum_j taps[:, j] x_(t - n + 1 + j); zeros before the start.  x [T, channels]."""
    n = taps.shape[1]
    padded = torch.cat([torch.zeros(n - 1, x.shape[1], dtype=x.dtype, device=x.device), x])
    return sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(n))


def silu(x):
    return x * torch.sigmoid(x)


def per_sequence(f, x, bounds):
    """f over each sequence's rows of x (or of several tensors), results under one another."""
    xs = x if isinstance(x, tuple) else (x,)
    return torch.cat([f(*(t[a:b] for t in xs)) for a, b in bounds])


def qwen_rows(cfg, W, tokens, bounds):
    width, eps, hd = cfg["hidden_size"], cfg["rms_norm_eps"], cfg["head_dim"]
    nq, nkv, inner = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["intermediate_size"]
    window = cfg["sliding_window"] if cfg["use_sliding_window"] else None
    # angles are 32-bit by the model's definition: float(position) / theta^(2i / d)
    denom = torch.tensor([cfg["rope_theta"]], dtype=torch.float32) ** (2.0 * torch.arange(hd // 2, dtype=torch.float32) / hd)

    def rope(x):
        a = (torch.arange(x.shape[0], dtype=torch.float32)[:, None] / denom).cuda().double()[:, None]
        u, w = x[..., :hd // 2], x[..., hd // 2:]
        return torch.cat([u * torch.cos(a) - w * torch.sin(a), u * torch.sin(a) + w * torch.cos(a)], dim=-1)

    def attend(q, k, v):
        q, k, v = (t.reshape(t.shape[0], -1, hd) for t in (q, k, v))
        return softmax_attention(rope(q), rope(k), v, hd ** -0.5, window).reshape(q.shape[0], -1)

    x = W("model.embed_tokens.weight", cfg["vocab_size"], width)[tokens]
    for i in range(cfg["num_hidden_layers"]):
        L = W.sub("model.layers.%d." % i)
        n = unit_rms(x, eps) * L("input_layernorm.weight", width, mean=1.0)
        q, k, v = (n @ L("self_attn.%s_proj.weight" % c, h * hd, width).T + L("self_attn.%s_proj.bias" % c, h * hd)
                   for c, h in (("q", nq), ("k", nkv), ("v", nkv)))
        x = x + per_sequence(attend, (q, k, v), bounds) @ L("self_attn.o_proj.weight", width, nq * hd).T
        n = unit_rms(x, eps) * L("post_attention_layernorm.weight", width, mean=1.0)
        for a in range(0, n.shape[0], 4096):
            part = n[a:a + 4096]
            act = silu(part @ L("mlp.gate_proj.weight", inner, width).T) * (part @ L("mlp.up_proj.weight", inner, width).T)
            x[a:a + 4096] += act @ L("mlp.down_proj.weight", width, inner).T
    return unit_rms(x, eps) * W("model.norm.weight", width, mean=1.0), W("lm_head.weight", cfg["vocab_size"], width)


def dapozen_rows(cfg, W, tokens, bounds):
    width, eps = cfg["width"], cfg["norm"]["eps"]

    def attention(h, m, L):
        heads, groups, d = m["heads"], m["kv_heads"], m["dim"]

        def projected(part, name, n):
            return causal_conv(part @ L(name, n * d, width).T + L(name + ".b", n * d), L(name + ".conv", n * d, m["conv"]))

        def mix(part):
            T = part.shape[0]
            q = unit_rms(rotate_pairs(projected(part, "q", heads).reshape(T, heads, d), m["rot"]), eps)
            k = unit_rms(rotate_pairs(projected(part, "k", groups).reshape(T, groups, d), m["rot"]), eps)
            v = projected(part, "v", groups).reshape(T, groups, d)
            return softmax_attention(q, k, v, m["scale"], run_size=m["mask"]["size"]).reshape(T, -1)
        return (per_sequence(mix, h, bounds) * torch.sigmoid(h @ L("g", heads * d, width).T)) @ L("o", width, heads * d).T

    def mamba2(h, m, L):
        heads, dv, n, groups = m["heads"], m["vdim"], m["state"], m["groups"]
        inner, gn = heads * dv, groups * n
        taps, tap_bias = L("conv", inner + 2 * gn, m["conv"]), L("conv.b", inner + 2 * gn)
        dt_bias, rate, skip = L("dt_bias", heads), torch.exp(L("A_log", heads)), L("D", heads)
        p = h @ L("in", 2 * inner + 2 * gn + heads, width).T

        def mix(part):
            T = part.shape[0]
            xbc = silu(causal_conv(part[:, inner:2 * inner + 2 * gn], taps) + tap_bias)
            x = xbc[:, :inner].reshape(T, heads, dv)
            B, C = xbc[:, inner:inner + gn].reshape(T, groups, n), xbc[:, inner + gn:].reshape(T, groups, n)
            dt = torch.nn.functional.softplus(part[:, 2 * inner + 2 * gn:] + dt_bias)
            fall = torch.cumsum(dt * rate, dim=0)                      # minus the logarithm of the decay since the start
            y = skip[:, None] * x
            for g in range(groups):
                pair = C[:, g] @ B[:, g].T
                for a in range(g * heads // groups, (g + 1) * heads // groups):
                    keep = torch.exp((fall[None, :, a] - fall[:, None, a]).tril()).tril()
                    y[:, a] += (pair * keep * dt[None, :, a]) @ x[:, a]
            return y.reshape(T, inner)
        y = per_sequence(mix, p, bounds) * silu(p[:, :inner])
        y = unit_rms(y.reshape(-1, m["norm_groups"], inner // m["norm_groups"]), eps).reshape(-1, inner)
        return (y * L("norm", inner, mean=1.0)) @ L("o", width, inner).T

    def clipped(h, F, ff, limit):
        g = (h @ F("gate", ff, width).T).clamp(max=limit)
        u = (h @ F("up", ff, width).T).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ F("down", width, ff).T

    def feed_forward(h, mlp, F):
        if mlp["kind"] == "dense":
            ff = mlp["ff"]
            return (silu(h @ F("gate", ff, width).T) * (h @ F("up", ff, width).T)) @ F("down", width, ff).T
        n, top = mlp["router"]["experts"], mlp["router"]["top"]
        chosen = F.ids("table", cfg["vocab"], top, n)[tokens]
        out = clipped(h, F.sub("shared."), mlp["shared"]["ff"], mlp["shared"]["limit"])
        for e in range(n):
            rows = (chosen == e).any(-1).nonzero()[:, 0]
            if rows.numel():
                out[rows] += clipped(h[rows], F.sub("e%d." % e), mlp["expert"]["ff"], mlp["expert"]["limit"]) / top
        return out

    x = W("embed", cfg["vocab"], width)[tokens] * cfg["embedding"]["scale"]
    for i, _ in run_order(cfg):
        layer, L = cfg["layers"][i], W.sub("l%d." % i)
        h = unit_rms(x, eps) * L("norm1", width, mean=1.0)
        y = (attention if layer["type"] == "attention" else mamba2)(h, layer["mixer"], L.sub("mix."))
        x = x + unit_rms(y, eps) * L("norm1b", width, mean=1.0)
        y = feed_forward(unit_rms(x, eps) * L("norm2", width, mean=1.0), layer["mlp"], L.sub("mlp."))
        x = x + unit_rms(y, eps) * L("norm2b", width, mean=1.0)
    return unit_rms(x, eps) * W("final.norm", width, mean=1.0), W("head", cfg["vocab"], width)


def beletar_rows(cfg, W, tokens, bounds):
    width, eps = cfg["width"], cfg["norm"]["eps"]

    def latent_attention(h, m, L):
        heads, d, rd, dv, rank = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        q, low = h @ L("q", heads * (d + rd), width).T, h @ L("dkv", rank + rd, width).T
        c = unit_rms(low[:, :rank], eps) * L("dkv.norm", rank, mean=1.0)
        k, v = c @ L("uk", heads * d, rank).T, c @ L("uv", heads * dv, rank).T
        sink = L("sink", heads)

        def mix(q, k, v, turned):
            T = q.shape[0]
            q, k, v = q.reshape(T, heads, d + rd), k.reshape(T, heads, d), v.reshape(T, heads, dv)
            turned = rotate_pairs(turned.reshape(T, 1, rd), m["rot"]).expand(T, heads, rd)
            q = torch.cat([q[..., :d], rotate_pairs(q[..., d:], m["rot"])], dim=-1)
            return softmax_attention(q, torch.cat([k, turned], dim=-1), v, m["scale"], sink=sink).reshape(T, -1)
        out = per_sequence(mix, (q, k, v, low[:, rank:]), bounds)
        gate = torch.sigmoid(h @ L("g", heads, width).T)
        return (out.reshape(-1, heads, dv) * gate[:, :, None]).reshape(-1, heads * dv) @ L("o", width, heads * dv).T

    def delta(h, m, L, per_channel):
        heads, groups, dk, dv, taps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]
        rows = h.shape[0]

        def short(name, n):
            w, t = L(name, n, width), L(name + ".conv", n, taps)
            return per_sequence(lambda part: silu(causal_conv(part @ w.T, t)), h, bounds)

        def unit(x):
            x = x.reshape(rows, groups, dk)
            x = x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
            return x.repeat_interleave(heads // groups, dim=1)
        q, k = unit(short("q", groups * dk)) * dk ** -0.5, unit(short("k", groups * dk))
        v = short("v", heads * dv).reshape(rows, heads, dv)
        beta, rate = torch.sigmoid(h @ L("b", heads, width).T), torch.exp(L("A_log", heads))
        if per_channel:
            raw = (h @ L("a1", m["decay_rank"], width).T) @ L("a2", heads * dk, m["decay_rank"]).T + L("dt_bias", heads * dk)
            decay = torch.exp(-rate[:, None] * torch.nn.functional.softplus(raw).reshape(rows, heads, dk))
            gate = torch.sigmoid((h @ L("g1", m["gate_rank"], width).T) @ L("g2", heads * dv, m["gate_rank"]).T)
        else:
            raw = h @ L("a", heads, width).T + L("dt_bias", heads)
            decay = torch.exp(-rate * torch.nn.functional.softplus(raw))[:, :, None].expand(rows, heads, dk)
            gate = silu(h @ L("g", heads * dv, width).T)
        # all sequences side by side, one token of each at a time
        n = len(bounds)
        first = torch.tensor([a for a, _ in bounds], device="cuda")
        length = torch.tensor([b - a for a, b in bounds], device="cuda")
        S = torch.zeros(n, heads, dk, dv, dtype=torch.float64, device="cuda")
        o = torch.zeros(rows, heads, dv, dtype=torch.float64, device="cuda")
        for t in range(int(length.max())):
            at = first + torch.minimum(length - 1, torch.full_like(length, t))     # a finished sequence: not kept below
            S = S * decay[at][..., None]
            u = beta[at][..., None] * (v[at] - torch.einsum("nhkv,nhk->nhv", S, k[at]))
            S = S + k[at][..., None] * u[:, :, None, :]
            live = t < length
            o[at[live]] = torch.einsum("nhkv,nhk->nhv", S, q[at])[live]
        o = unit_rms(o, eps) * L("norm", dv, mean=1.0)
        return (o.reshape(rows, heads * dv) * gate) @ L("o", width, heads * dv).T

    table = W("embed", cfg["vocab"], width)
    start = table[tokens] * cfg["embedding"]["scale"]
    x = start
    for i, again in run_order(cfg):
        layer, L = cfg["layers"][i], W.sub("l%d." % i)
        x = x + start if again else x
        h = layer_norm(x, L("norm1", width, mean=1.0), L("norm1.b", width), eps)
        if layer["type"] == "latent_attention":
            x = x + latent_attention(h, layer["mixer"], L.sub("mix."))
        else:
            x = x + delta(h, layer["mixer"], L.sub("mix."), layer["type"] == "channel_delta")
        h, ff = layer_norm(x, L("norm2", width, mean=1.0), L("norm2.b", width), eps), layer["mlp"]["ff"]
        F = L.sub("mlp.")
        x = x + (silu(h @ F("gate", ff, width).T) * (h @ F("up", ff, width).T)) @ F("down", width, ff).T
    return layer_norm(x, W("final.norm", width, mean=1.0), W("final.norm.b", width), eps), table


def exact(case, seed):
    cfg, lens = config_of(case), lengths_of(case)
    seqs = sequences_of(case, seed)
    bounds, at = [], 0
    for s in seqs:
        bounds.append((at, at + len(s)))
        at += len(s)
    tokens = torch.tensor([t for s in seqs for t in s], device="cuda")
    rows = {"dapozen": dapozen_rows, "beletar": beletar_rows}.get(case["model"], qwen_rows)
    h, head = rows(cfg, Weights(seed), tokens, bounds)

    def logits(places):
        z = h[torch.tensor([a + p for (a, _), p in zip(bounds, places)], device="cuda")] @ head.T
        cap = cfg.get("logit_softcap")
        return cap * torch.tanh(z / cap) if cap else z
    if case["what"] == "decode":
        return [logits([n + WARM for n in lens])]
    return [logits([n - 1 + k for n in lens]) for k in range(case["new"] + 1)]
