"""Latent attention of bf16 prompts with so many heads that several go through one launch: whole prompts, unequal batches, portions
after a cached prefix, a prompt whose scores hold fewer than all heads at a time; and the memory that a batch takes."""

import numpy as np
import pytest
import torch

import harness
import plain_beletar as plain
import test_beletar_gpu as beletar
from friday_inference_engine_b200 import Engine

pytestmark = pytest.mark.gpu

# the projection's rows are whole 16-byte pieces (heads * (dim + rot) + rank + rot + heads columns), as many heads at once need;
# one key or value size above and one below a tile of 64
CONFIGS = {
    "heads8": beletar.config(64, 150, [beletar.latent(8, 16, 8, 24, 40, 10000.0, (4.0, 64, 8.0, 1.0))], [32]),
    "heads16": beletar.config(96, 200, [beletar.latent(16, 64, 16, 72, 24, 500.0), beletar.latent(16, 8, 8, 16, 64)], [40, None], scale=2.0),
}
_made = {}


def model(tmp_path_factory, name):
    if name not in _made:
        d = beletar.write_folder(str(tmp_path_factory.mktemp("latent_" + name)), CONFIGS[name], {}, 90 + len(_made))
        _made[name] = (d,) + plain.load(d)
    return _made[name]


def run(folder, prompts, cuts, max_ctx):
    """Every prompt's logits, the batch taken in by one step per portion."""
    eng = Engine(model_path=folder, dtype="bfloat16", max_ctx=max_ctx, max_batch=len(prompts))
    slots, got, at = [eng.alloc_slot() for _ in prompts], [[] for _ in prompts], [0] * len(prompts)
    for cut in cuts:
        part = [p[a:int(len(p) * cut)] for p, a in zip(prompts, at)]
        out = eng.step(slots, part, [list(range(len(p))) for p in part], to="host")
        first = 0
        for i, p in enumerate(part):
            got[i].append(out[first:first + len(p)])
            first += len(p)
            at[i] += len(p)
    eng.check()
    return [np.concatenate(g) for g in got]


@pytest.mark.parametrize("name", list(CONFIGS))
@pytest.mark.parametrize("lengths,cuts", [([90], [1.0]), ([300, 33, 150, 64], [1.0]), ([260, 70, 131], [0.4, 1.0]), ([1100], [1.0])])
def test_prompts_with_several_heads_at_once(tmp_path_factory, name, lengths, cuts, monkeypatch):
    folder, cfg, tensors = model(tmp_path_factory, name)
    ps = beletar.prompts(lengths, cfg["vocab"], 12)
    got = run(folder, ps, cuts, 1200)
    monkeypatch.setenv("FRIDAY_LATENT_TC", "0")          # the kernels of the one-token steps, for every row
    other = run(folder, ps, cuts, 1200)
    for i, p in enumerate(ps):
        ref = plain.forward(cfg, tensors, p)
        for k in range(len(p)):
            ok, text = harness.bf16_ok(got[i][k], ref[k], "%s, prompt %d" % (name, i), harness.BF16_WIDE)
            assert ok, "place %d: %s" % (k, text)
        # two forms in the same precision: a few roundings to bf16 (2^-9) of the same numbers apart
        apart = np.linalg.norm(got[i].astype(np.float64) - other[i]) / np.linalg.norm(other[i].astype(np.float64))
        assert apart <= 8 * 2.0 ** -9, apart


def test_a_batch_takes_the_scores_memory_of_one_prompt(tmp_path):
    """16 heads x 512 x 512 scores are 17 MB and their weights as much again: held once, not once for each of 16 prompts."""
    cfg = beletar.config(64, 100, [beletar.latent(16, 8, 8, 8, 8)], [None])
    folder = beletar.write_folder(str(tmp_path / "model"), cfg, {}, 5)
    eng = Engine(model_path=folder, dtype="bfloat16", max_ctx=512, max_batch=16)
    ps = beletar.prompts([512] * 16, 100, 3)
    slots = [eng.alloc_slot() for _ in ps]
    eng.step(slots[:1], ps[:1], [[511]], to="host")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for s in slots:
        eng.free_slot(s)
    slots = [eng.alloc_slot() for _ in ps]
    eng.step(slots, ps, [[511]] * 16, to="host")
    grown = before - torch.cuda.mem_get_info()[0]
    # 8,192 rows of 64 to 300 columns in a dozen buffers, and what arenas and the driver round up; one pair of score buffers per
    # prompt would be 537 MB
    assert grown < 250 << 20, "%d MB" % (grown >> 20)
