"""32-bit rows that parts of a user's own read where they lie: normed, whether few rows (whose norm shipped parts leave to one another) or many."""
import os

import pytest
import torch

from friday_inference_engine_b200 import Engine, build_plugin, load_plugin

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
CONFIG = {"model_type": "qwen2", "num_hidden_layers": 3, "hidden_size": 96, "num_attention_heads": 3, "num_key_value_heads": 1, "head_dim": 32,
          "intermediate_size": 256, "vocab_size": 200, "rope_theta": 10000.0, "rms_norm_eps": 1e-5, "tie_word_embeddings": False,
          "use_sliding_window": False, "max_position_embeddings": 128, "torch_dtype": "float32"}


@pytest.fixture(scope="module")
def plugin(tmp_path_factory):
    load_plugin(build_plugin(os.path.join(HERE, "cpp", "plain_rows_parts.cu"), str(tmp_path_factory.mktemp("plugin") / "libplain_rows.so")))


@pytest.mark.parametrize("architecture", ["ToyReadsForCausalLM", "ToyWrapsForCausalLM", "Qwen2ForCausalLM"])
def test_few_rows_and_many_see_the_same_rows(plugin, architecture):
    eng = Engine(config=dict(CONFIG, architectures=[architecture]), seed=3, dtype="float32", max_ctx=64, max_batch=2)
    tokens = [int(t) for t in torch.randint(0, 200, (40,), generator=torch.Generator().manual_seed(1))]
    many, few = eng.alloc_slot(), eng.alloc_slot()
    all_at_once = torch.as_tensor(eng.step([many], [tokens], [list(range(40))])).double()
    in_fives = torch.cat([torch.as_tensor(eng.step([few], [tokens[a:a + 5]], [list(range(5))])).double() for a in range(0, 40, 5)])
    # fp32 sums in other orders: some 2^-20 of the rows' size, where a norm that is missing changes them as a whole
    assert (in_fives.cpu() - all_at_once.cpu()).norm() <= 2.0 ** -16 * all_at_once.cpu().norm()
