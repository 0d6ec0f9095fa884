"""Which form a prompt's rows take through the experts where nothing is forced: many experts per choice (more than 16 per choice,
where the dense form is no choice) run over gathered rows from 33 rows on, also below 256; others in the dense form up to 256 rows."""
import copy

import numpy as np
import pytest

import dapozen_models as models
import plain_dapozen as plain
import test_dapozen_gpu as dapozen
from friday_inference_engine_b200 import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("experts,top,form", [(40, 2, "grouped"), (20, 1, "grouped"), (8, 2, "dense")])
def test_default_form(tmp_path, experts, top, form, monkeypatch):
    cfg = copy.deepcopy(models.CONFIGS["R"])
    for layer in cfg["layers"]:
        if layer["mlp"] and layer["mlp"]["kind"] == "moe":
            layer["mlp"]["router"] = {"experts": experts, "top": top}
    folder = models.write_folder(str(tmp_path / "model"), cfg, models.tensors_of(cfg, np.random.default_rng(31)))
    loaded, tensors = plain.load(folder)
    eng = Engine(model_path=folder, dtype="bfloat16", max_ctx=512, max_batch=2)
    others = {"grouped": "pairs", "dense": "grouped"}
    for n in (33, 130, 256):
        (p,) = dapozen.prompts([n], cfg["vocab"], n)

        def run(forced):
            if forced:
                monkeypatch.setenv("FRIDAY_EXPERTS", forced)
            else:
                monkeypatch.delenv("FRIDAY_EXPERTS", raising=False)
            before, s = eng.stats()["launches"], eng.alloc_slot()
            out = eng.step([s], [p], [list(range(n))], to="host")
            eng.free_slot(s)
            return np.asarray(out), eng.stats()["launches"] - before
        got, launches = run(None)
        same, as_many = run(form)
        assert launches == as_many and np.array_equal(got, same), "%d rows" % n
        assert run(others[form])[1] != launches
        dapozen.compare(got, plain.forward(loaded, tensors, p), list(range(n)), "bfloat16", "%d of %d experts, %d rows" % (top, experts, n))
