"""Captured decode steps whose sublayers run as branches of the graph, against the same steps captured one kernel after
another: the same kernels on the same numbers, so every bit is the same, step after step."""

import tempfile

import pytest
import torch

import godotar_models
import tugodra_models
import zirurax_models
from harness import make_runner
from lily_b200.engine.batch import StepEntry

pytestmark = pytest.mark.gpu

DESIGNS = {"zirurax": (zirurax_models, 2), "godotar": (godotar_models, 1), "tugodra": (tugodra_models, 1)}      # and the lanes they ask for


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("config", ["VARIED", "WIDE"])
@pytest.mark.parametrize("design", sorted(DESIGNS))
def test_branches_give_the_bits_of_one_stream(monkeypatch, design, config, dtype):
    """Requests that leave between the steps (other batch sizes, so other graphs on the same lanes), the graphs replayed back to
    back."""
    from lily_b200.models.assembled import AssembledModel
    models, lanes = DESIGNS[design]
    cfg = getattr(models, config)
    with tempfile.TemporaryDirectory() as tmp:
        path = models.write_model_dir(tmp + "/m", cfg, models.make_weights(cfg, 5))

        def run(branches):
            with monkeypatch.context() as m:
                if not branches:
                    m.setattr(AssembledModel, "lanes", 0)
                runner = make_runner(path, dtype=dtype, device="cuda", max_tokens=2048, max_requests=4, context_length=512)
                assert runner.model.lanes == (lanes if branches else 0)
                ids = [models.tokens(60 + 7 * r, cfg["vocab"], r) for r in range(4)]
                slots = [runner.open_request() for _ in ids]
                out = [runner.step([StepEntry(s, t[:20 + 7 * r], [0]) for r, (s, t) in enumerate(zip(slots, ids))]).clone()]
                at = [20 + 7 * r for r in range(4)]
                for step in range(40):
                    live = [r for r in range(4) if step < 10 * (r + 1)]
                    out.append(runner.step([StepEntry(slots[r], [ids[r][at[r]]], [0]) for r in live]).clone())
                    for r in live:
                        at[r] += 1
                assert runner.graph_steps == 40 and all(len(g.batch.lanes) == (lanes if branches else 0) for g in runner._graphs.values())
                return out, [s[1:].clone() for s in runner.cache.states]          # row 0 is the padded rows'
        (one, states), (many, states_many) = run(False), run(True)
        assert all(torch.equal(a, b) for a, b in zip(one, many)) and all(torch.equal(a, b) for a, b in zip(states, states_many))
