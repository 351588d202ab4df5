"""Steps with prompt portions that come again in the same shape are replayed from a CUDA graph: the same bits as with every
step launched, for every design, and a graph per shape."""

import pytest
import torch

from bugapel_configs import BUGAPEL
from nisotar_configs import NISOTAR
from rematar_configs import REMATAR
from rodelorn_configs import RODELORN
from sipelorn_configs import SIPELORN
from tiny_configs import TINY
from todupel_configs import TODUPEL

pytestmark = pytest.mark.gpu

MODELS = {**{f"llama-{k}": TINY[k] for k in "ae"}, **{k: TODUPEL[k] for k in ("ta", "tc")}, **{k: REMATAR[k] for k in ("ra", "rd")},
          "oa": RODELORN["oa"], "ba": BUGAPEL["ba"], "sa": SIPELORN["sa"], **{k: NISOTAR[k] for k in ("na", "nc")}}


@pytest.mark.parametrize("name,dtype", [(n, "bfloat16") for n in MODELS] + [("llama-e", "float32"), ("na", "float32")])
def test_portions_replayed_give_the_same_bits(name, dtype, monkeypatch):
    from dynalm_b200 import Engine, StepEntry
    from dynalm_b200.engine.step import StepFunction
    monkeypatch.setattr(StepFunction, "GRAPH_AFTER", 3)
    cfg, seed = MODELS[name]
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    ids = torch.randint(0, vocab, (400,), generator=torch.Generator().manual_seed(9)).tolist()
    got = {}
    for graphs in (True, False):
        eng = Engine(config=cfg, random_seed=seed, dtype=dtype, ctx=1024, batch=160, max_running=4)
        fn = eng.step_fn
        assert fn.portion_graphs
        fn.use_graphs = graphs
        out = got[graphs] = []
        eng.step([StepEntry("a", ids[:37]), StepEntry("b", ids[40:50])])
        for again in range(6):
            # a request joins two live ones in portions of 24 (the last of another size, its end wanted), and leaves
            for i, (lo, hi) in enumerate(((0, 24), (24, 48), (48, 53))):
                live = [StepEntry(r, [ids[60 + 7 * again + i + k]], [0]) for k, r in enumerate("ab")]
                new = StepEntry("c", ids[100 + again + lo:100 + again + hi], [4] if i == 2 else [])
                out.append(eng.step(live + [new]).clone())
            eng.end("c")
        if graphs:
            assert 2 <= fn.graph_captures <= 4, "one graph a shape (the first two portions have one; a span may pass a power of two)"
            assert len(fn._shape_seen) <= fn.SHAPES_KEPT
        else:
            assert fn.graph_captures == 0
    for step, (a, b) in enumerate(zip(got[True], got[False])):
        assert torch.equal(a, b), f"step {step}"


def test_portions_that_leave_nothing_are_not_captured(monkeypatch):
    from dynalm_b200 import Engine, StepEntry
    from dynalm_b200.engine.step import StepFunction
    monkeypatch.setattr(StepFunction, "GRAPH_AFTER", 2)
    cfg, seed = TINY["a"]
    eng = Engine(config=cfg, random_seed=seed, dtype="bfloat16", ctx=512, batch=64, max_running=2)
    for _ in range(4):
        eng.step([StepEntry("r", list(range(20)))])
        eng.end("r")
    assert eng.step_fn.graph_captures == 0
    for _ in range(4):
        eng.step([StepEntry("r", list(range(20)), [19])])
        eng.end("r")
    assert eng.step_fn.graph_captures == 1


def test_shapes_that_pass_by_are_forgotten(monkeypatch):
    from dynalm_b200 import Engine, StepEntry
    from dynalm_b200.engine.step import StepFunction
    monkeypatch.setattr(StepFunction, "SHAPES_KEPT", 5)
    cfg, seed = TINY["a"]
    eng = Engine(config=cfg, random_seed=seed, dtype="float32", ctx=512, batch=64, max_running=2)
    for n in range(2, 30):
        eng.step([StepEntry("r", list(range(n)), [n - 1])])
        eng.end("r")
    assert len(eng.step_fn._shape_seen) == 5 and eng.step_fn.graph_captures == 0
