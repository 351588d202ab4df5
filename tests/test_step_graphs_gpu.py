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


# Sizes whose launches depend on what the step plans answer: expanded latents (heads of 128 + 64, values of 128), segments of
# the state-space recurrence, chunks with a sink and the two maps on tcgen05, dealt query tiles, planned units of the decode attention.
_LATENT = {"heads": 2, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 48, "scale": 0.07, "rot": {"base": 10000.0, "dims": 64}}
_SSM = {"heads": 2, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}
_DIFF = {"heads": 4, "kv_heads": 2, "dim": 64, "vdim": 128, "scale": 0.125, "softcap": 30.0, "diff": 0.4, "q_temp": {"coef": 0.2, "every": 256}}


def _gated(ff):
    return {"kind": "dense", "ff": ff, "limit": 7.0}


LARGE = {
    "rematar": {"architecture": "Rematar", "vocab": 300, "width": 128, "norm": {"eps": 1e-5}, "postln_alpha": 2.0, "embedding": {"scale": 8.0},
                "layers": [{"type": "mamba2", "mixer": dict(_SSM), "mlp": {"kind": "dense", "ff": 128}},
                           {"type": "latent_attention", "mixer": dict(_LATENT, q_rank=64, mask={"size": 150}), "mlp": {"kind": "dense", "ff": 128}},
                           {"type": "mamba2", "mixer": dict(_SSM), "mlp": {"kind": "dense", "ff": 128}},
                           {"type": "latent_attention", "mixer": dict(_LATENT, q_rank=64, mask={"size": 400}), "mlp": {"kind": "dense", "ff": 128}}]},
    "nisotar": {"architecture": "Nisotar", "vocab": 300, "width": 128, "norm": {"eps": 1e-5}, "embedding": {"scale": 8.0},
                "layers": [{"type": "latent_attention", "mixer": dict(_LATENT, mask={"size": 250}), "mlp": _gated(128)},
                           {"type": "parallel", "mixer": {
                               "left": {"heads": 4, "kv_heads": 2, "dim": 64, "vdim": 64, "scale": 0.2, "mask": {"size": 100},
                                        "rot": {"base": 5e5, "dims": 64}},
                               "right": {"heads": 2, "kv_heads": 1, "dim": 64, "vdim": 64, "conv": 4, "decay_rank": 16, "gate_rank": 16}},
                            "mlp": _gated(128)}]},
    "todupel": {"architecture": "Todupel", "vocab": 300, "width": 128, "norm": {"eps": 1e-5},
                "layers": [{"type": "attention", "mixer": dict(_DIFF), "mlp": {"kind": "dense", "ff": 128}} for _ in range(2)]},
    "llama": dict(TINY["e"][0], max_position_embeddings=8192),
}
TAKEN = {"rematar": {"latent_attention_tcgen05", "segments"}, "nisotar": {"latent_attention_tcgen05", "chunks"},
         "todupel": {"diff_attention_tcgen05"}, "llama": {"dealt", "paged_attention_decode_planned"}}


def _spy(monkeypatch, ops, seen):
    """Which of the kernels in question a step launches goes to `seen`."""
    def watch(name, label):
        real = getattr(ops, name)

        def call(*args, **kwargs):
            what = label(args, kwargs)
            if what:
                seen.add(what)
            return real(*args, **kwargs)
        monkeypatch.setattr(ops, name, call)
    for name in ("latent_attention_tcgen05", "diff_attention_tcgen05", "paged_attention_decode_planned"):
        watch(name, lambda a, k, name=name: name)
    watch("paged_attention_prefill_tcgen05", lambda a, k: "chunks" if k.get("chunk") else "dealt" if k.get("unit_parts") is not None else None)
    watch("ssm_scan", lambda a, k: "segments" if a[15] is not None and a[15][1][0] > 0 else None)


@pytest.mark.parametrize("name", list(LARGE))
def test_portions_whose_launches_follow_the_plans_replay_the_same_bits(name, monkeypatch):
    """Portions of 150 rows (Llama: 512, behind 3,560 keys and more, whose end passes 4,096) beside live requests, at another place
    in its prompt every time the shape comes again."""
    from dynalm_b200 import Engine, StepEntry
    from dynalm_b200.engine.step import StepFunction
    from dynalm_b200.kernels import ops
    monkeypatch.setattr(StepFunction, "GRAPH_AFTER", 2)
    ids = torch.randint(0, 256, (6000,), generator=torch.Generator().manual_seed(9)).tolist()
    long = name == "llama"
    live, portions = (13, (512, 100)) if long else (2, (150, 150, 37))
    got = {}
    for graphs in (True, False):
        seen = set()
        with monkeypatch.context() as m:
            _spy(m, ops, seen)
            eng = Engine(config=LARGE[name], random_seed=5, dtype="bfloat16", ctx=24576 if long else 4096, batch=600, max_running=live + 1)
            fn = eng.step_fn
            assert fn.portion_graphs
            fn.use_graphs = graphs
            out = got[graphs] = []
            for r in range(live):
                eng.step([StepEntry(r, ids[17 * r:17 * r + 30 + r])])
            for at in range(39, 3560, 512) if long else ():
                eng.step([StepEntry(0, ids[at:min(at + 512, 3560)])])
            for again in range(6):
                if long:
                    eng.step([StepEntry(0, ids[4000:4009])])           # (nothing wanted: launched in both)
                    fn.fork(0, "c")
                else:
                    eng.step([StepEntry("c", ids[500:501 + again])])
                at = 1000
                for n in portions:
                    step = [StepEntry(r, [ids[60 + 7 * again + 31 * r + at]], [0]) for r in range(live)]
                    out.append(eng.step(step + [StepEntry("c", ids[at:at + n], [n - 1])]).clone())
                    at += n
                eng.end("c")
        assert seen == TAKEN[name]
        assert fn.graph_kernel_launches > 0 and fn.graph_captures >= 2 if graphs else fn.graph_captures == 0
    for step, (a, b) in enumerate(zip(got[True], got[False])):
        assert torch.equal(a, b), f"step {step}"


def test_shapes_in_turn_beyond_the_places_are_not_captured_over_and_over(monkeypatch):
    """Portions of 40 lengths in turn: 32 graphs, one each, and the bits of steps launched; decode graphs stay."""
    from dynalm_b200 import Engine, StepEntry
    from dynalm_b200.engine.step import StepFunction
    monkeypatch.setattr(StepFunction, "GRAPH_AFTER", 2)
    cfg, seed = TINY["a"]
    ids = torch.randint(0, 256, (100,), generator=torch.Generator().manual_seed(3)).tolist()
    got, cfg = {}, dict(cfg, max_position_embeddings=512)
    for graphs in (True, False):
        eng = Engine(config=cfg, random_seed=seed, dtype="float32", ctx=1024, batch=64, max_running=2)
        eng.step_fn.use_graphs = graphs
        out = got[graphs] = []
        eng.step([StepEntry("live", ids[:3])])
        for again in range(5):
            for n in range(2, 42):
                out.append(eng.step([StepEntry("r", ids[again:again + n], [n - 1])]).clone())
                out.append(eng.step([StepEntry("live", [n], [0])]).clone())
                eng.end("r")
        if graphs:
            kept = eng.step_fn._graphs.graphs
            assert len(kept["portions"]) == 32 and 1 <= len(kept["decode"]) <= 2
            assert eng.step_fn.graph_captures == 32 + len(kept["decode"])
    assert all(torch.equal(a, b) for a, b in zip(got[True], got[False]))


@pytest.mark.parametrize("name", ["a", "e"])
def test_32_bit_portions_replay_the_same_bits_at_every_span(name, monkeypatch):
    """float32: portions of one size at spans of 64 to 1,024 keys, where rows and query tiles of the attention take turns."""
    from dynalm_b200 import Engine, StepEntry
    from dynalm_b200.engine.step import StepFunction
    from dynalm_b200.kernels import ops
    monkeypatch.setattr(StepFunction, "GRAPH_AFTER", 2)
    cfg, seed = dict(TINY[name][0], max_position_embeddings=2048), TINY[name][1]
    ids = torch.randint(0, 256, (1200,), generator=torch.Generator().manual_seed(5)).tolist()
    got, seen = {}, set()
    for graphs in (True, False):
        with monkeypatch.context() as m:
            if not graphs:
                for kernel in ("attention_f32_rows", "attention_f32_tiles"):
                    real = getattr(ops, kernel)
                    m.setattr(ops, kernel, lambda *a, real=real, kernel=kernel, **k: (seen.add(kernel), real(*a, **k))[1])
            eng = Engine(config=cfg, random_seed=seed, dtype="float32", ctx=4096, batch=256, max_running=2)
            eng.step_fn.use_graphs = graphs
            out = got[graphs] = []
            eng.step([StepEntry("live", ids[:9])])
            for again in range(3):
                for at in range(again, 1100, 100):
                    new = StepEntry("new", ids[at:at + 100], [99])
                    out.append(eng.step([StepEntry("live", [ids[at]], [0]), new]).clone())
                eng.end("new")
        assert eng.step_fn.graph_captures >= 4 if graphs else eng.step_fn.graph_captures == 0
    assert all(torch.equal(a, b) for a, b in zip(got[True], got[False]))
    assert seen == {"attention_f32_rows", "attention_f32_tiles"}
