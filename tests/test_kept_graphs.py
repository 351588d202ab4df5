"""Which launch shapes are kept as graphs (engine/kept_graphs.py): admission, eviction, places per kind of step."""

import pytest

from dynalm_b200.engine.kept_graphs import KeptGraphs


def _step(kept, kind, key, log):
    """One step of a shape, as the step function does it; log: (captures, replays) per (kind, key)."""
    counts = log.setdefault((kind, key), [0, 0])
    if kept.use(kind, key) is not None:
        counts[1] += 1
    elif kept.wants(kind, key):
        kept.keep(kind, key, object())
        counts[0] += 1


@pytest.mark.parametrize("shapes", [60, 64, 65, 70, 100, 1000])
def test_more_recurring_shapes_than_places(shapes):
    """In turn, 40 times each: every graph is captured once and replayed from then on, the other shapes never."""
    kept, log = KeptGraphs({"decode": 64, "portions": 32}, 8, 4096), {}
    for _ in range(40):
        for n in range(shapes):
            _step(kept, "decode", n, log)
    captured = [c for c in log.values() if c[0]]
    assert len(captured) == min(shapes, 64) and all(c == [1, 32] for c in captured)


def test_a_shape_takes_the_place_of_one_that_is_used_no_more():
    kept, log = KeptGraphs({"decode": 4}, 3, 100), {}
    for key in "abcd" * 3:
        _step(kept, "decode", key, log)
    for _ in range(3):                         # "a" stays in use; "b" was used longest ago
        for key in "aecd":
            _step(kept, "decode", key, log)
    assert set(kept.graphs["decode"]) == set("aecd")
    assert log[("decode", "e")][0] == 1
    for _ in range(2):                         # the one that went counts from nothing again, whoever else comes
        _step(kept, "decode", "b", log)
    assert log[("decode", "b")] == [1, 0] and "b" not in kept.graphs["decode"]


def test_no_capture_for_a_graph_still_in_use():
    """Two shapes with room for one, in turn and in runs."""
    kept, log = KeptGraphs({"decode": 1}, 8, 100), {}
    for _ in range(200):
        for key in "ab":
            _step(kept, "decode", key, log)
    assert log[("decode", "a")] == [1, 192] and log[("decode", "b")] == [0, 0]
    for _ in range(40):                        # from here on only b
        _step(kept, "decode", "b", log)
    assert log[("decode", "b")][0] == 1 and log[("decode", "b")][1] >= 24


def test_portions_do_not_push_out_decoding():
    kept, log = KeptGraphs({"decode": 64, "portions": 32}, 8, 4096), {}
    for n in range(2000):
        _step(kept, "decode", n % 3, log)
        _step(kept, "portions", n % 250 // 2, log)
        assert len(kept.graphs["portions"]) <= 32
    assert all(log[("decode", k)][0] == 1 for k in range(3))


def test_counts_of_shapes_that_pass_by_are_forgotten():
    kept, log = KeptGraphs({"decode": 2, "portions": 2}, 8, 5), {}
    for n in range(50):
        _step(kept, "portions", n, log)
    assert len(kept.seen) == 5 and not kept.graphs["portions"]
