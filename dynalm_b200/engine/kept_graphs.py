"""Which launch shapes of the step are kept as CUDA graphs, and which one goes for a new one.

A capture costs 5 to 15 ms on the host, some ten times what a replay saves, so a shape is captured when it has come `after`
times, and when all places are taken only in the place of a graph that was not used once while it came: with more recurring
shapes than places the ones in place stay and the others are launched kernel by kernel. (Dropping the graph used longest ago
for every shape seen often enough, 70 shapes coming in turn made a capture at nearly every step and no replay.) A shape that
was not let in, and one whose graph went, counts from nothing again.

Steps of single tokens and steps with prompt portions have places of their own: the shapes of the latter, which hold the
numbers of rows, can be many more, and must not push out the graphs that decoding runs on.

No CUDA in here: a graph is whatever `keep` is given.
"""

from __future__ import annotations

from typing import Any, Dict, Hashable, Optional


class KeptGraphs:
    def __init__(self, places: Dict[str, int], after: int, shapes_kept: int):
        self.places = dict(places)         # kind of step -> graphs kept
        self.after = int(after)
        self.shapes_kept = int(shapes_kept)
        self.graphs: Dict[str, Dict[Hashable, list]] = {kind: {} for kind in places}      # key -> [graph, last use]; used last goes last
        self.seen: Dict[Hashable, tuple] = {}      # (kind, key) -> (how often it has come, when first); the `shapes_kept` last new ones
        self.steps = 0

    def use(self, kind: str, key: Hashable) -> Optional[Any]:
        """The shape's graph, or None. Called once a step."""
        self.steps += 1
        got = self.graphs[kind].pop(key, None)
        if got is None:
            return None
        self.graphs[kind][key] = got
        got[1] = self.steps
        return got[0]

    def wants(self, kind: str, key: Hashable) -> bool:
        """Count a step of a shape without a graph; True when it is to be captured now (`keep` is called next)."""
        count, first = self.seen.pop((kind, key), (0, self.steps))
        count += 1
        if count >= self.after:
            kept = self.graphs[kind]
            if len(kept) < self.places[kind]:
                return True
            oldest = next(iter(kept))
            if kept[oldest][1] < first:
                del kept[oldest]
                return True
            return False
        self.seen[(kind, key)] = (count, first)
        if len(self.seen) > self.shapes_kept:
            del self.seen[next(iter(self.seen))]
        return False

    def keep(self, kind: str, key: Hashable, graph: Any) -> None:
        self.graphs[kind][key] = [graph, self.steps]
