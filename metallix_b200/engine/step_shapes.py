"""Which shapes of general steps are worth a captured graph.

A capture takes 3 to 8 ms, two or three launched steps, and pays by the
millisecond or so that each replay saves, so a shape has to come again before
it gets one, and room for a graph is limited. Where more shapes come again and
again than there is room for, graphs that make room for each other all the time
would cost more than they save (40 shapes picked evenly, 32 graphs, the oldest
making room: one step in five a capture; by the rule below one in forty, with as
many replays. 40 shapes of three prompts through four Sadosun layers: 1.8 ms a
step, some 2.5 launched). So a graph makes room only for a shape that comes as
often of late as its own, and that came again within a sixteenth of the time
that the graph has not been used.
"""
from __future__ import annotations

from typing import Container, Dict, Hashable, Iterable, List

HALF_LIFE = 256     # steps in which a sighting loses half its weight
IDLE_FACTOR = 16
REMEMBERED = 4096   # shapes at most
FAILED = 64         # further sightings that a shape needs whose capture failed


class StepShapes:
    """``room``: how many graphs are kept; ``sightings``: how often a shape has to have come before it is captured."""

    def __init__(self, room: int, sightings: int):
        self.room, self.sightings = room, sightings
        self._steps = 0
        self._seen: Dict[Hashable, List] = {}   # shape -> [sightings that count, their weight, step of the last one]

    def _weight(self, shape: Hashable) -> float:
        entry = self._seen.get(shape)
        return entry[1] * 0.5 ** ((self._steps - entry[2]) / HALF_LIFE) if entry else 0.0

    def came(self, shape: Hashable, kept: Container) -> bool:
        """Notes a step of this shape; whether it runs as a graph (one that is ``kept``, or is to be captured now)."""
        self._steps += 1
        before, _, last = self._seen.get(shape, (0, 0.0, None))
        weight = self._weight(shape) + 1.0
        self._seen[shape] = [before + 1, weight, self._steps]
        if len(self._seen) > REMEMBERED:
            self._forget_least(kept)
        if shape in kept:
            return True
        if before < self.sightings:
            return False
        if len(kept) < self.room:
            return True
        least = self.least(kept)
        idle = self._steps - self._seen[least][2] if least in self._seen else self._steps
        return last is not None and self._weight(least) <= weight and (self._steps - last) * IDLE_FACTOR < idle

    def least(self, kept: Iterable) -> Hashable:
        """The kept shape that makes room."""
        return min(kept, key=self._weight)

    def evicted(self, shape: Hashable) -> None:
        """The shape's graph is gone: it has to come as often again before it gets another."""
        if shape in self._seen:
            self._seen[shape][0] = 0

    def failed(self, shape: Hashable) -> None:
        """The shape could not be captured."""
        if shape in self._seen:
            self._seen[shape][0] = self.sightings - FAILED

    def _forget_least(self, kept: Container) -> None:
        ranked = sorted((shape for shape in self._seen if shape not in kept), key=self._weight)
        for shape in ranked[:REMEMBERED // 2]:
            del self._seen[shape]
