"""Which shapes of step are worth a captured graph.

A step is some two hundred launches issued from Python; when its kernels are fast the host becomes the limit, and a shape of
step that comes again is replayed from a graph instead.  A capture costs a step several times over (a run to warm up, the
collector, two synchronisations), and places are few, so a shape has to come again before it gets one, and once the places are
taken it has to come clearly more often than one that has a place, or find one that nobody uses any more.  More shapes in turn
than there are places would otherwise be captured at every single step: sixteen ragged prompts of up to 2,048 tokens
(Qwen2-1.5B sizes), whose pieces take turns in shape, 159 ms a request on a B200 with a capture at nearly every step, 94 without.
"""
from __future__ import annotations

from collections import deque
from typing import Any, Deque, Dict, Hashable, Optional, Tuple

COMINGS = 8               # a shape's last comings that are remembered
SHAPES_SEEN = 64          # shapes without a place that are remembered


class StepShapes:
    def __init__(self, sights: int):
        """`sights`: the coming at which a shape may be captured (at most `COMINGS`)."""
        self.sights = sights
        self.clock = 0
        self.kept: Dict[Hashable, Deque[int]] = {}        # shapes with a place: when they came, the least recent first
        self.seen: Dict[Hashable, Deque[int]] = {}        # shapes without

    def _pace(self, comings: Deque[int]) -> float:
        return (self.clock - comings[0]) / len(comings)   # steps from one coming to the next

    def coming(self, key: Hashable, places: int, idle: int) -> Tuple[bool, Optional[Any]]:
        """A step of this shape comes.  Returns whether it is to be captured (then `keep` follows, if the capture
        succeeds) and the shape that gives its place up for it, if one has to.  A shape that has a place is not captured again."""
        self.clock += 1
        if key in self.kept:
            comings = self.kept[key] = self.kept.pop(key)          # most recent last
            comings.append(self.clock)
            return False, None
        comings = self.seen[key] = self.seen.pop(key, None) or deque(maxlen=COMINGS)
        comings.append(self.clock)
        if len(self.seen) > SHAPES_SEEN:
            self.seen.pop(next(iter(self.seen)))
        if places < 1 or len(comings) < self.sights:
            return False, None
        if len(self.kept) < places:
            return True, None
        oldest = next(iter(self.kept))
        if self.clock - self.kept[oldest][-1] > idle:
            return True, oldest
        if len(comings) == COMINGS:
            slowest = max(self.kept, key=lambda k: self._pace(self.kept[k]))
            if self._pace(self.kept[slowest]) > 2.0 * self._pace(comings):
                return True, slowest
        return False, None

    def keep(self, key: Hashable, leaving: Optional[Any]) -> None:
        """The shape was captured; `leaving` is what `coming` returned with it."""
        if leaving is not None:
            self.kept.pop(leaving, None)
        self.kept[key] = self.seen.pop(key)
