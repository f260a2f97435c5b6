"""Page-locked staging buffers, so that small host arrays travel to the device without the host waiting for it."""
from __future__ import annotations

from typing import Dict

import torch

PINNED_RING = 4          # pinned staging buffers per size


class PinnedRings:
    """Page-locked staging buffers for what the host sends a step (its index arrays, page-table rows): ``PINNED_RING`` buffers in rotation
    per capacity, capacities being powers of two (at least ``MIN_CAPACITY`` values).  However many
    distinct lengths are asked for, at most ``PINNED_RING * log2(largest / MIN_CAPACITY)`` buffers
    ever exist.  An entry is ``[buffer, event]``; ``take`` waits for the event of the entry it hands
    out, so a buffer is never rewritten while a copy still reads it."""

    MIN_CAPACITY = 64

    def __init__(self, make=None):
        self._rings: Dict[int, dict] = {}
        self._make = make or (lambda cap: torch.empty(cap, dtype=torch.int32, pin_memory=True))

    @classmethod
    def capacity_for(cls, n: int) -> int:
        cap = cls.MIN_CAPACITY
        while cap < n:
            cap *= 2
        return cap

    def take(self, n: int) -> list:
        ring = self._rings.setdefault(self.capacity_for(n), {"next": 0, "slots": []})
        if len(ring["slots"]) < PINNED_RING:
            ring["slots"].append([self._make(self.capacity_for(n)), None])
            return ring["slots"][-1]
        entry = ring["slots"][ring["next"]]
        ring["next"] = (ring["next"] + 1) % PINNED_RING
        if entry[1] is not None:
            entry[1].synchronize()
        return entry

    def n_buffers(self) -> int:
        return sum(len(r["slots"]) for r in self._rings.values())
