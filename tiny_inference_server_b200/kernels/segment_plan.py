"""The first row of every request in a step, for kernels that walk a request's rows in order (a recurrence over
time) and want one CTA per request instead of one per row (``parts.base.StepPlanner``)."""
from __future__ import annotations

from typing import Dict, NamedTuple, Sequence, Tuple

import torch

from ..parts.base import StepPlanner


#: rows from which a request may be taken otherwise than token by token
LISTED_ROWS = 48


class Segments(NamedTuple):
    """The requests of a step, the longest first: their first rows (device), their number, the rows of the longest, the rows
    of each that has at least LISTED_ROWS, and of the longest that has fewer."""
    row0: torch.Tensor
    count: int
    longest: int
    rows: Tuple[int, ...]
    other: int


class SegmentPlanner(StepPlanner):
    key = ("segment_first_rows",)

    def max_words(self, rows: int) -> int:
        return rows

    def plan(self, segments: Sequence[Tuple[int, int]]):
        # the longest first: a request's rows are a chain, and the longest chain should not start last
        ordered = sorted(segments, key=lambda s: -s[1])
        lengths = [rows for _, rows in ordered]
        listed = [rows for rows in lengths if rows >= LISTED_ROWS]
        other = lengths[len(listed)] if len(listed) < len(lengths) else 0
        return {"row0": [first for first, _ in ordered]}, (len(ordered), max(lengths, default=0), other, *listed)

    def plan_decode(self, rows: int):
        return {"row0": list(range(rows))}, (rows, 1, 1)

    def bind(self, arrays: Dict[str, torch.Tensor], facts) -> Segments:
        return Segments(arrays["row0"], int(facts[0]), int(facts[1]), tuple(int(r) for r in facts[3:]), int(facts[2]))


_planner = SegmentPlanner()


def planner() -> SegmentPlanner:
    return _planner
