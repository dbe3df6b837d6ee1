"""How the tensor-core kernels of windowed attention want the rows of a step cut into tiles of consecutive rows of one
request: the mma.sync kernel (csrc/window_attention_mma.cu) takes as many rows as make 64 together with the query heads that
share a kv head (64 // group size); the tcgen05 kernel (csrc/window_attention_tc.cu) up to 128 rows of one query head.  Portions
of at least WIDE_MIN_ROWS rows are cut both ways, their mma.sync tiles first, so that a caller runs either the wide tiles and
the rest of the others, or all of the others.  The planner hands the tiles to the engine, which uploads them with the step's
own arrays (``parts.base.StepPlanner``)."""
from __future__ import annotations

from typing import Dict, NamedTuple, Sequence, Tuple

import torch

from ..parts.base import StepPlanner

PACKED_ROWS = 64
WIDE_MIN_ROWS = 64
WIDE_TILE_ROWS = 128


class WindowTiles(NamedTuple):
    """Tiles as (first rows, row counts, number of tiles); the first ``rows_in_wide`` of ``rows`` are those of ``wide``."""
    rows: Tuple[torch.Tensor, torch.Tensor, int]
    wide: Tuple[torch.Tensor, torch.Tensor, int]
    rows_in_wide: int


class WindowTilePlanner(StepPlanner):
    def __init__(self, tile_rows: int):
        self.tile_rows = tile_rows
        self.key = ("window_attention_tiles", tile_rows)

    def max_words(self, rows: int) -> int:
        return 4 * rows                      # at worst every row is a tile of its own, and once more in a wide tile

    def plan(self, segments: Sequence[Tuple[int, int]]):
        rest, covered, wide = [], [], []
        for first, n in segments:
            into = rest
            if n >= WIDE_MIN_ROWS:
                into = covered
                wide += [(first + a, min(WIDE_TILE_ROWS, n - a)) for a in range(0, n, WIDE_TILE_ROWS)]
            into += [(first + a, min(self.tile_rows, n - a)) for a in range(0, n, self.tile_rows)]
        tiles = covered + rest
        return {"row0": [t[0] for t in tiles], "rows": [t[1] for t in tiles], "wide0": [t[0] for t in wide],
                "wide": [t[1] for t in wide]}, (len(tiles), len(wide), len(covered))

    def plan_decode(self, rows: int):
        return {"row0": list(range(rows)), "rows": [1] * rows, "wide0": [], "wide": []}, (rows, 0, 0)

    def bind(self, arrays: Dict[str, torch.Tensor], facts) -> WindowTiles:
        count, wide, covered = (int(f) for f in facts)
        return WindowTiles((arrays["row0"], arrays["rows"], count), (arrays["wide0"], arrays["wide"], wide), covered)


_planners: Dict[int, WindowTilePlanner] = {}


def planner(group_size: int) -> WindowTilePlanner:
    """The planner for mixers with ``group_size`` query heads per kv head (at most 64)."""
    rows = max(1, PACKED_ROWS // group_size)
    if rows not in _planners:
        _planners[rows] = WindowTilePlanner(rows)
    return _planners[rows]
