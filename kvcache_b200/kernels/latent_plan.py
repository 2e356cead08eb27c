"""Work lists of latent attention: of the kernel over shared key rows (csrc/latent_flash.cu), and of portions whose keys and values
are expanded first (csrc/attention_pairs.cu, at the end).

All heads of a token read the same cached rows, so the kernel's rows are (token, head) pairs: a request that brings
`count` tokens has count * H rows, cut into tiles of BM rows; a tile sees the keys up to its last token's position.
Every tile is cut into the same number of splits over its keys - as many as bring the launch to about `blocks_wanted`
blocks, so that a few decoded tokens with long contexts still fill the GPU - and the splits of a tile are added up by
a second kernel in their order.  The number of splits follows from the number of tiles alone; steps of decoded tokens
with the same number of requests therefore have the same launches and can be replayed from one CUDA graph.
With a window a tile's keys start at the tile of 64 keys that holds the first key its first row sees; what lies before
is neither read nor expected in the cache (a windowed cache entry has given those pages back).
"""
from __future__ import annotations

import functools
from typing import Dict, Tuple

import numpy as np

from ..parts.base import StepPlanner
from .attention_plan import TC_PAIR_ROWS

KEY_TILE = 64
SMALL_TILE, LARGE_TILE = 16, 64      # rows of a tile: 16 while every request's rows fit one such tile, else 64
MAX_SPLITS = 32


@functools.lru_cache(maxsize=1024)
def _plan(segments: tuple, heads: int, blocks_wanted: int, large_tile: int = LARGE_TILE, window: int = 0):
    """segments: (segment index, tokens cached, tokens brought).  Returns (int32 [items, 4]: segment, first row, first
    key, end of keys; tiles; splits per tile; rows of a tile)."""
    bm = SMALL_TILE if all(count * heads <= SMALL_TILE for _, _, count in segments) else large_tile
    tiles = []
    for seg, start, count in segments:
        for m0 in range(0, count * heads, bm):
            last_token = min(count - 1, (m0 + bm - 1) // heads)
            first_key = max(0, start + m0 // heads - window + 1) // KEY_TILE * KEY_TILE if window else 0
            tiles.append((seg, m0, start + last_token + 1, first_key))
    tiles.sort(key=lambda t: t[3] - t[2])        # the tiles with the most keys first
    nsplit = max(1, min(MAX_SPLITS, blocks_wanted // len(tiles)))
    items = []
    for seg, m0, kv_end, first_key in tiles:
        per = -(-(-(-(kv_end - first_key) // KEY_TILE)) // nsplit) * KEY_TILE          # keys of a split: whole key tiles
        for s in range(nsplit):
            kb = min(first_key + s * per, kv_end)
            items.append((seg, m0, kb, min(kv_end, kb + per)))
    array = np.asarray(items, dtype=np.int32).reshape(-1, 4)
    array.setflags(write=False)
    return array, len(tiles), nsplit, bm


class LatentAttentionPlanner(StepPlanner):
    def __init__(self, heads: int, blocks_wanted: int, large_tile: int = LARGE_TILE, window: int = 0):
        """`large_tile`: rows of a tile in steps that bring more than `SMALL_TILE` rows of a request (64, or 32 where the
        kernel's shared memory holds two key stages only beside the smaller tile).  `window`: keys a query sees, its own
        included (0: all)."""
        self.heads, self.blocks_wanted, self.large_tile, self.window = heads, blocks_wanted, large_tile, int(window or 0)
        self.name = self.plan_name(heads, blocks_wanted, large_tile, self.window)

    @staticmethod
    def plan_name(heads: int, blocks_wanted: int, large_tile: int = LARGE_TILE, window: int = 0) -> str:
        return f"latent_attention.h{heads}.b{blocks_wanted}.t{large_tile}" + (f".w{window}" if window else "")

    def sections(self, num_tokens: int, num_segments: int) -> Dict[str, int]:
        tiles = num_tokens * self.heads // self.large_tile + 2 * num_segments
        return {"items": 4 * max(tiles, self.blocks_wanted + num_segments)}

    def plan(self, starts, counts) -> Tuple[Dict[str, np.ndarray], Dict[str, int]]:
        segments = tuple((i, int(s), int(c)) for i, (s, c) in enumerate(zip(starts, counts)))
        items, tiles, nsplit, bm = _plan(segments, self.heads, self.blocks_wanted, self.large_tile, self.window)
        return {"items": items.reshape(-1)}, {"items": len(items), "tiles": tiles, "nsplit": nsplit, "bm": bm}


EXPAND_BLOCK = 128               # keys of a block of expanded rows: the key tile of csrc/attention_pairs.cu
EXPAND_MAX_BLOCKS = 256          # blocks a step may bring
EXPAND_MAX_PAIRS = 128           # pairs of row tiles (csrc/attention_pairs.cu, MAX_TILES)
# Rows that every request of the step brings: an expanded key has to serve many.  A whole layer launched from Python on both sides, in us, keys
# as they are and expanded, 16 heads of 128 (rank 512) and 14 of 64 (rank 256): 64 rows 80 and 60, 70 and 61; 64 behind 2,000 87 and 78, 70 and 61;
# 128 behind 2,000 129 and 83, 77 and 61; 2,048 528 and 132, 261 and 80; four requests of 50 behind 2,000 (not taken) 189 and 126, 91 and 77: the line
# could lie lower.
EXPAND_MIN_ROWS = 64


class LatentExpandPlanner(StepPlanner):
    """Lists for steps of portions whose keys and values are expanded once per token and head before attention.

    `blocks`: (segment, first key) of every 128 keys that any row of the step sees; `key_row`: the row that a segment's key 0 has
    among the expanded rows, or would have; `pairs`: (segment, first row) of pairs of row tiles.  The count `blocks` is 0 where
    the step is not expanded: a request brings fewer than EXPAND_MIN_ROWS rows, or the step sees more than the lists hold."""

    def __init__(self, window: int = 0):
        self.window = int(window or 0)
        self.name = self.plan_name(self.window)

    @staticmethod
    def plan_name(window: int = 0) -> str:
        return "latent_expand" + (f".w{window}" if window else "")

    def sections(self, num_tokens: int, num_segments: int) -> Dict[str, int]:
        return {"blocks": 2 * EXPAND_MAX_BLOCKS, "key_row": num_segments, "pairs": 2 * (num_tokens // TC_PAIR_ROWS + num_segments)}

    def plan(self, starts, counts) -> Tuple[Dict[str, np.ndarray], Dict[str, int]]:
        none = np.zeros(0, dtype=np.int32)
        off = {"blocks": none, "key_row": none, "pairs": none}, {"blocks": 0, "pairs": 0}
        if int(min(counts)) < EXPAND_MIN_ROWS:
            return off
        blocks, key_row, pairs = [], [], []
        for i, (start, count) in enumerate(zip(starts, counts)):
            start, count = int(start), int(count)
            first = max(0, start - self.window + 1) // EXPAND_BLOCK * EXPAND_BLOCK if self.window else 0
            key_row.append(EXPAND_BLOCK * len(blocks) - first)
            blocks.extend((i, key) for key in range(first, start + count, EXPAND_BLOCK))
            pairs.extend((i, row) for row in range(0, count, TC_PAIR_ROWS))
        if len(blocks) > EXPAND_MAX_BLOCKS or len(pairs) > EXPAND_MAX_PAIRS:
            return off
        flat = lambda rows: np.asarray(rows, dtype=np.int32).reshape(-1)
        return {"blocks": flat(blocks), "key_row": flat(key_row), "pairs": flat(pairs)}, {"blocks": len(blocks), "pairs": len(pairs)}
