"""The work list of the tiled prompt-attention kernel: which CTA takes which queries and keys.

It belongs to the kernel (its tile sizes and how many of its CTAs the GPU runs at once decide
the cut); the attention mixer asks for it through ``CudaOps.plan_prompt_attention`` from its
``plan_step`` hook, and the step function carries it to the device with the step's other integers.
"""

from __future__ import annotations

import numpy as np

QUERY_TILE = 128       # most consecutive tokens of one request in a tile
KEY_CHUNK = 512        # key positions one work item walks over, where all items run at once
KEY_BLOCK = 64         # keys the kernel takes at a time
ITEM_BLOCKS = 4        # what a work item costs besides its key blocks, in key blocks
MERGE_BLOCKS = 3       # ... and what leaving its results to be merged adds
_LIMITS = np.array([*range(KEY_CHUNK, 2 * KEY_CHUNK + 1, QUERY_TILE), 1 << 30])   # most keys of an item: what is weighed


def query_tiles(q_lens, ctx_befores, slots=None):
    """Cut a ragged batch into work items ``(request, first row, rows, chunk, chunks)``.

    The tokens of each request are cut into runs of at most QUERY_TILE rows.  The keys a run
    may see (positions 0 .. its last token) are cut into ``chunks`` equal parts, of at most KEY_CHUNK
    positions where all items run at once, one work item each, so that a long context is spread over several CTAs; their
    partial results are merged afterwards.  Items of one run are consecutive, chunk 0 first; the
    runs come longest item first, so that when the grid does not fit the GPU at once, the CTAs
    that start last are the short ones.

    ``slots``: how many work items the GPU runs at once (per head).  Where parts of KEY_CHUNK do not all fit at once, longer
    parts (up to twice KEY_CHUNK) and whole runs are weighed against them: by the longest item, and the sum of all items
    over the slots where there are several rounds, with ITEM_BLOCKS for what an item costs besides its key blocks and
    MERGE_BLOCKS more where its results have to be merged.  (16 heads, 2,048 tokens, one CTA an SM: 9 slots a head; whole
    runs, 16 items of up to 32 blocks, take 0.6 of the time of 40 parts.)"""

    runs = []                                     # (request, first row, rows, keys it may see)
    row = 0
    for r, (n, before) in enumerate(zip(q_lens, ctx_befores)):
        for b in range(0, n, QUERY_TILE):
            rows = min(QUERY_TILE, n - b)
            runs.append((r, row + b, rows, before + b + rows))
        row += n

    limit = KEY_CHUNK
    # (where no run sees more than KEY_CHUNK keys there is nothing to weigh)
    if (slots and max((keys for _, _, _, keys in runs), default=0) > KEY_CHUNK
            and sum(-(-keys // limit) for _, _, _, keys in runs) > slots):
        keys = np.array([keys for _, _, _, keys in runs])
        blocks, limits = -(-keys // KEY_BLOCK), _LIMITS
        chunks = -(-keys // limits[:, None])                  # [limit, run], as the three below
        besides = ITEM_BLOCKS + MERGE_BLOCKS * (chunks > 1)
        items, total = chunks.sum(1), blocks.sum() + (chunks * besides).sum(1)
        longest = (-(-blocks // chunks) + besides).max(1)
        cost = np.where(items <= slots, longest, np.maximum(longest, total / slots) + 0.3 * longest)
        limit = int(limits[cost.argmin()])                    # (the shortest of equals)
    cut = []
    for i, (r, row0, rows, keys) in enumerate(runs):
        chunks = max(1, -(-keys // limit))
        cut.append((-(keys / chunks), i, r, row0, rows, chunks))
    cut.sort()
    return [(r, row0, rows, c, chunks) for _, _, r, row0, rows, chunks in cut for c in range(chunks)]
