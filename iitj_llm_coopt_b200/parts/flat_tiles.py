"""The per-step plan of the mixers whose attention runs over flat-page caches (`Kernels.attention_flat`): the step's tokens cut
into runs of neighbouring tokens of one request, as many as one block of the tensor-core kernel takes beside the heads of a
key/value group, and, for a step of single decoded tokens, over how many blocks each run's keys are shared out.  In float32 the
lists of the float32 attention kernels stand beside them where these serve the layer (`Kernels.flat_f32_runs`) and the step is
faster on them than on the kernel that walks a row a warp (`_float32_lists`).

Layers with equal head counts, sizes and window share one plan per step (`prepare_key`)."""
from __future__ import annotations

import math

import torch

from .base import StepPlan


def flat_prepare_key(heads, kv_heads, key_dim, value_dim, window) -> str:
    return f"flat_attention.{heads}.{kv_heads}.{key_dim}.{value_dim}.{window}"


# us, per head size: the longest chain of a step (its start, and per key or tile of 32 keys), and what the step's keys add up to over all SMs (per
# row or run and head, and per key or tile of it).  Measured over 1 to 300 requests of 1 to 64 tokens behind 8 to 8000 keys, with
# 4 to 32 heads; a step takes about the root of the sum of both squares.
_WARP = {64: (5.0, 0.272, 0.0, 0.103e-3), 128: (5.0, 0.305, 0.0, 0.185e-3)}           # attention_flat.cu: a row of a head a warp
_SINGLE = {64: (3.5, 0.026, 9.5e-3, 0.112e-3), 128: (3.8, 0.036, 19e-3, 0.24e-3)}      # attention_f32.cu: a row of a head a block
_TILE = {64: (3.5, 4.0, 3e-3, 17.7e-3), 128: (4.0, 6.1, 5e-3, 35e-3)}                  # attention_f32.cu: up to 64 rows of a head a block


def _estimate(costs, heads, longest, count, total) -> float:
    start, chain, each, key = costs
    return math.hypot(start + chain * longest, heads * (each * count + key * total)) if count else 0.0


def _float32_lists(heads, dim, window, run, query_lens, seq_lens):
    """(token rows of requests that bring one token, runs of up to `run` tokens of the others) for the kernels of float32 attention,
    or None where a warp a row is the faster way: a block a row or run pays its way while a step waits for its longest chain of keys (one
    token of 32 heads of 64 behind 500 keys 16 us for 139, 100 of them 200 for 241), not once the SMs are full of warps (300 of them 582
    for 478; 300 behind 8 keys 94 for 17; 100 requests of 4 tokens behind 300 keys 562 for 409)."""
    seen = [min(total, window) for total in seq_lens] if window > 0 else seq_lens
    items, runs, row = [], [], 0
    item_keys, tiles, all_keys = [], [], 0
    for b, (n, total, keys) in enumerate(zip(query_lens, seq_lens, seen)):
        all_keys += n * keys
        if n == 1:
            items.append(row)
            item_keys.append(keys)
        else:
            if keys == total:
                all_keys -= n * (n - 1) // 2              # the rows before the last see fewer
            for s in range(0, n, run):
                rows, last = min(run, n - s), total - n + min(s + run, n)
                runs.append((row + s, rows, total - n + s, b))
                tiles.append((min(last, window + rows - 1) if window > 0 else last) / 32 + 0.5)
        row += n
    lists = _estimate(_SINGLE[dim], heads, max(item_keys, default=0), len(items), sum(item_keys)) + \
        _estimate(_TILE[dim], heads, max(tiles, default=0), len(runs), sum(tiles))
    if lists >= _estimate(_WARP[dim], heads, max(seen), row, all_keys):
        return None
    runs.sort(key=lambda r: r[2] + r[1])              # the kernel starts at the list's end: the longest contexts first
    return items, [v for r in runs for v in r]


def plan_flat_tiles(kernels, shape, heads, kv_heads, key_dim, value_dim, window, shared_value=False, dtype=None):
    """StepPlan with `tiles` (first token row, tokens, position of the first, request) and `.splits`, or None when the
    kernel set plans nothing (it then walks a row per warp)."""
    per_tile = getattr(kernels, "flat_tokens_per_tile", None)
    if per_tile is None:
        return None
    run = per_tile(heads, kv_heads)
    tiles, row, longest = [], 0, 0
    for b, (n, total) in enumerate(zip(shape.query_lens, shape.seq_lens)):
        for s in range(0, n, run):
            tiles += [row + s, min(run, n - s), total - n + s, b]
        row += n
        longest = max(longest, min(total, window + n - 1) if window > 0 else total)
    splits = 1
    if shape.num_tokens == len(shape.query_lens):
        # single decoded tokens: few blocks, long key ranges.  The longest range is rounded up to 512 keys, so that a captured
        # graph (which freezes the count) serves the steps while contexts grow.
        splits = kernels.flat_key_splits(len(shape.query_lens), heads, kv_heads, key_dim, value_dim, shared_value,
                                         -(-longest // 512) * 512)
    run = kernels.flat_f32_runs(heads, kv_heads, key_dim, value_dim, shared_value) if dtype == torch.float32 else 0
    lists = _float32_lists(heads, key_dim, window, run, shape.query_lens, shape.seq_lens) if run else None
    arrays = {"tiles": tiles}
    if lists is not None:
        arrays.update({name: rows for name, rows in zip(("items", "runs"), lists) if rows})
    plan = StepPlan(arrays=arrays, graph_key=(splits, lists is not None))
    plan.splits = splits
    return plan
