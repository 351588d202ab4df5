"""Chooses the latent-attention kernel for a step, and cuts the step into query tiles for the tensor-core one.

float32 always runs the plain kernel (csrc/latent_attention.cu), whose arithmetic for a row is fixed by the row
alone. bfloat16 runs the tensor-core kernel (csrc/latent_attention_flash.cu) when the record's two pieces are
multiples of 8 numbers and the latent has at most 512: its blocks take 32 query units, a unit being (row, head), so
the host cuts every request of the step into tiles of 32 / heads-to-a-block consecutive rows (a step plan, sent with
the step's integers). Prompt portions and single decoded tokens go through the same launch, unless the heads have the sizes
EXPAND_SIZES: then a portion's keys and values are worked out for every head (one product over the records its rows see) and
attended by the tcgen05 flash kernel (csrc/attention_prefill_tcgen05.cu), a fifth of the operations a row and key.
"""

from __future__ import annotations

import numpy as np
import torch

from . import ops
from .device import sm_count

UNITS = 32          # query units (row, head) to a block of the tensor-core kernel


NUMPY_TILES = 64    # more tiles than this are worked out in numpy (two rows a tile: 258 rows 27 us against 54, 708 rows 33 against 142)


def heads_per_block(heads: int) -> int:
    """Heads to a block: all of them up to 32, else the heads dealt evenly over the fewest blocks."""
    groups = -(-heads // UNITS)
    return -(-heads // groups)


class LatentTilePlan:
    """Every request of the step cut into tiles of at most `rows` consecutive rows: int32 [tiles, 4] = (request slot,
    first row of the step, rows, first position), the tiles that see the most keys first. `fill` returns the number
    of tiles."""

    def __init__(self, rows: int):
        self.rows = int(rows)
        self.name = f"latent_query_tiles:{self.rows}"

    def ints(self, max_tokens: int, max_requests: int) -> int:
        return 4 * (max_tokens // self.rows + max_requests)

    def fill(self, host, shape) -> int:
        if sum(shape.q_len) > NUMPY_TILES * self.rows:
            n, r0, start, slot = (np.asarray(v, dtype=np.int32) for v in (shape.q_len, shape.q_start, shape.pos_start, shape.slots))
            count = -(-n // self.rows)
            of = np.repeat(np.arange(len(n)), count)
            t0 = (np.arange(len(of), dtype=np.int32) - np.repeat(np.cumsum(count) - count, count)) * self.rows
            rows, pos = np.minimum(self.rows, n[of] - t0), start[of] + t0
            order = np.argsort(-(pos + rows), kind="stable")
            host[:4 * len(of)].reshape(-1, 4)[:] = np.stack([slot[of], r0[of] + t0, rows, pos], axis=1)[order]
            return len(of)
        tiles = []
        for n, r0, start, slot in zip(shape.q_len, shape.q_start, shape.pos_start, shape.slots):
            for t0 in range(0, n, self.rows):
                tiles.append((slot, r0 + t0, min(self.rows, n - t0), start + t0))
        tiles.sort(key=lambda t: -(t[3] + t[2]))
        flat = [v for t in tiles for v in t]
        host[:len(flat)] = flat
        return len(tiles)


class LatentExpandPlan:
    """Prompt portions whose keys and values are worked out for the heads before the attention: for every request behind the
    single tokens at the head of the step, the keys its rows may see, from a multiple of 16 on, as pieces of 16. On the
    device: per request slot what a key's position is added to for its row among the expanded ones, then int32 [pieces, 4] =
    (request slot, first key, keys, 0). `fill` returns the pieces, 0 when the step is to go the other way: no portions, one
    of fewer than EXPAND_MIN_ROWS rows, or more keys than there is room for: 2 x the most tokens of a step + 2,048, as many as
    the expanded keys and values have scratch for (6,144 keys take 50 MB with 16 heads where a step brings up to 2,048 tokens).
    A layer without a window so goes back to the records once a prompt is longer than that."""

    def __init__(self, window: int, max_requests: int = 0, max_tokens: int = 0):
        self.window = int(window)
        self.max_requests, self.max_tokens = int(max_requests), int(max_tokens)
        self.name = f"latent_expand:{self.window}"

    @staticmethod
    def most_pieces(max_tokens: int) -> int:
        return (2 * max_tokens + 2048) // 16

    def ints(self, max_tokens: int, max_requests: int) -> int:
        # (the same in the buffers of small steps: which way a prompt goes must not change with the size of its portions)
        return (max_requests + 3) // 4 * 4 + 4 * self.most_pieces(max(max_tokens, self.max_tokens))

    def fill(self, host, shape) -> tuple:
        requests = (self.max_requests + 3) // 4 * 4
        room = (len(host) - requests) // 4
        lead = 0
        while lead < len(shape.q_len) and shape.q_len[lead] == 1:
            lead += 1
        portions = list(zip(shape.q_len, shape.pos_start, shape.slots))[lead:]
        if not portions or min(n for n, _, _ in portions) < EXPAND_MIN_ROWS:
            return 0, requests
        spans, total = [], 0
        for n, start, slot in portions:
            lo = max(0, start - self.window + 1) // 16 * 16 if self.window > 0 else 0
            count = -(-(start + n - lo) // 16)
            spans.append((slot, lo, start + n, count))
            total += count
        if total > room:
            return 0, requests
        at = 0
        pieces = host[requests:requests + 4 * total].reshape(total, 4)
        for slot, lo, hi, count in spans:
            keys = np.arange(lo, lo + 16 * count, 16, dtype=np.int32)
            host[slot] = 16 * at - lo
            part = pieces[at:at + count]
            part[:, 0], part[:, 1], part[:, 2], part[:, 3] = slot, keys, np.minimum(16, hi - keys), 0
            at += count
        return total, requests


# Rows of a portion from which its keys and values are expanded: expanding costs a key 2 R heads (d + e) operations once, and
# saves a row 2 heads (2 R - d - e) for every key it sees, on a kernel four times as fast: even at some 45 rows when all keys
# are new to the step. Measured on B200, three steps of a Rematar model (width 2,048) that bring a prompt in portions beside
# four single tokens, expanded / absorbed: portions of 64 1,685 / 1,843 us, of 256 2,019 / 2,170; two prompts of 394 and 1,383
# tokens, the attention of a layer 38 + 4 us and the product / 299 us. The longer the context, the more it gains, small portions
# too (a step of one portion through eight layers, 16 heads, 64 rows / 400 rows): at the start 642 against 786 / 927 against 1,262,
# behind 1,500 keys 1,175 against 1,834 / 1,431 against 3,135, behind 5,500 2,411 against 4,364 / 2,715 against 8,047.
EXPAND_MIN_ROWS = 64
EXPAND_SIZES = (128, 64, 128)      # (own numbers of a key, turned piece, values) of the tcgen05 kernel

_expand_plans = {}


def expand_plan(spec, max_requests: int, max_tokens: int):
    """The plan for a layer of these sizes, or None where the tcgen05 kernel has no such sizes, or not its scale: it takes a row's
    largest score before it scales the scores, the kernel over the records after."""
    if (spec.head_dim, spec.rot_dim, spec.value_dim) != EXPAND_SIZES or spec.kv_rank % 8 or not float(spec.scale) > 0:
        return None
    key = (int(spec.get("window", 0)), int(max_requests), int(max_tokens))
    plan = _expand_plans.get(key)
    if plan is None:
        plan = _expand_plans[key] = LatentExpandPlan(*key)
    return plan


_plans = {}


def tile_plan(spec) -> LatentTilePlan:
    rows = max(1, UNITS // heads_per_block(spec.num_heads))
    plan = _plans.get(rows)
    if plan is None:
        plan = _plans[rows] = LatentTilePlan(rows)
    return plan


def flash_applies(spec, dtype) -> bool:
    return (dtype == torch.bfloat16 and spec.kv_rank % 8 == 0 and spec.rot_dim % 8 == 0 and spec.kv_rank <= 512
            and ops.latent_flash_fits(spec.kv_rank, spec.rot_dim))


KEY_TILE = 64           # keys to a tile of the tensor-core kernel
PART_ROWS = 64          # steps of single tokens up to this many rows may deal their keys over several blocks
MAX_PARTS = 16


def key_parts(ctx, spec, sms: int = 0, single_rows: int = 0) -> int:
    """Into how many parts the keys of every query tile are dealt. Only steps in which every request brings one token (or the
    single_rows single tokens of a step by themselves), and few of them: such a step has one block per request and group of
    heads, each walking all of its keys alone. The count follows the step's longest span of keys in powers of two (cut off at the window), so that a growing context
    keeps its launch shape, gives every part at least two key tiles, and aims at two blocks per SM."""
    rows = single_rows or (ctx.num_tokens if ctx.decode_only else PART_ROWS + 1)
    if rows > PART_ROWS:
        return 1
    window = int(spec.get("window", 0))
    span = 256
    while span < ctx.max_kv_len:
        span *= 2
    if window > 0:
        span = min(span, window)
    tiles = span // KEY_TILE + 1
    blocks = rows * -(-spec.num_heads // heads_per_block(spec.num_heads))
    want = -(-2 * (sms or sm_count()) // blocks)
    return max(1, min(want, tiles // 2, MAX_PARTS))


def attend(wide: torch.Tensor, cache, ctx, out: torch.Tensor, spec, sink, runtime=None, single=None) -> bool:
    """The tensor-core kernel over the step's tiles, or over `single` = (tiles, number) of one row each, the first rows of the
    step; False (nothing done) when it does not take this model or step."""
    if not flash_applies(spec, wide.dtype):
        return False
    planned = single or ctx.extras.get(tile_plan(spec).name)
    if planned is None:
        return False
    tiles, n_tiles = planned
    (records,) = cache.arrays
    parts = key_parts(ctx, spec, single_rows=n_tiles if single else 0) if runtime is not None else 1
    scratch = None
    if parts > 1:
        scratch = runtime.flat(f"latent_parts_{spec.num_heads}_{spec.kv_rank}",
                               PART_ROWS * spec.num_heads * MAX_PARTS * (spec.kv_rank + 2))
    ops.latent_attention_flash(wide, records, cache.block_table, tiles, n_tiles, sink, out, spec.num_heads, spec.kv_rank,
                               spec.rot_dim, cache.page_size, float(spec.scale), int(spec.get("window", 0)),
                               heads_per_block(spec.num_heads), parts, scratch)
    return True
