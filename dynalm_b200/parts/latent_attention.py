"""Attention whose keys and values are projections of a cached latent: the "latent_attention" mixer.

Per token the layer's input h gives a query latent and a key/value latent:

    c_q = rmsnorm(dq h) * dq_norm,   q = uq c_q                  H heads of [d unrotated | r rotated] numbers
    c   = rmsnorm((dkv h)[:R]) * dkv_norm,   k_rot = (dkv h)[R:]    one rotated key part of r numbers for all heads
    k_h = uk_h c,  v_h = uv_h c                                    (d and e numbers per head)
    s   = scale * (q_h[:d] . k_h + rot(q_h[d:]) . rot(k_rot))
    p   = exp(s) / (sum over the window of exp(s) + exp(sink_h))   the sink has no key and no value
    out = o( concat_h(sum p v_h) * sigmoid(g h) )

With q_rank 0 there is no query latent: q = q h (tensor "q" instead of dq, dq_norm and uq), one product with the rest.

Only c and rot(k_rot) are cached, as one record per token, and the attention runs on the records themselves: since
q_h . uk_h c = (uk_h^T q_h) . c, every head gets a "wide" query [uk_h^T q_h | rot(q_h[d:])] of R + r numbers that is
scored against the records, the softmax weights sum the records' latents, and uv_h is applied to that sum. The two
per-head products are block-diagonal (ops.head_linear). The window (0: every earlier key) also tells the cache
manager which pages may be given back.

All sizes and constants come from the spec: num_heads, head_dim (d), rot_dim (r), value_dim (e), q_rank, kv_rank (R),
scale, window, eps, position (a PositionSpec of kind "rotary_interleaved" or "rotary_halves", or None); the sinks and the
output gate are there when the model has their tensors. The kernels turn neighbours: for a rotation by halves the rows of
the projections that make the rotated parts of queries and keys are put in another order at load time, pair by pair, which
changes no score.
"""

from __future__ import annotations

from typing import Dict, Optional

import torch

from ..errors import Unsupported
from ..kernels import linear, ops
from ..kernels.attention import QUERY_TILES
from ..kernels.gemm import linear_partial, linear_short
from .base import POSITIONS, CacheSpec, TensorDecl, register_mixer


@register_mixer("latent_attention")
class LatentAttention:
    replay_safe = True     # all device work goes through the recorded launches of kernels/ops.py (engine/launch_memo.py)
    graph_safe = True      # launches depend on row counts only
    portions_graph_safe = True      # the same of steps with prompt portions, given the plans' answers and the span (engine/step.py)

    @staticmethod
    def declare(spec) -> Dict[str, TensorDecl]:
        H, d, r, e = spec.num_heads, spec.head_dim, spec.rot_dim, spec.value_dim
        query = {"q": TensorDecl((H * (d + r), spec.width))} if spec.q_rank == 0 else {
            "dq": TensorDecl((spec.q_rank, spec.width)),
            "dq_norm": TensorDecl((spec.q_rank,), role="vector", init="around_one"),
            "uq": TensorDecl((H * (d + r), spec.q_rank))}
        return {
            **query,
            "dkv": TensorDecl((spec.kv_rank + r, spec.width)),
            "dkv_norm": TensorDecl((spec.kv_rank,), role="vector", init="around_one"),
            "uk": TensorDecl((H * d, spec.kv_rank)),
            "uv": TensorDecl((H * e, spec.kv_rank)),
            "sink": TensorDecl((H,), role="vector", required=False, init="bias"),
            "gate": TensorDecl((H * e, spec.width), required=False),
            "o": TensorDecl((spec.width, H * e)),
        }

    def __init__(self, spec, tensors: Dict[str, torch.Tensor], runtime):
        H, d, r, e, R = spec.num_heads, spec.head_dim, spec.rot_dim, spec.value_dim, spec.kv_rank
        if R > 1024 or R + r > 8192:
            raise Unsupported(f"latent_attention: a latent of {R} numbers has no kernel (1,024 at most)")
        self.spec = spec
        self.rt = runtime
        self.has_gate = "gate" in tensors
        # one product for everything that reads the layer's input: [query latent or queries | latent | key part | gate]
        self.q_cols = spec.q_rank or H * (d + r)
        pos = spec.get("position")
        self.position = POSITIONS.get(pos.kind)(pos, runtime) if pos is not None else None
        w_q, w_dkv = tensors["uq"] if spec.q_rank else tensors["q"], tensors["dkv"]
        if getattr(self.position, "halves", False):
            order = self.position.neighbours(r).to(w_q.device)
            per_head = w_q.reshape(H, d + r, -1)
            w_q = torch.cat([per_head[:, :d], per_head[:, d:][:, order]], dim=1).reshape(H * (d + r), -1).contiguous()
            w_dkv = torch.cat([w_dkv[:R], w_dkv[R:][order]], dim=0)
        elif self.position is not None and not getattr(self.position, "interleaved", False):
            raise Unsupported(f"latent_attention: position encoding '{pos.kind}' has no kernel here (rotary_interleaved and "
                              f"rotary_halves have)")
        down = [tensors["dq"] if spec.q_rank else w_q, w_dkv] + ([tensors["gate"]] if self.has_gate else [])
        self.w_down = torch.cat(down, dim=0).contiguous()
        self.dq_norm, self.dkv_norm = tensors.get("dq_norm"), tensors["dkv_norm"]
        self.w_uq = w_q if spec.q_rank else None
        self.joined_col = self.w_down.shape[0]
        self.w_uk = tensors["uk"].reshape(H, d, R).contiguous()                          # [H, in = d, out = R] as stored
        self.w_uv = tensors["uv"].reshape(H, e, R).transpose(1, 2).contiguous()          # [H, in = R, out = e]
        # for prompt portions at the sizes of the tcgen05 kernel: one product gives every head's keys and values of a record
        from ..kernels import latent_attention as fast
        self.expand = None
        if self.rt.dtype == torch.bfloat16 and fast.flash_applies(spec, self.rt.dtype):
            self.expand = fast.expand_plan(spec, runtime.max_requests, runtime.max_tokens)
        self.w_kv = torch.cat([tensors["uk"], tensors["uv"]], dim=0).contiguous() if self.expand is not None else None
        self.sink = tensors.get("sink")
        self.w_o = tensors["o"]
        self.eps = float(spec.eps)
        self.rot = self.position.rotary_dim if self.position is not None else 0
        self.freq = self.position.frequencies if self.position is not None else None
        self.mag = self.position.magnitude if self.position is not None else 1.0

    def join_input(self, w: torch.Tensor) -> bool:
        """Takes the rows of another product over the same input into this part's first one; `joined` gives its result."""
        self.w_down = torch.cat([self.w_down, w], dim=0).contiguous()
        return True

    def joined(self, rows: int) -> torch.Tensor:
        return self.rt.buffer("latent_down", (rows, self.w_down.shape[0]))[:, self.joined_col:]

    def first_weights(self) -> torch.Tensor:
        return self.w_down

    def step_plans(self) -> list:
        """The query tiles of the step, for the tensor-core kernel (kernels/latent_attention.py)."""
        from ..kernels import latent_attention as fast
        plans = [fast.tile_plan(self.spec)] if fast.flash_applies(self.spec, self.rt.dtype) else []
        return plans + ([QUERY_TILES, self.expand] if self.expand is not None else [])

    def graph_key(self, ctx) -> tuple:
        from ..kernels import latent_attention as fast
        return (("latent_parts", fast.key_parts(ctx, self.spec)),) if fast.flash_applies(self.spec, self.rt.dtype) else ()

    def cache_spec(self) -> Optional[CacheSpec]:
        s = self.spec
        return CacheSpec(kind="pages", entry_shape=(s.kv_rank + s.rot_dim,), tensors=1, window=int(s.get("window", 0)))

    def forward(self, x: torch.Tensor, ctx, cache, owns_cache: bool = True) -> torch.Tensor:
        """x: [rows, width] in the compute dtype -> [rows, width] (or split-K partial sums of it)."""
        s, rt = self.spec, self.rt
        if not owns_cache:
            raise Unsupported("latent_attention: every run of the layer writes records of its own")
        H, d, r, e, R = s.num_heads, s.head_dim, s.rot_dim, s.value_dim, s.kv_rank
        rows = x.shape[0]
        (records,) = cache.arrays
        down = rt.buffer("latent_down", (rows, self.w_down.shape[0]))
        linear(x, self.w_down, down, runtime=rt)
        if s.q_rank:
            cq = rt.buffer("latent_cq", (rows, s.q_rank))
            ops.latent_prep(down, s.q_rank, R, r, self.rot, self.dq_norm, self.dkv_norm, self.eps, self.freq, ctx.positions,
                            ctx.row_slot, cache.block_table, records, cache.page_size, cq, self.mag)
            q = rt.buffer("latent_q", (rows, H * (d + r)))
            linear(cq, self.w_uq, q, runtime=rt)
        else:
            q = down[:, :self.q_cols]
            ops.latent_prep(down[:, self.q_cols:], 0, R, r, self.rot, None, self.dkv_norm, self.eps, self.freq, ctx.positions,
                            ctx.row_slot, cache.block_table, records, cache.page_size, None, self.mag)
        heads = rt.buffer("latent_heads", (rows, H * e))
        gate = down[:, self.q_cols + R + r:] if self.has_gate else None
        if not self._expanded(q, gate, cache, ctx, heads):
            self._absorbed(q, gate, cache, ctx, heads, rows, None)
        return linear_partial(heads, self.w_o, rt, "mixer_out")

    def _absorbed(self, q: torch.Tensor, gate: Optional[torch.Tensor], cache, ctx, heads: torch.Tensor, rows: int, single) -> None:
        """The first `rows` rows with the up-projections on the queries' and the results' side, over the records as they are."""
        s, rt = self.spec, self.rt
        H, d, r, e, R = s.num_heads, s.head_dim, s.rot_dim, s.value_dim, s.kv_rank
        q, heads = q[:rows], heads[:rows]
        wide = rt.buffer("latent_wide_q", (rows, H * (R + r)))
        ops.head_linear(q, d + r, d, self.w_uk, wide, R + r)
        if r:
            ops.rotate_pairs(q, d + r, d, wide, R + r, R, r, self.rot, self.freq, ctx.positions, H, self.mag)
        mixed = rt.buffer("latent_mixed", (rows, H * R))
        self.attend(wide, cache, ctx, mixed, single)
        ops.head_linear(mixed, R, R, self.w_uv, heads, e, gate, e)

    def _expanded(self, q: torch.Tensor, gate: Optional[torch.Tensor], cache, ctx, heads: torch.Tensor) -> bool:
        """A step whose portions' keys and values are worked out first (kernels/latent_attention.LatentExpandPlan): the portions
        through the tcgen05 kernel, the single tokens at the step's head beside them the other way. False: nothing done."""
        planned = ctx.extras.get(self.expand.name) if self.expand is not None else None
        tiles = ctx.extras.get(QUERY_TILES.name)
        if planned is None or tiles is None or planned[1][0] == 0 or cache.page_size < 16 or cache.page_size & (cache.page_size - 1) \
                or q.stride(0) % 8 or q.data_ptr() % 16:
            return False
        s, rt = self.spec, self.rt
        H, d, r, e, R = s.num_heads, s.head_dim, s.rot_dim, s.value_dim, s.kv_rank
        (records,) = cache.arrays
        ints, (pieces, first_piece) = planned
        most = 16 * self.expand.most_pieces(rt.max_tokens)
        latents = rt.spare(f"latent_rows_{R + r}", most * (R + r), torch.bfloat16)
        kv = rt.spare(f"latent_kv_{H * (d + e)}", most * H * (d + e), torch.bfloat16) if latents is not None else None
        if kv is None:
            return False
        q_tiles, (_, n_tiles, lead) = tiles
        from ..kernels import attention
        side = rt.side_stream if lead > 0 and attention.SIDE_BY_SIDE else None
        if side is not None:
            ops.stream_fork(side)
            with ops.on_stream(side):
                self._absorbed(q, gate, cache, ctx, heads, lead, (q_tiles[4 * n_tiles:], lead))
        elif lead > 0:
            self._absorbed(q, gate, cache, ctx, heads, lead, (q_tiles[4 * n_tiles:], lead))
        keys = 16 * pieces
        latents = latents[:keys * (R + r)].view(keys, R + r)
        kv = kv[:keys * H * (d + e)].view(keys, H * (d + e))
        ops.latent_gather(records, cache.block_table, cache.page_size, ints[first_piece:], pieces, latents)
        linear_short(latents[:, :R], self.w_kv, kv)
        rows = q.shape[0]
        q_rot = rt.buffer("latent_q_rot", (rows, H * r))
        ops.rotate_pairs(q, d + r, d, q_rot, r, 0, r, self.rot, self.freq, ctx.positions, H, self.mag)
        ops.latent_attention_tcgen05(q, q_rot, latents, R, kv, ints, q_tiles, n_tiles, heads, H, float(s.scale),
                                     int(s.get("window", 0)), self.sink)
        if gate is not None:
            ops.sigmoid_gate(heads[lead:], gate[lead:])
        if side is not None:
            ops.stream_join(side)
        return True

    def attend(self, wide: torch.Tensor, cache, ctx, out: torch.Tensor, single=None) -> None:
        s = self.spec
        (records,) = cache.arrays
        from ..kernels import latent_attention as fast
        if fast.attend(wide, cache, ctx, out, s, self.sink, self.rt, single):
            return
        ops.latent_attention(wide, records, cache.block_table, ctx.positions, ctx.row_slot, self.sink, out, s.num_heads,
                             s.kv_rank, s.rot_dim, cache.page_size, float(s.scale), int(s.get("window", 0)))
