"""A step's pre-norm layers launched by one native call.

A step that brings a prompt portion is launched kernel by kernel from the host, and with few rows the host is what it waits
for: at the 3B sizes 77 rows take the GPU 60 to 90 us a layer and the host, from Python, 110 to 140.  Where a model's layers are
all of the common kind (:class:`~inferflux_b200.parts.block.PreNormBlock` of grouped-query attention and SwiGLU with RMSNorm,
bfloat16, head size 128, no window) such a step's layers are launched by ``ops.prenorm_layers``: the same kernels with the same
arguments, so the same results.  Everything else goes through the blocks; so does a model of which a block or one of its parts has
been given a method of its own since it was made (to watch it, say) or been replaced.
"""
from __future__ import annotations

from typing import Optional

import numpy as np
import torch

from ..kernels import ops
from ..parts.attention import GQAttention, prefill_plan
from ..parts.base import PartialSums
from ..parts.block import PreNormBlock
from ..parts.feed_forward import FUSED_PRODUCT_ROWS, SwiGLU
from ..parts.linear import FEW_ROWS, FEW_ROWS_MIN_K, GEMV_ROWS, Linear
from ..parts.norm import RMSNorm

#: The rows for which the parts take the kernels of the call: more than the weight-streaming product's, no more than the few-row kernels'.
MIN_ROWS, MAX_ROWS = GEMV_ROWS + 1, min(FEW_ROWS, FUSED_PRODUCT_ROWS)

#: What the call stands in for: the kinds of a layer's parts with the methods that launch their kernels, as they are here.
_STANDS_FOR = {cls: {name: getattr(cls, name) for name in names} for cls, names in (
    (PreNormBlock, ("forward",)), (RMSNorm, ("forward",)), (SwiGLU, ("forward",)), (Linear, ("forward",)),
    (GQAttention, ("forward", "attend", "decode", "_fused_qkv", "_share_by_tiles")))}


_MIXERS_OWN = frozenset(_STANDS_FOR[GQAttention])


def _sizes(block) -> tuple:
    m = block.mixer
    return block.position_name, m.hidden, m.n_heads, m.n_kv, m.head_dim, m.scale, m.window, m.kv_shared, block.feed_forward.intermediate


class PrenormRun:
    """The layers of a model that one call can launch: all of its runs or none."""

    def __init__(self, blocks):
        self.blocks = blocks                            # one per run, in schedule order (the model holds this, not the other way round too)
        self.sizes = _sizes(blocks[0])

    @staticmethod
    def of(model) -> Optional["PrenormRun"]:
        blocks = [model.blocks[r.layer] for r in model.spec.schedule]
        if model.dtype != torch.bfloat16 or not blocks:
            return None
        shapes = set()
        for block, info in zip(blocks, model.runs):
            if type(block) is not PreNormBlock or type(block.mixer) is not GQAttention or type(block.feed_forward) is not SwiGLU:
                return None
            if type(block.mixer_norm) is not RMSNorm or type(block.feed_forward_norm) is not RMSNorm:
                return None
            a = block.mixer
            if a.window or a.kv_shared or not info.writes_kv or a.head_dim != ops.UMMA_ATTENTION_HEAD_DIM or a.params.get("o_bias"):
                return None
            shapes.add((info.kv_group, *_sizes(block)))
        # (a shorter down projection goes to the library, which the call does not reach)
        if len(shapes) != 1 or blocks[0].mixer.hidden % 8 or blocks[0].feed_forward.intermediate % 8 or blocks[0].feed_forward.intermediate < FEW_ROWS_MIN_K:
            return None
        return PrenormRun(blocks)

    def takes(self, model, ctx) -> bool:
        step = ctx.extras[GQAttention.describe_key]
        return MIN_ROWS <= ctx.n_tokens <= MAX_ROWS and step.n_decode != ctx.n_tokens and self._as_made(model)

    def _as_made(self, model) -> bool:
        """Whether blocks and parts are still of the kinds that the call stands in for, with these kinds' own methods (a microsecond a
        layer)."""
        for cls, methods in _STANDS_FOR.items():
            if any(getattr(cls, name) is not method for name, method in methods.items()):
                return False
        for b, run in zip(self.blocks, model.spec.schedule):
            if model.blocks[run.layer] is not b:
                return False
            m, f = b.mixer, b.feed_forward
            if not (type(b) is PreNormBlock and type(m) is GQAttention and type(f) is SwiGLU and type(b.mixer_norm) is RMSNorm
                    and type(b.feed_forward_norm) is RMSNorm and _MIXERS_OWN.isdisjoint(m.__dict__) and _sizes(b) == self.sizes):
                return False
            for linear in (m.qkv, m.o, f.gate_up, f.down):
                if type(linear) is not Linear or "forward" in linear.__dict__:
                    return False
            for part in (b, f, b.mixer_norm, b.feed_forward_norm):
                if "forward" in part.__dict__:
                    return False
        return True

    def forward(self, residual: torch.Tensor, ctx, runs) -> Optional[PartialSums]:
        """All layers; the last one's pending delta.  None (nothing done): weights, angles or a cache of which the kernels of the call
        take no such form; the blocks choose others, or refuse them."""
        first, n, dev = self.blocks[0].mixer, ctx.n_tokens, residual.device
        hidden, inter, nh, nkv, hd = first.hidden, self.blocks[0].feed_forward.intermediate, first.n_heads, first.n_kv, first.head_dim
        width, g, page = (nh + 2 * nkv) * hd, runs[0].kv_group, nkv * ctx.page_size * hd
        position = ctx.position_tables.get(self.blocks[0].position_name) if self.blocks[0].position_name else None
        if not isinstance(position, (tuple, list)) or len(position) != 2:
            return None
        cos, sin = position
        if any(t.shape != (n, hd // 2) or t.dtype != torch.float32 or not t.is_contiguous() for t in position):
            return None
        if not residual.is_contiguous() or residual.dtype != torch.float32 or ctx.slot_maps[g].dtype != torch.int32 or ctx.slot_maps[g].numel() != n:
            return None
        tables = ctx.block_tables[g]
        if tables.dtype != torch.int32 or tables.stride(1) != 1:
            return None
        shapes = ((width, hidden), (hidden, nh * hd), (2 * inter, hidden), (hidden, inter))
        words = []
        for block, info in zip(self.blocks, runs):
            a, f = block.mixer, block.feed_forward
            k, v, page_stride = ctx.kv.layer_views(info.kv_group, info.kv_index)
            if k.dtype != torch.bfloat16 or v.dtype != torch.bfloat16 or (not words and ops.paged_pool_pages(k, v, page_stride, page) < 1):
                return None
            at = []
            for linear, shape in zip((a.qkv, a.o, f.gate_up, f.down), shapes):
                w = linear.weight
                at.append(w.data_ptr())
                if w.dtype != torch.bfloat16 or w.shape != shape or at[-1] & 15 or not w.is_contiguous() or linear.bias is not None:
                    return None
            bias, norms = a.qkv_bias, (block.mixer_norm.weight, block.feed_forward_norm.weight)
            if bias is not None and (bias.dtype != torch.float32 or bias.numel() != width or not bias.is_contiguous()):
                return None
            if any(w.dtype != torch.float32 or w.numel() != hidden for w in norms):
                return None
            words.append((norms[0].data_ptr(), at[0], 0 if bias is None else bias.data_ptr(), k.data_ptr(), v.data_ptr(), at[1],
                          norms[1].data_ptr(), at[2], at[3], 0, 0))
        layers = np.array(words, dtype=np.int64)
        eps = layers.view(np.float64)
        eps[:, 9] = [b.mixer_norm.eps for b in self.blocks]
        eps[:, 10] = [b.feed_forward_norm.eps for b in self.blocks]

        step = ctx.extras[GQAttention.describe_key]
        s = ops.PrenormStep()
        keep = []                                       # scratch stays until the kernels are launched (then the stream orders its reuse)

        def scratch(dtype, count):
            t = torch.empty(count, dtype=dtype, device=dev)
            keep.append(t)
            return t.data_ptr()
        bf16, f32 = torch.bfloat16, torch.float32
        s.rows, s.hidden, s.inter, s.n_heads, s.n_kv, s.page_size = n, hidden, inter, nh, nkv, ctx.page_size
        s.qkv_parts = ops.gemm_umma_skinny_parts(width, hidden, n)
        s.o_parts = ops.gemm_umma_skinny_parts(hidden, nh * hd, n)
        s.down_parts = ops.gemm_umma_skinny_parts(hidden, inter, n)
        delta = torch.empty((max(s.o_parts, s.down_parts), n, hidden), dtype=f32, device=dev)
        s.residual, s.delta = residual.data_ptr(), delta.data_ptr()
        s.x, s.qkv, s.attn, s.act = (scratch(bf16, n * w) for w in (hidden, width, nh * hd, inter))
        s.qkv_sums = scratch(f32, s.qkv_parts * n * width)
        s.cos_t, s.sin_t, s.slot_map = cos.data_ptr(), sin.data_ptr(), ctx.slot_maps[g].data_ptr()
        s.block_tables, s.bt_stride, s.page_stride = tables.data_ptr(), tables.stride(0), page_stride
        s.entry_q_start, s.entry_q_len, s.entry_ctx_start = (t.data_ptr() for t in (ctx.entry_q_start, ctx.entry_q_len, ctx.entry_ctx_start))
        s.num_pages = ops.paged_pool_pages(k, v, page_stride, page)
        s.gate_up_streams = n <= ops.GEMV_MAX_ROWS
        s.scale = first.scale
        s.n_tiles, s.tile_rows = step.n_umma_tiles, step.umma_tile_rows
        s.tile_entry, s.tile_q0 = step.umma_tile_entry.data_ptr(), step.umma_tile_q0.data_ptr()
        s.n_splits = prefill_plan(ctx, 2, step.umma_tile_rows, nh, ctx.max_ctx_len, 0)[0]
        if s.n_splits > 1:
            rows = ops.attn_prefill_cut_units(s.n_tiles, nh) * s.n_splits * ops.UMMA_ATTENTION_TILE
            s.part_o, s.part_ml = scratch(f32, rows * hd), scratch(f32, rows * 2)
        s.n_dec, s.dec_splits = step.n_decode, 1
        if step.n_decode:
            s.dec_entries = step.decode_entries.data_ptr()
            if first._share_by_tiles(step):
                s.dec_pieces = ops.attn_decode_pieces(nh, nkv, hd, ctx.max_ctx_len)
                s.piece_count = scratch(torch.int32, step.n_decode * nh)
            else:
                s.dec_splits = ops.attn_decode_splits(step.n_decode, nh, nkv, hd, ctx.max_ctx_len)
            rows = step.n_decode * nh * max(s.dec_pieces, s.dec_splits)
            s.dec_o, s.dec_ml = scratch(f32, rows * hd), scratch(f32, rows * 2)
        ops.prenorm_layers(s, layers, dev)
        return PartialSums(delta[:s.down_parts])
