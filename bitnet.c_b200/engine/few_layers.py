"""All layers of a Llama-style model for few tokens in bfloat16, launched from one native call (csrc/few_layers.cu)."""
from __future__ import annotations

import ctypes
from ctypes import c_float, c_int, c_void_p
from typing import Optional

import torch

from ..csrc import build, ops
from ..parts.attention import Attention
from ..parts.base import Normed
from ..parts.block import PreNormBlock
from ..parts.mlp import GatedMlp
from ..parts.norm import RmsNorm
from ..parts.position import Rotary


class _Layer(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in ("w_qkv", "w_o", "w_gate_up", "w_down", "gain_ffn", "gain_next", "k_cache", "v_cache", "page_table")] + \
               [(n, c_int) for n in ("gain_ffn_dtype", "gain_next_dtype", "pt_stride", "n_cache_pages")] + [("eps_ffn", c_float), ("eps_next", c_float)]


class _Step(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in (
        "layers", "linear_tc", "resident", "rope", "decode", "decode_items", "prefill", "x", "h", "qkv", "attn", "act", "mid", "next", "delta", "mid_ss",
        "next_ss", "tok_pos", "tok_seq", "slots", "tile_seq", "tile_row0", "seq_start", "seq_pos0", "items", "part_o", "part_ml", "tickets", "status")] + \
        [(n, c_int) for n in (
            "n_layers", "M", "n_seqs", "width", "inter", "n_heads", "n_kv_heads", "head_dim", "act_code", "rotary_dims", "window", "decoding", "n_splits",
            "pages_per_block", "n_tickets", "n_items", "item_group", "n_tiles", "res_qkv", "res_o", "res_gate_up", "res_down", "cluster_o",
            "cluster_down")] + [("scale", c_float), ("theta_scale", c_float)]


def _layers(model):
    """The blocks of ``model`` in the order they run, of each the addresses of its matrices (QKV, O, gate and up, down), and of all norms (the mixers' and the
    feed-forwards' in turn, then the last one) address, type and eps; None unless all blocks are alike and of the kinds that ``bn_few_layers`` knows, with
    parameters of the types and shapes that its kernels read without another look."""
    spec = model.spec
    if (model.dtype is not torch.bfloat16 or not spec.schedule or model.embedding_norm is not None or getattr(spec, "streams", 1) != 1
            or type(model.final_norm) is not RmsNorm):
        return None
    runs, matrices, norms, blocks, bf16, gains = [], [], [], model.blocks, torch.bfloat16, (spec.width,)
    s = None
    for e in spec.schedule:
        b = blocks[e.block]
        if e.cache_of is not None or type(b) is not PreNormBlock:
            return None
        m, f = b.mixer, b.ffn
        n1, n2 = b.mixer_norm, b.ffn_norm
        if type(m) is not Attention or type(f) is not GatedMlp or type(n1) is not RmsNorm or type(n2) is not RmsNorm:
            return None
        qkv, o, gate_up, down = m.w_qkv, m.w_o, f.w_gate_up, f.w_down
        if s is None:
            s, act, inter = m.spec, f.act, down.shape[1]
            if s.head_dim > 128 or type(m.position) is not Rotary or (s.q_dim | s.kv_dim | spec.width | inter) % 8:
                return None
            shapes = ((s.q_dim + 2 * s.kv_dim, spec.width), (spec.width, s.q_dim), (2 * inter, spec.width), (spec.width, inter))
        if (m.spec is not s and m.spec != s) or f.act != act or not b.build.resident or getattr(f.spec, "wide_output", False):
            return None
        if (qkv.shape, o.shape, gate_up.shape, down.shape) != shapes:
            return None
        at = []
        for w in (qkv, o, gate_up, down):
            if w.dtype is not bf16 or not w.is_cuda or not w.is_contiguous():
                return None
            at.append(w.data_ptr())
        if (at[0] | at[1] | at[2] | at[3]) & 15:
            return None
        runs.append(b)
        matrices.append(at)
        norms += (n1, n2)
    norms.append(model.final_norm)
    for i, n in enumerate(norms):
        w = n.weight
        code = ops._DT.get(w.dtype) if w is not None else None
        if code is None or w.shape != gains or not w.is_cuda or not w.is_contiguous():
            return None
        norms[i] = (w.data_ptr(), code, n.spec.eps)
    return runs, matrices, norms


class FewLayers:
    """Runs the layers of a model from one native call.  It keeps nothing of the model, and what the kernels rely on is looked at for every step: a
    weight set anew or a cache of another shape goes the way of the parts, which take it or refuse it."""

    @staticmethod
    def of(model) -> Optional["FewLayers"]:
        """Called when all parameters are bound; None for a model whose layers are not of this kind."""
        return FewLayers() if _layers(model) is not None else None

    def __init__(self):
        self.entries = None

    def _entry_points(self):
        if self.entries is None:
            names = (("linear_tc", "bn_linear_tc_ex"), ("linear_resident", "bn_linear_resident"), ("rope", "bn_rope_append"),
                     ("attention_decode_tc", "bn_attention_decode_tc"), ("attention_decode_tc", "bn_attention_decode_tc_items"),
                     ("attention_prefill_tc", "bn_attention_prefill_tc"))
            self.entries = [ctypes.cast(getattr(build.library(lib), name), c_void_p).value for lib, name in names]
        return self.entries

    def takes(self, model, cache, ctx):
        """What ``run`` needs for a step of these tokens: the layers, where their matrices lie, and where their keys and values lie.  None if the step does not go this
        way; every switch that sends a part elsewhere sends the step there too."""
        if not (ctx.n_tokens <= ops.TC_MAX_ROWS and ctx.diag is None and ops.PROFILE is None and ops.USE_TCGEN05 and ops.USE_FUSED_NORM
                and (ctx.decode or (ctx.wide_tile_seq is not None and ops.USE_TCGEN05_ATTENTION))):
            return None
        layers = _layers(model)
        if layers is None:
            return None
        m = layers[0][0].mixer
        planes = cache.own_planes(len(layers[0]), m.spec.n_kv_heads, m.spec.head_dim, torch.bfloat16, m.w_qkv.device)
        return (*layers, planes) if planes is not None else None

    def run(self, taken, x, h, ctx, last_norm):
        """The layers on the residual x [T, width] from the first one's normed rows h; ``taken`` is what ``takes`` answered, ``last_norm`` the norm
        behind the last layer, if that layer's product is to prepare it.  Returns what is pending (as the last block would)."""
        runs, matrices, norms, planes = taken
        attention, ffn = runs[0].mixer, runs[0].ffn
        spec, T, dev = attention.spec, x.shape[0], x.device
        shapes = [tuple(w.shape) for w in (attention.w_qkv, attention.w_o, ffn.w_gate_up, ffn.w_down)]
        (n_qkv, _), (width, q_dim), (n_gu, _), (_, inter) = shapes
        steps = ("tok_pos", "slots") if ctx.decode else ("tok_pos", "slots", "tok_seq", "wide_tile_seq", "wide_tile_row0", "seq_start", "seq_pos0")
        for name in steps:
            ops._need(getattr(ctx, name), name, torch.int32, 1)
        if ctx.tok_pos.shape[0] < T or ctx.slots.shape[0] < ctx.n_seqs:
            raise ops.KernelError(f"few_layers: {ctx.tok_pos.shape[0]} positions and {ctx.slots.shape[0]} slots do not fit {T} tokens of {ctx.n_seqs} sequences")
        s = _Step()
        s.linear_tc, s.resident, s.rope, s.decode, s.decode_items, s.prefill = self._entry_points()
        sms = ops.n_sms(dev)
        s.res_qkv, s.res_o, s.res_gate_up, s.res_down = (int(ops.linear_resident_pays(T, n, k, sms)) for n, k in shapes)
        s.cluster_o, s.cluster_down = ops._auto_cluster(width, q_dim), ops._auto_cluster(width, inter)
        tiles = (width + 127) // 128
        mid_parts = (width + 15) // 16 if s.res_o else tiles * s.cluster_o
        next_parts = (width + 15) // 16 if s.res_down else tiles * s.cluster_down
        part_o = part_ml = 0
        if ctx.decode:
            if ctx.decode_items is not None:
                ops._need(ctx.decode_items, "items", torch.int32, 1)
                if not 1 <= ctx.decode_item_group <= 8 or ctx.decode_items.shape[0] % ctx.decode_item_group or ctx.decode_items.shape[0] == 0:
                    raise ops.KernelError(f"few_layers: {ctx.decode_items.shape[0]} items in groups of {ctx.decode_item_group}")
                s.items, s.n_items, s.item_group = ctx.decode_items.data_ptr(), ctx.decode_items.shape[0], ctx.decode_item_group
                splits = ctx.decode_item_group
            else:
                s.n_splits, s.pages_per_block = ops.decode_grid(ctx.max_len, T, spec.n_heads, spec.n_kv_heads)
                splits = s.n_splits
            part_o, part_ml = T * spec.n_heads * splits * spec.head_dim * 4, T * spec.n_heads * splits * 8
            counters = ops._split_scratch(dev)[1]
            s.tickets, s.n_tickets, s.decoding = counters.data_ptr(), counters.numel(), 1
        else:
            s.tok_seq, s.tile_seq, s.tile_row0 = ctx.tok_seq.data_ptr(), ctx.wide_tile_seq.data_ptr(), ctx.wide_tile_row0.data_ptr()
            s.seq_start, s.seq_pos0, s.n_tiles = ctx.seq_start.data_ptr(), ctx.seq_pos0.data_ptr(), ctx.wide_tile_seq.shape[0]
        # everything between the kernels from one allocation, pieces on 256-byte borders
        sizes = {"qkv": 2 * T * n_qkv, "attn": 2 * T * q_dim, "act": 2 * T * inter, "mid": 2 * T * width, "mid_ss": 4 * T * mid_parts, "part_o": part_o,
                 "part_ml": part_ml}
        room = torch.empty(sum((n + 255) & ~255 for n in sizes.values()), dtype=torch.uint8, device=dev)
        at = room.data_ptr()
        for name, n in sizes.items():
            setattr(s, name, at)
            at += (n + 255) & ~255
        nxt = torch.empty((T, width), dtype=torch.bfloat16, device=dev)  # rows for the next layer, or the last product itself
        ss = torch.empty((next_parts, T), dtype=torch.float32, device=dev)
        delta = torch.empty((T, width), dtype=torch.bfloat16, device=dev) if last_norm is None else None
        behind = norms[2::2] if last_norm is not None else norms[2:-1:2] + [(None, 0, 0.0)]
        layers = (_Layer * len(runs))(*[
            (*w, gain, gain_next, k, v, table, dtype, dtype_next, row, pages, eps, eps_next)
            for w, (gain, dtype, eps), (gain_next, dtype_next, eps_next), (k, v, table, row, pages) in zip(matrices, norms[1::2], behind, planes)])
        s.layers = ctypes.addressof(layers)
        s.x, s.h, s.next, s.next_ss, s.delta = x.data_ptr(), h.data_ptr(), nxt.data_ptr(), ss.data_ptr(), delta.data_ptr() if delta is not None else None
        s.tok_pos, s.slots, s.status = ctx.tok_pos.data_ptr(), ctx.slots.data_ptr(), ops.tc_status(dev).data_ptr()
        s.n_layers, s.M, s.n_seqs, s.width, s.inter, s.n_heads, s.n_kv_heads = len(runs), T, ctx.n_seqs, width, inter, spec.n_heads, spec.n_kv_heads
        s.head_dim, s.act_code, s.window, s.scale = spec.head_dim, ffn.act, spec.window, spec.softmax_scale
        s.rotary_dims, s.theta_scale = attention.position.rotary_params()
        ops.few_layers(s, len(runs) * (5 if ctx.decode else 6))
        if delta is not None:
            return delta
        return Normed(ops.RowScaled(nxt, ss, width, last_norm.spec.eps))
