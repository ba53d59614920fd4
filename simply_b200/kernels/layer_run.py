"""The layers of a step in one call from the host (csrc/layer_run.cu), for models whose layers are all of one shape.

`UniformLayers` says whether a model's blocks are such (sandwich or pre-norm blocks of `paged_attention` and `gated`, RMS
norms, every layer run once with a cache of its own); `run` hands their tensors and the step's over.  The launches are
the ones the parts would make.  What a step or a model needs beyond that (another kernel table, float32, captured
steps of single tokens, an option of the table) goes layer by layer through the parts.
"""

from __future__ import annotations

import ctypes
from typing import Any

import numpy as np
import torch

from simply_b200.kernels.ops import CudaOps
from simply_b200.parts.attention import PagedAttention
from simply_b200.parts.block import PreNormBlock, SandwichNormBlock
from simply_b200.parts.feedforward import GatedFeedForward
from simply_b200.parts.linear import Linear
from simply_b200.parts.norm import RMSNorm

_P, _I, _F, _L = ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_longlong
_OTHER = ctypes.CFUNCTYPE(_I, _I, _I)


class _Attention(ctypes.Structure):
  _fields_ = ([(n, _P) for n in ("prefill_items", "decode_items", "split_start", "split_count", "part_o", "part_ml")]
              + [(n, _I) for n in ("num_prefill", "num_decode", "chunk", "rows_max", "window", "unused")])


class _Step(ctypes.Structure):
  _fields_ = ([(n, _P) for n in ("token_seq", "positions", "cu_q", "q_start", "h", "y", "qkv", "q", "attended", "mixed",
                                 "gate_up", "z", "down", "library_workspace")]
              + [("library_bytes", _L)] + [(n, _P) for n in ("work_counter", "err", "prefill", "decode")]
              + [(n, _I) for n in ("tokens", "width", "hidden", "num_q_heads", "num_kv_heads", "head_dim", "page_size",
                                   "activation", "scales_f32", "plus_one", "older_keys_settled", "few_rows", "mid_qkv",
                                   "mid_gated", "mid_plain", "gated_tc_rows")]
              + [(n, _F) for n in ("limit", "q_scale", "cap", "eps")])


LAYER_WORDS = 16  # numbers of 64 bits per layer

# Operations of a layer's products from which the parts issue a step's launches as fast as the device runs them (about
# 90 us a layer).  Beyond it nothing is gained, and a queue that is always full was measured to cost 0.3 to 0.5 % (us,
# parts and one call, Gemma 2 2B: 13 tokens 2,478 and 1,660, 90 3,507 and 2,215, 2,048 8,715 and 8,763; 7 prompts of
# 3,300 in all 13,982 and 14,025; 9B, 300 tokens 10,953 and 10,941, 3,001 50,544 and 50,746).
MOST_OPERATIONS = 1e11

# What the one call stands for: where one of these has been replaced, on the kernel table, its class, a part or a part's
# class (a tracer's or a test's), the layers go part by part.
STANDS_FOR = frozenset(("residual_norm", "project_rotate_store", "rope_and_cache_write", "paged_attention", "linear",
                        "gated_linear", "gated_activation", "_call"))
OWN_CALLS = [(CudaOps, name, vars(CudaOps)[name]) for name in STANDS_FOR] + [
    (c, "forward", c.forward) for c in (SandwichNormBlock, PreNormBlock, PagedAttention, GatedFeedForward)] + [
    (Linear, "__call__", Linear.__call__)]


class UniformLayers:

  def __init__(self, blocks: list, names: list[str]):
    self.blocks, self.names = blocks, names
    m, f = blocks[0].mixer, blocks[0].feed_forward
    self.head_dim, self.group = m.head_dim, m.num_heads // m.num_kv_heads
    # 2 operations per weight and token: q, k, v, output, gate, up, down
    self.operations_per_token = 2.0 * m.width * (2 * (m.num_heads + m.num_kv_heads) * m.head_dim + 3 * f.hidden)

  @classmethod
  def of(cls, model: Any) -> "UniformLayers | None":
    """The model's layers, or None where they are not all of one such shape."""
    calls = model.spec.run_order
    blocks = [model.blocks[c.layer] for c in calls]
    if len({c.layer for c in calls}) < len(calls) or any(
        c.add_embedding or c.stream_input is not None or c.mixer_cache is not None or not c.writes_cache for c in calls):
      return None
    for b in blocks:
      m, f = b.mixer, getattr(b, "feed_forward", None)
      if (type(b) not in (SandwichNormBlock, PreNormBlock) or type(m) is not PagedAttention or not m.project_kv
          or type(f) is not GatedFeedForward or any(type(n) is not RMSNorm for n in b._norms())):
        return None
    def alike(get) -> bool:
      return len({get(b) for b in blocks}) == 1
    if not all(alike(g) for g in (
        type, lambda b: (b.mixer.width, b.mixer.num_heads, b.mixer.num_kv_heads, b.mixer.head_dim, b.mixer.query_scale,
                         b.mixer.logit_softcap),
        lambda b: (b.feed_forward.hidden, b.feed_forward.activation, b.feed_forward.limit))):
      return None
    norms = [n for b in blocks for n in b._norms()]
    if len({(n.eps, n.plus_one) for n in norms}) != 1:
      return None
    return cls(blocks, list(model.cache_names))

  def takes(self, ctx: Any) -> bool:
    """Whether this step goes this way (its table's options at their defaults)."""
    o = ctx.ops
    return (o.layer_runs and ctx.num_tokens * self.operations_per_token <= MOST_OPERATIONS and o.dtype == torch.bfloat16
            and ctx.max_q_len > 1 and o.fused_qkv_rope and o.direct_library_products and o.gated_tc_pairs
            and not (o.skinny_warps or o.gated_tc_blocks or o.mid_split or o.mid_stages or o.decode_variant)
            and STANDS_FOR.isdisjoint(vars(o)) and all(getattr(c, name) is call for c, name, call in OWN_CALLS)
            and not any("forward" in vars(part) for b in self.blocks for part in (b, b.mixer, b.feed_forward))
            and all(type(b.mixer.o_proj) is Linear and type(b.feed_forward.down_proj) is Linear for b in self.blocks)
            and o._uses_tensor_core_attention(self.head_dim, self.group)
            and o._prefill_uses_tcgen05(self.head_dim, self.group, ctx.page_size))

  def run(self, h: torch.Tensor, ctx: Any, caches: dict[str, Any]):
    """Runs the layers over the stream h (float32, updated in place); returns the last layer's branch, which is
    still to be added (with that layer's post norm), or None: nothing has run, the parts are to do it."""
    o, t = ctx.ops, ctx.num_tokens
    first = self.blocks[0]
    m, f = first.mixer, first.feed_forward
    heads, kv_heads, dim, width, hidden = m.num_heads, m.num_kv_heads, m.head_dim, m.width, f.hidden
    group = self.group
    scales = first.pre_mixer.weight.dtype
    for b in self.blocks:
      products = (b.mixer.qkv_weight, b.mixer.o_proj.weight, b.feed_forward.gate_up_weight, b.feed_forward.down_proj.weight)
      if any(w.dtype != torch.bfloat16 or not w.is_contiguous() for w in products) or any(
          n.weight.dtype != scales for n in b._norms()):
        return None
    pair = o._prefill_uses_pairs(dim, group, ctx.page_size)
    fns = o._attention_lib(dim)
    prefill, decode = fns[4] if pair else fns[3], fns[1]
    new = lambda *shape: torch.empty(shape, dtype=torch.bfloat16, device=o.device)
    kinds: dict[int | None, int] = {}
    attentions, held = [], []
    for b in self.blocks:
      if b.mixer.window in kinds:
        continue
      kinds[b.mixer.window] = len(kinds)
      plan = o._attention_plan(ctx, b.mixer.window, group, 256 if pair else 128, kv_heads, dim)
      n = plan["num_decode"] * kv_heads * plan["rows_max"]
      part_o = torch.empty(n * dim, dtype=torch.float32, device=o.device)
      part_ml = torch.empty(n * 2, dtype=torch.float32, device=o.device)
      held += [plan, part_o, part_ml]
      attentions.append(_Attention(
          plan["prefill_items"].data_ptr(), plan["decode_items"].data_ptr(), plan["split_start"].data_ptr(),
          plan["split_count"].data_ptr(), part_o.data_ptr(), part_ml.data_ptr(), plan["num_prefill"], plan["num_decode"],
          plan["chunk"], plan["rows_max"], int(b.mixer.window or 0), 0))
    any_decode = any(a.num_decode for a in attentions)
    at = lambda x: 0 if x is None else x.data_ptr()
    rows = []
    for b, name in zip(self.blocks, self.names):
      cache = caches[name]
      if cache.storage.dtype != torch.bfloat16 or cache.need.num_kv_heads != kv_heads:
        return None
      cos, sin = b.mixer.position.rotation_tables(ctx, dim) or (None, None)
      table = ctx.block_tables[cache.group]
      tensor_map = o._tensor_map(cache.storage, dim, ctx.page_size) if any_decode else None
      rows.append((at(b.mixer.qkv_weight), at(b.mixer.o_proj.weight), at(b.feed_forward.gate_up_weight),
                   at(b.feed_forward.down_proj.weight), at(b.pre_mixer.weight),
                   at(b.post_mixer.weight) if b.post_mixer is not None else 0, at(b.pre_feed_forward.weight),
                   at(b.post_feed_forward.weight) if b.post_feed_forward is not None else 0, at(cache.storage), at(table),
                   at(cos), at(sin), (tensor_map.value or 0) if tensor_map is not None else 0, cache.storage.shape[0],
                   table.shape[1], kinds[b.mixer.window]))
    layers = np.array(rows, dtype=np.int64)
    assert layers.shape[1] == LAYER_WORDS
    y, q, attended, mixed = new(t, width), new(t, heads, dim), new(t, heads * dim), new(t, width)
    z, down = new(t, hidden), new(t, width)
    # (what a product stores that no fused kernel takes; steps are short here, so all of it is always there)
    qkv, gate_up = new(t, (heads + 2 * kv_heads) * dim), new(t, 2 * hidden)
    mid = o.mid_rows if o.mid_rows_kernel else dict.fromkeys(o.mid_rows, 0)
    workspace = o._library_workspace()
    step = _Step(
        at(ctx.token_seq), at(ctx.positions), at(ctx.cu_q), at(ctx.q_start), at(h), at(y), at(qkv), at(q), at(attended),
        at(mixed), at(gate_up), at(z), at(down), at(workspace), workspace.numel(), at(o._attn_counter), at(o.err),
        ctypes.cast(prefill, _P).value, ctypes.cast(decode, _P).value, t, width, hidden, heads, kv_heads, dim, ctx.page_size,
        f.activation, int(scales == torch.float32), int(first.pre_mixer.plus_one),
        int(getattr(ctx, "older_keys_settled", False)), o.skinny_max_rows, mid["qkv"], mid["gated"], mid["plain"],
        o.gated_tc_min_rows, f.limit, m.query_scale, m.logit_softcap, first.pre_mixer.eps)
    failed = []

    def other(layer: int, which: int) -> int:
      # (the library has no algorithm of its own choosing for this shape: through the tensor library, as `linear` does)
      try:
        b = self.blocks[layer]
        x, w, out = ((y, b.mixer.qkv_weight, qkv), (attended, b.mixer.o_proj.weight, mixed),
                     (y, b.feed_forward.gate_up_weight, gate_up), (z, b.feed_forward.down_proj.weight, down))[which]
        torch.mm(x, w.t(), out=out)
        return 0
      except Exception as e:  # (an exception cannot pass through the caller)
        failed.append(e)
        return -1

    launches = ctypes.c_int(0)
    callback = _OTHER(other)
    rc = o.lib.sb_layer_run(layers.ctypes.data, len(rows), ctypes.byref((_Attention * len(attentions))(*attentions)),
                            ctypes.byref(step), callback, ctypes.byref(launches), o._stream())
    o.launches += launches.value
    if failed:
      raise failed[0]
    if rc:
      o._raise("sb_layer_run", rc)
    del held
    return down
