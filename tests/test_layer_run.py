"""When a model's layers go to the device in one call (kernels/layer_run.py), and the structs that it hands over.  No GPU is needed."""

import ctypes
import types

import pytest

from simply_b200.config import preset
from simply_b200.kernels import build, layer_run
from simply_b200.kernels.ops import CudaOps
from simply_b200.parts.model import DecoderModel


class OwnProducts(CudaOps):

  def linear(self, x, w):
    return super().linear(x, w)


@pytest.mark.parametrize("table,replaced,want", [(CudaOps, None, True), (OwnProducts, None, False), (CudaOps, "linear", False),
                                                 (CudaOps, "paged_attention", False)])
def test_a_table_with_entry_points_of_its_own_goes_part_by_part(monkeypatch, table, replaced, want):
  ops = object.__new__(table)
  ops.dtype = layer_run.torch.bfloat16
  ops.prefill_tcgen05 = True
  ops.layer_runs = ops.tensor_core_attention = ops.fused_qkv_rope = ops.direct_library_products = ops.gated_tc_pairs = True
  ops.skinny_warps = ops.gated_tc_blocks = ops.mid_split = ops.mid_stages = ops.decode_variant = 0
  if replaced:
    setattr(ops, replaced, lambda *a, **kw: None)
  ran = []
  monkeypatch.setattr(layer_run.UniformLayers, "run", lambda self, *a: ran.append(a))
  model = DecoderModel(preset("gemma2-2b").model_spec())
  model._run_layers(types.SimpleNamespace(h=None), types.SimpleNamespace(ops=ops, num_tokens=20, max_q_len=20, page_size=64), {})
  assert bool(ran) == want


def test_the_mirrors_of_the_structs_have_their_sizes():
  lib = ctypes.CDLL(build.build(verbose=False))
  sizes = (8 * layer_run.LAYER_WORDS, ctypes.sizeof(layer_run._Attention), ctypes.sizeof(layer_run._Step))
  assert tuple(lib.sb_layer_run_bytes(i) for i in range(3)) == sizes


@pytest.mark.parametrize("replaced", ["block", "mixer", "feed_forward", "class of a mixer", "class of a block", "class of the table",
                                      "product"])
def test_replaced_calls_of_parts_and_classes_are_made(monkeypatch, replaced):
  ops = object.__new__(CudaOps)
  ops.dtype = layer_run.torch.bfloat16
  ops.layer_runs = ops.tensor_core_attention = ops.prefill_tcgen05 = ops.fused_qkv_rope = ops.direct_library_products = ops.gated_tc_pairs = True
  ops.skinny_warps = ops.gated_tc_blocks = ops.mid_split = ops.mid_stages = ops.decode_variant = 0
  model = DecoderModel(preset("gemma2-2b").model_spec())
  ctx = types.SimpleNamespace(ops=ops, num_tokens=20, max_q_len=20, page_size=64)
  uniform = layer_run.UniformLayers.of(model)
  assert uniform.takes(ctx)
  block = uniform.blocks[3]
  if replaced == "product":
    monkeypatch.setattr(block.mixer, "o_proj", lambda x, ctx: None)
    assert not uniform.takes(ctx)
    return
  part = {"block": block, "mixer": block.mixer, "feed_forward": block.feed_forward, "class of a mixer": type(block.mixer),
          "class of a block": type(block), "class of the table": CudaOps}[replaced]
  monkeypatch.setattr(part, "linear" if part is CudaOps else "forward", lambda *a, **kw: None)
  assert not uniform.takes(ctx)
