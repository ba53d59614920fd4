"""Work lists of bfloat16 attention: layers of different kinds share one step, and each has to hand every request's rows
to a kernel, once.  The kernels are stand-ins that read the lists they are given, so no GPU is needed."""

import ctypes
import itertools
import types

import numpy as np
import pytest
import torch

from simply_b200.kernels.ops import CudaOps

HEADS, KV_HEADS, DIM, PAGE = 8, 4, 128, 64
GROUP = HEADS // KV_HEADS


class Launches:
  """Stand-ins for the kernels: `covered` counts how often each (token, kv head) is computed."""

  def __init__(self, lengths):
    self.cu = np.concatenate([[0], np.cumsum(lengths)])
    self.clear()

  def clear(self):
    self.covered = np.zeros((self.cu[-1], KV_HEADS), dtype=int)

  @staticmethod
  def _read(address, count):
    return np.ctypeslib.as_array((ctypes.c_int * count).from_address(address))

  def _tiles(self, items, tokens_per_tile):
    for b, i0, *head in items.tolist():
      first = self.cu[b] + i0
      assert first < self.cu[b + 1]
      self.covered[first:min(first + tokens_per_tile, self.cu[b + 1]), head or slice(None)] += 1

  def tcgen05(self, rows):  # (six pointers, out, tokens, six sizes, items, their number)
    return lambda *a: self._tiles(self._read(a[14], 3 * a[15]).reshape(-1, 3), rows // GROUP) or 0

  def mma_sync(self, *a):  # (six pointers, out, six sizes, items, their number, rows of a tile)
    self._tiles(self._read(a[13], 2 * a[14]).reshape(-1, 2), a[15] // GROUP)
    return 0

  def decode(self, *a):  # (six pointers, token_seq, out, tokens, six sizes, items, their number)
    for b in set(self._read(a[15], 2 * a[16])[::2].tolist()):
      self.covered[self.cu[b]:self.cu[b + 1]] += 1
    return 0


def host_table(launches):
  ops = object.__new__(CudaOps)
  ops.dtype, ops.device, ops.launches, ops._step_stream = torch.bfloat16, torch.device("cpu"), 0, ctypes.c_void_p(0)
  ops.tensor_core_attention = ops.prefill_tcgen05 = ops.prefill_pairs = ops.few_rows_in_tiles = True
  ops.decode_chunk = ops.decode_variant = ops.prefill_rows = 0
  ops.prefill_single_key_group, ops.attention_rows, ops._tensor_maps = False, None, {}
  ops.err = ops._attn_counter = torch.zeros(1, dtype=torch.int32)
  ops._decode_slots = {(DIM, DIM): 444}
  tile = launches.mma_sync
  ops._attn_fns = {(DIM, DIM): (tile, launches.decode, lambda *a: 0, launches.tcgen05(128), launches.tcgen05(256), None, tile,
                                launches.tcgen05(128), None)}
  return ops


# what a layer has beside the window, and its score cap
KINDS = {"plain": ({}, 0.0), "capped": ({}, 30.0), "sink": (dict(sink=torch.zeros(HEADS)), 0.0),
         "distance": (dict(distance_bias=torch.zeros(2, HEADS)), 0.0), "linear": (dict(distance_bias=torch.zeros(1, HEADS)), 0.0),
         "capped distance": (dict(distance_bias=torch.zeros(2, HEADS)), 30.0)}


@pytest.mark.parametrize("window", [None, 256])
@pytest.mark.parametrize("seqs", [[(300, 1), (0, 200), (700, 2), (64, 8)], [(0, 150), (40, 9)], [(5, 1), (90, 3)]])
def test_every_row_is_computed_once_whatever_layers_share_a_step(seqs, window):
  history, lengths = np.array([h for h, _ in seqs]), np.array([n for _, n in seqs])
  launches = Launches(lengths)
  ops = host_table(launches)
  tokens = int(lengths.sum())
  q, storage = torch.zeros(tokens, HEADS, DIM, dtype=torch.bfloat16), torch.zeros(16, 2, KV_HEADS, PAGE, DIM, dtype=torch.bfloat16)
  ints = torch.zeros(tokens, dtype=torch.int32)
  for first, second in itertools.permutations(KINDS, 2):
    ctx = types.SimpleNamespace(
        host=dict(cu_q=launches.cu, q_start=history), memo={}, page_size=PAGE, num_seqs=len(seqs), num_tokens=tokens,
        max_q_len=int(lengths.max()), max_kv_len=int((history + lengths).max()), cu_q=ints, q_start=ints, token_seq=ints, positions=ints)
    for name in (first, second, first):
      options, cap = KINDS[name]
      launches.clear()
      ops.paged_attention(q, storage, torch.zeros(len(seqs), 16, dtype=torch.int32), ctx, num_heads=HEADS, num_kv_heads=KV_HEADS,
                          head_dim=DIM, logit_softcap=cap, window=window, **options)
      assert (launches.covered == 1).all(), (first, second, name)


def test_steps_of_few_tokens_alone_have_one_list():
  """Without prompts there are no tiles, and every kind of layer reads the same split keys: they are listed once."""
  launches = Launches([1, 1, 2])
  ops = host_table(launches)
  q, storage = torch.zeros(4, HEADS, DIM, dtype=torch.bfloat16), torch.zeros(16, 2, KV_HEADS, PAGE, DIM, dtype=torch.bfloat16)
  ints = torch.zeros(4, dtype=torch.int32)
  ctx = types.SimpleNamespace(
      host=dict(cu_q=launches.cu, q_start=np.array([300, 0, 700])), memo={}, page_size=PAGE, num_seqs=3, num_tokens=4, max_q_len=2,
      max_kv_len=702, cu_q=ints, q_start=ints, token_seq=ints, positions=ints)
  for name, (options, cap) in KINDS.items():
    launches.clear()
    ops.paged_attention(q, storage, torch.zeros(3, 16, dtype=torch.int32), ctx, num_heads=HEADS, num_kv_heads=KV_HEADS,
                        head_dim=DIM, logit_softcap=cap, window=None, **options)
    assert (launches.covered == 1).all(), name
  assert len(ctx.memo) == 1


def test_only_the_general_kernel_asks_how_many_tokens_share_a_block(monkeypatch):
  def refused(*a):
    raise AssertionError("asked for a tensor-core kernel")
  monkeypatch.setattr("simply_b200.kernels.ops.tokens_per_attention_block", refused)
  test_steps_of_few_tokens_alone_have_one_list()
