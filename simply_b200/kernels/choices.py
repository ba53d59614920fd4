"""Which of two ways a step's call takes, from its sizes alone: the lines between kernels that are drawn on the host.

Times are of a B200 (148 SMs), measured on both sides of each line.
"""

from __future__ import annotations

import math
from typing import Sequence

SMS = 148


def experts_on_tensor_memory(pairs: int, width: int, hidden: int, gated: bool) -> bool:
  """Whether the routed experts' products of a step go through the grouped tcgen05 kernels (csrc/moe_tc.cu) or the
  mma.sync kernel (csrc/moe.cu); `pairs`: (token, choice) pairs.

  A tcgen05 launch starts and ends slower (2 us, 6 us with the exponential of a gate's silu on its sums), then
  streams rows of weights about 1.7 times as fast and multiplies five times as fast: it pays for long chains of
  k (width + hidden) and for much to multiply.  us, mma.sync against tcgen05, sorting to sum, weights from DRAM
  (experts, width x hidden, pairs):

      silu with a gate                     exact gelu without
      8, 64 x 128, 4,096       21 / 31     8, 64 x 128, 2,048      16 / 23
      8, 512 x 512, 512        31 / 36     8, 256 x 512, 80        17 / 18
      8, 512 x 512, 1,024      40 / 36     1, 512 x 512, 1,024     27 / 28
      2, 1,024 x 1,024, 128    37 / 45     64, 512 x 256, 768      30 / 32
      2, 1,024 x 1,024, 256    47 / 41     64, 512 x 256, 3,072    40 / 36
      256, 1,024 x 256, 320   103 / 106    256, 1,024 x 256, 64    48 / 48
      16, 1,536 x 1,536, 32    71 / 73     2, 1,024 x 1,024, 8     28 / 24
      16, 2,048 x 2,048, 32    97 / 87     16, 2,048 x 2,048, 32   70 / 60
      64, 2,048 x 1,408, 48   148 / 126    64, 2,048 x 1,408, 48  116 / 97
      8, 512 x 3,584, 16       62 / 63     16, 2,560 x 2,560, 64  130 / 109
      16, 4,096 x 3,584, 64   307 / 261    16, 4,096 x 3,584, 64  219 / 178
  """
  work = pairs * width * hidden
  if gated:
    return width + hidden >= 3400 or work >= 1 << 28
  return width + hidden >= 1280 or work > 1 << 28


def tokens_per_attention_block(tokens: int, requests: int, heads: int) -> int:
  """How many neighbouring tokens of a request share a block of the general attention kernel (float32 storage,
  csrc/attention_generic.cu), and with it every key and value that is fetched: as many as leave every SM two blocks, where
  requests bring that many tokens on average (a request's last tokens and single ones have blocks of their own).  us of 1,
  2, 4 and 8 (16 heads of 128): 20 tokens 11.4, 11.3, 13.0, 15.7; 64 27.6, 16.9, 16.7, 20.4; 130 58.5, 34.2, 30.8, 31.0;
  600 694, 329, 244, 212; 3 requests of 20 to 150 88, 47, 38, 38; 8 of 9 to 70 70.1, 33.4, 31.6, 35.8; 7 of one token and
  2,000 keys beside a prompt of 256 439, 360, 287, 232; 31 of one and 4,000 beside 600 1,482, 1,047, 1,009, 1,368."""
  for together in (8, 4, 2):
    if tokens >= together * requests and -(-tokens // together) * heads >= 2 * SMS:
      return together
  return 1


def attention_cluster(requests: int, kv_heads: int, group: int, dim: int, keys: int) -> int:
  """Blocks per (request, kv head) of the one-launch decode attention (csrc/attention_rows.cu) for single tokens that
  see up to `keys` keys, or 0: the split-key kernel (csrc/attention_mma.cu), which streams long contexts better.

  64 blocks where clusters are 8 or 16 wide (more clusters of 8 than two per GPC wait for one another), else up to
  148, one per SM.  us of a decode step, split keys against one launch (Gemma 2 2B unless said; its requests' keys):

      1 x 1,000 1,530 / 1,470    2 x 1,900 1,577 / 1,551    8 x 900   1,690 / 1,657    24 x 300 2,501 / 2,238
      1 x 4,000 1,614 / 1,570    2 x 3,900 1,663 / 1,690    8 x 2,000 1,807 / 1,849    24 x 800 2,498 / 2,486
      1 x 7,000 1,637 / 1,640    4 x 900   1,631 / 1,547    16 x 300  1,986 / 1,851    32 x 700 2,718 / 2,582
                                 4 x 1,900 1,641 / 1,685    16 x 900  2,119 / 2,068    40 x 900 3,088 / 3,365
      Gemma 2 9B: 1 x 900 4,201 / 4,070, 8 x 900 4,634 / 4,572
      heads of 128, four to a kv head: 8 kv heads 1 x 900 487 / 468, 2 x 900 478 / 470, 3 x 900 472 / 473, 4 x 900 475 / 483
      (4 x 300 497 / 484), 6 x 900 509 / 509, 8 x 900 545 / 558; 4 kv heads 1 x 900 594 / 602
  Other heads and groups that the kernel is compiled for have no measured step: they stay with the split keys."""
  pairs = requests * kv_heads
  cluster = max((c for c in (1, 2, 4, 8, 16) if pairs * c <= (64 if c >= 8 else 128)), default=0) or int(pairs <= SMS)
  if not cluster or keys > (256 * cluster if cluster >= 4 else 1024):
    return 0
  if dim == 256 and group == 2:
    return cluster
  return cluster if dim == 128 and group == 4 and 8 <= pairs <= 16 else 0


def few_rows_join_tiles(keys: Sequence[int], kv_heads: int, prompt_keys: Sequence[int] = (100,), rows: int = 0,
                        key_bytes: int = 1024) -> bool:
  """Whether the requests of a step that bring only a few tokens beside prompts (`keys`: how many each sees) are tiles of
  the prompts' attention kernel too (csrc/attention_tc_pair.cu), in place of a split-key launch and its merge behind
  it.  `prompt_keys`: the keys of each of the prompts' tiles (one short prompt where they are not given); `rows`: the step's
  tokens times query heads; `key_bytes`: of a key and its value (heads of 256).

  A tile is walked from end to end by one of 74 pairs of blocks: 9 us and 14.5 us per 1,000 keys (19 with a prompt's
  full rows), for heads of 128 and 256 alike.  So a lone request of many keys is the longest walk of the step unless a
  prompt's is longer, and many requests take several rounds of pairs.  The split keys take 8 us, 1 us per 1,000 rows (the
  merge looks at each) and what their keys need at 5 TB/s.  us of the attention of a layer, split keys and tiles (requests
  of one token x keys; 8 and 4 heads of 256 | 32 and 8 of 128):

                  beside 60 tokens         beside 400                beside 4,000
      1 x 1,000   32, 29  | 26, 30         38, 29  | 42, 30          142, 95  | 396, 255
      1 x 8,000   47, 128 | 35, 120        46, 126 | 50, 121         151, 135 | 405, 267
      4 x 4,000   42, 74  | 40, 72         50, 74  | 56, 71          154, 112 | 409, 283
      16 x 300    34, 24  | 32, 35         40, 34  | 48, 45          144, 109 | 401, 280
      32 x 600    44, 47  | 46, 77         52, 48  | 63, 82          156, 131 | 417, 317

  A step of Gemma 2 2B: 1 x 7,000 beside 60 2,680 and 4,357, beside 5,000 21,547 and 20,042; 8 x 300 beside 400 3,900
  and 3,284; prompts of 3 to 1,500 tokens together 14,001 and 13,230."""
  pairs = 74

  def rounds(costs: list[float]) -> float:  # when the last pair is done
    costs.sort(reverse=True)
    tiles = len(costs) * kv_heads  # (of j * pairs + 1 tiles one pair has j + 1)
    return max([sum(costs) * kv_heads / pairs] + [(j + 1) * costs[pairs * j // kv_heads] for j in range(-(-tiles // pairs))])

  prompts = [9 + 0.019 * k for k in prompt_keys]
  split = 8 + 0.001 * rows + sum(keys) * kv_heads * key_bytes / 5e6
  return rounds(prompts + [9 + 0.0145 * k for k in keys]) < rounds(prompts) + split


def walks_by_chunks(kind: int, lengths: Sequence[int], heads: int, dim: int, value_dim: int) -> bool:
  """Whether a step's walks through recurrent states go by chunks of tokens (csrc/chunk_walks.cu) or token by token
  (csrc/state_scans.cu): `lengths` new tokens per request, states of dim x value_dim.  One kernel walks all
  requests of a step, so what a request of one token costs it counts too."""
  longest, tokens, requests = max(lengths), sum(lengths), len(lengths)
  if longest < 64 or dim > (128, 64)[kind]:  # (larger states the kernels do not take)
    return False
  if kind == 0:
    # State space.  Chunks: a block takes 32 columns and an SM holds one; a chunk of 64 tokens takes 7.3 us, a
    # request's start and end half as long; one of a few tokens takes 1.9 chunks' time in all (its rows are
    # fetched over and over).  Token by token: the longest request's chain, or 0.097 us per token and block of
    # 512 / (rows' lanes) columns and SM, and 4.4 us of fetching and storing per 64 states of 128 x 64.
    # Chunks only where they come out 15 % ahead: the estimate is that good.  us, tokens / chunks (64 heads of
    # 128 x 64 unless said; 1 x 64 + 31: a prompt of 64 tokens beside 31 single tokens):
    #   1 x 64            28 / 19    1 x 64 + 3         44 / 57     1 x 64 + 31        164 / 387
    #   1 x 256 + 3      108 / 75    1 x 256 + 15      163 / 212    1 x 1,024 + 15     470 / 278
    #   8 x 64           118 / 75    20 x 100          394 / 318    1 x 2,048 + 31     912 / 556
    #   16 x 64 states: 1 x 2,048 389 / 234, 8 x 300 98 / 269; 128 heads: 1 x 255 52 / 66
    #   64 x 64 states: 1 x 2,048 499 / 236, 8 x 300 217 / 274; 128 heads of 128 x 64: 1 x 512 + 15 355 / 501
    blocks = heads * math.ceil(value_dim / 32)
    chunks = lambda n: 0.0 if n == 0 else 1.9 if n < 32 else math.ceil(n / 64) + 0.45
    mean = sum(map(chunks, lengths)) / requests
    by_chunks = 7.3 * max(chunks(longest) * math.ceil(blocks / SMS), mean * math.ceil(requests * blocks / SMS))
    columns, chain = next(way for rows, *way in ((15, 128, 0.52), (16, 128, 0.187), (32, 64, 0.225), (64, 32, 0.24), (128, 16, 0.26))
                          if dim <= rows)
    by_tokens = (4.4 * requests * heads * dim * value_dim / (64 * 128 * 64)
                 + max(chain * longest, 0.097 * tokens * heads * math.ceil(value_dim / columns) / SMS))
    return 1.15 * by_chunks <= by_tokens
  # Delta rule.  Chunks of 16 tokens are ahead while the token walk waits for its own chain: where the blocks of
  # both leave SMs to spare, or a long request outlasts the work of all (0.31 us of its chain per token
  # against 0.52 us of work per token, head and SM, measured to pay from 128 tokens and heads of more than 48
  # channels on).  us, tokens / chunks (32 heads of 64 unless said):
  #   1 x 64   28 / 25    1 x 64 + 15  48 / 51    1 x 128 + 7   64 / 47    1 x 256 + 15  134 / 89
  #   8 x 64   72 / 67    20 x 100    258 / 274   10 x 100     127 / 141   1 x 1,024 + 31 467 / 327
  #   64 heads: 1 x 64 + 7 51 / 54, 1 x 255 99 / 70, 8 x 300 551 / 560; 128 heads: 1 x 64 39 / 42
  #   64 heads of 32: 1 x 64 25 / 24, 8 x 300 221 / 357; 64 heads of 40: 1 x 128 + 7 64 / 66
  # Heads of fewer than 32 channels stay with the token walk, whose short sums are nearer to 64 bits (heads of
  # 20: 1.28e-7 against 1.31e-7; of 32 and 64 the two are level).
  if dim < 32:
    return False
  if requests * heads * math.ceil(dim / 16) <= SMS:
    return True
  return dim > 48 and longest >= 128 and tokens * heads <= 88 * longest and tokens >= 16 * requests
