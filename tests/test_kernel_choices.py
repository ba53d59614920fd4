"""Which kernel a size goes to, at sizes whose times were measured on both sides of each line (B200).  The rules are
plain functions of sizes, so no GPU is needed."""

import ctypes
import os
import subprocess
import sys

import pytest

from simply_b200.kernels import build
from simply_b200.kernels.choices import attention_cluster, experts_on_tensor_memory, few_rows_join_tiles, tokens_per_attention_block, walks_by_chunks


@pytest.fixture(scope="module")
def lib():
  return ctypes.CDLL(build.build(verbose=False))


# rows, gate and up rows, width: us with 4 and with 8 warps per block
@pytest.mark.parametrize("rows,n,k,times", [
    (16, 9728, 1024, (7.1, 8.9)), (9, 11264, 2048, (11.9, 13.2)), (16, 14208, 4096, (23.7, 26.9)),
    (16, 14336, 2048, (19.6, 15.0)), (9, 18432, 2304, (23.2, 17.0)), (16, 28672, 4096, (59.3, 51.2)),
    (16, 24576, 768, (10.7, 12.1)), (16, 49152, 1024, (25.2, 26.1)), (16, 28672, 1536, (24.2, 22.3))])
def test_warps_of_the_gated_product(lib, rows, n, k, times):
  assert lib.sb_skinny_warps(rows, n, k, 2) == (4 if times[0] < times[1] else 8)


@pytest.mark.parametrize("rows,n,k,epilogue,want", [(17, 28672, 4096, 2, 4), (8, 28672, 4096, 2, 4), (16, 28672, 4096, 0, 4),
                                                    (16, 2048, 2048, 0, 16), (16, 2048, 512, 0, 4), (16, 4096, 1024, 0, 8)])
def test_warps_of_other_products(lib, rows, n, k, epilogue, want):
  assert lib.sb_skinny_warps(rows, n, k, epilogue) == want


# tokens, channels, taps: us with one number per thread and with eight tokens
@pytest.mark.parametrize("tokens,channels,taps,times", [
    (256, 64, 2, (3.5, 6.1)), (2048, 64, 2, (4.3, 6.1)), (2048, 128, 3, (4.8, 6.8)), (512, 256, 4, (4.6, 7.1)),
    (300, 1024, 4, (6.1, 8.1)), (512, 1024, 4, (7.7, 8.2)), (2048, 1024, 4, (19.6, 10.1)), (6000, 256, 4, (15.3, 8.8)),
    (256, 2048, 3, (6.8, 7.1)), (300, 2048, 3, (7.5, 7.1)), (2048, 2048, 3, (31.7, 12.7)), (256, 4352, 4, (12.2, 8.6)),
    (256, 8192, 3, (17.6, 8.1))])
def test_tokens_per_thread_of_the_short_convolution(lib, tokens, channels, taps, times):
  assert bool(lib.sb_short_conv_by_rows(tokens, channels, taps)) == (times[1] < times[0])


# tokens, router rows, width: us with one token and with four per block
@pytest.mark.parametrize("tokens,rows,width,times", [
    (592, 8, 64, (3.9, 4.4)), (700, 8, 64, (3.8, 4.7)), (900, 8, 64, (6.4, 4.6)), (1500, 8, 64, (9.0, 5.5)),
    (700, 8, 2048, (8.1, 8.4)), (900, 8, 2048, (14.0, 8.7)), (592, 16, 256, (8.6, 5.7)), (592, 19, 2048, (13.8, 9.1)),
    (640, 32, 64, (14.5, 9.3)), (700, 128, 2048, (75.1, 62.7)), (592, 256, 4096, (169.2, 101.1))])
def test_tokens_per_block_of_the_router(lib, tokens, rows, width, times):
  bytes_per_token = ctypes.c_longlong(4 * (width + 2 * rows + 2))
  assert lib.sb_moe_route_together(tokens, rows, bytes_per_token) == (4 if times[1] < times[0] else 1)


# rows, columns, k: us with tiles of 128, 64 and 32
@pytest.mark.parametrize("m,n,k,times", [
    (1500, 3100, 31, (26.4, 12.1, 15.6)), (300, 9000, 32, (20.5, 7.8, 9.7)), (300, 9000, 4096, (741, 502, 705)),
    (256, 16384, 2048, (383, 352, 497)), (44, 32768, 2048, (377, 207, 250)), (256, 2048, 8192, (809, 273, 315)),
    (44, 2048, 8192, (807, 270, 212)), (4000, 3100, 2048, (1090, 1031, 1433)), (1500, 9000, 2048, (1096, 1121, 1571)),
    (1500, 9000, 256, (181, 151, 206)), (2048, 16384, 2048, (2505, 2697, 3864)), (2048, 16384, 512, (705, 696, 985)),
    (6000, 16384, 64, (516, 304, 417)), (600, 1600, 1024, (110, 77, 74)), (300, 500, 1024, (110, 36, 26))])
def test_tiles_of_the_float32_product(lib, m, n, k, times):
  got = lib.sb_gemm_f32_tile(m, n, k, int(k % 4 == 0))
  assert times[(128, 64, 32).index(got)] <= 1.05 * min(times)


# the same with the groups of threads that the tiles now have
@pytest.mark.parametrize("m,n,k,times", [
    (1500, 3100, 31, (29.2, 12.5, 18.1)), (300, 9000, 32, (21.2, 8.4, 11.8)), (300, 9000, 4096, (726, 504, 713)),
    (256, 16384, 2048, (376, 351, 508)), (44, 32768, 2048, (374, 203, 253)), (256, 2048, 8192, (809, 207, 303)),
    (44, 2048, 8192, (803, 202, 96)), (4000, 3100, 2048, (1075, 1024, 1471)), (1500, 9000, 2048, (1079, 1116, 1611)),
    (1500, 9000, 1024, (569, 569, 820)), (1500, 9000, 256, (188, 156, 225)), (2048, 16384, 2048, (2467, 2678, 3971)),
    (2048, 16384, 512, (716, 701, 1035)), (6000, 16384, 64, (536, 308, 571)), (600, 1600, 1024, (115, 57.9, 68.1)),
    (300, 500, 1024, (115, 30.2, 21.9))])
def test_tiles_of_the_float32_product_with_their_groups(lib, m, n, k, times):
  got = lib.sb_gemm_f32_tile(m, n, k, int(k % 4 == 0))
  assert times[(128, 64, 32).index(got)] <= 1.05 * min(times)


# rows, columns, k, tile: us with one and four groups of threads per tile
@pytest.mark.parametrize("m,n,k,tile,times", [
    (256, 2048, 64, 64, (5.4, 5.4)), (256, 2048, 100, 64, (7.9, 7.2)), (256, 2048, 256, 64, (12.5, 10.7)), (256, 2048, 2048, 64, (72, 56)),
    (44, 16384, 512, 64, (31.2, 32.0)), (44, 16384, 2048, 64, (110, 107)), (256, 3000, 515, 64, (35.3, 37.1)), (256, 3072, 2048, 64, (112, 108)),
    (600, 1600, 1024, 64, (58.6, 57.9)), (600, 2048, 64, 64, (9.6, 11.5)), (600, 2048, 100, 64, (16.5, 16.9)), (600, 2048, 256, 64, (27.6, 26.8)), (600, 2048, 512, 64, (50, 46)),
    (600, 2048, 8192, 64, (726, 593)), (600, 3072, 2048, 64, (209, 208)), (44, 32768, 2048, 64, (203, 208)), (256, 16384, 2048, 64, (351, 369)),
    (6000, 16384, 64, 64, (308, 525)), (44, 2048, 2048, 32, (56, 26)), (300, 500, 1024, 32, (31, 22)), (20, 2048, 64, 32, (4.5, 3.8)),
    (20, 2048, 32, 32, (3.6, 3.6))])
def test_groups_of_the_float32_product(lib, m, n, k, tile, times):
  assert times[(1, 4).index(lib.sb_gemm_f32_groups(m, n, k, tile))] <= 1.01 * min(times)


def _beside(prompt, singles):
  return [prompt] + [1] * singles


# kind (0 state space, 1 delta rule), lengths, heads, state rows, columns: us token by token and by chunks
@pytest.mark.parametrize("kind,lengths,heads,dim,cols,times", [
    (0, [64], 64, 128, 64, (28.3, 19.2)), (0, [2048], 64, 128, 64, (620, 241)), (0, [64] * 8, 64, 128, 64, (118, 75)),
    (0, [100] * 20, 64, 128, 64, (394, 318)), (0, _beside(1024, 15), 64, 128, 64, (470, 278)),
    (0, _beside(2048, 31), 64, 128, 64, (912, 556)), (0, _beside(64, 3), 64, 128, 64, (44, 57)),
    (0, _beside(64, 31), 64, 128, 64, (164, 387)), (0, _beside(256, 15), 64, 128, 64, (163, 212)),
    (0, _beside(512, 31), 64, 128, 64, (318, 425)), (0, [64] * 4 + [1] * 28, 64, 128, 64, (187, 377)),
    (0, [200] * 3 + [1] * 29, 64, 128, 64, (255, 442)), (0, _beside(512, 15), 128, 128, 64, (355, 501)),
    (0, [300] * 8, 128, 128, 64, (803, 548)), (0, [255], 128, 16, 64, (52, 66)), (0, [300] * 8, 64, 16, 64, (98, 269)),
    (0, [2048], 64, 16, 64, (389, 234)), (0, [300] * 8, 64, 64, 64, (217, 274)), (0, [300] * 8, 64, 128, 16, (130, 165)),
    (0, [300] * 8, 64, 8, 64, (176, 269)), (0, [300] * 8, 4, 16, 32, (61, 42)), (0, _beside(512, 15), 64, 128, 36, (208, 240)),
    (1, [64], 32, 64, 64, (27.9, 25.2)), (1, _beside(64, 15), 32, 64, 64, (48, 51)), (1, _beside(64, 31), 32, 64, 64, (63, 94)),
    (1, _beside(256, 15), 32, 64, 64, (134, 89)), (1, _beside(1024, 31), 32, 64, 64, (467, 327)),
    (1, [100] * 20, 32, 64, 64, (258, 281)), (1, [100] * 10, 32, 64, 64, (127, 141)), (1, _beside(64, 7), 64, 64, 64, (51, 54)),
    (1, [255], 64, 64, 64, (99, 70)), (1, [64], 128, 64, 64, (39, 42)), (1, [300] * 8, 64, 32, 32, (221, 357)),
    (1, [300] * 8, 32, 20, 20, (124, 190)), (1, [64], 128, 32, 32, (27, 28)), (1, _beside(128, 7), 64, 40, 40, (63, 66)),
    (1, [300] * 8, 4, 48, 48, (105, 51)), (1, [300] * 8, 64, 16, 16, (195, 271))])
def test_walks_by_chunks_where_they_are_faster(kind, lengths, heads, dim, cols, times):
  assert walks_by_chunks(kind, lengths, heads, dim, cols) == (times[1] < times[0])


# what the kernels do not take, walks that are short, heads so small that a chain of their channels rounds less
@pytest.mark.parametrize("kind,lengths,dim", [(0, [500], 132), (1, [500], 68), (0, [63], 128), (1, [1, 63], 64), (1, [500], 20)])
def test_walks_that_stay_token_by_token(kind, lengths, dim):
  assert not walks_by_chunks(kind, lengths, 8, dim, 64)


# pairs, experts, width, hidden, gate: us on the mma.sync and on the tcgen05 products
@pytest.mark.parametrize("pairs,experts,width,hidden,gated,times", [
    (16, 8, 64, 128, True, (11.5, 24.0)), (4096, 8, 64, 128, True, (21, 31)), (512, 8, 512, 512, True, (31, 36)),
    (1024, 8, 512, 512, True, (40, 36)), (2, 8, 1024, 1024, True, (29, 35)), (128, 2, 1024, 1024, True, (37, 45)),
    (256, 2, 1024, 1024, True, (47, 41)), (256, 8, 1024, 1024, True, (59, 40)), (128, 256, 1024, 256, True, (73.5, 81.6)),
    (32, 16, 1536, 1536, True, (71, 73)), (256, 16, 1536, 1536, True, (92, 78)), (4, 16, 2048, 2048, True, (56, 48)),
    (32, 16, 2048, 2048, True, (97, 87)), (160, 16, 2048, 2048, True, (104, 94)), (8192, 16, 2048, 2048, True, (1326, 251)),
    (48, 64, 2048, 1408, True, (148, 126)), (64, 16, 4096, 3584, True, (307, 261)), (1024, 128, 2048, 768, True, (281, 235)),
    (2048, 8, 64, 128, False, (16, 23)), (80, 8, 256, 512, False, (17.1, 18.1)), (16, 8, 512, 512, False, (19.3, 19.5)),
    (1024, 1, 512, 512, False, (26.6, 27.6)), (768, 64, 512, 256, False, (30.0, 31.6)), (3072, 64, 512, 256, False, (40, 36)),
    (6144, 64, 512, 256, False, (62, 45)), (8, 256, 1024, 256, False, (38.3, 35.9)), (8, 2, 1024, 1024, False, (28, 24)),
    (128, 2, 1024, 1024, False, (34.4, 34.0)), (32, 16, 2048, 2048, False, (70, 60)), (48, 64, 2048, 1408, False, (116, 97)),
    (64, 16, 2560, 2560, False, (130, 109)), (64, 16, 4096, 3584, False, (219, 178)), (8192, 16, 2048, 2048, False, (913, 199))])
def test_experts_products_where_they_are_faster(pairs, experts, width, hidden, gated, times):
  assert experts_on_tensor_memory(pairs, width, hidden, gated) == (times[1] < times[0])


# requests, kv heads, query heads per kv head, head size, most keys: us of a decode step by split keys and in one launch
@pytest.mark.parametrize("requests,kv_heads,group,dim,keys,times", [
    (1, 4, 2, 256, 1024, (1530, 1470)), (1, 4, 2, 256, 4096, (1614, 1570)), (1, 4, 2, 256, 8192, (1637, 1640)),
    (2, 4, 2, 256, 2048, (1577, 1551)), (2, 4, 2, 256, 4096, (1663, 1690)), (4, 4, 2, 256, 1024, (1631, 1547)),
    (4, 4, 2, 256, 2048, (1641, 1685)), (8, 4, 2, 256, 1024, (1690, 1657)), (8, 4, 2, 256, 2048, (1807, 1849)),
    (16, 4, 2, 256, 1024, (2119, 2068)), (24, 4, 2, 256, 1024, (2498, 2486)), (32, 4, 2, 256, 1024, (2718, 2582)),
    (40, 4, 2, 256, 1024, (3088, 3365)), (1, 8, 2, 256, 1024, (4201, 4070)), (8, 8, 2, 256, 1024, (4634, 4572)),
    (1, 8, 4, 128, 1024, (487, 468)), (2, 8, 4, 128, 1024, (478, 470)), (8, 8, 4, 128, 1024, (545, 558)),
    (1, 4, 4, 128, 1024, (594, 602))])
def test_decode_attention_in_one_launch_where_it_is_faster(requests, kv_heads, group, dim, keys, times):
  assert bool(attention_cluster(requests, kv_heads, group, dim, keys)) == (times[1] < times[0])


# (heads of 128 in groups of 4, 8 kv heads: nothing is gained between 16 and 64 pairs)
@pytest.mark.parametrize("requests,times", [(3, (471.5, 472.5)), (4, (475, 483)), (6, (508.7, 509.1))])
def test_heads_of_128_stay_with_the_split_keys_from_17_pairs_on(requests, times):
  assert bool(attention_cluster(requests, 8, 4, 128, 1024)) == (times[1] < times[0])


def test_decode_attention_in_one_launch_is_refused_where_no_cluster_fits():
  """A device that holds no cluster of the size that is asked for (here: no device at all) is a shape the kernel does not
  take, status -9, and the split keys take the step."""
  call = ("import ctypes; from simply_b200.kernels import build; lib = ctypes.CDLL(build.build_attention(256, verbose=False)); "
          "p = ctypes.c_void_p(1 << 20); z = ctypes.c_void_p(0); f = lib.sb_attn_rows_hd256; "
          "print([f(p, p, p, 8, p, p, 1, 8, 4, 64, 8, ctypes.c_float(0), 0, c, 0, p, z) for c in (1, 2, 4, 8, 16)])")
  done = subprocess.run([sys.executable, "-c", call], env={**os.environ, "CUDA_VISIBLE_DEVICES": ""}, capture_output=True, text=True)
  assert done.stdout.split("\n")[-2] == str([-9] * 5), done.stdout + done.stderr


# requests of one token, their keys: us of a step with them on split keys and as tiles beside a prompt
@pytest.mark.parametrize("requests,keys,times", [
    (8, 200, (2673, 2295)), (8, 600, (3579, 3141)), (16, 200, (2872, 2464)), (16, 600, (3898, 3541)), (39, 100, (3013, 3034)),
    (39, 300, (3213, 3305)), (39, 600, (3492, 3590)), (1, 3, (14001, 13230))])
def test_few_rows_are_tiles_where_that_is_faster(requests, keys, times):
  assert few_rows_join_tiles([keys] * requests, 4) == (times[1] < times[0])


# heads, kv heads, head size, the prompt, requests of one token and their keys: us of a layer's attention by split keys and
# as tiles
@pytest.mark.parametrize("heads,kv_heads,dim,prompt,requests,keys,times", [
    (8, 4, 256, 60, 1, 200, (29.7, 18.4)), (8, 4, 256, 60, 1, 2000, (31.7, 45.9)), (8, 4, 256, 60, 1, 8000, (47.0, 127.8)),
    (8, 4, 256, 60, 4, 4000, (42.0, 73.7)), (8, 4, 256, 60, 8, 300, (31.6, 21.5)), (8, 4, 256, 60, 32, 600, (43.9, 47.1)),
    (8, 4, 256, 400, 1, 1000, (37.9, 28.7)), (8, 4, 256, 400, 1, 4000, (39.9, 71.7)), (8, 4, 256, 400, 16, 300, (39.9, 33.8)),
    (8, 4, 256, 1500, 1, 4000, (70.7, 72.7)), (8, 4, 256, 1500, 1, 8000, (76.8, 127.0)), (8, 4, 256, 1500, 32, 600, (82.9, 65.5)),
    (8, 4, 256, 4000, 1, 8000, (150.5, 135.2)), (8, 4, 256, 4000, 32, 600, (155.6, 131.1)),
    (16, 8, 256, 60, 8, 1500, (48.1, 43.7)), (16, 8, 256, 60, 32, 100, (35.9, 54.2)), (16, 8, 256, 400, 32, 100, (46.1, 54.3)),
    (16, 8, 256, 400, 32, 600, (70.7, 85.0)), (16, 8, 256, 1500, 1, 8000, (97.0, 131.9)), (16, 8, 256, 1500, 32, 600, (113.7, 109.6)),
    (32, 8, 128, 60, 1, 8000, (34.9, 119.9)), (32, 8, 128, 60, 8, 300, (27.6, 20.5)), (32, 8, 128, 400, 8, 1500, (52.2, 47.1)),
    (32, 8, 128, 400, 32, 600, (62.5, 82.1)), (32, 8, 128, 1500, 1, 4000, (126.0, 71.7)), (32, 8, 128, 4000, 32, 600, (416.8, 317.4)),
    (16, 4, 128, 60, 1, 1000, (25.6, 28.7)), (16, 4, 128, 60, 16, 1000, (31.7, 30.7)), (16, 4, 128, 400, 1, 8000, (41.7, 120.8)),
    (16, 4, 128, 1500, 1, 4000, (76.8, 70.5)), (16, 4, 128, 4000, 1, 8000, (216.1, 140.3))])
def test_few_rows_are_tiles_where_a_layer_is_faster_for_it(heads, kv_heads, dim, prompt, requests, keys, times):
  tile = 256 // (heads // kv_heads)
  prompts = [min(i + tile, prompt) for i in range(0, prompt, tile)]
  joined = few_rows_join_tiles([keys + 1] * requests, kv_heads, prompts, (prompt + requests) * heads, 4 * dim)
  assert times[joined] <= 1.04 * min(times)


# tokens, requests: us of float32 attention (16 heads of 128) with 1, 2, 4 and 8 tokens per block
@pytest.mark.parametrize("tokens,requests,times", [
    (20, 1, (11.4, 11.3, 13.0, 15.7)), (64, 1, (27.6, 16.9, 16.7, 20.4)), (130, 1, (58.5, 34.2, 30.8, 31.0)),
    (256, 1, (162, 82, 70, 69)), (600, 1, (694, 329, 244, 212)), (247, 3, (87.6, 47.2, 38.0, 38.4)),
    (283, 8, (70.1, 33.4, 31.6, 35.8)), (263, 8, (439, 360, 287, 232)), (615, 16, (808, 421, 332, 322)),
    (631, 32, (1482, 1047, 1009, 1368))])
def test_tokens_per_block_of_float32_attention(tokens, requests, times):
  got = times[(1, 2, 4, 8).index(tokens_per_attention_block(tokens, requests, 16))]
  # (the last: single tokens with 6 times the prompt's keys, whose blocks then are few to an SM)
  assert got <= (1.15 if requests < 32 else 1.4) * min(times)
