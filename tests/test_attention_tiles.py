"""Which form of the prompt attention a step takes, asked of the C rule (no GPU): sizes whose forms were measured more than 5 %
apart."""
import pytest

from janus_b200.kernels import ops


def two_tiles(nh, nkv, hd, lens, past=0, window=0, chunk=0, capped=0):
    lib = ops._lib("attention_tc", ops._attention_tc_row(hd), lambda h: dict({"JB_HEAD_DIM": h}, **ops._ATTN_TC_DEFINES))
    longest = -(-(max(lens) + past) // 64) * 64
    return bool(lib.jb_attention_tc_two_tiles(sum(lens), len(lens), max(lens), longest, nh, nkv, hd, window, chunk, capped))


@pytest.mark.parametrize("nh, nkv, lens, past, how, two", [
    (32, 8, [2000] + [1] * 63, 0, {}, True), (32, 8, [4096] + [1] * 33, 0, {}, True), (16, 16, [2000] + [1] * 31, 0, {}, True),
    (16, 1, [2000] + [1] * 15, 0, {}, True), (32, 8, [8190], 0, {}, True), (32, 8, [701, 600, 500, 400, 300, 250, 200, 150], 0, {}, True),
    (16, 16, [500] * 12, 0, {}, True), (32, 8, [100] * 8, 4000, {}, True), (32, 8, [2049, 1023], 0, dict(window=512), True),
    (16, 4, [400, 333, 266, 199, 132, 65], 0, {}, False), (16, 16, [33] * 64, 0, {}, False), (32, 16, [64] * 16, 2000, {}, False),
    (16, 4, [1500], 0, {}, False), (8, 2, [4000], 0, {}, False), (16, 1, [2049, 1023], 0, dict(capped=1), False), (16, 16, [5], 0, {}, False)])
def test_heads_of_more_than_64_numbers(nh, nkv, lens, past, how, two):
    assert two_tiles(nh, nkv, 128, lens, past, **how) is two


@pytest.mark.parametrize("lens", [[1], [8190], [2000] + [1] * 63, [100] * 64])
@pytest.mark.parametrize("hd", [8, 64, 192, 256])
def test_heads_that_go_by_one_tile(hd, lens):
    """Up to 64 numbers one tile is the faster form; beyond 128 there is no other."""
    assert not two_tiles(32, 8, hd, lens)
