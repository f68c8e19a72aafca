"""Where the chunks of a step lie in the scratch, and how much of it is asked for (no GPU)."""
import random

import pytest

from janus_b200.kernels import ops


@pytest.mark.parametrize("seed", range(20))
def test_packed_chunks_do_not_meet(seed):
    """A sequence's chunks begin at floor(q_start / 32) + its place: never before the end of the one before it, never past
    what is asked for."""
    g = random.Random(seed)
    lens = [g.choice((0, 1, 2, 31, 32, 33, g.randint(0, 200))) for _ in range(g.randint(1, 300))]
    slots, tiles = ops._chunk_slots(len(lens), sum(lens), 1 << 20, 32, 4, 1 << 60)       # (were one of them that long)
    assert tiles == 0 and slots == sum(lens) // 32 + len(lens)
    at, free = 0, 0
    for s, n in enumerate(lens):
        first = at // 32 + s
        assert first >= free
        free, at = first + -(-n // 32), at + n
    assert free <= slots


def test_scratch_is_bounded():
    """Beyond the bound a step goes in slabs of as many chunks a sequence as fit it, at least one."""
    per = 4 * ops._STATE_KINDS["mamba"][1] * 128
    for n, tokens, longest in ((8, 8 * 4096, 4096), (64, 64 * 4096, 4096), (2000, 2000 * 600, 600)):
        slots, tiles = ops._chunk_slots(n, tokens, longest, 32, per, ops.STATE_SCRATCH_BYTES)
        assert tiles >= 1 and slots == n * tiles and (tiles == 1 or slots * per <= ops.STATE_SCRATCH_BYTES)
    slots, tiles = ops._chunk_slots(256, 8192 + 255, 8192, 32, per, ops.STATE_SCRATCH_BYTES)
    assert tiles == 0 and slots * per <= ops.STATE_SCRATCH_BYTES


@pytest.mark.parametrize("lens, floats", [([1500], True), ([1500] + [1] * 7, True), ([200] + [1] * 63, False), ([100] + [1] * 15, False),
                                          ([64] * 8, True), ([100] + [2] * 3, False)])
def test_delta_rule_scratch_goes_by_the_work(lens, floats):
    asked = ops.delta_rule_scratch(len(lens), 16, max(lens), 4096, 0, 512, 128, sum(lens), 128)
    chunks = min(len(lens) * -(-max(lens) // 32), sum(lens) // 32 + len(lens))
    assert asked == 0 if not floats else chunks * 16 * ops._DELTA_CHUNK_FLOATS <= asked <= 2 * chunks * 16 * ops._DELTA_CHUNK_FLOATS
