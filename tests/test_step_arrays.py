"""The arrays that a step copies to the device, and the check that a step passes before it runs (no GPU)."""
import random
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from janus_b200.cache import PAGE_SIZE, SequenceCache
from janus_b200.engine import StepEntry
from janus_b200.engine.step import FROM_DEVICE, Engine, StepError
from janus_b200.engine.workspace import Workspace
from janus_b200.parts.base import KVSpec

CPU = torch.device("cpu")
V = 100


@pytest.fixture
def engine(monkeypatch):
    """An engine without a device: the cache's books, and an index buffer that is not pinned."""
    monkeypatch.setattr(torch.cuda, "Event", lambda: SimpleNamespace(record=lambda: None))
    e = Engine.__new__(Engine)
    e.model, e.device, e.dtype, e.max_seq_len = SimpleNamespace(vocab_size=V), CPU, torch.float32, 300
    e.cache = SequenceCache([KVSpec(2, 16), KVSpec(2, 16, 100)], PAGE_SIZE * 40, 8, torch.float32, CPU)
    e.workspace, e._pinned = Workspace(CPU), torch.empty(1 << 16, dtype=torch.int32)
    return e


def bring(engine, entries):
    for x in entries:
        engine.cache.reserve(x.slot, len(x.tokens))
    ctx, want, _ = engine.build_context(entries)
    got = {n: getattr(ctx, n).tolist() for n in ("token_ids", "positions", "token_seq", "q_start", "kv_len", "seq_slot", "kv_start")}
    got.update(want=want.tolist(), dest=[g.dest_rows.tolist() for g in ctx.groups], tables=[g.block_table.tolist() for g in ctx.groups])
    return ctx, got


@pytest.mark.parametrize("seed", range(10))
def test_arrays_of_a_step_against_one_entry_at_a_time(engine, seed):
    """Prompts beside single tokens, starts inside a page and at its edges, pages given back behind a window, wanted places
    as a tuple, a list, an array and ranges with steps, none among them."""
    r = random.Random(seed)
    slots = [engine.cache.alloc_slot() for _ in range(6)]
    for _ in range(4):
        chosen = r.sample(slots, r.randint(1, 6))
        entries = []
        for s in chosen:
            n = min(r.choice((1, 1, 2, PAGE_SIZE - 1, PAGE_SIZE, PAGE_SIZE + 1, r.randint(1, 70))), 300 - engine.cache.lengths[s])
            if n < 1:
                continue
            tokens = [r.randrange(V) for _ in range(n)]
            want = r.choice(((n - 1,), (), [0, n - 1], np.array([n // 2]), range(n), range(n - 1, -1, -2), range(0, n, 3)))
            entries.append(StepEntry(s, r.choice((tokens, tuple(tokens), np.array(tokens))), want))
        if not entries:
            continue
        engine._validate(entries)
        ctx, got = bring(engine, entries)
        lens = [len(x.tokens) for x in entries]
        starts = [engine.cache.lengths[x.slot] for x in entries]
        q = [sum(lens[:i]) for i in range(len(lens) + 1)]
        after = [s + n for s, n in zip(starts, lens)]
        assert got["token_ids"] == [int(t) for x in entries for t in x.tokens]
        assert got["positions"] == [p for s, n in zip(starts, lens) for p in range(s, s + n)]
        assert got["token_seq"] == [i for i, n in enumerate(lens) for _ in range(n)]
        assert got["q_start"] == q and got["kv_len"] == after and got["seq_slot"] == [x.slot for x in entries]
        assert got["kv_start"] == [sum(after[:i]) for i in range(len(after) + 1)] and ctx.kv_total == sum(after)
        assert got["want"] == [q[i] + int(w) for i, x in enumerate(entries) for w in x.want]
        for g, dest, table in zip(engine.cache.groups, got["dest"], got["tables"]):
            assert dest == [g.pages[x.slot][p // PAGE_SIZE] * PAGE_SIZE + p % PAGE_SIZE
                            for x, s, n in zip(entries, starts, lens) for p in range(s, s + n)]
            for x, row in zip(entries, table):
                pages = list(g.pages[x.slot])
                assert row == pages + [-1] * (len(row) - len(pages))
        for x in entries:
            engine.cache.advance(x.slot, len(x.tokens))


def test_the_look_at_a_whole_step_agrees_with_the_one_entry_by_entry(engine):
    a, b, full, dead = (engine.cache.alloc_slot() for _ in range(4))
    engine.cache.free_slot(dead)
    engine.cache.reserve(full, 299)
    engine.cache.advance(full, 299)
    good = [StepEntry(a, [1, 2, 3], range(3)), StepEntry(b, (V - 1,), (0,)), StepEntry(full, [0], [0]), StepEntry(a, np.arange(5), (4, 0)),
            StepEntry(b, [5, 6], ()), StepEntry(b, [5, 6], range(1, -1, -1)), StepEntry(a, [0, 0], range(5, 5))]
    bad = [StepEntry(dead, [1], [0]), StepEntry(a, [], []), StepEntry(a, [V], [0]), StepEntry(a, [-1], [0]), StepEntry(a, [1, V], [0]),
           StepEntry(a, [1, -2], [0]), StepEntry(a, [1, FROM_DEVICE], [0]), StepEntry(full, [1, 2], [0]), StepEntry(a, [1, 2], (2,)),
           StepEntry(a, [1, 2], (0, -1)), StepEntry(a, [1, 2], range(3)), StepEntry(a, [1, 2], range(1, -2, -1)), StepEntry(a, [1], range(2)),
           StepEntry(a, list(range(V)) + [V], ())]
    for entries in [[x] for x in good + bad] + [[good[1], x] for x in bad] + [[good[0], good[3]], [], [good[0], good[1], good[2]]]:
        for device_tokens in (False, True):
            def each(entries=entries):
                try:
                    engine._validate_each([StepEntry(x.slot, x.tokens, x.want) for x in entries], device_tokens)
                except StepError as e:
                    return str(e)
            said = each()
            fresh = [StepEntry(x.slot, x.tokens, x.want) for x in entries]
            assert engine._passes(fresh, device_tokens) == (said is None), (entries, device_tokens, said)
            fresh = [StepEntry(x.slot, x.tokens, x.want) for x in entries]
            if said is None:
                engine._validate(fresh, device_tokens)
            else:
                with pytest.raises(StepError) as e:
                    engine._validate(fresh, device_tokens)
                assert str(e.value) == said
