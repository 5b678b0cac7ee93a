"""How many shares a decode step's keys are cut into, and when a step counts as uneven."""
import copy
import types

import pytest
import torch


@pytest.mark.parametrize("n,heads,table,uneven,want", [
    (1, 8, 1024, False, 16), (1, 1, 100000, False, 32), (4, 8, 1024, True, 4),             # one or two; a short table stays as it was
    (8, 8, 4096, False, 4), (8, 8, 4096, True, 4), (8, 8, 8192, True, 6), (12, 8, 4096, False, 3), (12, 8, 4096, True, 4),
    (16, 8, 4096, True, 3), (16, 8, 3072, True, 3), (16, 8, 2048, True, 2), (24, 8, 3072, True, 2), (24, 8, 2048, True, 1),
    (30, 8, 4096, True, 1), (37, 8, 4096, True, 1), (38, 8, 2048, False, 1), (48, 8, 2048, True, 1), (48, 8, 1024, False, 1),
    (40, 8, 3072, False, 7), (40, 8, 3072, True, 2), (48, 8, 4096, False, 2), (64, 8, 4096, False, 1), (64, 8, 4096, True, 1)])
def test_shares_of_a_step(n, heads, table, uneven, want):
    from pulsar_b200 import ops
    assert ops.decode_shares(n, heads, table, uneven) == want
    for batch in range(1, 200, 7):
        for tokens in (16, 300, 2048, 100000):
            assert 1 <= ops.decode_shares(batch, heads, tokens, uneven) <= 32


@pytest.mark.parametrize("lens,want", [([5], False), ([100, 100], False), ([100, 40], False), ([100, 39], True), ([1, 1, 1000], True)])
def test_uneven_steps(lens, want):
    from pulsar_b200.parts.base import HostBatch, StepContext
    ctx = StepContext(types.SimpleNamespace(dtype=torch.float32, device="cpu"), len(lens), len(lens),
                      HostBatch([1] * len(lens), lens, [-1] * len(lens)))
    assert ctx.uneven is want


# more pairs than slots over a short table: sequences of like length behind 1,024 tokens take two where ``decode_splits`` takes two or more
@pytest.mark.parametrize("n,table,uneven,want", [(38, 2048, False, 1), (40, 2048, False, 1), (41, 2048, False, 2), (44, 2048, False, 2), (48, 2048, False, 2),
                                                 (55, 2048, False, 2), (56, 2048, False, 1), (64, 2048, False, 1), (44, 2048, True, 1), (48, 1040, False, 2),
                                                 (48, 1024, False, 1), (44, 600, False, 1), (37, 2048, False, 1)])
def test_shares_of_more_pairs_than_slots_over_a_short_table(n, table, uneven, want):
    from pulsar_b200 import ops
    assert ops.decode_shares(n, 8, table, uneven) == want


def test_unevenness_counts_only_where_shares_follow_it():
    from pulsar_b200 import ops
    assert not ops.unevenness_matters(8, [(8, 1024)]) and not ops.unevenness_matters(8, [(8, 4096)]) and not ops.unevenness_matters(8, [])
    assert ops.unevenness_matters(16, [(8, 4096)]) and ops.unevenness_matters(44, [(8, 2048)]) and not ops.unevenness_matters(44, [(8, 1024)])
    assert ops.unevenness_matters(16, [(8, 1024), (8, 4096)]) and not ops.unevenness_matters(16, [(2, 4096)])


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", ["dense", "general"])
def test_a_step_stays_captured_while_its_lengths_become_even(sizes, tmp_path):
    """Four sequences that begin uneven and become even: one capture, whatever the share of keys they hold together."""
    import helpers
    from pulsar_b200.engine.engine import Engine
    from pulsar_b200.engine.runner import StepEntry
    if sizes == "dense":
        raw, seed, page = helpers.TINY["F"]
    else:
        from test_bubotar import CONFIGS
        raw, seed, page = CONFIGS["A"]
    helpers.make_folder(str(tmp_path), copy.deepcopy(raw), seed, store_dtype=torch.bfloat16)
    engine = Engine(str(tmp_path), dict(dtype="bfloat16", page_size=page, num_pages=128, max_sessions=4, max_running=4, max_chunk_size=256, eos_id=-1))
    assert engine.model.shares_keys is (sizes == "dense")
    assert engine.runner._sharing == ([(0, 8)] if sizes == "dense" else [])
    runner = engine.runner
    runner.step([StepEntry(i, [1 + i] * n, []) for i, n in enumerate((30, 30, 30, 60))])
    seen = set()
    for i in range(30):
        runner.step([StepEntry(r, [5], [0]) for r in range(4)])
        lens = [31 + i] * 3 + [61 + i]
        seen.add(10 * sum(lens) < 7 * max(lens) * 4)
    assert seen == {True, False}
    assert len(runner._graphs) == 1 and runner.graph_replays >= 26          # a few eager steps first, while buffers grow
