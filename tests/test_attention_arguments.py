"""What the attention of a step hands to its kernels (on the CPU: the kernels are the test's own)."""
import types

import pytest
import torch


@pytest.mark.parametrize("tcgen05", [True, False])
@pytest.mark.parametrize("q_lens", [[5], [2, 7], [1, 1, 4], [1, 6, 1], [1, 1, 1, 3, 2]])
def test_prompts_get_the_steps_tensors_and_portions_what_is_behind_the_single_tokens(q_lens, tcgen05, monkeypatch):
    from pulsar_b200 import ops
    calls = []
    monkeypatch.setattr(ops, "prefill_tcgen05_supported", lambda *a: tcgen05)
    monkeypatch.setattr(ops, "prefill_tc_supported", lambda *a: True)
    monkeypatch.setattr(ops, "decode_tc_supported", lambda *a: tcgen05)
    monkeypatch.setattr(ops, "prefill_tcgen05_tiles", lambda lens: ("tiles", tuple(lens)))
    monkeypatch.setattr(ops, "prefill_tc_tiles", lambda lens: ("tiles", tuple(lens)))
    for name in ("paged_attention_prefill_tcgen05", "paged_attention_prefill_tc"):
        monkeypatch.setattr(ops, name, lambda q, k, v, out, *rest, name=name: calls.append((name, rest)))
    monkeypatch.setattr(ops, "paged_attention_decode", lambda q, k, v, out, partial, table, kv, *rest, beside: calls.append(("decode", (table, kv, beside))))
    n, s = sum(q_lens), len(q_lens)
    q = torch.zeros(n, 4, 128, dtype=torch.bfloat16)
    pool = torch.zeros(3, 2, 16, 128, dtype=torch.bfloat16)
    table, cu = torch.arange(s * 2, dtype=torch.int32).view(s, 2), torch.tensor([sum(q_lens[:i]) for i in range(s + 1)], dtype=torch.int32)
    kv = torch.arange(10, 10 + s, dtype=torch.int32)
    ctx = types.SimpleNamespace(all_decode=False, n_seqs=s, host=types.SimpleNamespace(q_lens=q_lens), cu_q=cu, kv_len=kv,
                                scratch=lambda tag, shape, dtype: torch.empty(1))
    ops.attention(ctx, q, types.SimpleNamespace(k_pool=pool, v_pool=pool, block_table=table), torch.empty_like(q), 0.1, None)
    n_dec = next(i for i, x in enumerate(q_lens) if x > 1)
    name, (got_table, got_cu, got_kv, tiles, scale, window) = [c for c in calls if c[0] != "decode"][0]
    assert name.endswith("tcgen05") is tcgen05 and tiles == ("tiles", tuple(q_lens[n_dec:])) and (scale, window) == (0.1, None)
    assert torch.equal(got_table, table[n_dec:]) and torch.equal(got_cu, cu[n_dec:]) and torch.equal(got_kv, kv[n_dec:])
    if n_dec == 0:                          # a prompt step takes no slices: they cost the host more than a microsecond each, every layer
        assert got_table is table and got_cu is cu and got_kv is kv and len(calls) == 1
    else:
        decode = [c for c in calls if c[0] == "decode"]
        assert len(decode) == 1 and torch.equal(decode[0][1][0], table[:n_dec]) and torch.equal(decode[0][1][1], kv[:n_dec]) and decode[0][1][2] is tcgen05
        assert (calls[0][0] == "decode") is not tcgen05
