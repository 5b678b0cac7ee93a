"""Attention of a step of single tokens and portions: the decode kernel beside the prefill kernel gives what each gives alone."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


# portions of one tile and of many, fewer blocks than SMs and more; one split (written by the kernel) and several (merged by another);
# groups of two (two heads a block) and of one (the one-head kernel); what comes next reads all rows
@pytest.mark.parametrize("decoding,portions", [([900], [2]), ([2900, 1, 64, 700], [505]), ([30] * 40, [129, 700]), ([4000] * 3, [2500])])
@pytest.mark.parametrize("hq,hkv,page,window", [(32, 8, 16, None), (6, 6, 8, 300)])
def test_decoding_beside_portions(decoding, portions, hq, hkv, page, window):
    from pulsar_b200 import ops
    d, cached = 128, 77
    q_lens = [1] * len(decoding) + portions
    kv_lens = decoding + [p + cached for p in portions]
    width = -(-max(kv_lens) // page)
    g = torch.Generator(device="cuda").manual_seed(sum(q_lens) + hq)
    need = [-(-k // page) for k in kv_lens]
    ids = torch.randperm(sum(need), generator=torch.Generator().manual_seed(1)).to(torch.int32)
    table = torch.zeros(len(need), width, dtype=torch.int32)
    for i, n in enumerate(need):
        table[i, :n] = ids[sum(need[:i]):sum(need[:i + 1])]
    table = table.cuda()
    pools = [torch.randn(sum(need), hkv, page, d, generator=g, device="cuda").bfloat16() for _ in range(2)]
    q = torch.randn(sum(q_lens), hq, d, generator=g, device="cuda").bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")                          # noqa: E731
    cu, kv = i32([sum(q_lens[:i]) for i in range(len(q_lens) + 1)]), i32(kv_lens)
    buffers = {}

    def scratch(tag, shape, dtype):
        return buffers.setdefault((tag, shape), torch.empty(shape, dtype=dtype, device="cuda"))
    ctx = types.SimpleNamespace(all_decode=False, n_seqs=len(q_lens), host=types.SimpleNamespace(q_lens=q_lens), cu_q=cu, kv_len=kv, scratch=scratch)
    cache = types.SimpleNamespace(k_pool=pools[0], v_pool=pools[1], block_table=table)
    n = len(decoding)
    want = torch.empty_like(q)
    ops.paged_attention_prefill_tcgen05(q, *pools, want, table[n:], cu[n:], kv[n:], ops.prefill_tcgen05_tiles(portions), 0.088, window)
    shares = ops.decode_shares(n, hkv, width * page)
    partial = torch.empty(n * hq * shares * (d + 2), device="cuda")
    ops.paged_attention_decode(q[:n], *pools, want[:n], partial, table[:n], kv[:n], 0.088, window, shares)
    torch.cuda.synchronize()
    for _ in range(3):
        out = torch.full_like(q, float("nan"))
        ops.attention(ctx, q, cache, out, 0.088, window)
        after = out.float() + 1                             # the next kernel on the stream finds every row written
        assert torch.equal(out, want) and torch.equal(after, want.float() + 1)
    ops.check_wait_words()
