"""The float32 path's products at the edges of their kernels' tiles, against float64 and, bit for bit, against the general kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _unaligned(t):
    """The same values on an address that is no multiple of 16 bytes: the general kernel takes them."""
    buf = torch.empty(t.numel() + 4, dtype=t.dtype, device=t.device)
    off = next(o for o in range(1, 4) if (buf.data_ptr() + 4 * o) % 16)
    view = buf[off:off + t.numel()].view(t.shape)
    view.copy_(t)
    return view


# n: one block, a remainder, blocks for more than one an SM (4800); k: less than a stage, whole stages, tails; the last: many blocks
@pytest.mark.parametrize("n,k", [(1, 4), (33, 64), (130, 68), (321, 516), (4800, 132), (153600, 8)])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 33, 65, 100])
def test_products_of_rows_and_tiles(m, n, k):
    from pulsar_b200 import ops
    if n == 153600 and m not in (3, 17, 65, 100):
        pytest.skip("large outputs at a few row counts only")
    g = torch.Generator(device="cuda").manual_seed(m * 1000 + k)
    a, w = (torch.randn(r, k, generator=g, device="cuda") for r in (m, n))
    out = torch.full((m, n), float("nan"), device="cuda")
    ops.gemm_simt(a, w, out)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert bool(((out.double() - ref).abs() <= (k + 1) * 2.0 ** -24 * size).all())       # a chain of k rounded multiply-adds
    want = torch.empty_like(out)
    ops.gemm_simt(_unaligned(a), w, want)
    assert torch.equal(out, want), "the sums are the general kernel's, bit for bit"
    if n <= 4800:
        half = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
        ops.gemm_simt(a, w, half)
        assert torch.equal(half, out.bfloat16())


# every ring of stages turns more than twice, with a ragged tail: four stages of 256 and of 128 k, two of 256, for every number of rows that
# streams the weights, two of 32 k of the tiles
@pytest.mark.parametrize("m,n,k", [(m, 130, 2116) for m in range(1, 17)] + [(m, 4800, 1092) for m in range(1, 17)]
                         + [(65, 153600, 132), (100, 153600, 132), (33, 130, 1092), (100, 321, 2116)])
def test_products_whose_stages_are_used_again(m, n, k):
    from pulsar_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(m * 1000 + k)
    a, w = (torch.randn(r, k, generator=g, device="cuda") for r in (m, n))
    out, want = torch.full((m, n), float("nan"), device="cuda"), torch.empty(m, n, device="cuda")
    ops.gemm_simt(_unaligned(a), w, want)
    for loaded in (False, True):
        out.fill_(float("nan"))
        torch.cuda.synchronize()
        ops.gemm_simt(a, w, out, loaded)
        assert torch.equal(out, want), "the sums are the general kernel's, bit for bit"
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert bool(((out.double() - ref).abs() <= (k + 1) * 2.0 ** -24 * size).all())       # a chain of k rounded multiply-adds


# 16 rows a block (many rows; head sizes up to 64 and 128), 8 (wider heads), 4 and 1 (few rows); groups of one to more heads than a
# block has rows, tokens of several sequences, windows that begin inside a tile
@pytest.mark.parametrize("q_lens,kv_lens,hq,hkv,d,page,window", [
    ([387], [420], 16, 4, 128, 16, None), ([300, 1, 41, 3], [300, 70, 500, 3], 20, 4, 64, 16, 150), ([700], [700], 8, 2, 208, 8, 40),
    ([5, 1, 70], [5, 90, 200], 6, 2, 32, 4, None), ([33], [164], 40, 2, 80, 16, 50), ([260], [261], 36, 1, 48, 4, 33)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_attention_of_rows_that_share_keys(q_lens, kv_lens, hq, hkv, d, page, window, dtype):
    from pulsar_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(hq * 100 + d)
    need = [-(-k // page) for k in kv_lens]
    ids = torch.randperm(sum(need) + 3, generator=torch.Generator().manual_seed(d)).to(torch.int32)
    table = torch.full((len(need), max(need)), -1, dtype=torch.int32)
    for s, n in enumerate(need):
        table[s, :n] = ids[sum(need[:s]):sum(need[:s]) + n]
        if window:
            table[s, :max(0, kv_lens[s] - q_lens[s] - window + 1) // page] = -1        # released pages are never looked at
    pools = [torch.randn(len(ids), hkv, page, d, generator=g, device="cuda").to(dtype) for _ in range(2)]
    q = torch.randn(sum(q_lens), hq, d, generator=g, device="cuda").to(dtype)
    out = torch.full_like(q, float("nan"))
    as_i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")                       # noqa: E731
    cu = as_i32([sum(q_lens[:i]) for i in range(len(q_lens) + 1)])
    seq = torch.repeat_interleave(torch.arange(len(q_lens), device="cuda"), as_i32(q_lens)).to(torch.int32)
    ops.paged_attention_generic(q, pools[0], pools[1], out, table.cuda(), cu, as_i32(kv_lens), seq, d ** -0.5, window)
    at = 0
    for s, (n, kl) in enumerate(zip(q_lens, kv_lens)):
        key = torch.arange(kl)
        k, v = (p[table[s, key // page].clamp_min(0).long().cuda(), :, (key % page).cuda()].double() for p in pools)
        k, v = (t.repeat_interleave(hq // hkv, dim=1) for t in (k, v))
        pos = torch.arange(kl - n, kl, device="cuda")[:, None]
        hidden = key.cuda()[None] > pos
        if window:
            hidden |= key.cuda()[None] <= pos - window
        scores = torch.einsum("ihd,jhd->hij", q[at:at + n].double(), k) * d ** -0.5
        want = torch.einsum("hij,jhd->ihd", torch.softmax(scores.masked_fill(hidden, -float("inf")), dim=-1), v)
        # float32: scores a few units off in the last place and a few hundred rounded additions; bfloat16: the one rounding
        tol = 2e-5 if dtype == torch.float32 else 2.0 ** -8
        assert float((out[at:at + n].double() - want).abs().max() / want.abs().max()) < tol
        at += n


@pytest.mark.parametrize("kv_lens,hkv,dtype", [([1000], 8, torch.bfloat16), ([130], 2, torch.float32), ([1, 700], 4, torch.bfloat16)])
def test_decode_attention_of_a_sequence_or_two(kv_lens, hkv, dtype):
    """As many shares as ``decode_shares`` gives: one per tile of keys, some without a key."""
    from pulsar_b200 import ops
    hq, d, page, s = 4 * hkv, 128, 16, len(kv_lens)
    width = 64 * -(-max(kv_lens) // (64 * page))
    shares = ops.decode_shares(s, hkv, width * page)
    assert shares == min(16 if width == 64 else 32, 128 // (s * hkv))
    assert ops.decode_shares(1, 1, 100000) == 32               # the kernels take no more than 64, the rule no more than 32
    g = torch.Generator(device="cuda").manual_seed(hkv)
    table = torch.full((s, width), -1, dtype=torch.int32)
    for i, n in enumerate(kv_lens):
        table[i, :-(-n // page)] = torch.arange(-(-n // page)) + i * width
    pools = [torch.randn(s * width, hkv, page, d, generator=g, device="cuda").to(dtype) for _ in range(2)]
    q = torch.randn(s, hq, d, generator=g, device="cuda").to(dtype)
    out, partial = torch.empty_like(q), torch.full((s * hq * shares * (d + 2),), float("nan"), device="cuda")
    ops.paged_attention_decode(q, pools[0], pools[1], out, partial, table.cuda(), torch.tensor(kv_lens, dtype=torch.int32, device="cuda"),
                               d ** -0.5, None, shares)
    for i, n in enumerate(kv_lens):
        key = torch.arange(n)
        k, v = (p[table[i, key // page].long().cuda(), :, (key % page).cuda()].double().repeat_interleave(4, dim=1) for p in pools)
        w = torch.softmax(torch.einsum("hd,jhd->hj", q[i].double(), k) * d ** -0.5, dim=-1)
        want = torch.einsum("hj,jhd->hd", w, v)
        tol = 2e-5 if dtype == torch.float32 else 2.0 ** -6      # bfloat16: the weights and the output rounded once each
        assert float((out[i].double() - want).abs().max() / want.abs().max()) < tol


# single tokens and portions of several sequences, whose rows never share a block: one row a block (few rows), four, and sixteen or eight
# with tokens that begin anywhere; groups of one, of a part of a block's rows, and of more
@pytest.mark.parametrize("q_lens,cached", [([3], 40), ([1, 2, 1], 7), ([1] * 9 + [30, 1, 5], 300), ([1] * 33 + [37, 2, 5, 1, 260], 90)])
@pytest.mark.parametrize("hq,hkv,d,window", [(32, 8, 128, None), (16, 16, 64, 50), (20, 1, 48, None), (6, 2, 32, 33), (18, 6, 256, None)])
def test_attention_of_a_sequence_does_not_depend_on_the_others(q_lens, cached, hq, hkv, d, window):
    from pulsar_b200 import ops
    page, n = 16, sum(q_lens)
    kv_lens = [q + (cached * (i % 5 + 1)) // 5 for i, q in enumerate(q_lens)]
    g = torch.Generator(device="cuda").manual_seed(n + d)
    width = -(-max(kv_lens) // page)
    table = torch.randperm(len(q_lens) * width, generator=torch.Generator().manual_seed(n)).to(torch.int32).view(len(q_lens), width).cuda()
    pools = [torch.randn(len(q_lens) * width, hkv, page, d, generator=g, device="cuda") for _ in range(2)]
    q = torch.randn(n, hq, d, generator=g, device="cuda")
    as_i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")                       # noqa: E731

    def run(rows, seqs):
        lens = [q_lens[s] for s in seqs]
        out = torch.full_like(rows, float("nan"))
        seq = torch.repeat_interleave(torch.arange(len(seqs), device="cuda"), as_i32(lens)).to(torch.int32)
        ops.paged_attention_generic(rows, pools[0], pools[1], out, table[seqs].contiguous(), as_i32([sum(lens[:i]) for i in range(len(lens) + 1)]),
                                    as_i32([kv_lens[s] for s in seqs]), seq, d ** -0.5, window)
        return out

    whole, at = run(q, list(range(len(q_lens)))), 0
    assert bool(torch.isfinite(whole).all())
    for s, m in enumerate(q_lens):
        assert torch.equal(run(q[at:at + m].contiguous(), [s]), whole[at:at + m])
        at += m
