"""The general attention's form for a few rows on the tensor cores against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _paged(q_lens, kv_lens, page, pools, dtype, gen):
    """A shuffled block table and random pools [pages, heads, page, width], one per (heads, width)."""
    need = [-(-k // page) for k in kv_lens]
    ids = torch.randperm(sum(need) + 2, generator=gen).to(torch.int32)
    table = torch.full((len(need), max(need) + 1), -1, dtype=torch.int32)
    for s, n in enumerate(need):
        table[s, :n] = ids[sum(need[:s]):sum(need[:s]) + n]
    made = [torch.randn(len(ids), h, page, w, generator=gen).to(dtype).cuda() for h, w in pools]
    return table, made


def _keys_of(pool, table, s, kl, page):
    key = torch.arange(kl)
    return pool[table[s, key // page].long().cuda(), :, (key % page).cuda()].double()


class _Ctx:
    """What the general attention asks of a step."""

    def __init__(self, q_lens, kv_lens):
        self.host = type("Host", (), {"q_lens": q_lens})()
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")                      # noqa: E731
        self.cu_q, self.kv_len = i32([sum(q_lens[:i]) for i in range(len(q_lens) + 1)]), i32(kv_lens)
        self.seq_of_token = torch.repeat_interleave(torch.arange(len(q_lens), device="cuda"), i32(q_lens)).to(torch.int32)

    def scratch(self, tag, shape, dtype):
        return torch.full(shape, float("nan"), dtype=dtype, device="cuda")


# every instance of the kernel at its largest and at an odd size; one long row of keys (what an MMA cuts off must not add up)
@pytest.mark.parametrize("q_lens,kv_lens,hq,hkv,dk,dv,opts", [
    ([1, 1], [1900, 70], 16, 1, 576, 512, {}), ([3, 1], [40, 70], 5, 1, 576, 512, dict(sinks=True)),
    ([1, 2], [1000, 64], 32, 1, 320, 256, {}), ([1, 15], [190, 333], 6, 2, 192, 128, dict(page=5)),
    ([1] * 3, [100, 1024, 1025], 16, 4, 128, 128, dict(slopes=True, chunk=64)), ([1, 7], [90, 333], 8, 1, 80, 48, dict(sinks=True)),
    ([1, 5, 2], [64, 37, 300], 12, 4, 64, 64, dict(window=50, keep_first=4, softcap=20.0, sinks=True)),
    ([2, 1], [90, 33], 8, 2, 64, 128, dict(sigmoid=True, turn=True)), ([1, 1], [90, 2333], 8, 4, 64, 64, dict(sigmoid=True, v_share=2)),
    ([1], [1], 2, 1, 16, 16, {}), ([1, 2], [300, 40], 4, 1, 32, 32, {}), ([1, 2], [300, 40], 3, 1, 32, 32, {}),
    ([2, 1], [70, 500], 8, 1, 16, 48, dict(sinks=True))])
def test_few_rows_on_the_tensor_cores(q_lens, kv_lens, hq, hkv, dk, dv, opts):
    from pulsar_b200 import ops
    gen = torch.Generator().manual_seed(dk + hq)
    page, share, n = opts.get("page", 16), opts.get("v_share", 1), sum(q_lens)
    latent = dk in (576, 320)                                # the value is part of the key's row
    table, pools = _paged(q_lens, kv_lens, page, [(hkv, dk)] if latent else [(hkv, dk), (hkv // share, dv)], torch.bfloat16, gen)
    k_pool, v_pool = pools[0], pools[-1]
    q = torch.randn(n, hq, dk, generator=gen).cuda()
    vec = lambda on: torch.randn(hq, generator=gen).cuda() if on else None                     # noqa: E731
    slopes, sinks, bias = vec(opts.get("slopes")), vec(opts.get("sinks")), vec(opts.get("sigmoid"))
    slopes = slopes.abs() * 0.1 if slopes is not None else None
    angle = (torch.rand(n, dv // 2, generator=gen) * 6).cuda()
    turn = (angle.cos(), angle.sin()) if opts.get("turn") else None
    ctx = _Ctx(q_lens, kv_lens)
    got = {}
    for dtype in (torch.float32, torch.bfloat16):
        got[dtype] = torch.full((n, hq, dv), float("nan"), dtype=dtype, device="cuda")
        ops.paged_attention_general(ctx, q, k_pool, v_pool, got[dtype], table.cuda(), dk ** -0.5, opts.get("window"), opts.get("chunk"), slopes,
                                    value_width=dv, tensor_cores=False, keep_first=opts.get("keep_first", 0), softcap=opts.get("softcap"),
                                    sinks=sinks, v_share=share, sigmoid=bool(opts.get("sigmoid")), score_bias=bias, turn_back=turn)
    at = 0
    want = torch.empty(n, hq, dv, dtype=torch.float64, device="cuda")
    for s, (m, kl) in enumerate(zip(q_lens, kv_lens)):
        k = _keys_of(k_pool, table, s, kl, page).repeat_interleave(hq // hkv, dim=1)
        v = _keys_of(v_pool, table, s, kl, page)[..., :dv].repeat_interleave(hq // hkv * share, dim=1)
        pos, key = torch.arange(kl - m, kl, device="cuda")[:, None], torch.arange(kl, device="cuda")[None]
        low = torch.zeros_like(pos)
        if opts.get("window"):
            low = torch.maximum(low, pos - opts["window"] + 1)
        if opts.get("chunk"):
            low = torch.maximum(low, pos // opts["chunk"] * opts["chunk"])
        seen = (key <= pos) & ((key >= low) | (key < opts.get("keep_first", 0)))
        sc = torch.einsum("ihd,jhd->hij", q[at:at + m].double(), k) * dk ** -0.5
        if opts.get("softcap"):
            sc = opts["softcap"] * torch.tanh(sc / opts["softcap"])
        if slopes is not None:
            sc = sc - slopes.double()[:, None, None] * (pos - key)
        if opts.get("sigmoid"):
            w = torch.sigmoid(sc + bias.double()[:, None, None]) * seen
        else:
            sc = sc.masked_fill(~seen, -math.inf)
            if sinks is not None:
                sc = torch.cat([sc, sinks.double()[:, None, None].expand(hq, m, 1)], dim=-1)
            w = torch.softmax(sc, dim=-1)[..., :kl]
        out = torch.einsum("hij,jhv->ihv", w, v)
        if turn is not None:
            c, sn = turn[0][at:at + m].double()[:, None], turn[1][at:at + m].double()[:, None]
            u, t = out[..., 0::2], out[..., 1::2]
            out = torch.stack([u * c + t * sn, t * c - u * sn], dim=-1).flatten(-2)
        want[at:at + m] = out
        at += m
    # float32 rows: scores of up to 576 products and sums over the keys, each a few units in the last place off
    assert float((got[torch.float32].double() - want).norm() / want.norm()) < 1.5e-6
    assert float((got[torch.bfloat16].double() - want).abs().max() / want.abs().max()) < 2.0 ** -8


# queries at the ends of float32: infinite ones (with sigmoid weights, which are then zero or one), and finite ones that round to an
# infinite bfloat16 and meet keys as small
@pytest.mark.parametrize("large,sigmoid", [(math.inf, True), (torch.finfo(torch.float32).max, True), (torch.finfo(torch.float32).max, False),
                                           (3.39e38, False), (-3.4e38, False)])
def test_queries_at_the_ends_of_float32(large, sigmoid):
    from pulsar_b200 import ops
    q_lens, kv_lens, hq, hkv, d, page = [1, 2], [70, 33], 4, 2, 64, 16
    gen = torch.Generator().manual_seed(3)
    table, (k_pool, v_pool) = _paged(q_lens, kv_lens, page, [(hkv, d)] * 2, torch.bfloat16, gen)
    q = torch.randn(3, hq, d, generator=gen).cuda() * 0.1
    q[:, :, 5] = large
    k_pool[..., 5] = torch.where(k_pool[..., 5] > 0, 1.0, -1.0) * (1.0 if math.isinf(large) else 2.0 ** -125)       # products of about 8
    ctx, got, want = _Ctx(q_lens, kv_lens), torch.empty(3, hq, d, device="cuda"), torch.empty(3, hq, d, dtype=torch.float64, device="cuda")
    ops.paged_attention_general(ctx, q, k_pool, v_pool, got, table.cuda(), 1.0, tensor_cores=False, sigmoid=sigmoid)
    at = 0
    for s, (m, kl) in enumerate(zip(q_lens, kv_lens)):
        k, v = (_keys_of(p, table, s, kl, page).repeat_interleave(2, dim=1) for p in (k_pool, v_pool))
        hidden = torch.arange(kl, device="cuda")[None] > torch.arange(kl - m, kl, device="cuda")[:, None]
        sc = torch.einsum("ihd,jhd->hij", q[at:at + m].double(), k)
        w = torch.sigmoid(sc) * ~hidden if sigmoid else torch.softmax(sc.masked_fill(hidden, -math.inf), dim=-1)
        want[at:at + m] = torch.einsum("hij,jhv->ihv", w, v)
        at += m
    assert bool(torch.isfinite(got).all())
    assert float((got.double() - want).norm() / want.norm()) < 1e-5       # scores near 9, known to 2^-21 of that: the weights to 5e-6


# infinite numbers in the cache: a key whose score is -infinity weighs nothing (with sigmoid weights one at +infinity weighs one), an
# infinite value makes its column infinite and no other.  Queries of one bfloat16 (0.25) and of three parts of both signs (0.3); one
# that is no number beside them takes its own head's row and no other.
@pytest.mark.parametrize("hq,hkv,dk,dv", [(4, 2, 64, 64), (16, 1, 576, 512)])
@pytest.mark.parametrize("sigmoid", [False, True])
def test_infinite_keys_and_values(hq, hkv, dk, dv, sigmoid):
    from pulsar_b200 import ops
    kv_lens, page = [70, 33], 16
    gen = torch.Generator().manual_seed(5)
    table, (k_pool, v_pool) = _paged([1, 1], kv_lens, page, [(hkv, dk), (hkv, dv)], torch.bfloat16, gen)
    q = torch.randn(2, hq, dk, generator=gen).cuda() * 0.1
    q[0, :, 5], q[1, :, 5], q[1, -1, 6] = 0.25, 0.3, math.nan
    first = table[:, 0].long().cuda()                        # both sequences' first pages
    k_pool[first, :, 3, 5] = -math.inf
    if sigmoid:
        k_pool[first, :, 4, 5] = math.inf
    v_pool[first, :, 7, 9], v_pool[first, :, 8, 17] = math.inf, -math.inf
    ctx, got, want = _Ctx([1, 1], kv_lens), torch.empty(2, hq, dv, device="cuda"), torch.empty(2, hq, dv, dtype=torch.float64, device="cuda")
    ops.paged_attention_general(ctx, q, k_pool, v_pool, got, table.cuda(), 0.5, tensor_cores=False, sigmoid=sigmoid)
    for s, kl in enumerate(kv_lens):
        k, v = (_keys_of(p, table, s, kl, page).repeat_interleave(hq // hkv, dim=1) for p in (k_pool, v_pool))
        sc = torch.einsum("hd,jhd->hj", q[s].double(), k) * 0.5
        w = torch.sigmoid(sc) if sigmoid else torch.softmax(sc, dim=-1)
        want[s] = torch.einsum("hj,jhv->hv", w, v)
    assert bool(torch.isnan(got[1, -1]).all())
    got, want = (x.view(2 * hq, dv)[:-1] for x in (got, want))
    fin = torch.isfinite(want)
    assert not bool(torch.isnan(want).any()) and int((~fin).sum()) == 2 * (2 * hq - 1)
    assert torch.equal(got[~fin].double(), want[~fin])
    assert float((got[fin].double() - want[fin]).norm() / want[fin].norm()) < 1e-5       # as at the ends of float32


@pytest.mark.parametrize("q_lens,kv_lens,hq,hkv,dk,dv", [([1, 1], [1900, 70], 16, 1, 576, 512), ([1, 3], [500, 64], 8, 4, 64, 64)])
def test_partial_results_at_any_float(q_lens, kv_lens, hq, hkv, dk, dv):
    """Scratch that begins at an odd float (a view of a caller's own buffer)."""
    from pulsar_b200 import ops
    gen = torch.Generator().manual_seed(dk)
    table, pools = _paged(q_lens, kv_lens, 16, [(hkv, dk)] if dk == 576 else [(hkv, dk), (hkv, dv)], torch.bfloat16, gen)
    q, n = torch.randn(sum(q_lens), hq, dk, generator=gen).cuda(), sum(q_lens)

    class Shifted(_Ctx):
        def scratch(self, tag, shape, dtype):
            assert tag == "attn.general.partial"
            self.asked = torch.full((shape[0] + 1,), float("nan"), dtype=dtype, device="cuda")
            return self.asked[1:]

    got = []
    for ctx in (_Ctx(q_lens, kv_lens), Shifted(q_lens, kv_lens)):
        out = torch.full((n, hq, dv), float("nan"), device="cuda")
        ops.paged_attention_general(ctx, q, pools[0], pools[-1], out, table.cuda(), dk ** -0.5, value_width=dv, tensor_cores=False)
        got.append(out)
    assert bool(torch.isfinite(ctx.asked[1:3]).all())
    assert float((got[0] - got[1]).norm() / got[0].norm()) < 3e-6         # the two forms, each 1.5e-6 from float64


# 16 tokens and fewer: one and two token tiles, outputs around a block's 64, odd counts, k around the slices and behind their end
@pytest.mark.parametrize("n,heads,k,m", [(1, 2, 1, 1), (8, 3, 16, 64), (9, 2, 17, 65), (16, 5, 100, 66), (3, 2, 512, 128), (5, 2, 1024, 63)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_heads_linear_of_a_few_tokens(n, heads, k, m, dtype):
    from pulsar_b200 import ops
    gen = torch.Generator().manual_seed(n * k + m)
    wide = torch.randn(n, heads * (k + 5), generator=gen).to(dtype).cuda()
    a = wide.view(n, heads, k + 5)[:, :, :k]                 # strided rows, not all on 16-byte addresses
    w, gate = (torch.randn(*s, generator=gen).to(dtype).cuda() for s in ((heads, k, m), (n, heads * m)))
    want = torch.einsum("nhk,hkm->nhm", a.double(), w.double())
    size = torch.einsum("nhk,hkm->nhm", a.double().abs(), w.double().abs())
    out = torch.full((n, heads, m), float("nan"), device="cuda")
    ops.heads_linear(a, w, out)
    assert bool(((out.double() - want).abs() <= (k + 8) * 2.0 ** -24 * size).all())
    gated = torch.empty(n, heads, m, dtype=dtype, device="cuda")
    ops.heads_linear(a, w, gated, gate)
    want = want * torch.sigmoid(gate.double()).view(n, heads, m)
    assert bool(((gated.double() - want).abs() <= ((k + 16) * 2.0 ** -24 + (0 if dtype == torch.float32 else 2.0 ** -8)) * size).all())


# many rows, widths below, at and above one round of a block
@pytest.mark.parametrize("width", [36, 2048, 4100, 8192])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_add_rmsnorm_of_many_rows(width, dtype):
    from pulsar_b200 import ops
    n, gen = 593, torch.Generator().manual_seed(width)
    residual, delta, weight = (torch.randn(*s, generator=gen).cuda() for s in ((n, width), (n, width), (width,)))
    delta = delta.to(dtype)
    out, stream = torch.empty(n, width, dtype=dtype, device="cuda"), residual.clone()
    ops.add_rmsnorm(stream, delta, weight, 1e-6, out)
    assert torch.equal(stream, residual + delta.float())
    x = stream.double()
    want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6) * weight.double()
    tol = 2e-6 if dtype == torch.float32 else 2.0 ** -8         # a sum of up to 8,192 squares, a square root and two products; one rounding
    assert bool(((out.double() - want).abs() <= tol * want.abs() + 1e-30).all())


# The order of a row's sum of squares comes from the width alone: a row has the same bits in a step of a few rows as in one of many,
# so that a float32 prompt's logits do not depend on how it was cut into steps.
@pytest.mark.parametrize("width", [36, 2044, 2048, 3000, 4000, 4096, 4100, 8192, 8196])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_add_rmsnorm_does_not_depend_on_the_number_of_rows(width, dtype):
    from pulsar_b200 import ops
    n, gen = 1300, torch.Generator().manual_seed(width)
    residual, delta, weight = (torch.randn(*s, generator=gen).cuda() for s in ((n, width), (n, width), (width,)))
    delta = delta.to(dtype)
    whole, stream = torch.empty(n, width, dtype=dtype, device="cuda"), residual.clone()
    ops.add_rmsnorm(stream, delta, weight, 1e-6, whole)
    for first, rows in ((0, 1), (3, 2), (7, 591), (500, 592), (700, 593)):
        cut, part = residual[first:first + rows].clone(), torch.empty(rows, width, dtype=dtype, device="cuda")
        ops.add_rmsnorm(cut, delta[first:first + rows].clone(), weight, 1e-6, part)
        assert torch.equal(part, whole[first:first + rows]) and torch.equal(cut, stream[first:first + rows])


# the merge of a row's splits: every round length at its edges and more than one round of 32, one and two columns a thread; most of
# many splits hold no key
@pytest.mark.parametrize("splits", [2, 4, 5, 8, 9, 16, 17, 32, 33, 64, 70])
@pytest.mark.parametrize("hq,hkv,dk,dv,opts", [(4, 4, 16, 16, {}), (8, 1, 576, 512, dict(sinks=True)), (6, 2, 320, 256, dict(sigmoid=True, turn=True)),
                                               (2, 1, 64, 272, dict(turn=True))])
def test_merge_of_splits(splits, hq, hkv, dk, dv, opts, monkeypatch):
    from pulsar_b200 import ops
    q_lens, kv_lens, gen = [1, 3], [530, 40], torch.Generator().manual_seed(splits + dv)
    table, pools = _paged(q_lens, kv_lens, 16, [(hkv, dk), (hkv, dv)], torch.bfloat16, gen)
    q, n = torch.randn(4, hq, dk, generator=gen).cuda(), 4
    sinks = torch.randn(hq, generator=gen).cuda() if opts.get("sinks") else None
    angle = torch.rand(n, dv // 2, generator=gen).cuda()
    options = dict(value_width=dv, tensor_cores=False, sinks=sinks, sigmoid=bool(opts.get("sigmoid")),
                   turn_back=(angle.cos(), angle.sin()) if opts.get("turn") else None)
    got = []
    for k in (1, splits):
        monkeypatch.setattr(ops, "general_splits", lambda blocks, tokens: k)
        out = torch.full((n, hq, dv), float("nan"), device="cuda")
        ops.paged_attention_general(_Ctx(q_lens, kv_lens), q, pools[0], pools[1], out, table.cuda(), dk ** -0.5, **options)
        got.append(out.double())
    assert float((got[0] - got[1]).norm() / got[0].norm()) < 3e-6         # the same sums in another grouping, each 1.5e-6 from float64
