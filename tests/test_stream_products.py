"""The weight-streaming tcgen05 product at the edges of its cuts: shares of tokens, remainders of tiles, rounds of clusters."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m * 1000 + n + k)
    a = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(n, k, generator=g, device="cuda") / k ** 0.5).bfloat16()
    return a, w, a.double() @ w.double().T, a.double().abs() @ w.double().abs().T


# m: one token, a last quad of one to four tokens, one and two passes; n, k: fewer tiles than clusters, several rounds of them with a
# remainder, one k-tile, a k-tile that ends inside an atom, more slices than k-tiles of a block
@pytest.mark.parametrize("m", [1, 18, 35, 63, 66, 128])
@pytest.mark.parametrize("n,k", [(16, 8), (136, 136), (40000, 264), (2064, 4096), (30002, 1000)])
@pytest.mark.parametrize("loaded", [True, False])
def test_products(m, n, k, loaded):
    from pulsar_b200 import ops
    a, w, ref, size = _operands(m, n, k)
    out = torch.full((m, n), float("nan"), device="cuda")
    assert ops.gemm_tcgen05_stream(a, w, out, loaded=loaded)
    # k products, exact in float32, added in float32 (the tensor core may cut instead of rounding): an ulp of the sum of sizes each
    assert bool(((out.double() - ref).abs() <= k * 2.0 ** -23 * size).all())
    half = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    assert ops.gemm_tcgen05_stream(a, w, half, loaded=loaded)
    assert torch.equal(half, out.bfloat16())                # the same sums, rounded once
    again = torch.empty_like(out)
    assert ops.gemm_tcgen05_stream(a, w, again, loaded=loaded)
    assert torch.equal(again, out)
    ops.check_wait_words()


@pytest.mark.parametrize("m", [17, 64, 97])
@pytest.mark.parametrize("inter,k", [(24, 512), (1000, 4096), (12288, 2048)])
@pytest.mark.parametrize("gating", [None, (7.0, 1.702, 1.0), (0.5, float("inf"), 0.0)])
def test_gated_products(m, inter, k, gating):
    from pulsar_b200 import ops
    a, w, ref, _ = _operands(m, 2 * inter, k)
    act = torch.full((m, inter), float("nan"), device="cuda")
    assert ops.gemm_tcgen05_stream(a, w, act, swiglu=True, gating=gating)
    gate, up = ref[:, :inter], ref[:, inter:]
    limit, alpha, shift = gating or (float("inf"), 1.0, 0.0)
    gate, up = gate.clamp(max=limit), up.clamp(-limit, limit)
    slope = torch.sigmoid(alpha * gate) if alpha < float("inf") else (gate > 0).double()
    # the sums are off by 1e-5 of their size at most, the gating's slopes are small numbers, expf a few units in the last place
    assert float((act.double() - gate * slope * (up + shift)).abs().max()) < 2e-4
    ops.check_wait_words()


@pytest.mark.parametrize("m,n,k", [(17, 640, 2048), (33, 160, 4096), (64, 4096, 4096), (65, 2048, 8192), (96, 512, 8200)])
def test_linear_takes_it_and_gives_the_library_products_result(m, n, k, monkeypatch):
    from pulsar_b200 import ops
    a, w, ref, _ = _operands(m, n, k)
    assert ops._stream_wanted(m, n, k)
    taken = []
    kernel = ops.gemm_tcgen05_stream
    monkeypatch.setattr(ops, "gemm_tcgen05_stream", lambda *args, **kw: taken.append(kernel(*args, **kw)) or taken[-1])
    out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    ops.linear(a, w, out)
    assert taken == [True]
    assert float((out.double() - ref).abs().max() / ref.abs().max()) < 2.0 ** -8
    # weights on an address that is no multiple of 16 bytes: the library product, as before
    buf = torch.empty(n * k + 8, dtype=torch.bfloat16, device="cuda")
    odd = buf[1:n * k + 1].view(n, k)
    odd.copy_(w)
    ops.linear(a, odd, out)
    assert taken == [True, False]
    assert float((out.double() - ref).abs().max() / ref.abs().max()) < 2.0 ** -8


# every block's epilogue takes all of a tile's sums, however many slices share them: no more slices than the walk over a tile pays for
@pytest.mark.parametrize("gated,m,n,k,most", [(1, 111, 28672, 4096, 2), (1, 111, 22016, 4096, 2), (1, 97, 16384, 2048, 1), (0, 128, 76000, 2048, 1),
                                              (0, 112, 128256, 2048, 1), (1, 48, 24576, 4096, 2), (0, 48, 4096, 12288, 4), (0, 17, 160, 4096, 8)])
def test_a_product_is_cut_into_no_more_slices_than_its_sums_allow(gated, m, n, k, most):
    import ctypes
    from pulsar_b200 import ops
    slices, rows = ctypes.c_int(), ctypes.c_int()
    assert ops.fn("pb_gemm_tcgen05_stream_cut")(gated, m, n, k, ctypes.byref(slices), ctypes.byref(rows)) > 0
    assert 1 <= slices.value <= most and rows.value % 16 == 0 and 48 <= rows.value <= 128
    a, w, ref, size = _operands(m, n, k)
    out = torch.full((m, n // 2 if gated else n), float("nan"), device="cuda")
    assert ops.gemm_tcgen05_stream(a, w, out, swiglu=bool(gated))
    if gated:
        ref = torch.nn.functional.silu(ref[:, :n // 2]) * ref[:, n // 2:]
        assert float((out.double() - ref).abs().max()) < 2e-4
    else:
        assert bool(((out.double() - ref).abs() <= k * 2.0 ** -23 * size).all())
    ops.check_wait_words()
