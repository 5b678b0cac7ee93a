"""Weights that are views into larger buffers: contiguous, but not on the boundaries that wide loads need."""
import pytest
import torch


@pytest.mark.parametrize("dtype,code,size", [(torch.float32, 0, 4), (torch.bfloat16, 1, 2)])
def test_pairs_of_weights_are_read_where_they_stand_on_pair_boundaries(dtype, code, size):
    """Which form ``heads_linear`` takes, asked on the host: the address counts, not only the number of outputs."""
    from pulsar_b200 import ops
    pairs = ops.fn("pb_heads_linear_pairs")
    for outputs in (1, 2, 63, 64):
        for offset in range(4):
            assert pairs(code, 4096 + offset * size, outputs) == int(outputs % 2 == 0 and offset % 2 == 0), (outputs, offset)


@pytest.mark.gpu
@pytest.mark.parametrize("n,heads,k,m", [(1, 2, 16, 64), (9, 3, 17, 66), (16, 2, 128, 512), (3, 1, 5, 2), (20, 2, 24, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_heads_linear_takes_weights_at_any_element(n, heads, k, m, dtype):
    from pulsar_b200 import ops
    gen = torch.Generator().manual_seed(n * k)
    a, w = (torch.randn(*s, generator=gen).to(dtype).cuda() for s in ((n, heads, k), (heads, k, m)))
    want = torch.empty(n, heads, m, device="cuda")
    ops.heads_linear(a, w, want)
    buf = torch.empty(w.numel() + 3, dtype=dtype, device="cuda")
    for offset in (1, 2, 3):
        view = buf[offset:offset + w.numel()].view(w.shape)
        view.copy_(w)
        assert view.is_contiguous() and view.data_ptr() % (2 * view.element_size()) == (offset % 2) * view.element_size()
        out = torch.empty_like(want)
        ops.heads_linear(a, view, out)
        assert torch.equal(out, want)


def test_only_loaded_weights_are_read_before_the_kernels_ahead_have_ended(monkeypatch):
    """The float32 products and ``heads_linear`` take a ``w`` that an earlier kernel may still be writing unless the caller says
    that it is a loaded weight."""
    from pulsar_b200 import ops
    asked = []
    monkeypatch.setattr(ops, "fn", lambda name: lambda *args: asked.append(name) or 0)
    monkeypatch.setattr(ops, "_cuda", lambda *tensors: None)
    monkeypatch.setattr(ops, "stream", lambda: 0)
    a, w, out = torch.zeros(2, 8), torch.zeros(4, 8), torch.zeros(2, 4)
    scratch = type("Ctx", (), {"scratch": lambda self, tag, shape, dtype=None: torch.zeros(shape)})()
    for call in (lambda **kw: ops.gemm_simt(a, w, out, **kw), lambda **kw: ops.linear(a, w, out, **kw),
                 lambda **kw: ops.gated_linear(scratch, a, w, torch.zeros(2, 2), **kw)):
        for kw, name in (({}, "pb_gemm_simt"), (dict(loaded=False), "pb_gemm_simt"), (dict(loaded=True), "pb_gemm_simt_loaded")):
            asked.clear()
            call(**kw)
            assert [n for n in asked if "simt" in n] == [name]


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 3, 16])
def test_a_product_with_a_matrix_that_was_just_computed(m):
    """``w`` comes from the kernel just before, which lets its successor onto the SMs at its first instruction."""
    from pulsar_b200 import ops
    n, k = 4096, 1024
    gen = torch.Generator(device="cuda").manual_seed(m)
    a, ones = torch.randn(m, k, generator=gen, device="cuda"), torch.ones(k, device="cuda")
    w, out = torch.zeros(n, k, device="cuda"), torch.empty(m, n, device="cuda")
    heads = torch.empty(m, 4, 1024, device="cuda")
    for i in range(20):
        rows = torch.randn(n, k, generator=gen, device="cuda")
        ops.add_rmsnorm(rows, None, ones, 1e-6, w)
        ops.linear(a, w, out)
        first = out.clone()
        torch.cuda.synchronize()
        ops.linear(a, w, out)
        assert torch.equal(out, first)
        ops.add_rmsnorm(rows, None, ones * 2, 1e-6, w)
        ops.heads_linear(a.view(m, 1, k).expand(m, 4, k), w.view(4, 1024, 1024), heads)
        first = heads.clone()
        torch.cuda.synchronize()
        ops.heads_linear(a.view(m, 1, k).expand(m, 4, k), w.view(4, 1024, 1024), heads)
        assert torch.equal(heads, first)
