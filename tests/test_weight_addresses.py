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
