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


# n: one block, a remainder, blocks for more than one an SM (4800); k: less than a stage, whole stages, tails; the last: 64 rows a block
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
