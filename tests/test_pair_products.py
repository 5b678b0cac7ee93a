"""float32 products whose tiles compute neighbouring columns in pairs: edges of the tiles, against the general kernel bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# n: blocks for more than one an SM, columns that are no multiple of 4 or of a tile; k: less than a stage, a remainder, many stages;
# m: more than half a tile of rows, a last tile of a few
@pytest.mark.parametrize("n,k", [(19200, 4), (19201, 68), (9602, 260), (19330, 1028)])
@pytest.mark.parametrize("m", [17, 32, 49, 60, 90])
def test_pairs(m, n, k):
    from pulsar_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(m * 1000 + k)
    a, w = (torch.randn(r, k, generator=g, device="cuda") for r in (m, n))
    odd = torch.empty(m * k + 4, device="cuda")[1:m * k + 1].view(m, k).copy_(a)         # an address the general kernel takes
    out, want = torch.full((m, n), float("nan"), device="cuda"), torch.empty(m, n, device="cuda")
    ops.gemm_simt(a, w, out)
    ops.gemm_simt(odd, w, want)
    assert torch.equal(out, want)
    half = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    ops.gemm_simt(a, w, half)
    assert torch.equal(half, want.bfloat16())
    a[m // 2, k // 2] = float("inf")
    w[n - 1, 0] = float("nan")
    odd.copy_(a)
    ops.gemm_simt(a, w, out)
    ops.gemm_simt(odd, w, want)
    assert torch.equal(out.nan_to_num(1.5), want.nan_to_num(1.5))
