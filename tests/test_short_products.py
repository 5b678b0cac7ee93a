"""float32 products of up to 16 rows over a short K, whose stages are 64 k: both sides of the rule, against the general kernel bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# k: up to two stages, a remainder, whole long stages, a ring that turns, the last before long stages; n: few blocks, more than one an SM
@pytest.mark.parametrize("k", [4, 60, 64, 68, 128, 132, 192, 256, 320, 380, 384, 512, 576, 636, 640])
@pytest.mark.parametrize("n", [130, 4800])
def test_products_over_a_short_k(n, k):
    from pulsar_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(n + k)
    w = torch.randn(n, k, generator=g, device="cuda")
    for m in (1, 2, 3, 4, 5, 8, 9, 16):
        a = torch.randn(m, k, generator=g, device="cuda")
        odd = torch.empty(m * k + 4, device="cuda")[1:m * k + 1].view(m, k).copy_(a)         # an address the general kernel takes
        out, want = torch.full((m, n), float("nan"), device="cuda"), torch.empty(m, n, device="cuda")
        ops.gemm_simt(odd, w, want)
        for loaded in (False, True):
            out.fill_(float("nan"))
            torch.cuda.synchronize()
            ops.gemm_simt(a, w, out, loaded)
            assert torch.equal(out, want), (m, loaded)
        half = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
        ops.gemm_simt(a, w, half)
        assert torch.equal(half, want.bfloat16()), m
