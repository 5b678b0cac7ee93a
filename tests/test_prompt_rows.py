"""Kernels of prompt portions that move 16 bytes at a time where their rows allow it: the same bits as one element at a time."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def _at(t, off):
    """A contiguous copy of ``t`` on the GPU, ``off`` elements behind a 16-byte address."""
    flat = torch.empty(t.numel() + off, dtype=t.dtype, device="cuda")
    flat[off:].copy_(t.reshape(-1))
    return flat[off:].view(t.shape)


# one token, tokens around a span of 256 and behind it, two sequences; channels in and beside blocks of eight; states around the four
# vectors that are read together
@pytest.mark.parametrize("lens,inner,state", [((1,), 8, 16), ((255, 7), 24, 8), ((256, 1), 16, 4), ((300, 513), 40, 16), ((40,), 20, 16)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_chunked_scan_of_aligned_rows(lens, inner, state, dtype):
    from pulsar_b200 import ops
    if not ops.selective_scan_chunked_supported(state):
        pytest.skip("a state size that the kernel does not take")
    n, gen = sum(lens), torch.Generator().manual_seed(sum(lens) + inner)
    x, xz, bc = (torch.randn(n, w, generator=gen).to(dtype) for w in (inner, 2 * inner, 2 * state + 8))
    dt_pre, start = torch.randn(n, inner, generator=gen), torch.randn(len(lens) + 1, inner * (state + 3), generator=gen)
    a_log, d_skip, dt_bias = torch.rand(inner, state, generator=gen), torch.randn(inner, generator=gen), torch.randn(inner, generator=gen)
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    ctx = types.SimpleNamespace(cu_q=cu, state_slots=torch.arange(len(lens), dtype=torch.int32, device="cuda").flip(0).contiguous(), n_seqs=len(lens))
    got = []
    for off in (0, 1):
        arena, y = start.cuda(), _at(torch.full((n, inner), float("nan"), dtype=dtype), off)
        ops.selective_scan_prompt(ctx, _at(x, off), _at(xz, off), _at(bc, off), _at(dt_pre, off), dt_bias.cuda(), a_log.cuda(), d_skip.cuda(),
                                  arena, inner * state, 4, y, chunked=True)
        got.append((y.clone(), arena))
    assert bool(torch.isfinite(got[0][0].float()).all())
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("n,heads,dim,rot", [(1, 1, 8, 8), (3, 5, 24, 16), (65, 16, 128, 64), (7, 3, 20, 4)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rows_of_the_expanded_form(n, heads, dim, rot, dtype):
    from pulsar_b200 import ops
    gen = torch.Generator().manual_seed(n + dim)
    plain, shared = torch.randn(n, heads, dim, generator=gen).to(dtype), torch.randn(n, rot, generator=gen).to(dtype)
    want = torch.cat([plain, shared[:, None].expand(n, heads, rot)], dim=-1)
    q, turn = torch.randn(n, heads * (dim + rot) + 8, generator=gen).to(dtype), torch.rand(n, rot // 2, generator=gen).cuda()
    for off in (0, 1):
        keys = _at(torch.zeros(n, heads, dim + rot, dtype=dtype), off)
        ops.latent_expand_keys(_at(plain, off), _at(shared, off), keys)
        assert torch.equal(keys.cpu(), want)
        rows = _at(torch.full((n, heads, dim + rot), float("nan")), off)
        ops.latent_prepare(_at(q, off)[:, :heads * (dim + rot)], None, None, 1e-6, turn.cos(), turn.sin(), None, None, rows, heads, dim, rot,
                           8, 16, plain_too=True)
        assert torch.equal(rows.cpu()[..., :dim], q[:, :heads * (dim + rot)].view(n, heads, dim + rot)[..., :dim].float())
        assert bool(torch.isfinite(rows).all())


@pytest.mark.parametrize("n,width,behind", [(1, 8, 0), (3, 4104, 8), (700, 2048, 2048), (5, 12, 4), (5, 16, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sigmoid_gate_of_aligned_rows(n, width, behind, dtype):
    from pulsar_b200 import ops
    gen = torch.Generator().manual_seed(n + width)
    x, wide = torch.randn(n, width, generator=gen).to(dtype), (8 * torch.randn(n, width + behind, generator=gen)).to(dtype)
    wide[0, :4] = torch.tensor([float("inf"), -float("inf"), 200.0, -200.0])
    got = []
    for off in (0, 1):
        y = _at(x, off)
        ops.sigmoid_gate(y, _at(wide, off)[:, :width])
        got.append(y.clone())
    assert torch.equal(got[0], got[1])
    want = x.double() * torch.sigmoid(wide[:, :width].double())
    tol = 4e-6 if dtype == torch.float32 else 2.0 ** -8         # an exponential, a sum and a quotient in float32; one rounding
    assert bool(((got[0].cpu().double() - want).abs() <= tol * want.abs() + 1e-38).all())
