"""Draws from rows short enough for one block (up to 2,048 tokens), at the edges of the threads' ranges."""
import pytest
import torch

from plain import qwen3_plain as plain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [1, 2, 255, 256, 257, 336, 513, 2047, 2048, 2049])
@pytest.mark.parametrize("top_k,top_p", [(0, 1.0), (1, 1.0), (7, 1.0), (0, 0.6), (40, 0.95), (5000, 0.999)])
def test_rows_follow_the_inverse_cdf_of_the_survivors(vocab, top_k, top_p):
    from pulsar_b200 import ops
    g = torch.Generator().manual_seed(vocab * 7 + top_k)
    logits = torch.randn(vocab, generator=g) * 2.0
    logits[::5] = logits[0]                                  # equal probabilities, some of them at the cut
    if vocab > 3:
        logits[vocab // 2] = -float("inf")
    rows, temperature = 40, 0.9
    uniform = (torch.arange(rows, dtype=torch.float32) + 0.5) / rows
    uniform[0] = 0.0
    args = [t.cuda() for t in (logits.repeat(rows, 1), torch.full((rows,), temperature), torch.full((rows,), top_k, dtype=torch.int32),
                               torch.full((rows,), top_p), uniform)]
    out = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    ops.sample(args[0], out, *args[1:], any_greedy=False)
    keep = torch.zeros(vocab, dtype=torch.bool)
    keep[plain.sample_filter(logits, temperature, top_k, top_p)[1]] = True
    p = torch.softmax(logits.double() / temperature, 0) * keep
    cdf = torch.cumsum(p, 0)
    got = out.cpu().long()
    for r in range(rows):
        assert bool(keep[got[r]]), "a token outside the surviving set was drawn"
        want = min(int(torch.searchsorted(cdf, float(uniform[r]) * float(p.sum()), right=True)), vocab - 1)
        # the device adds float32 probabilities: a draw on the border of two tokens may fall to either side
        assert got[r] == want or abs(float(cdf[min(got[r], want)]) - float(uniform[r]) * float(p.sum())) < 1e-5, (r, int(got[r]), want)
    # greedy rows beside them, and the same call again
    mixed = args[1].clone()
    mixed[::3] = 0.0
    again = torch.full_like(out, -1)
    ops.sample(args[0], again, mixed, *args[2:])
    top = int(torch.argmax(logits))
    assert again.cpu().tolist() == [top if r % 3 == 0 else int(got[r]) for r in range(rows)]
