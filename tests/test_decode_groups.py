"""Decode attention on the CUDA cores for query heads in groups of every size up to nine: whole passes, passes with places left over, several."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# few blocks (tiles staged in shared memory) and many; a sequence without keys, one key, tiles that end early
@pytest.mark.parametrize("kv_lens", [[0, 1, 33, 200], [70, 31] * 40])
@pytest.mark.parametrize("d", [16, 80, 256])
@pytest.mark.parametrize("group", [1, 2, 3, 4, 5, 6, 7, 9])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_groups(kv_lens, d, group, dtype):
    from pulsar_b200 import ops
    hkv, page, splits, scale = 3, 8, 2, 0.2
    g = torch.Generator(device="cuda").manual_seed(d * 10 + group)
    need = [-(-k // page) for k in kv_lens]
    ids = torch.randperm(sum(need), generator=torch.Generator().manual_seed(group)).to(torch.int32)
    table = torch.zeros(len(need), max(need), dtype=torch.int32)
    for i, n in enumerate(need):
        table[i, :n] = ids[sum(need[:i]):sum(need[:i + 1])]
    pools = [torch.randn(sum(need), hkv, page, d, generator=g, device="cuda").to(dtype) for _ in range(2)]
    q = torch.randn(len(kv_lens), hkv * group, d, generator=g, device="cuda").to(dtype)
    out = torch.full_like(q, float("nan"))
    partial = torch.empty(q.shape[0] * q.shape[1] * splits * (d + 2), device="cuda")
    ops.paged_attention_decode(q, *pools, out, partial, table.cuda(), torch.tensor(kv_lens, dtype=torch.int32, device="cuda"), scale, None,
                               splits, tensor_cores=False)
    for i, n in enumerate(kv_lens):
        if n == 0:
            assert not out[i].any()
            continue
        rows = [p[table[i, :need[i]].long().cuda()].transpose(1, 2).reshape(-1, hkv, d)[:n].double() for p in pools]
        for h in range(hkv * group):
            s = torch.softmax(rows[0][:, h // group] @ q[i, h].double() * scale, 0)
            want, size = s @ rows[1][:, h // group], s @ rows[1][:, h // group].abs()
            # a score is a chain of d products (its error moves the weight by its size), a sum one of n; then the rounding of the output
            score = d * 2.0 ** -24 * float((rows[0][:, h // group].abs() @ q[i, h].double().abs()).max()) * scale
            bound = (4 * score + (n + 8) * 2.0 ** -23) * size + (want.abs() * 2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
            assert bool(((out[i, h].double() - want).abs() <= bound + 1e-30).all()), (i, h)
