"""Prompt attention whose running maximum moves: the reference of a row's scores follows it only past a factor of 2^8.

Values lie in [0.5, 1.5], so nothing cancels: probabilities rounded to bf16 (8 significant bits: 2^-8 relative at most), the
result rounded to bf16 (2^-8) and fp32 sums in between bound every output's relative error by 2^-7.
"""
import pytest
import torch

from conftest import load

pytestmark = pytest.mark.gpu


# growth of the scores per key, in powers of two of a probability: none, within the factor over blocks, past it at some
# blocks and rows only, past it everywhere, falling
@pytest.mark.parametrize("growth", [0.0, 0.01, 0.07, 0.5, -0.05])
@pytest.mark.parametrize("lens", [[1], [127, 128, 129], [700], [64, 513]])
@pytest.mark.parametrize("Dk,Dv", [(128, 128), (64, 128), (128, 64)])
def test_scores_that_grow(growth, lens, Dk, Dv):
    ops = load("ops")
    H, T = 3, sum(lens)
    g = torch.Generator(device="cuda").manual_seed(T)
    q = torch.randn(T, H, Dk, generator=g, device="cuda") * 0.3
    k = torch.randn(T, H, Dk, generator=g, device="cuda") * 0.3
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    q[:, :, 0], k[:, :, 0] = 8.0, (pos * growth * 0.6931 / 8.0)[:, None].expand(T, H)
    v = torch.rand(T, H, Dv, generator=g, device="cuda") + 0.5
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    kv = torch.cat([k.flatten(1), v.flatten(1)], 1).contiguous()
    tiles, base = [], 0
    for n in lens:
        tiles += [(base, base + o, min(128, n - o), o) for o in range(0, n, 128)]
        base += n
    out = torch.full((T, H * Dv), float("nan"), device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.prefill_attention_dense(q.flatten(1).contiguous(), kv, H * Dk, torch.tensor(tiles, dtype=torch.int32, device="cuda"), len(tiles), H, Dk, Dv,
                                1.0, out, status=status)
    assert int(status) == 0
    base = 0
    for n in lens:
        s = torch.einsum("qhd,khd->hqk", q[base:base + n].double(), k[base:base + n].double())
        s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
        want = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v[base:base + n].double()).flatten(1)
        got = out[base:base + n].double()
        assert ((got - want).abs() / want).max().item() < 2.0 ** -7
        base += n
