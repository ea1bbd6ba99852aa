"""Prompt attention whose running maximum moves: a row's sum and output are rescaled at every block that raises it.

Values lie in [0.5, 1.5], so nothing cancels: probabilities rounded to bf16 (8 significant bits: 2^-8 relative at most), the
result rounded to bf16 (2^-8) and fp32 sums in between bound every output's relative error by 2^-7.
"""
import pytest
import torch

from conftest import load

pytestmark = pytest.mark.gpu


# growth of the scores per key, in powers of two of a probability: none, little over a block, 2^9 over a block, past what fp32
# holds, falling
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


# Two keys share a row's probability, the later one with the larger score, and only that one has a value: its probability is 1,
# which bf16 holds exactly, the sum is fp32, so the output is the 64-bit value rounded once: off by half a unit of its last of 8
# bits, plus 2^-18 for exponential, sum and quotient in fp32.  (A reference that lags behind the maximum would round the
# probability a second time.)
@pytest.mark.parametrize("late", [131, 200, 300])
def test_the_largest_probability_is_exact(late):
    ops = load("ops")
    H, D, T = 24, 64, 384
    g = torch.Generator(device="cuda").manual_seed(late)
    q, k, v = (torch.zeros(T, H, D, device="cuda") for _ in range(3))
    q[:, :, 0], k[:, :, 0] = 1.0, -64.0
    growth = torch.linspace(0.05, 5.5, H, device="cuda").bfloat16()
    k[5, :, 0], k[late, :, 0] = 0.0, growth.float()
    v[late] = torch.rand(H, D, generator=g, device="cuda") + 0.5
    kv = torch.cat([k.flatten(1), v.flatten(1)], 1).bfloat16().contiguous()
    tiles = torch.tensor([(0, o, 128, o) for o in range(0, T, 128)], dtype=torch.int32, device="cuda")
    out = torch.zeros(T, H * D, device="cuda").bfloat16()
    ops.prefill_attention_dense(q.flatten(1).bfloat16().contiguous(), kv, H * D, tiles, 3, H, D, D, 1.0, out)
    want = v[late].bfloat16().double() / (1 + torch.exp(-growth.double()))[:, None]
    got = out.view(T, H, D)[late:].double()
    assert ((got - want).abs() <= 2.0 ** (want.log2().floor() - 8) + want * 2.0 ** -18).all()


# tiles without rows, at position 0 and further on, in front of, between and behind others: nothing happens, nothing is reported
@pytest.mark.parametrize("paged", [False, True])
def test_tiles_without_rows(paged):
    ops = load("ops")
    H, D, n = 2, 64, 200
    g = torch.Generator(device="cuda").manual_seed(3)
    q, kv = torch.randn(n, H * D, generator=g, device="cuda").bfloat16(), torch.randn(208, 2 * H * D, generator=g, device="cuda").bfloat16()
    k, v = (t.reshape(13, 16, H, D).transpose(1, 2).contiguous() for t in (kv[:, :H * D], kv[:, H * D:]))
    table = torch.arange(13, dtype=torch.int32, device="cuda")[None]
    outs = []
    for tiles in ([(0, 0, 128, 0), (0, 128, 72, 128)], [(0, 0, 0, 0), (0, 0, 128, 0), (0, 128, 0, 128), (0, 128, 72, 128), (0, 0, 0, 0), (0, 0, -5, 0)]):
        t = torch.tensor(tiles, dtype=torch.int32, device="cuda")
        out, status = torch.full((n, H * D), 7.0, device="cuda").bfloat16(), torch.zeros(1, dtype=torch.int32, device="cuda")
        if paged:
            ops.prefill_attention_masked(q, k, v, table, t, len(tiles), H, D ** -0.5, out, status=status)
        else:
            ops.prefill_attention_dense(q, kv, H * D, t, len(tiles), H, D, D, D ** -0.5, out, status=status)
        assert int(status) == 0
        outs.append(out)
    assert torch.equal(*outs)


# pages of a sequence one after the other in the pool are fetched eight at a time: the same bytes as page by page
@pytest.mark.parametrize("n", [1, 112, 128, 129, 640, 1000])
@pytest.mark.parametrize("D,Hq,Hkv", [(128, 4, 2), (64, 3, 3)])
def test_pages_in_runs_and_scattered(n, D, Hq, Hkv):
    ops = load("ops")
    g = torch.Generator(device="cuda").manual_seed(n)
    pages = -(-n // 16)
    q = torch.randn(n, Hq * D, generator=g, device="cuda").bfloat16()
    k, v = (torch.full((3 * pages, Hkv, 16, D), float("nan"), device="cuda").bfloat16() for _ in range(2))
    rows = torch.randn(2, n, Hkv, D, generator=g, device="cuda").bfloat16()
    tables = [torch.arange(pages) + pages, torch.randperm(3 * pages, generator=torch.Generator().manual_seed(n))[:pages],
              torch.arange(pages).flip(0), torch.arange(pages) * 2]
    tables.append(tables[0].clone())
    tables[4][pages // 2:] += 1  # a run that breaks off inside a block
    tiles = torch.tensor([(0, o, min(128, n - o), o) for o in range(0, n, 128)], dtype=torch.int32, device="cuda")
    outs = []
    for table in tables:
        k.fill_(float("nan")), v.fill_(float("nan"))
        at = table.cuda()[torch.arange(n, device="cuda") // 16], torch.arange(n, device="cuda") % 16
        k[at[0], :, at[1]], v[at[0], :, at[1]] = rows[0], rows[1]
        out = torch.zeros(n, Hq * D, device="cuda").bfloat16()
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        ops.prefill_attention_masked(q, k, v, table[None].to(torch.int32).cuda(), tiles, len(tiles), Hq, D ** -0.5, out, status=status)
        assert int(status) == 0
        outs.append(out)
    s = torch.einsum("qhd,khd->hqk", q.view(n, Hq, D).double(), rows[0].double().repeat_interleave(Hq // Hkv, 1)) * D ** -0.5
    s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    want = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), rows[1].double().repeat_interleave(Hq // Hkv, 1)).flatten(1)
    assert ((outs[0].double() - want).norm() / want.norm()).item() < 2.0 ** -7  # two roundings to bf16, as above
    for o in outs[1:]:
        assert torch.equal(o, outs[0])
