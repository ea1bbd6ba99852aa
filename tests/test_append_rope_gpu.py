"""Rotation and append of prompt rows: more heads than one trip of the 16-byte kernel takes, and key pages off a 16-byte border,
against the rotation in 64 bits.

An angle is below 1000 and carries the fp32 rounding of its frequency and of the product (2^-22 of it: 2^-12); sines, cosines and
sums add less, twice that is allowed.  The result is rounded to bf16: half a unit is 2^-8 of it at most."""
import pytest
import torch

from conftest import load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,D", [(40, 40, 128), (64, 8, 128), (56, 8, 128), (128, 128, 64), (4, 2, 64), (1, 1, 128), (128, 64, 128)])
@pytest.mark.parametrize("page", [16, 32])
def test_heads_and_key_page_alignment(Hq, Hkv, D, page):
    ops = load("ops")
    T, theta, max_pages = 50, 10000.0, 1000 // page
    g = torch.Generator(device="cuda").manual_seed(Hq + D)
    pos = torch.randint(0, max_pages * page, (T,), generator=g, device="cuda")
    slot = torch.arange(T, device="cuda")
    pos[7], pos[11] = -1, max_pages * page  # no entry in the table: nothing is written
    table = torch.randint(0, T, (T, max_pages), generator=g, device="cuda").to(torch.int32)
    live = (pos >= 0) & (pos < max_pages * page)
    at = torch.arange(T, device="cuda") % T
    table[slot[live], pos[live] // page] = at[live].to(torch.int32)  # a page of its own for every row
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, generator=g, device="cuda").bfloat16()
    x = qkv.double().view(T, Hq + 2 * Hkv, D)[:, :Hq + Hkv]
    a = pos[:, None] * theta ** (-torch.arange(D // 2, device="cuda", dtype=torch.float64) * 2 / D)
    lo, hi, c, s = x[..., :D // 2], x[..., D // 2:], a.cos()[:, None], a.sin()[:, None]
    want = torch.cat([lo * c - hi * s, hi * c + lo * s], -1)
    bound = 2.0 ** -8 * want.abs() + 2.0 ** -11 * torch.cat([lo.abs() + hi.abs()] * 2, -1)
    results = []
    for off in (0, 2):  # elements: key pages on a 16-byte border, and 4 bytes off it
        rows = qkv.clone()
        n = T * Hkv * page * D
        k = torch.full((n + 8,), 7.0, device="cuda").bfloat16()[off:off + n].view(T, Hkv, page, D)
        v = torch.full((T, Hkv, page, D), 7.0, device="cuda").bfloat16()
        assert (k.data_ptr() % 16 == 0) == (off == 0)
        ops.kv_append_rope(rows, k, v, table, slot.to(torch.int32), pos.to(torch.int32), Hq, Hkv, D, page, theta)
        results.append((rows, k.clone(), v))
    in_page = (pos % page).clamp(min=0)
    written = torch.zeros(T, page, dtype=torch.bool, device="cuda")
    written[at[live], in_page[live]] = True
    for rows, k, v in results:
        got = torch.cat([rows.view(T, -1, D)[:, :Hq], k[at, :, in_page]], 1).double()
        assert ((got - want).abs() <= bound)[live].all()
        assert torch.equal(v[at[live], :, in_page[live]], qkv.view(T, -1, D)[live][:, Hq + Hkv:])
        assert torch.equal(rows[~live], qkv[~live]) and torch.equal(rows.view(T, -1, D)[:, Hq:], qkv.view(T, -1, D)[:, Hq:])
        assert (k.transpose(1, 2)[~written] == 7).all() and (v.transpose(1, 2)[~written] == 7).all()


def test_the_same_key_whoever_appends_it():
    """Decode of single heads, of four and of two that share a key head, and both kernels for prompt rows."""
    ops = load("ops")
    T, Hkv, D, page, theta = 1024, 8, 128, 16, 10000.0
    g = torch.Generator(device="cuda").manual_seed(3)
    kv = torch.randn(T, 2 * Hkv * D, generator=g, device="cuda").bfloat16()
    pos = torch.randint(0, 200 * page, (T,), generator=g, device="cuda").to(torch.int32)
    table = torch.arange(T, device="cuda", dtype=torch.int32)[:, None].repeat(1, 200)  # (a row sees its own page alone)
    slot, at, got = torch.arange(T, device="cuda", dtype=torch.int32), torch.arange(T, device="cuda"), []
    for Hq, off in ((8, 0), (32, 0), (16, 0), (8, None), (8, 2)):
        rows = torch.cat([torch.randn(T, Hq * D, generator=g, device="cuda").bfloat16(), kv], 1)
        n, v = T * Hkv * page * D, torch.zeros(T, Hkv, page, D, device="cuda").bfloat16()
        k = torch.zeros(n + 8, device="cuda").bfloat16()[off or 0:(off or 0) + n].view(T, Hkv, page, D)
        if got and Hq == 8:
            ops.kv_append_rope(rows, k, v, table, slot, pos, Hq, Hkv, D, page, theta)
        else:
            ops.paged_attention(rows, k, v, table, slot, pos, Hq, Hkv, D, page, theta, True, n_splits=1)
        got.append(k[at, :, (pos % page).long()].view(torch.int16))
    assert all(torch.equal(k, got[0]) for k in got)
