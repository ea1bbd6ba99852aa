"""Decode attention of query heads that share a key head: the same rows one by one, which run the kernel for single heads."""
import pytest
import torch

from conftest import load

pytestmark = pytest.mark.gpu


def _case(cuda, T, Hq, Hkv, ps, lens, seed):
    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g).to(cuda)
    max_pages = max(lens) // ps + 2
    K, V = (r(T * max_pages, Hkv, ps, 128).bfloat16() for _ in range(2))
    bt = torch.randperm(T * max_pages - 1, generator=g)[:T * max_pages - 1].add(1)
    bt = torch.cat([bt, bt[:1]]).int().view(T, max_pages)
    for t, n in enumerate(lens):  # whatever lies behind a sequence's last key
        K[bt[t, n // ps], :, n % ps + 1:], V[bt[t, n // ps], :, n % ps + 1:] = float("nan"), float("inf")
    return r, K, V, bt.to(cuda), torch.arange(T, dtype=torch.int32, device=cuda), torch.tensor(lens, dtype=torch.int32, device=cuda)


def _same(out, one):
    # fp32 scores and sums in another order, then rounded to bf16: neighbouring values at most, half of 2^-7 each
    assert bool(torch.isfinite(out).all())
    diff = (out.float() - one.float()).abs()
    assert float((diff - 2 ** -7 * one.float().abs()).max()) <= 1e-5
    assert float(diff.norm() / one.float().norm()) < 1e-3


LENS = [0, 1, 14, 15, 16, 17, 31, 32, 33, 63, 64, 65, 100, 127, 128, 129, 250, 300]


@pytest.mark.parametrize("Hq,Hkv,ps", [(32, 8, 16), (32, 16, 16), (64, 8, 32), (36, 18, 32), (48, 4, 16)])
@pytest.mark.parametrize("n_splits", [1, 3])
@pytest.mark.parametrize("chunk", [0, 48])
def test_masked(cuda, Hq, Hkv, ps, n_splits, chunk):
    ops = load("ops")
    if chunk % ps:
        chunk = 64
    lens = [LENS[i % len(LENS)] for i in range(18)]
    T = len(lens)
    r, K, V, bt, rs, rp = _case(cuda, T, Hq, Hkv, ps, lens, Hq + ps)
    q, sink = r(T, Hq * 128).bfloat16(), r(Hq)
    out, one = torch.zeros_like(q), torch.zeros_like(q)

    def run(rows, o):
        w = torch.zeros(max(ops.paged_attention_workspace(T, Hq, 128, n_splits), 16), dtype=torch.uint8, device=cuda)
        ops.paged_attention_masked(q[rows], K, V, bt, rs[rows], rp[rows], Hq, 128 ** -0.5, o[rows], chunk=chunk, sink=sink, n_splits=n_splits, work=w)

    run(slice(0, T), out)
    for t in range(T):
        run(slice(t, t + 1), one)
    _same(out, one)


@pytest.mark.parametrize("Hq,Hkv,ps,dim,rot", [(32, 8, 16, 128, 128), (32, 16, 32, 120, 64), (40, 10, 16, 128, 0)])
@pytest.mark.parametrize("n_splits", [1, 2])
def test_new_token_with_bias_rotation_and_norm(cuda, Hq, Hkv, ps, dim, rot, n_splits):
    ops = load("ops")
    lens = [LENS[i % len(LENS)] for i in range(18)]
    T = len(lens)
    r, K, V, bt, rs, rp = _case(cuda, T, Hq, Hkv, ps, lens, dim + rot)
    x, bias, sink = r(T, (Hq + Hkv) * dim).bfloat16(), r((Hq + Hkv) * dim), r(Hq)
    inv = 500000.0 ** (-torch.arange(max(rot // 2, 1), device=cuda) / max(rot // 2, 1))
    got = []
    for rows in ([slice(0, T)], [slice(t, t + 1) for t in range(T)]):
        k, v, o = K.clone(), V.clone(), torch.zeros(T, Hq * 128, dtype=torch.bfloat16, device=cuda)
        w = torch.zeros(max(ops.paged_attention_workspace(T, Hq, 128, n_splits), 16), dtype=torch.uint8, device=cuda)
        for s in rows:
            ops.paged_attention_rms(x[s], bias, inv, rot, dim, 1e-6, k, v, bt, rs[s], rp[s], Hq, dim ** -0.5, o[s], sink=sink, n_splits=n_splits, work=w)
        got.append((k, v, o))
    assert all(torch.equal(a.view(torch.int16), b.view(torch.int16)) for a, b in zip(got[0][:2], got[1][:2]))  # what is appended: the same bits
    _same(got[0][2], got[1][2])


@pytest.mark.parametrize("Hq,Hkv,ps", [(32, 8, 16), (32, 16, 32)])
@pytest.mark.parametrize("fused", [True, False])
def test_rotary(cuda, Hq, Hkv, ps, fused):
    ops = load("ops")
    lens = [LENS[i % len(LENS)] for i in range(18)]
    T = len(lens)
    r, K, V, bt, rs, rp = _case(cuda, T, Hq, Hkv, ps, lens, 7)
    x, got = r(T, (Hq + 2 * Hkv) * 128).bfloat16(), []
    for rows in ([slice(0, T)], [slice(t, t + 1) for t in range(T)]):
        k, v, o = K.clone(), V.clone(), torch.zeros(T, Hq * 128, dtype=torch.bfloat16, device=cuda)
        for s in rows:
            ops.paged_attention(x[s], k, v, bt, rs[s], rp[s], Hq, Hkv, 128, ps, 10000.0, fused, out=o[s], n_splits=1)
        got.append((k, v, o))
    assert torch.equal(got[0][0].view(torch.int16), got[1][0].view(torch.int16))  # what is appended: the same bits
    assert torch.equal(got[0][1].view(torch.int16), got[1][1].view(torch.int16))
    _same(got[0][2], got[1][2])


@pytest.mark.parametrize("Hq,Hkv,ps", [(32, 8, 16), (32, 16, 32), (32, 8, 32), (32, 16, 16)])
@pytest.mark.parametrize("n_splits", [1, 3])
def test_keys_with_a_score_of_minus_infinity(cuda, Hq, Hkv, ps, n_splits):
    """They are left out, whatever their value is, for the heads that score them so; a row of nothing else (or of no scores at all) is zero."""
    ops = load("ops")
    lens = [LENS[i % len(LENS)] for i in range(18)]
    T, D = len(lens), 128
    r, K, V, bt, rs, rp = _case(cuda, T, Hq, Hkv, ps, lens, Hq + ps + 1)
    q = r(T, Hq, D).bfloat16()
    q[:, ::2, 5], q[:, 1::2, 5] = 1.0, 0.25  # (both heads of a pair see column 5 with a plus sign)
    q[:, :, 6] = 0.0
    q = q.view(T, Hq * D)
    for t, n in enumerate(lens):
        for key in range(n + 1):
            if (n > 200 and key % 5 == 3) or n in (15, 33, 64) or (n == 100 and key < 40):
                K[bt[t, key // ps], :, key % ps, 5] = float("-inf")
                V[bt[t, key // ps], :, key % ps] = float("inf") if key % 2 else float("nan")
            if n == 17:
                K[bt[t, key // ps], :, key % ps, 6] = float("nan")
    out, one = torch.zeros_like(q), torch.zeros_like(q)

    def run(rows, o):
        w = torch.zeros(max(ops.paged_attention_workspace(T, Hq, D, n_splits), 16), dtype=torch.uint8, device=cuda)
        ops.paged_attention_masked(q[rows], K, V, bt, rs[rows], rp[rows], Hq, D ** -0.5, o[rows], n_splits=n_splits, work=w)

    run(slice(0, T), out)
    for t in range(T):
        run(slice(t, t + 1), one)
    _same(out, one)
    assert all(bool((out[t] == 0).all()) == (n in (15, 17, 33, 64)) for t, n in enumerate(lens))
