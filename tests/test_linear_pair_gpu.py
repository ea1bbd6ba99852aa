"""Projections of prompt-size batches on pairs of CTAs, at the edges of their tiles, against fp32 torch on the same values.

Sums are fp32 and the result is rounded once to bf16 (8 significant bits), so 2^-8 of the result's norm bounds the distance;
fp32 outputs differ by the order of the sums only.
"""
import pytest
import torch

from conftest import load

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -8


def _err(y, ref):
    return ((y.float() - ref).norm() / ref.norm()).item()


def _setup(T, K, N, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    W = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    return g, x, W, x.float() @ W.float().t()


# 9473 = 74 pairs' worth of 128-token tiles and one row; out: an odd number of row tiles, a ragged last one; in: less than a
# k-block, and one that is not a multiple of it
@pytest.mark.parametrize("T,K,N", [(9473, 64, 128), (9473, 200, 136), (160, 320, 12288), (257, 8, 12288 + 64), (1100, 320, 1920), (4096, 64, 640)])
@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("form", ["bf16", "f32", "relu2"])
def test_base(T, K, N, packed, form):
    ops = load("ops")
    _, x, W, ref = _setup(T, K, N, T + N)
    flags = {"bf16": 0, "f32": ops.OUT_F32, "relu2": ops.ACT_RELU2}[form]
    if form == "relu2":
        ref = ref.clamp(min=0) ** 2
    work = ops.new_workspace(load("_lib").lib().mlora_linear_workspace(T, K, N), x.device)
    y = ops.linear(x, ops.PackedWeight(W) if packed else W, flags=flags, work=work)
    assert ops.status_word(work) == 0
    assert _err(y, ref) < (1e-5 if form == "f32" else TOL)


# element by element: rounding to bf16 (2^-8 of the value), fp32 sums of K products (K 2^-24 of the sum of their magnitudes), and
# what either activation makes of them (its slope is at most 1.13; a gelu of erff is good to 2^-20 of its argument)
@pytest.mark.parametrize("T,K,N", [(9473, 200, 136), (160, 320, 12288), (257, 8, 12288 + 64), (1100, 320, 1920), (1999, 512, 2688)])
@pytest.mark.parametrize("form", ["bf16", "gelu"])
def test_every_element(T, K, N, form):
    ops = load("ops")
    _, x, W, _ = _setup(T, K, N, T + K)
    z, slack = x.double() @ W.double().t(), (x.double().abs() @ W.double().abs().t()) * (K * 2.0 ** -24)
    if form == "gelu":
        slack = 1.13 * slack + 2.0 ** -20 * z.abs()
        z = torch.nn.functional.gelu(z)
    y = ops.linear(x, ops.PackedWeight(W), flags=ops.ACT_GELU if form == "gelu" else 0)
    assert ((y.double() - z).abs() <= 2.0 ** -8 * z.abs() + (1 + 2.0 ** -8) * slack).all()


# modules with odd numbers of row tiles (a pair must not span two of them); few adapters in runs, runs that start inside a
# 16-row block, more than a run table holds, every row another adapter, none at all
@pytest.mark.parametrize("rank", [16, 32, 64, 128])
@pytest.mark.parametrize("adapters,layout", [(1, "runs"), (7, "runs"), (300, "runs"), (40, "scattered"), (5, "none")])
@pytest.mark.parametrize("T,mods,packed", [(1999, [0, 384, 640, 1152], True), (1999, [0, 384, 640, 1152], False), (5000, [0, 136], False)])
def test_lora(T, mods, packed, rank, adapters, layout):
    ops = load("ops")
    K, N, n_mod = 192, mods[-1], len(mods) - 1
    g, x, W, ref = _setup(T, K, N, rank + adapters)
    A = (torch.randn(adapters, n_mod * rank, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    B = (torch.randn(adapters, N, rank, generator=g, device="cuda") * 0.2).bfloat16()
    scales = torch.rand(adapters, generator=g, device="cuda") + 0.5
    stack = ops.LoraStack(A, B, torch.full((adapters,), rank, dtype=torch.int32, device="cuda"), scales, rank, n_mod, tuple(mods), n_out=N)
    if layout == "runs":
        slots = torch.arange(T, device="cuda") * adapters // T
    else:
        slots = torch.randint(-1, adapters if layout == "scattered" else 0, (T,), generator=g, device="cuda")
    slots = slots.to(torch.int32)
    u = ops.lora_shrink(x, stack, slots)
    live = slots >= 0
    if live.any():
        s = slots[live].long()
        su = (u[live].view(-1, n_mod, rank) * scales[s][:, None, None]).bfloat16().float()  # the expand's operand is bf16
        for m in range(n_mod):
            ref[live, mods[m]:mods[m + 1]] += torch.einsum("tr,tor->to", su[:, m], B[s, mods[m]:mods[m + 1]].float())
    if packed:
        stack.pack_b()
    work = ops.new_workspace(load("_lib").lib().mlora_linear_workspace(T, K, N), x.device)
    y = ops.linear(x, ops.PackedWeight(W), stack, slots, u, work=work)
    again = ops.linear(x, ops.PackedWeight(W), stack, slots, u, work=work)
    assert ops.status_word(work) == 0
    assert _err(y, ref) < TOL
    assert torch.equal(y, again)


@pytest.mark.parametrize("T,N", [(2500, 1024), (9473, 128), (300, 8192)])
def test_silu_of_interleaved_rows(T, N):
    ops = load("ops")
    _, x, W, ref = _setup(T, 256, N, N)
    pre = ref.view(T, N // 16, 2, 8)
    ref = (torch.nn.functional.silu(pre[:, :, 0]) * pre[:, :, 1]).flatten(1)
    assert _err(ops.linear(x, ops.PackedWeight(W), flags=ops.SILU_MUL), ref) < TOL


# groups of 256-row tiles: whole tiles, ragged chunks, an odd number of row tiles; column slices per group with a gate
@pytest.mark.parametrize("T,K,N,groups", [(256, 128, 256, 3), (700, 64, 384, 2), (301, 192, 136, 5)])
def test_grouped(T, K, N, groups):
    ops = load("ops")
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, groups * K, generator=g, device="cuda").bfloat16()
    W = (torch.randn(groups, N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    gate = torch.randn(T, groups, generator=g, device="cuda").bfloat16()
    y = torch.full((T, groups * N), 7.0, device="cuda").bfloat16()
    work = ops.new_workspace(load("_lib").lib().mlora_grouped_linear_workspace(256), x.device)
    ops.grouped_linear(x, ops.GroupedWeight(W), y, T=T, x_cols=K, y_cols=N, tile_rows=256, gate=gate, work=work)
    ref = torch.cat([x[:, i * K:(i + 1) * K].float() @ W[i].float().t() * torch.sigmoid(gate[:, i:i + 1].float()) for i in range(groups)], 1)
    assert ops.status_word(work) == 0
    assert _err(y, ref) < TOL


# the same sums as the one-CTA kernel, bit for bit, where its plan has whole tiles (the last three) and where it splits them.  A
# rank pitch of 24 keeps a call on that kernel; no row has an adapter.
@pytest.mark.parametrize("T,K,N", [(300, 2048, 8192), (1000, 512, 4096), (2048, 8192, 2048), (3000, 4096, 4096), (1184, 256, 2048),
                                   (5000, 128, 6144), (9473, 200, 136)])
def test_stable_sums_are_those_of_the_one_cta_kernel(T, K, N):
    ops = load("ops")
    g, x, W, _ = _setup(T, K, N, T)
    stack = ops.LoraStack(torch.zeros(1, 24, K, device="cuda").bfloat16(), torch.zeros(1, N, 24, device="cuda").bfloat16(),
                          torch.full((1,), 24, dtype=torch.int32, device="cuda"), torch.ones(1, device="cuda"), 24, 1, (0, N))
    slots = torch.full((T,), -1, dtype=torch.int32, device="cuda")
    want = ops.linear(x, ops.PackedWeight(W), stack, slots, torch.zeros(T, 24, device="cuda"), flags=ops.OUT_F32)
    got = ops.linear(x, ops.PackedWeight(W), flags=ops.OUT_F32 | ops.STABLE_SUMS)
    assert torch.equal(got, want)
