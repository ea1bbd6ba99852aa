"""The per-row expand of the rank-compact layout at the edges of its spans of 1024 features, bit for bit against the row-major
layout (the same sums in the same order), which other tests hold against torch."""
import pytest
import torch

from conftest import load

pytestmark = pytest.mark.gpu


# one whole span, a span of 8 features behind it, two spans and one of 8, module borders inside the second and third span
@pytest.mark.parametrize("mods", [[0, 1024], [0, 1032], [0, 2056], [0, 1152, 2304, 3456], [0, 264, 1296, 1304]])
@pytest.mark.parametrize("ranks", [[8, 16, 32, 64, 128, 0], [8], [16], [24, 40], [128, 0]])
@pytest.mark.parametrize("f32", [True, False])
def test_against_the_row_major_layout(mods, ranks, f32):
    ops = load("ops")
    T, K, N, n_mod, n_ad = 37, 64, mods[-1], len(mods) - 1, 12
    pitch = max(ranks)
    g = torch.Generator(device="cuda").manual_seed(N + len(ranks))
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, W, A, B = rnd(T, K), rnd(N, K), rnd(n_ad, n_mod * pitch, K), rnd(n_ad, N, pitch)
    of = [ranks[i % len(ranks)] for i in range(n_ad)]
    for i, r in enumerate(of):
        A[i].view(n_mod, pitch, K)[:, r:], B[i, :, r:] = 0, 0
    slots = torch.randint(-1, n_ad, (T,), generator=g, device="cuda").to(torch.int32)
    stack = ops.LoraStack(A, B, torch.tensor(of, dtype=torch.int32, device="cuda"), torch.rand(n_ad, generator=g, device="cuda") + 0.5,
                          pitch, n_mod, tuple(mods), n_out=N)
    u = ops.lora_shrink(x, stack, slots)
    flags = ops.LORA_PER_ROW | (ops.OUT_F32 if f32 else 0)
    want = ops.linear(x, W, stack, slots, u, flags=flags)
    plain = ops.linear(x, W, flags=flags & ops.OUT_F32)
    stack.split_b(of)
    got = ops.linear(x, W, stack, slots, u, flags=flags)
    assert torch.equal(got, want)
    used = [int(s) >= 0 and of[int(s)] > 0 for s in slots]
    assert all(torch.equal(want[t], plain[t]) != used[t] for t in range(T))
