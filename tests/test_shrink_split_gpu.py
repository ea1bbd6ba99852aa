"""The prompt-size shrink with the k-blocks of a tile shared by the CTAs of a cluster, at the edges of its splits, against fp64 on
the same values.  Products of bf16 are exact in fp32, so the error is that of fp32 sums of ``in`` terms: below in * 2^-24 of the
sum of magnitudes, and of the order of sqrt(in) * 2^-24 of the norm; 1e-5 leaves an order of magnitude."""
import pytest
import torch

from conftest import load

pytestmark = pytest.mark.gpu


# tiles of 128 rows: 2 (whole, ragged); 18 | 19, 37 | 38 and 74 | 75 are where eight, four and two CTAs last share one and
# fewer do (148 SMs); in: fewer k-blocks than two CTAs take, a count that does not divide, a ragged last block
@pytest.mark.parametrize("T", [256, 257, 1152, 1153, 2304, 2305, 2432, 4736, 4737, 9472, 9473, 9500])
@pytest.mark.parametrize("K", [64, 1000, 4104])
@pytest.mark.parametrize("rank,n_mod,adapters,layout", [(16, 3, 2, "runs"), (64, 1, 1, "runs"), (8, 1, 40, "mixed"), (64, 3, 3, "mixed"), (16, 1, 5, "none")])
def test_against_fp64(T, K, rank, n_mod, adapters, layout):
    ops = load("ops")
    g = torch.Generator(device="cuda").manual_seed(T + K)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    A = (torch.randn(adapters, n_mod * rank, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    B = torch.zeros(adapters, 128 * n_mod, rank, device="cuda").bfloat16()
    ranks = torch.full((adapters,), rank, dtype=torch.int32, device="cuda")
    stack = ops.LoraStack(A, B, ranks, torch.ones(adapters, device="cuda"), rank, n_mod, tuple(range(0, 128 * n_mod + 1, 128)))
    if layout == "runs":
        slots = torch.arange(T, device="cuda") * adapters // T
    else:
        slots = torch.randint(-1, adapters if layout == "mixed" else 0, (T,), generator=g, device="cuda")
    slots = slots.to(torch.int32)
    u = torch.full((T, n_mod * rank), float("nan"), device="cuda")
    ops.lora_shrink(x, stack, slots, out=u)
    want = torch.zeros(T, n_mod * rank, dtype=torch.float64, device="cuda")
    for s in range(adapters):
        rows = slots == s
        want[rows] = x[rows].double() @ A[s].double().t()
    assert torch.equal(u[slots < 0], torch.zeros_like(u[slots < 0]))
    assert ((u.double() - want).norm() <= 1e-5 * want.norm()).item()
    again = torch.empty_like(u)
    ops.lora_shrink(x, stack, slots, out=again)
    assert torch.equal(u, again)
