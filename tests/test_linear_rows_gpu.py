"""The decode-size projection that gives every CTA whole output rows (``MLORA_ANY_SUMS``): against float64 and the stream-K kernel."""
import ctypes as C

import pytest
import torch

from conftest import load

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    return load("ops")


def _plan(ops, T, K, N, flags, rank=0, n_mod=1, offs=None):
    v, o = (C.c_int32 * 6)(), None if offs is None else (C.c_int32 * len(offs))(*offs)
    assert load("_lib").lib().mlora_linear_rows_plan(T, K, N, rank, n_mod, o, flags | ops.ANY_SUMS | ops.W_PACKED | (ops.B_PACKED if rank else 0), v) == 0
    return dict(zip(("passes", "grid", "groups", "multiplied", "kb", "slots"), list(v)))


def _run(ops, cuda, T, K, N, flags=0, rank=0, n_mod=1, n_ad=5, seed=0, ids=None):
    """(output of this kernel, of stream-K, float64 reference, bound of one output's error)."""
    offs = (0, N) if flags & ops.SILU_MUL or n_mod == 1 else tuple(N // 128 * i // n_mod * 128 for i in range(n_mod)) + (N,)
    assert _plan(ops, T, K, N, flags, rank, n_mod, offs)["passes"], "another kernel than the one under test"
    g = torch.Generator().manual_seed(seed + T * 131 + K + N)
    x = torch.randn(T, K, generator=g).bfloat16()
    W = (torch.randn(N, K, generator=g) * K ** -0.5).bfloat16()
    want = x.double() @ W.double().T
    st = slots = u = None
    if rank:
        silu = flags & ops.SILU_MUL
        pitch = 2 * rank if silu else rank  # (interleaved gate / up rows: one operand over both modules' ranks)
        B = (torch.randn(n_ad, N, pitch, generator=g) * 0.1).bfloat16()
        u = torch.randn(T, rank * n_mod, generator=g)
        slots = torch.randint(-1, n_ad + 1, (T,), generator=g).int() if ids is None else torch.tensor(ids).int()  # n_ad: no such adapter
        scales = torch.linspace(0.5, 2.0, n_ad)
        for t in range(T):
            s = int(slots[t])
            if not 0 <= s < n_ad:
                continue
            su = (scales[s] * u[t]).bfloat16().double()  # (the operand both kernels multiply)
            for m in range(1 if silu else n_mod):
                lo, hi = (0, N) if silu else (offs[m], offs[m + 1])
                want[t, lo:hi] += B[s, lo:hi].double() @ (su if silu else su[m * rank:(m + 1) * rank])
        st = ops.LoraStack(torch.zeros(n_ad, rank * n_mod, K, dtype=torch.bfloat16, device=cuda), B.to(cuda),
                           torch.full((n_ad,), rank, dtype=torch.int32, device=cuda), scales.to(cuda), rank, n_mod, offs).pack_b()
        u, slots = u.to(cuda), slots.to(cuda)
    if flags & ops.SILU_MUL:
        v = want.view(T, -1, 2, 8)
        want = (v[:, :, 0] * torch.sigmoid(v[:, :, 0]) * v[:, :, 1]).reshape(T, -1)
    elif flags & ops.ACT_RELU2:
        want = want.clamp(min=0) ** 2
    elif flags & ops.ACT_GELU:
        want = 0.5 * want * (1 + torch.erf(want / 2 ** 0.5))
    work = ops.new_workspace(load("_lib").lib().mlora_linear_workspace(T, K, N), cuda)
    got, old = (ops.linear(x.to(cuda), ops.PackedWeight(W.to(cuda)), st, slots, u=u, flags=flags | f, work=work) for f in (ops.ANY_SUMS, 0))
    again = ops.linear(x.to(cuda), ops.PackedWeight(W.to(cuda)), st, slots, u=u, flags=flags | ops.ANY_SUMS, work=work)
    assert ops.status_word(work) == 0
    assert torch.equal(got, again)  # a fixed order of sums
    return got.double().cpu(), old.double().cpu(), want


def _check(got, old, want, f32):
    # fp32 sums of some thousand products: below 2^-16 of the result's size; bf16 outputs: half a unit in the last of 8 bits, 2^-8 of a
    # value.  No further off than stream-K, but for sums so short that both are at fp32's own rounding (2^-20 of the result)
    size = want.abs().max()
    err, err_old = (got - want).abs(), (old - want).abs()
    assert float((err - (0 if f32 else 2 ** -8) * want.abs()).max()) <= 2 ** -16 * float(size)
    assert float(err.norm()) <= (1.0 if f32 else 1.01) * float(err_old.norm()) + 2 ** -20 * float(want.norm())


@pytest.mark.parametrize("K,N,left", [(8, 1184, ()), (72, 1200, ()), (512, 2048, ()), (1032, 4096, ()), (4096, 7000, ()), (4096, 9600, ()), (4096, 12288, ()),
                                      (3072, 20104, ()), (4096, 28416, ()), (4096, 28424, (17, 32)), (6144, 2048, (4, 15, 16)), (16384, 4096, (4, 15, 16, 17, 32))])
@pytest.mark.parametrize("T", [1, 4, 15, 16, 17, 32])
def test_plain(ops, cuda, T, K, N, left):
    """One row group per CTA and several, one and two passes, odd numbers of k-blocks, ragged last rows, slots of 2 to 8 k-blocks
    (``left``: rows with which the shape stays on another kernel)."""
    if T in left:
        assert not _plan(ops, T, K, N, ops.OUT_F32)["passes"]
        return
    _check(*_run(ops, cuda, T, K, N, ops.OUT_F32), True)


@pytest.mark.parametrize("T", [1, 16])
@pytest.mark.parametrize("N", [48000, 72000])
def test_three_passes_and_more(ops, cuda, T, N):
    """Few enough columns that one CTA's rows are read in several passes: plain, SiLU*up, adapters with module boundaries inside a pass."""
    assert _plan(ops, T, 72, N, 0)["passes"] == (3 if N == 48000 else 4)
    _check(*_run(ops, cuda, T, 72, N, ops.OUT_F32), True)
    _check(*_run(ops, cuda, T, 72, N, ops.SILU_MUL), False)
    _check(*_run(ops, cuda, T, 136, N, ops.OUT_F32, 16, 8), True)
    _check(*_run(ops, cuda, T, 72, N, ops.SILU_MUL, 32, 2), False)


@pytest.mark.parametrize("T", [17, 32])
def test_two_passes_beyond_16_rows(ops, cuda, T):
    assert _plan(ops, T, 200, 28416, 0)["passes"] == 2 and _plan(ops, T, 200, 28416, ops.SILU_MUL)["passes"] == 2
    _check(*_run(ops, cuda, T, 200, 28416, ops.SILU_MUL), False)
    _check(*_run(ops, cuda, T, 200, 28416, ops.OUT_F32, 32, 3), True)
    _check(*_run(ops, cuda, T, 200, 28416, ops.SILU_MUL, 16, 2), False)


@pytest.mark.parametrize("T", [3, 32])
@pytest.mark.parametrize("flag", ["SILU_MUL", "ACT_RELU2", "ACT_GELU", None])
@pytest.mark.parametrize("K,N", [(256, 1200), (640, 2064), (2048, 22016)])
def test_activations_and_bf16(ops, cuda, T, flag, K, N):
    _check(*_run(ops, cuda, T, K, N, getattr(ops, flag) if flag else 0), False)


@pytest.mark.parametrize("T,rank,n_mod,K,N", [(1, 16, 1, 4096, 4096), (16, 16, 3, 1024, 12288), (17, 32, 3, 512, 1536), (32, 64, 3, 4096, 12288),
                                              (32, 128, 1, 256, 1208), (9, 64, 1, 8192, 4096), (2, 64, 1, 11008, 8192), (32, 16, 8, 128, 2048)])
def test_adapters(ops, cuda, T, rank, n_mod, K, N):
    """Module boundaries inside a CTA's rows, adapters over several slots, rows without adapter or with one that does not exist."""
    _check(*_run(ops, cuda, T, K, N, ops.OUT_F32, rank, n_mod), True)


def test_adapters_all_distinct_none_and_gate_up(ops, cuda):
    _check(*_run(ops, cuda, 32, 512, 4096, ops.OUT_F32, 16, 1, 32, ids=list(range(32))), True)
    _check(*_run(ops, cuda, 32, 512, 4096, ops.OUT_F32, 16, 1, 4, ids=[-1] * 32), True)
    for T in (5, 32):
        _check(*_run(ops, cuda, T, 512, 22016, ops.SILU_MUL, 64, 2), False)


def test_rows_and_outputs_of_other_pitches(ops, cuda):
    """x as a slice of wider rows; y likewise, also where four outputs are no aligned store."""
    g = torch.Generator().manual_seed(1)
    X, W = torch.randn(7, 520, generator=g).bfloat16().to(cuda), (torch.randn(1192, 256, generator=g) / 16).bfloat16().to(cuda)
    x, Y = X[:, 8:264], torch.full((7, 1229), 9.0, dtype=torch.bfloat16, device=cuda)
    work = ops.new_workspace(load("_lib").lib().mlora_linear_workspace(7, 256, 1192), cuda)
    ops.linear(x, ops.PackedWeight(W), flags=ops.ANY_SUMS, out=Y[:, 3:1195], work=work)
    want = x.double() @ W.double().T
    assert float(((Y[:, 3:1195].double() - want).abs() - 2 ** -8 * want.abs()).max()) < 1e-4
    assert bool((Y[:, :3] == 9).all()) and bool((Y[:, 1195:] == 9).all())


def test_calls_that_keep_the_plans_sums(ops, cuda):
    """Without the flag, or with STABLE_SUMS, the bits are those of the stream-K plan."""
    got = {}
    g = torch.Generator().manual_seed(2)
    x, W = torch.randn(4, 4096, generator=g).bfloat16().to(cuda), ops.PackedWeight(torch.randn(4096, 4096, generator=g).bfloat16().to(cuda))
    for f in (0, ops.STABLE_SUMS, ops.STABLE_SUMS | ops.ANY_SUMS):
        got[f] = ops.linear(x, W, flags=f | ops.OUT_F32)
    assert torch.equal(got[0], got[ops.STABLE_SUMS]) and torch.equal(got[0], got[ops.STABLE_SUMS | ops.ANY_SUMS])


@pytest.mark.parametrize("T,rank,n_mod", [(16, 64, 3), (32, 16, 1), (20, 64, 1)])
@pytest.mark.parametrize("silu", [False, True])
def test_many_distinct_adapters_keep_their_fp32_operands(ops, cuda, T, rank, n_mod, silu):
    """``LORA_PER_ROW``: scale * u is not rounded to bf16, and an adapter that holds infinities reaches the rows that use it alone."""
    g = torch.Generator().manual_seed(T + rank)
    K, N = 1024, 3072
    n_mod, pitch = (2, 2 * rank) if silu else (n_mod, rank)
    x, W = torch.randn(T, K, generator=g).bfloat16(), (torch.randn(N, K, generator=g) * K ** -0.5).bfloat16()
    B, u = (torch.randn(T, N, pitch, generator=g) * 0.1).bfloat16(), torch.randn(T, rank * n_mod, generator=g)
    offs = (0, N) if silu or n_mod == 1 else tuple(N // n_mod * i for i in range(n_mod + 1))
    want = x.double() @ W.double().T
    for m in range(1 if silu else n_mod):
        lo, hi = (0, N) if silu else offs[m:m + 2]
        want[:, lo:hi] += torch.einsum("tor,tr->to", B[:, lo:hi].double(), 0.5 * (u if silu else u[:, m * rank:(m + 1) * rank]).double())
    if silu:
        v = want.view(T, -1, 2, 8)
        want = (v[:, :, 0] * torch.sigmoid(v[:, :, 0]) * v[:, :, 1]).reshape(T, -1)
    got = []
    for bad in (False, True):
        b = B.clone()
        if bad:
            b[3, ::7] = float("inf")
        st = ops.LoraStack(torch.zeros(T, rank * n_mod, K, dtype=torch.bfloat16, device=cuda), b.to(cuda), torch.full((T,), rank, dtype=torch.int32, device=cuda),
                           torch.full((T,), 0.5, device=cuda), rank, n_mod, offs).pack_b()
        flags = ops.ANY_SUMS | ops.LORA_PER_ROW | (ops.SILU_MUL if silu else ops.OUT_F32)
        work = ops.new_workspace(load("_lib").lib().mlora_linear_workspace_flags(T, K, N, flags), cuda)
        got.append(ops.linear(x.to(cuda), ops.PackedWeight(W.to(cuda)), st, torch.arange(T, dtype=torch.int32, device=cuda), u=u.to(cuda), flags=flags, work=work).cpu())
    others = [t for t in range(T) if t != 3]
    assert torch.equal(got[0][others], got[1][others]) and not torch.isfinite(got[1][3]).all()
    # fp32 sums as in _check; SiLU*up leaves as bf16: half a unit, 2^-8 of a value.  A bf16 operand would be 2^-9 of the adapters' share off
    err = (got[0].double() - want).abs() - (2 ** -8 * want.abs() if silu else 0)
    assert float(err.max()) <= 2 ** -16 * float(want.abs().max())
