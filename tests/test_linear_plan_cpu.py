"""Host-side planning of the tensor-core projection (``mlora_linear_plan`` of the one-CTA kernel, ``mlora_linear_pair_plan``
of pairs of CTAs): whatever the shape, every tile -- or, at decode sizes, every k-block of every tile -- is dealt to exactly one
CTA or pair.  No GPU: the plan is arithmetic on the shape (the SM
count falls back to a B200's 148 without a device)."""
import ctypes as C

import pytest

from conftest import load

SHAPES = [
    # T, in, out
    (1, 4096, 4096), (8, 4096, 12288), (32, 4096, 22016), (32, 11008, 4096), (32, 4096, 32000), (64, 4096, 22016),
    (128, 5120, 5120), (200, 256, 384), (512, 4096, 12288), (1000, 320, 12288), (1100, 128, 24576), (2048, 256, 12288),
    (4096, 4096, 4096), (4096, 11008, 4096), (5000, 128, 6144), (8192, 4096, 12288), (8192, 4096, 22016),
    (8192, 11008, 4096), (8192, 4096, 4096), (8200, 4096, 12288 + 64), (16384, 4096, 12288), (40000, 4096, 12288),
]


def _plan(T, K, N):
    lib = load("_lib").lib()
    v = (C.c_int32 * 12)()
    assert lib.mlora_linear_plan(T, K, N, v) == 0
    keys = ("bn", "grid", "row_tiles", "tok_tiles", "k_blocks", "per_cta", "gt", "lanes", "steps", "groups", "ch_last")
    return dict(zip(keys, list(v)))


def _walk(p, cta):
    """Tiles CTA ``cta`` visits, in order (the kernel's wave_tile, restated)."""
    out = []
    if p["lanes"] > 0:  # lane form
        j, lane = cta % p["gt"], cta // p["gt"]
        for g in range(p["groups"]):
            for s in range(p["steps"]):
                row, tok = lane + s * p["lanes"], g * p["gt"] + j
                if lane < p["lanes"] and row < p["row_tiles"] and tok < p["tok_tiles"]:
                    out.append(tok * p["row_tiles"] + row)
        return out
    full = p["groups"]  # chunk form: full groups of gt token tiles, then one narrower group
    for g in range(full + 1):
        gt = p["gt"] if g < full else p["tok_tiles"] - full * p["gt"]
        ch = p["steps"] if g < full else p["ch_last"]
        for qi in range(ch):
            q = cta * ch + qi
            if q < p["row_tiles"] * gt:
                j = q // p["row_tiles"]
                out.append((g * p["gt"] + j) * p["row_tiles"] + q % p["row_tiles"])
    return out


@pytest.mark.parametrize("T,K,N", SHAPES)
def test_every_tile_is_dealt_exactly_once(T, K, N):
    p = _plan(T, K, N)
    assert p["bn"] in (16, 32, 64, 128, 256) and 1 <= p["grid"] <= 148
    assert p["row_tiles"] == -(-N // 128) and p["tok_tiles"] == -(-T // p["bn"]) and p["k_blocks"] == -(-K // 64)
    n_tiles = p["row_tiles"] * p["tok_tiles"]
    if p["gt"] == 0:
        # contiguous ranges of k-block steps: CTA c owns [c * per_cta, (c + 1) * per_cta) of tiles * k_blocks
        total = n_tiles * p["k_blocks"]
        assert (p["grid"] - 1) * p["per_cta"] < total <= p["grid"] * p["per_cta"]
        assert p["bn"] <= 128
        return
    seen = []
    for c in range(p["grid"]):
        seen += _walk(p, c)
    assert sorted(seen) == list(range(n_tiles)), "a tile is missing or dealt twice"
    if p["lanes"] > 0:
        assert p["lanes"] == p["grid"] // p["gt"]
        assert p["gt"] == 1 or p["gt"] * p["bn"] * K * 2 <= 48e6  # the group's token rows stay L2-resident
        # at every step the CTAs of one lane -- one per token tile of the group -- read the same row tile (from HBM once)
        for lane in range(p["lanes"]):
            ctas = [c for c in range(p["grid"]) if c // p["gt"] == lane]
            assert len(ctas) == p["gt"]
            for s_ in range(p["steps"]):
                row = lane + s_ * p["lanes"]
                if row < p["row_tiles"]:
                    toks = sorted(t // p["row_tiles"] for c in ctas for t in _walk(p, c) if t % p["row_tiles"] == row)
                    assert toks == list(range(p["tok_tiles"]))  # every token tile, through this lane only
    slots = p["grid"] * (p["groups"] * p["steps"] + p["ch_last"])
    assert n_tiles / slots > 0.6, "more than 40 % of the slots idle"


# (of the one-CTA plan: prompt sizes run on it only where the expand is on CUDA cores, the others on pairs, below)
def test_prompt_passes_take_256_token_tiles_and_decode_sizes_do_not():
    assert _plan(8192, 4096, 12288)["bn"] == 256
    assert _plan(8192, 4096, 4096)["bn"] == 256
    assert _plan(4096, 4096, 4096)["bn"] == 256      # 512 tiles >= 3 rounds of the grid
    assert _plan(1024, 4096, 4096)["bn"] == 128      # too few whole tiles for 256-token ones
    assert _plan(32, 4096, 4096)["bn"] == 32 and _plan(32, 4096, 4096)["gt"] == 0
    assert _plan(16, 4096, 4096)["bn"] == 16
    p = _plan(8192, 4096, 12288)
    assert (p["gt"], p["lanes"], p["steps"], p["groups"]) == (16, 9, 11, 2)


def _pair_plan(T, K, N, mods=None, rank=0, flags=0):
    lib = load("_lib").lib()
    v, offs = (C.c_int32 * 6)(), (C.c_int32 * len(mods))(*mods) if mods else None
    assert lib.mlora_linear_pair_plan(T, K, N, rank, len(mods) - 1 if mods else 1, offs, flags, v) == 0
    return dict(zip(("bn", "pairs", "row_tiles", "tok_tiles", "row_pairs", "gt"), list(v)))


def _pair_rows(p, mods, row_pair):
    """Row tiles of a row pair (the kernel's pair_rows, restated): never of two modules."""
    first, end, m = 0, p["row_tiles"], 0
    if len(mods) > 2:
        while True:
            first, end = mods[m] // 128, mods[m + 1] // 128 if m + 2 < len(mods) else p["row_tiles"]
            n = (end - first + 1) // 2
            if row_pair < n or m + 2 >= len(mods):
                break
            row_pair, m = row_pair - n, m + 1
    return [t for t in (first + 2 * row_pair, first + 2 * row_pair + 1) if t < end], m


@pytest.mark.parametrize("mods", [None, [0, 384, 640], [0, 128, 256, 1280], [0, 128, 384, 512, 896]])
@pytest.mark.parametrize("T,K,N", SHAPES + [(129, 64, 20000), (333, 4096, 12288), (700, 16384, 9000), (9473, 64, 128), (70000, 16384, 264)])
def test_pairs_compute_every_tile_exactly_once(T, K, N, mods):
    mods = [0, N] if mods is None else mods + [N]
    if mods[-2] >= N:
        pytest.skip("fewer outputs than module offsets")
    p = _pair_plan(T, K, N, mods, 16 if len(mods) > 2 else 0)
    if p["bn"] == 0:
        assert T <= 128 or 4 * -(-T // 128) * sum((-(-b // 128) - a // 128 + 1) // 2 for a, b in zip(mods, mods[1:])) < 3 * 74
        return
    assert p["bn"] % 32 == 0 and 64 <= p["bn"] <= 256 and p["tok_tiles"] == -(-T // p["bn"]) and p["row_tiles"] == -(-N // 128)
    n_tiles = p["tok_tiles"] * p["row_pairs"]
    assert p["pairs"] == min(n_tiles, 74) and p["gt"] >= 1
    seen = []
    for w in range(p["pairs"]):
        for idx in range(w, n_tiles, p["pairs"]):  # the kernel's pair_tile, restated
            grp, rem = divmod(idx, p["gt"] * p["row_pairs"])
            width = min(p["gt"], p["tok_tiles"] - grp * p["gt"])
            rows, m = _pair_rows(p, mods, rem // width)
            assert rows and all(mods[m] <= t * 128 < mods[m + 1] for t in rows)
            seen += [(t, grp * p["gt"] + rem % width) for t in rows]
    assert sorted(seen) == [(r, t) for r in range(p["row_tiles"]) for t in range(p["tok_tiles"])]


@pytest.mark.parametrize("T,K,N", SHAPES)
def test_stable_sums_take_pairs_only_where_no_tile_is_split(T, K, N):
    p = _plan(T, K, N)
    whole = p["gt"] > 0 or p["per_cta"] % p["k_blocks"] == 0
    stable = load("ops").STABLE_SUMS
    assert (_pair_plan(T, K, N, flags=stable)["bn"] > 0) == (whole and _pair_plan(T, K, N)["bn"] > 0)


def _rows_plan(T, K, N, flags, mods=None, rank=0):
    lib, ops = load("_lib").lib(), load("ops")
    v, offs = (C.c_int32 * 6)(), (C.c_int32 * len(mods))(*mods) if mods else None
    n_mod = len(mods) - 1 if mods else 2 if flags & ops.SILU_MUL and rank else 1
    assert lib.mlora_linear_rows_plan(T, K, N, rank, n_mod, offs, flags | ops.W_PACKED | (ops.B_PACKED if rank else 0), v) == 0
    return dict(zip(("passes", "grid", "groups", "multiplied", "kb", "slots"), list(v)))


@pytest.mark.parametrize("silu", [False, True])
@pytest.mark.parametrize("rank", [0, 16])
@pytest.mark.parametrize("T", [1, 16, 17, 32])
def test_whole_rows_are_dealt_exactly_once(T, rank, silu):
    ops = load("ops")
    unit = 2 if silu else 1
    for N in (1184, 1200, 2048, 4096, 5120, 7008, 9600, 12288, 15360, 20112, 22016, 28416, 32000, 48000, 100000):
        for K in (8, 72, 1032, 4096, 6144):
            p = _rows_plan(T, K, N, ops.ANY_SUMS | (ops.SILU_MUL if silu else 0), rank=rank)
            units = -(-N // (8 * unit))
            if (N + 7) // 8 < 148 or T > 16 and units > 2 * (12 // unit) * 148:
                assert p["passes"] == 0
                continue
            if p["passes"] == 0 and K > 2048 and N < 7104:  # (by measurement: see the test below)
                continue
            assert p["passes"] >= 1 and p["grid"] == min(148, units) and p["groups"] <= p["multiplied"] <= (12 if T > 16 else 20)
            seen = []
            for c in range(p["grid"]):  # the kernel's ranges, restated
                u0, u1 = units * c // p["grid"], units * (c + 1) // p["grid"]
                at = [(u0 + (u1 - u0) * i // p["passes"]) * unit for i in range(p["passes"] + 1)]
                assert all(0 < b - a <= p["groups"] for a, b in zip(at, at[1:])) and at[0] == u0 * unit and at[-1] == u1 * unit
                # a pass's groups are copied in three pieces at most, each inside a tile of 16
                assert all((b - 1) // 16 - a // 16 < 3 for a, b in zip(at, at[1:]))
                seen += range(at[0], at[-1])
            assert seen == list(range(units * unit))
            # what the ring, the sums and the adapters' side take fits the SM
            rows = 32 if T > 16 else 16
            slot = p["kb"] * (p["groups"] * 1024 + rows * 128)
            assert 3 <= p["slots"] <= 16 and p["kb"] in (2, 4, 8)
            assert p["slots"] * slot + 1024 * rows + 1024 + (rows * 400 if rank else 0) <= 227 * 1024 - 64


def test_which_calls_get_whole_rows():
    ops = load("ops")
    some = ops.ANY_SUMS
    taken = [(1, 6144, 2048), (1, 16384, 4096), (2, 4096, 2048), (4, 16384, 8192), (4, 3072, 2048), (7, 4096, 4096), (8, 6144, 4096), (16, 2048, 5120), (16, 8192, 6144),
             (17, 6144, 2048), (32, 4096, 4096), (32, 5120, 5120), (17, 4096, 28416), (32, 6144, 12288), (16, 4096, 200000)]
    # (each of these was slower there than on stream-K, or was not measured)
    left = [(1, 8192, 2048), (2, 8192, 2048), (4, 8192, 2048), (16, 8192, 2048), (4, 11008, 4096), (4, 4096, 5120), (5, 8192, 4096), (16, 5120, 5120), (16, 11008, 4096),
            (5, 8200, 12288), (32, 6144, 3072), (32, 6144, 4096), (17, 6152, 12288), (32, 8192, 2048), (33, 4096, 4096), (17, 4096, 28424), (8, 4096, 1176)]
    assert all(_rows_plan(*c, some)["passes"] for c in taken) and not any(_rows_plan(*c, some)["passes"] for c in left)
    for flags in (0, ops.STABLE_SUMS, ops.STABLE_SUMS | some):
        assert not any(_rows_plan(*c, flags)["passes"] for c in taken)
    assert _rows_plan(16, 8192, 4096, some, rank=16)["passes"] and not _rows_plan(1, 6144, 4096, some, rank=16)["passes"]
    assert _rows_plan(32, 6144, 8192, some, rank=16)["passes"] and not _rows_plan(32, 6144, 6144, some, rank=16)["passes"]
    # adapters: rank pitches of the packed layout, rows of shrink outputs that fit, modules of whole row tiles
    assert all(_rows_plan(8, 4096, 4096, some, rank=r)["passes"] for r in (16, 32, 64, 128))
    assert not any(_rows_plan(8, 4096, 4096, some, rank=r)["passes"] for r in (8, 24, 48))
    assert _rows_plan(8, 4096, 12288, some, [0, 4096, 8192, 12288], 64)["passes"]
    assert not _rows_plan(8, 4096, 12288, some, [0, 4096, 8192, 12288], 128)["passes"]
    assert not _rows_plan(8, 4096, 12288, some, [0, 4096, 8200, 12288], 64)["passes"]
    assert _rows_plan(8, 4096, 22016, some | ops.SILU_MUL, rank=64)["passes"] and not _rows_plan(8, 4096, 22016, some | ops.SILU_MUL, rank=128)["passes"]
