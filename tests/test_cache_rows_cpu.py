"""Rows of a forward as the host builds them: row by row against a plain list, over everything a caller may pass."""
import random
from types import SimpleNamespace

import numpy as np
import pytest

from conftest import load


def _cache():
    kv = load("kv_cache").PagedCache(6, 960, 64, 16, "cpu", max_seq_len=320)
    kv._push = lambda dst, src: dst.copy_(load("kv_cache").torch.from_numpy(np.ascontiguousarray(src)))  # (no pinned memory here)
    return kv


@pytest.mark.parametrize("seed", range(8))
def test_rows_of_random_forwards(seed):
    rng, kv = random.Random(seed), _cache()
    for sid in rng.sample(range(20), 6):
        kv.add_sequence(sid)
    have = {sid: 0 for sid in kv._slot_of}
    for _ in range(12):
        sids = rng.sample(sorted(have), rng.randint(1, 6))
        lens = [rng.choice([0, 1, 2, 15, 16, 17, rng.randint(0, 40), -rng.randint(0, have[s])]) for s in sids]
        lens = [min(n, 300 - have[s]) for s, n in zip(sids, lens)]
        row_slot, row_pos = kv.begin_rows(sids, lens)
        assert row_slot.dtype == row_pos.dtype == np.int32
        assert row_slot.tolist() == [kv.slot(s) for s, n in zip(sids, lens) for _ in range(n)]
        assert row_pos.tolist() == [have[s] + i for s, n in zip(sids, lens) for i in range(n)]
        kv.end_forward()
        for s, n in zip(sids, lens):
            have[s] += n
        assert {s: kv.length(s) for s in have} == have
        assert all(kv.tokens_reserved(s) >= n for s, n in have.items())
        assert kv.block_table.tolist() == kv._bt_host.tolist()


def test_one_list_longer_than_the_other_and_none_at_all():
    kv = _cache()
    for sid in range(3):
        kv.add_sequence(sid)
    for sids, lens, want in (([0, 1, 2], [4], [0] * 4), ([2], [2, 9, 9], [2] * 2), ([], [], [])):
        row_slot, row_pos = kv.begin_rows(sids, lens)
        assert row_slot.tolist() == [kv.slot(s) for s in want]
        assert row_pos.tolist() == list(range(len(want)))


def test_unknown_sequences_and_too_many_pages_are_refused():
    kv = _cache()
    kv.add_sequence(0)
    with pytest.raises(KeyError):
        kv.begin_rows([0, 9], [1, 1])
    with pytest.raises(RuntimeError):
        kv.begin_rows([0], [400])


@pytest.mark.parametrize("slot", [1 << 32, 1 << 40, -(1 << 31) - 1])
def test_adapter_slots_beyond_32_bits_are_refused(slot):
    """... before anything is reserved, and not taken for what is left of them in 32 bits."""
    base = load("engine").EngineBase
    eng = base.__new__(base)
    eng.kv, eng.m, eng.max_rows = _cache(), SimpleNamespace(device="cpu", V=8), 64
    eng.tokens = eng.slots = eng.row_slot = eng.row_pos = eng.last_rows = None
    eng.kv.add_sequence(4)
    eng._stage_all = lambda *parts: pytest.fail("taken")
    with pytest.raises(OverflowError):
        eng.extend([4], [[1, 2, 3]], [slot])
    assert eng.kv.tokens_reserved(4) == 0


def test_sequences_of_a_cache_without_a_gpu():
    """Adding a sequence clears its length in place: no pinned memory, which a machine without a GPU does not have."""
    kv = load("kv_cache").PagedCache(3, 96, 64, 16, "cpu")
    kv.seq_lens.fill_(7)
    assert [kv.seq_lens[kv.add_sequence(s)].item() for s in (5, 9)] == [0, 0]
    assert kv.seq_lens.sum().item() == 7
    kv.remove_sequence(5)
    assert kv.slot(9) == 1
