"""Rows and page table of a forward: what the host knows is what the device has, however the table's rows travel."""
import pytest
import torch

from conftest import load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_copy", [0, 16384])  # a copy per sequence / one over all changed rows
def test_rows_positions_and_pages(per_copy):
    kvc = load("kv_cache")
    kv = kvc.PagedCache(8, 640, 64, 16, "cuda", max_seq_len=200)
    kv._ROWS_PER_COPY = per_copy
    have = {}
    for sid in (5, 1, 7, 3):
        kv.add_sequence(sid)
        have[sid] = 0
    for sids, lens in (([5, 7], [33, 1]), ([1, 5, 3], [16, 15, 100]), ([7], [1]), ([3, 7, 1], [28, 62, 1])):
        row_slot, row_pos = kv.begin_forward(sids, lens)
        assert row_slot.tolist() == [kv.slot(s) for s, n in zip(sids, lens) for _ in range(n)]
        assert row_pos.tolist() == [have[s] + i for s, n in zip(sids, lens) for i in range(n)]
        kv.end_forward()
        for s, n in zip(sids, lens):
            have[s] += n
    used = []
    for sid, n in have.items():
        pages = kv.block_table[kv.slot(sid), :-(-n // 16)].tolist()
        assert kv.length(sid) == n == kv.seq_lens[kv.slot(sid)].item() and kv.tokens_reserved(sid) == len(pages) * 16
        used += pages
    assert len(set(used)) == len(used)
    # a forward that finds no page for its last sequence: those before keep theirs, on both sides
    with pytest.raises(RuntimeError):
        kv.begin_forward([1, 5], [40, 400])
    assert kv.tokens_reserved(1) == 64
    assert kv.block_table[kv.slot(1), :4].tolist() == kv._bt_host[kv.slot(1), :4].tolist()
    for sid in (5, 1, 7, 3):
        kv.remove_sequence(sid)
    assert sorted(kv._free) == list(range(kv.n_pages))
    slot = kv.add_sequence(9)
    assert kv.seq_lens[slot].item() == 0
