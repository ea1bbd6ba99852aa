"""Tables on their way to the device: what does not fit its destination is refused before anything is launched."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from conftest import load


def _i32(n):
    return torch.zeros(n, dtype=torch.int32)


@pytest.mark.parametrize("n,repeat,room", [(1, 1, 0), (3, 1, 2), (2, 5, 9), (1792, 1, 1791)])
def test_values_beyond_the_table(n, repeat, room):
    with pytest.raises(RuntimeError, match=f"{n * repeat} values into a table of {room}"):
        load("ops").put_i32(_i32(room), np.arange(n), repeat)


def test_rows_beyond_one_of_the_tables():
    seqs = np.array([[0, -1, 4, 0], [1, -1, 3, 9]])
    for short in range(3):
        tables = [_i32(6 if i == short else 7) for i in range(3)]
        with pytest.raises(RuntimeError, match="7 values into a table of 6"):
            load("ops").put_rows(seqs, *tables)
    with pytest.raises(ValueError, match="four numbers"):
        load("ops").put_rows(seqs[:, :3], *[_i32(9)] * 3)


def test_tables_of_another_type_or_layout():
    ops = load("ops")
    for bad in (torch.zeros(8), torch.zeros(8, dtype=torch.int64), _i32(16)[::2]):
        with pytest.raises(ValueError, match="contiguous int32"):
            ops.put_i32(bad, [1, 2])
        with pytest.raises(ValueError, match="contiguous int32"):
            ops.put_rows([[0, 0, 2, 0]], _i32(8), bad, _i32(8))
    with pytest.raises(ValueError, match="CUDA"):
        ops.put_i32(_i32(2), [1, 2])


def test_nothing_to_put():
    load("ops").put_i32(_i32(4)[2:2], [])
    load("ops").put_rows(np.zeros((0, 4)), _i32(0), _i32(0), _i32(0))
    load("ops").put_rows([[0, 0, 0, 0]], _i32(0), _i32(0), _i32(0))


def test_more_segments_than_the_engine_has_room_for():
    """One sequence listed more often than the batch has places, as ``extend`` takes it."""
    engine = object.__new__(load("relidra").RelidraEngine)
    engine.segs, engine.tiles = _i32(8).view(2, 4), _i32(16).view(4, 4)
    engine.kv = SimpleNamespace(slot=lambda sid: 0)
    with pytest.raises(RuntimeError, match="12 values into a table of 8"):
        engine._begin_prompt_pass([(0, 0, 1, 0), (0, 1, 1, 1), (0, 2, 1, 2)])
