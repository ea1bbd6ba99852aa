"""Host tables that travel in launch parameters: against plain lists, at the edges of a launch."""
import random

import numpy as np
import pytest
import torch

from conftest import load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 255, 256, 257, 895, 896, 897, 1792, 2000])
@pytest.mark.parametrize("repeat", [1, 3, 512])
def test_values(cuda, n, repeat):
    values = np.random.default_rng(n + repeat).integers(-2 ** 31, 2 ** 31, n).astype(np.int32)
    dst = torch.full((n * repeat + 2,), 7, dtype=torch.int32, device=cuda)
    load("ops").put_i32(dst[1:], values, repeat)
    values_before = values.copy()
    values[:] = 0  # the launch holds its own copy
    assert dst.tolist() == [7] + np.repeat(values_before, repeat).tolist() + [7]


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 300])
def test_rows(cuda, n):
    rng = random.Random(n)
    seqs = [(rng.randrange(99), rng.randrange(-1, 9), rng.choice([0, 1, 2, 31, 300]), rng.randrange(4000)) for _ in range(n)]
    want = [[a for s, a, k, p in seqs for _ in range(k)], [s for s, a, k, p in seqs for _ in range(k)], [p + i for s, a, k, p in seqs for i in range(k)]]
    T = len(want[0])
    got = [torch.full((T + 1,), -9, dtype=torch.int32, device=cuda) for _ in range(3)]
    load("ops").put_rows(np.array(seqs, dtype=np.int32), *got)
    assert [t.tolist() for t in got] == [w + [-9] for w in want]


def test_refusals(cuda):
    lib, d = load("_lib").lib(), torch.zeros(4, dtype=torch.int32, device=cuda)
    bad = np.array([[0, 0, -1, 0]], dtype=np.int32)
    assert lib.mlora_put_rows(bad.ctypes.data, 1, d.data_ptr(), d.data_ptr(), d.data_ptr(), None) < 0
    assert lib.mlora_put_i32(d.data_ptr(), bad.ctypes.data, 4, 0, None) < 0
    assert lib.mlora_put_i32(d.data_ptr(), bad.ctypes.data, 4, 2 ** 30, None) < 0
