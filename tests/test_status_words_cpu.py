"""The two status words of an engine: one of the projections, one of its own kernels with bounded waits, in one scratch header."""
import os
import re
from types import SimpleNamespace

import pytest
import torch

from conftest import PKG, ROOT, load


def _engine():
    base = load("engine").EngineBase
    eng = base.__new__(base)
    eng.ws_linear, eng.kv, eng.m, eng.max_rows = load("ops").new_workspace(4096, "cpu"), None, SimpleNamespace(device="cpu", V=8), 64
    return eng


@pytest.mark.parametrize("projection,own", [(5, 0), (0, 1), (64, 2)])
def test_a_failure_is_told_once_and_leaves_a_clear_scratch(projection, own):
    eng = _engine()
    word = eng._own_status_word()
    eng.check_status()
    eng.ws_linear[:4].view(torch.int32)[0], word[0] = projection, own
    eng.ws_linear[300] = 9  # an arrival counter that a late contributor has bumped
    with pytest.raises(RuntimeError) as told:
        eng.check_status()
    assert (f"{projection:#x}" in str(told.value)) == bool(projection) and ("attention" in str(told.value)) == bool(own)
    assert not eng.ws_linear.any()
    eng.check_status()


def test_the_word_is_reserved_in_the_header():
    with open(os.path.join(ROOT, "include", "mlora.h")) as f:
        at = int(re.search(r"#define MLORA_WORK_CALLER_OFFSET (\d+)", f.read()).group(1))
    eng = _engine()
    assert eng._own_status_word().data_ptr() == eng.ws_linear.data_ptr() + at
    for name in ("linear_tc.cuh", "chain_tc.cu"):
        with open(os.path.join(ROOT, PKG, "csrc", name)) as f:
            assert re.search(r"static_assert\([^;]*MLORA_WORK_CALLER_OFFSET", f.read()), name


def test_engines_with_a_check_of_their_own_are_asked():
    eng, asked = _engine(), []
    eng._check_prompt_status = lambda: asked.append(1)
    eng.extend([], [])
    assert asked == [1]
