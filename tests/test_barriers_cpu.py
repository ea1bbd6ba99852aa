"""What no run may show, read from the source: barriers that a warp reaches diverged, or that a part of their warps never reaches."""
import os
import re

import pytest

from conftest import PKG, ROOT


def _source(name):
    with open(os.path.join(ROOT, PKG, "csrc", name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_cluster_barriers_are_reached_by_whole_warps():
    """``.aligned`` wants every thread of the warp to execute it together, after whatever loop came before."""
    src = _source("tc_ptx.cuh")
    body = src[src.index("void cluster_sync() {"):]
    body = body[:body.index("\n}")]
    assert re.search(r"__syncwarp\(\);\s*asm volatile\(\"barrier\.cluster\.arrive", body)
    for name in os.listdir(os.path.join(ROOT, PKG, "csrc")):
        if name != "tc_ptx.cuh":
            assert "barrier.cluster" not in _source(name)
