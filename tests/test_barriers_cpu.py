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


def test_a_failed_share_of_the_shrink_is_told_outside_the_ring():
    """Copies still in flight may land on whatever a CTA that gave up writes into its ring; and whoever gave up, the CTA waits for
    what the producer has requested."""
    src = _source("shrink_tc.cu")
    tail = src[src.index("__syncthreads();\n  if (s_abort && tid == 0)"):]
    assert "part[" in tail and not re.search(r"part\[[^\]]*\]\s*=", tail)  # (read, not written)
    first = tail.index("cluster_sync();")
    assert tail.index("mbar_wait(&full_bar") < first < tail.index("ld_cluster(&s_abort") < tail.index("ld_cluster4(&part")


@pytest.mark.parametrize("name", ["linear_pair_tc.cu", "linear_tc.cuh", "chain_tc.cu"])
def test_output_warps_share_a_verdict(name):
    """A warp that leaves by itself after a wait that ran out keeps the others at their next named barrier for good."""
    waits = re.findall(r"^.*mbar_wait\w*\(&acc_full.*$", _source(name), flags=re.M)
    assert waits and all("bar_all(1, mbar_wait" in w for w in waits), waits


def test_operand_builders_of_a_pair_share_a_verdict():
    src = _source("linear_pair_tc.cu")
    role = src[src.index("const uint32_t cache_lead"):src.index("__syncthreads();\n  if (s_abort)")]
    assert role.count("mbar_wait_pair(") == 1  # in `wait` alone, which returns the role's verdict
    assert "return bar_all(2, w != 0);" in role


def test_a_cta_of_a_pair_leaves_after_its_last_arrivals():
    """Commits of the even CTA arrive at the odd one's barriers too: whoever uses a barrier waits for its last phase before the pair
    parts (accumulators: the output warps wait for every one)."""
    src = _source("linear_pair_tc.cu")
    assert sorted(set(re.findall(r"umma_commit_pair\((?!uint32_t)(?:smem_u32\(&?)?(\w+)", src))) == ["acc_full", "cache_empty", "empty0"]
    producer = src[src.index("const uint32_t full0 = lead_addr"):src.index("else if (warp == 1)")]
    tail = producer[producer.index("mbar_arrive(info_empty)"):]
    assert "i < NS" in tail and "mbar_wait_pair(&empty_bar[s], par" in tail
    builders = src[src.index("const uint32_t cache_lead"):src.index("__syncthreads();\n  if (s_abort)")]
    assert builders.index("++n_batch;") < builders.rindex("wait(cache_empty, (n_batch - 1) & 1);")
    assert builders.rindex("wait(cache_empty") > builders.rindex("mbar_arrive_cluster(cache_lead)")


def test_lanes_read_behind_a_warp_barrier_what_one_lane_waited_for():
    """A shuffle hands over the verdict of the waiting lane and orders no memory for the others."""
    src = _source("linear_rows.cu")
    copies = src[src.index("else if (warp < kRwProducts)") - 6000:src.index("else if (warp < kRwProducts)")]
    wait = copies[copies.index("mbar_wait(list_bar"):]
    assert "__syncwarp();" in wait[:wait.index("n_seg = s_nseg")].split("break;")[-1]
