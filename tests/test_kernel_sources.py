"""What kernels do with a wait that ran out or a value that another CTA may overwrite, checked on the sources: no entry point
can bring either about without holding up a GPU."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bamboo_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_a_compute_warp_that_gave_up_adds_nothing_to_dq():
    """`drain` of the backward at head dimension 64: between its wait and its add-reduction it leaves when the wait ran out."""
    text = source("attention_tc.cu")
    body = text[text.index("auto drain = "):]
    body = body[:body.index("tma_reduce_add_2d")]
    assert re.search(r"mbar_wait_warp\(&dq_full.*alive = false", body)
    assert re.search(r"if \([^)]*!alive[^)]*\) return;", body[body.index("alive = false"):])


def test_hand_backs_without_release_wait_for_what_was_read():
    """An arrival without release orders no earlier read.  A scheduling entry goes back under a branch on the value that was read, an
    accumulator behind the fence that orders tensor-memory reads before barrier operations."""
    text = source("gemm_tcgen05.cu")
    calls = [m.start() for m in re.finditer(r"mbar_arrive_cluster_relaxed\(", text)]
    assert len(calls) >= 2
    for at in calls:
        call, before = text[at:at + 80], text[:at]
        if "sched_empty" in call:
            read = before.rindex("tile = __shfl_sync(0xffffffffu, sched_tile[r], 0);")
            assert re.search(r"if \(tile >= -1\) bb::$", before[read:])
        else:
            assert "tmem_empty" in call
            load = before.rindex("tmem_ld_wait();")
            assert "tc_fence_before_sync();" in before[load:] and "__syncwarp();" in before[load:]
