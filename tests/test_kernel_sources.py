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
