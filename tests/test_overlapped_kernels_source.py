"""Kernels that may be resident while their predecessor still writes (they call pdl_sync) must not read that
predecessor's results through the read-only data path, whose contract is data that does not change during the kernel.
Checked on the sources: a violation shows as a wrong value only when timing and code generation happen to allow it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bamboo_b200", "csrc")
# parameters: written by the optimizer, whose kernel does not let a successor in early
PARAMETERS = {"gamma", "beta", "bias"}
# the GEMM's bias, under the name it has inside add_bias
PARAMETER_LOADS = {("gemm_tcgen05.cu", "reinterpret_cast<const uint4*>(b + i)")}


def functions(text):
    """Device code of a source file, one piece per __global__ / __device__ function."""
    text = re.sub(r"//[^\n]*", "", text)
    starts = [m.start() for m in re.finditer(r"^\s*(?:template[^\n]*\n)?\s*(?:__global__|(?:static )?__device__)[^\n;]*", text, re.M)]
    return [text[a:b] for a, b in zip(starts, starts[1:] + [len(text)])]


def read_only_loads(name, body):
    bad = [m.group(0) for m in re.finditer(r"const\s+\w[\w ]*\*\s*__restrict__\s+(\w+)", body) if m.group(1) not in PARAMETERS]
    # (a load through a restricted pointer may be moved in front of the wait: the wait is not based on that pointer)
    for m in re.finditer(r"(?<!const )\b\w+\s*\*\s*__restrict__\s+(\w+)", body.split("{")[0]):
        if re.search(rf"\b{m.group(1)}\[[^\]]*\]\s*\+=", body) or (m.group(1).startswith("out") and re.search(r"\bout\[[^\]]*\]\s*\+=", body)):
            bad.append(m.group(0))
    for m in re.finditer(r"__ldg\(", body):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(body[i], 0)
            i += 1
        arg = body[m.end():i - 1]
        if (name, arg) not in PARAMETER_LOADS and not any(re.search(rf"\b{p}\b", arg) for p in PARAMETERS):
            bad.append(f"__ldg({arg})")
    return bad + re.findall(r"ld\.global\.nc", body)


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_overlapped_kernels_read_results_coherently(path):
    with open(path) as f:
        text = f.read()
    if "pdl_sync" not in text:
        return
    name, bad = os.path.basename(path), []
    for body in functions(text):
        # a kernel that waits for its predecessor, or a helper that one may call
        if "pdl_sync" in body or not body.lstrip().startswith(("template", "__global__")) or "__device__" in body.split("{")[0]:
            bad += read_only_loads(name, body)
    assert not bad, f"{name}: {bad}"
