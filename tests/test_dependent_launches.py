"""CPU test of the rules that dependent launches (launch_pdl, csrc/common.cuh) rest on: a kernel launched that
way waits for its predecessor before anything else, and reads what that one wrote by plain loads, not
through the read-only path, which asks for data that is constant over the kernel's whole life."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "votca_gb300", "csrc")


def _sources():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            src = open(os.path.join(CSRC, f)).read()
            yield f, re.sub(r"//[^\n]*", "", src)


def test_kernels_wait_first():
    """Every kernel that does not begin with the wait is launched in another way."""
    kernels, waits, text = set(), set(), ""
    for f, src in _sources():
        text += src
        for m in re.finditer(r"__global__[^{;]*?\b(\w+)\s*\((?:[^()]|\([^()]*\))*\)\s*\{\s*((?:vgb::)?pdl_wait\(\);)?",
                             src):
            kernels.add(m.group(1))
            if m.group(2):
                waits.add(m.group(1))
    assert len(waits) > 40
    for k in kernels - waits:
        other = re.findall(r"\b%s\s*<<<|cudaLaunchCooperativeKernel\([^;]*\b%s\b" % (k, k), text)
        assert other, k
        assert not re.search(r"launch_(?:pdl|jobs)\([^;]*\b%s\b" % k, text), k


def test_no_read_only_loads():
    for f, src in _sources():
        assert "__ldg(" not in src, f
        assert not re.search(r"const [\w ]+\*\s*__restrict__", src), f
