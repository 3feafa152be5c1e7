"""Waits on barriers in the kernels that hand work from warp to warp, checked on the CPU: a barrier tells two phases apart by their parity
only, so whoever waits must not be able to fall two phases behind."""
import os
import re

import pytest

from conftest import PKG

CSRC = os.path.join(PKG, "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu") and "elect_one()" in open(os.path.join(CSRC, f)).read())


def issuing_branches(text):
    """The warp roles in which all lanes run a loop and one of them issues."""
    roles = re.split(r"(?:\} else )?if \(warp [<=]", re.sub(r"//[^\n]*", "", text))
    return [r for r in roles[1:] if "elect_one()" in r]


def test_there_are_issuing_warps():
    assert {"dense_tc.cu", "gemm.cu", "latent_tc.cu", "softmax_tc.cu"} <= set(FILES)


@pytest.mark.parametrize("name", FILES)
def test_issuing_warps_leave_their_waits_together(name):
    """Between a wait and what is issued after it the lanes converge: else the one that issues can move the barrier two phases past a lane that
    has not looked yet, which then waits for the parity of the phase before its own."""
    branches = issuing_branches(open(os.path.join(CSRC, name)).read())
    assert branches
    for b in branches:
        for m in re.finditer(r"\bmbar_wait\(", b):
            rest = b[m.end():]
            sync, issue = rest.find("__syncwarp()"), re.search(r"elect_one\(\)|\(one\)|\(!one\)", rest)
            assert sync >= 0 and (issue is None or sync < issue.start()), (name, rest[:120])
