"""Waits on barriers in the kernels that hand work from warp to warp, checked on the CPU: a barrier tells two phases apart by their parity
only, so whoever waits must not be able to fall two phases behind."""
import ctypes
import os
import re
import subprocess

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


@pytest.mark.parametrize("name", FILES)
def test_tensor_memory_is_taken_before_the_next_kernel_is_let_in(name):
    """A kernel that is launched early and takes its tensor memory waits for the one before it to end; one that has yet to take its own would
    wait for the other's. So it is taken ahead of griddep_launch(), behind a barrier of the CTA."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    kernels = [k for k in re.split(r"__global__", text)[1:] if re.search(r"\b(tc_alloc|tmem_alloc)\(", k)]
    assert kernels
    for k in kernels:
        alloc, let_in = re.search(r"\b(tc_alloc|tmem_alloc)\(", k).start(), k.index("griddep_launch()")
        assert alloc < k.index("__syncthreads()", alloc) < let_in, name


@pytest.mark.parametrize("in_smem", [0, 1])
@pytest.mark.parametrize("wanted", range(8))
def test_a_stage_of_expanded_weights_belongs_to_one_group(tmp_path_factory, in_smem, wanted):
    """A group that waits for a use of a stage has to take part in the next one: then no use can pass it by."""
    lib = host_lib(tmp_path_factory)
    stages = lib.b2_host_gemm_stages(in_smem, wanted)
    assert 2 <= stages <= (2 if in_smem else 4)
    owners = {}
    for block in range(64):
        owners.setdefault(lib.b2_host_gemm_stage(block, stages), set()).add(lib.b2_host_gemm_group(block))
    assert len(owners) == stages and all(len(o) == 1 for o in owners.values())
    assert set.union(*owners.values()) == {0, 1}


def host_lib(tmp_path_factory, made=[]):
    if not made:
        out = str(tmp_path_factory.mktemp("ring") / "ring.so")
        subprocess.run(["g++", "-O2", "-fPIC", "-shared", os.path.join(CSRC, "host_selftest.cpp"), "-o", out], check=True)
        made.append(ctypes.CDLL(out))
    return made[0]


CLUSTER_FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu") and "cluster_address(" in open(os.path.join(CSRC, f)).read())


def test_arrivals_at_another_ctas_barrier_order_for_the_cluster():
    """An arrival without a scope orders for its own CTA only: reads of what the other CTA then overwrites could still be under way."""
    text = open(os.path.join(CSRC, "ptx.cuh")).read()
    arrivals = re.findall(r"mbarrier\.arrive[\w.:]*shared::cluster[\w.:]*", text)
    assert arrivals and all(".release.cluster." in a for a in arrivals)
    assert "mbarrier.try_wait.parity.acquire.cluster." in text[text.index("void mbar_wait_cluster"):]


@pytest.mark.parametrize("name", CLUSTER_FILES)
def test_barriers_that_another_cta_reaches_are_waited_for_in_the_cluster(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    barriers = set(re.findall(r"cluster_address\(smem_u32\(&?(\w+)", text)) & set(re.findall(r"mbar_init\(&(\w+)", text))
    assert barriers or "st_async_16(" not in text
    for b in barriers:
        waits = re.findall(r"\b(mbar_wait\w*)\(&%s\b" % b, text)
        assert waits and set(waits) == {"mbar_wait_cluster"}, (b, waits)


def test_score_parts_are_given_back_after_they_have_been_read():
    """latent_tc.cu: each warp's own arrival at x_taken comes after its reads of the other CTA's parts, and the arrival there after all of these."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "latent_tc.cu")).read())
    read, taken = text.rindex("xs["), text.index("mbar_arrive(&x_taken")
    assert read < text.index("__syncwarp()", read) < taken
    wait, give = text.index("mbar_wait_warp(&x_taken"), text.index("mbar_arrive_cluster(")
    assert wait < give and text.count("mbar_arrive_cluster(") == 1 and "(&x_empty" in text[give:]


@pytest.mark.parametrize("name", FILES)
def test_a_wait_that_gave_up_names_itself(name):
    codes = re.findall(r"mbar_wait\w*\([^;]*?\b(0x[0-9a-f]+)u", re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read()))
    assert codes and len(codes) == len(set(codes))
