"""Engines on several GPUs share one process, and a kernel's limit of dynamic shared memory belongs to the kernel on one device: it has to be
raised on each. Checked on the CPU: the flag that remembers it (csrc/per_device.h) and, in the sources, that nothing raises it once per process."""
import ctypes
import os
import re
import subprocess

import pytest

from conftest import PKG

CSRC = os.path.join(PKG, "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h")) and "cudaFuncSetAttribute" in open(os.path.join(CSRC, f)).read())


@pytest.fixture(scope="module")
def host_lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("per_device") / "host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", os.path.join(CSRC, "host_selftest.cpp"), "-o", out], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("calls,times", [([0, 0, 1, 0, 1, 7], {0: 1, 1: 1, 7: 1}), ([-1, 0, 0, -2, -2, 1], {0: 2, 1: 3}), ([63, 64, 64, 63, 70], {63: 1, 64: 2, 70: 1})])
def test_each_device_once_and_again_after_a_refusal(host_lib, calls, times):
    """A call -1 - d is one that device d refuses. (Devices past the 64 that are remembered are set up by every call.)"""
    got, ready = (ctypes.c_int * 128)(), (ctypes.c_int * len(calls))()
    host_lib.b2_host_per_device((ctypes.c_int * len(calls))(*calls), len(calls), got, ready)
    assert {d: n for d, n in enumerate(got) if n} == times
    done = set()
    for call, ok in zip(calls, ready):
        if call >= 0:
            done.add(call)
        assert bool(ok) == ((call if call >= 0 else -1 - call) in done)


@pytest.mark.parametrize("name", FILES)
def test_limits_are_raised_for_every_device(name):
    """Either through allow_smem (kernels.h), which remembers the device, or in one of the functions that every engine calls for its own."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    per_engine = r"(?:cudaError_t|static cudaError_t) (?:\w+_init|set_smem_attrs)\([^)]*\) \{.*?\n\}"
    rest = re.sub(per_engine, "", text, flags=re.S)
    for m in re.finditer(r"[^\n]*cudaFuncSetAttribute", rest):
        assert name == "kernels.h" and "limits.ready(device" in m.group(0), (name, m.group(0))


def test_every_engine_raises_its_devices_limits():
    text = open(os.path.join(CSRC, "engine.cu")).read()
    create, finalize = text.index("static int engine_create_impl(b2_engine* e, const b2_config* c) {"), text.index('extern "C" int b2_engine_finalize(')
    for name, at in (("mv_init", create), ("attn_init", create), ("attn_mma_init", create), ("gemm_init", finalize)):
        assert f"CK({name}())" in text[at:text.index("\n}\n", at)], name
