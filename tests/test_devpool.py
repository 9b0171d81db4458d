"""The device memory pool behind the solvers' buffers, on the host: devpool.cu
compiled with a fake CUDA runtime (tests/devpool_check.cpp).  Reuse across
threads and devices, the bound, the way back of the memory, the waits before a
block is handed on, and failures of host memory."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "fastmbcui_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers not available")
    out = str(tmp_path_factory.mktemp("devpool") / "check")
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(CUDA, "include"), "-x", "c++", os.path.join(CSRC, "devpool.cu"),
                    os.path.join(HERE, "devpool_check.cpp"), "-o", out], check=True, timeout=300)
    return out


@pytest.mark.parametrize("check", ["reuse", "bound", "trim", "trim_unpooled", "leave", "room", "spare", "waits",
                                   "host_memory"])
def test_pool(exe, check):
    r = subprocess.run([exe, check], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stderr)


def test_every_call_hands_its_result_through_its_scope():
    """A call that fails may leave work on its stream; CallScope::end waits for
    it before the pool hands the call's buffers on."""
    import re

    seen = 0
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith(".cu"):
            continue
        src = open(os.path.join(CSRC, f)).read()
        for body in re.findall(r'^extern "C" .*?^}', src, re.S | re.M):
            if "CallScope " in body:
                seen += 1
                assert "scope.end(" in body, body.split("(")[0]
    assert seen >= 9
