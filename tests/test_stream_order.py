"""Host calls that touch one buffer from two streams without a wait between
them (stream_order.cpp: the library's host code against a stand-in for the
CUDA runtime; no GPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "diablo3_b200", "csrc")
CUDA = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("stream_order") / "stream_order")
    srcs = [os.path.join(HERE, "stream_order.cpp")] + [os.path.join(CSRC, f) for f in ("db_api.cu", "db_sgs.cu")]
    # what the program never calls (other launchers) stays unresolved
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", CUDA, "-x", "c++", *srcs, "-x", "none", "-static", "-o", exe,
                    "-Wl,--unresolved-symbols=ignore-all", "-lpthread"], check=True)
    return exe


@pytest.mark.parametrize("what", ["init", "init mixed", "sgs", "targets"])
def test_no_two_streams_on_one_buffer(program, what):
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
