"""The host side of a build, checked without a GPU: the orchestration (csrc/ooc_api.cu) compiled as
plain C++ against a stand-in for the CUDA runtime and the kernels (fake_cuda.h), whose streams run
their work as late as CUDA allows.  Failures are refused allocations and callbacks that return an
error, at every point of every kind of call."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "ooc_svo_builder_gb300", "csrc")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    cxx = shutil.which("g++")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if cxx is None or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or no CUDA headers")
    exe = str(tmp_path_factory.mktemp("host_build") / "check")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I", cuda,
                    "-x", "c++", os.path.join(CSRC, "ooc_api.cu"), os.path.join(HERE, "host_build_check.cpp"),
                    "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("what", [
    "drained",  # nothing of a failed call is still queued, on any stream, when it returns
    "clean",    # the build after one whose layout check failed starts from clean buffers
    "recovered",  # every kind of build succeeds after a failure
    "freed",    # a destroyed context has given everything back
    "aligned",  # destinations that the records' stores cannot reach are refused, the others are not
    "admitted",  # a request's footprint covers what its build allocates
])
def test_host_build(check, what):
    p = subprocess.run([check, what], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr
