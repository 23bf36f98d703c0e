"""csrc/host_copy.cpp, which carries parameters between device and pageable host memory, on a host-only stand-in for the CUDA
runtime (host_copy_check.cpp): what a GPU run would show only by chance or only when memory runs out."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "vdnn_implementation_b200", "csrc")
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    binary = str(tmp_path_factory.mktemp("host_copy") / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CUDA_INCLUDE, "-I", CSRC, os.path.join(HERE, "host_copy_check.cpp"),
                    os.path.join(CSRC, "host_copy.cpp"), "-o", binary, "-lpthread"], check=True)
    return lambda *what: subprocess.run([binary] + [str(w) for w in what], timeout=120).returncode


def test_concurrent_copies_keep_their_bytes_apart(check):
    assert check("concurrent") == 0


@pytest.mark.parametrize("pinned,streams", [(0, 99), (1, 99), (2, 99), (3, 99), (99, 0), (99, 1)])
def test_copies_go_on_when_pinned_memory_or_streams_run_out(check, pinned, streams):
    assert check("scarce", pinned, streams) == 0


def test_the_current_device_of_the_caller_stays(check):
    assert check("device") == 0
