"""csrc/once.h: what precedes a kernel's first launch on a device, when several host threads make it."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "vdnn_implementation_b200", "csrc")


def test_no_thread_goes_on_before_the_preparation(tmp_path):
    binary = str(tmp_path / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, os.path.join(HERE, "once_check.cpp"), "-o", binary, "-lpthread"], check=True)
    for _ in range(5):
        assert subprocess.run([binary], timeout=60).returncode == 0
