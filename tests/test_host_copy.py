"""Staged host copies on a stand-in for the CUDA runtime (tests/cpp/host_copy.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")))
    exe = str(tmp_path_factory.mktemp("host_copy") / "host_copy")
    csrc = os.path.join(ROOT, "gianduia_b200", "csrc")
    subprocess.run(["/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++", "-std=c++17", "-O1", "-pthread", "-ldl",
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(csrc, "include"), "-I", os.path.join(csrc, "cuda"),
                    "-I", os.path.join(cuda, "include"), "-x", "c++", os.path.join(csrc, "cuda", "hostcopy.cu"),
                    os.path.join(ROOT, "tests", "cpp", "host_copy.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("case", ["pageable", "pinned", "no-pinned-memory", "no-threads", "one-thread", "device-pointers"])
def test_copies(program, case):
    assert subprocess.run([program, case], timeout=60).returncode == 0
